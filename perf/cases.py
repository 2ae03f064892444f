"""The workloads this framework is timed on.

Each case is a call a simulation makes through the public Python entry points
(chui_treepm): one force evaluation, one KDK step, one force VJP, or a
differentiable KDK integration with its backward pass. The listed cases span
4096 to 16.8 million particles; `draw` gives further cases of the same kinds
and ranges (odd particle counts, odd and rectangular meshes included).

A case is a dict of plain values:
  kind       "force" | "step" (kick, drift, force, kick) | "vjp" | "train"
             (KDK steps, CIC density loss, gradient to the displacements)
  n          particles: floor(((1 - halo_fraction) n)^(1/3))^3 of them on a
             Zel'dovich-displaced lattice, the rest in NFW halos
  halo_fraction, halos, decades   the halo population (0 halos: none)
  rms        rms lattice displacement in lattice spacings
  mx, my, mz mesh cells per axis; box is the x length, cells are cubic
  theta, leaf, eps, tsc, deconv   solver knobs (eps in units of box / n^(1/3))
  fp64       FP64 solver instead of mixed precision
  host       inputs and outputs in host (numpy) memory
  masses     1: one mass per particle, log-uniform over a factor of 8; 0: equal
  soft       1: per-particle softening lanes
  open       1: isolated/open boundaries
  active     fraction of the particles that are targets (1: all of them); an
             active subset reuses the PM field of an earlier full solve
  adaptive   1: relative-monopole acceptance with |a| history (the fast deck)
  steps, dt  KDK steps and step
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "chui-dev_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import chui_treepm as ct  # noqa: E402
from chui_treepm import adjoint  # noqa: E402

ASMTH, RCUT = 1.25, 6.25  # r_s and r_cut in mesh cells (the solver's defaults)
F64 = torch.float64

_DEFAULT = dict(kind="force", n=4096, halo_fraction=0.0, halos=0, decades=3.0, rms=0.2, mx=16, my=16, mz=16, box=10.0,
                theta=0.5, leaf=16, eps=0.0, tsc=0, deconv=1, fp64=0, host=0, masses=0, soft=0, open=0, active=1.0,
                adaptive=0, steps=0, dt=0.0)


def _case(name=None, **kw):
    c = dict(_DEFAULT, **kw)
    if name is not None:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest call: a test-sized box, where launches and waits are the cost
        _case("lattice16", n=16 ** 3, eps=0.016),
        # the plain configuration: 32^3 lattice, mesh twice as fine, one KDK step
        _case("step32", kind="step", n=32 ** 3, mx=64, my=64, mz=64, dt=0.05),
        # odd and rectangular mesh, TSC, unequal masses and per-particle softening
        # lanes: a zoom-like species mix
        _case("species50k", n=50021, halo_fraction=0.5, halos=12, rms=0.5, mx=40, my=36, mz=45, box=10.0, tsc=1,
              eps=0.05, masses=1, soft=1),
        # isolated/open boundaries: a collapsing cloud, zero-padded convolution
        _case("open70k", n=70001, halo_fraction=0.4, halos=20, rms=0.3, mx=48, my=48, mz=48, eps=0.05, open=1, deconv=0),
        # a host program with its particles in host memory (the C++ host's call)
        _case("host200k", n=200003, halo_fraction=0.4, halos=40, rms=0.5, mx=64, my=64, mz=64, box=50.0, eps=0.01,
              host=1),
        # the FP64 solver, as the accuracy comparator of a run
        _case("fp64_64", n=64 ** 3, rms=0.3, mx=64, my=64, mz=64, box=50.0, eps=0.1, fp64=1),
        # differentiable run: 10 KDK steps, CIC density loss, backward pass
        _case("train64", kind="train", n=64 ** 3, rms=0.3, mx=64, my=64, mz=64, box=50.0, eps=0.1, steps=10, dt=0.05),
        # clustered force at 2.1 M particles (300 halos over 3 decades)
        _case("clustered128", n=128 ** 3, halo_fraction=0.4, halos=300, rms=0.5, mx=128, my=128, mz=128, box=100.0,
              eps=0.00128),
        # the same state, 3 % of the particles active between two PM refreshes
        # (block time steps)
        _case("active128", n=128 ** 3, halo_fraction=0.4, halos=300, rms=0.5, mx=128, my=128, mz=128, box=100.0,
              theta=0.7, eps=0.00128, active=0.03),
        # the adaptive fast deck (relative monopole, COM-distance cutoff nodes)
        _case("deck128", n=128 ** 3, halo_fraction=0.4, halos=300, rms=0.5, mx=128, my=128, mz=128, box=100.0, theta=0.7,
              eps=0.00128, adaptive=1),
        # one force VJP of the clustered state
        _case("vjp128", kind="vjp", n=128 ** 3, halo_fraction=0.4, halos=300, rms=0.5, mx=128, my=128, mz=128, box=100.0,
              eps=0.05),
        # the largest: one KDK step of the 256^3 clustered box (2000 halos)
        _case("step256", kind="step", n=256 ** 3, halo_fraction=0.5, halos=2000, rms=0.5, mx=256, my=256, mz=256,
              box=200.0, theta=0.6, eps=0.00128, dt=0.002),
    ]


def draw(rng):
    kind = rng.choice(["force", "force", "force", "force", "step", "vjp", "train"])
    form = rng.choice(["plain", "plain", "species", "open", "host", "fp64", "active", "adaptive"]) if kind == "force" else "plain"
    top = {"train": 40 ** 3, "vjp": 1_500_000}.get(kind, {"species": 400_000, "open": 300_000, "host": 1_000_000,
                                                           "fp64": 150_000}.get(form, 3_000_000))
    n = int(math.exp(rng.uniform(math.log(3000), math.log(top))))
    clustered = kind != "train" and form != "fp64" and rng.random() < 0.6
    side = n ** (1 / 3)
    if kind == "train":
        n = int(side) ** 3
    # 0.6 to 2 mesh cells per mean particle spacing, and at least 16 per axis
    m = max(16, min(256, int(side * math.exp(rng.uniform(math.log(0.6), math.log(2.0))))))
    c = _case(kind=kind, n=n, mx=m, my=m, mz=m, box=round(rng.uniform(5.0, 250.0), 3), rms=round(rng.uniform(0.1, 0.5), 3),
              theta=rng.choice([0.5, 0.6, 0.7]), leaf=rng.choice([16, 16, 32]), eps=round(rng.choice([0.0, 0.01, 0.05, 0.1]), 3),
              deconv=rng.randint(0, 1), tsc=1 if rng.random() < 0.25 else 0)
    if clustered:
        c.update(halo_fraction=round(rng.uniform(0.2, 0.6), 3), halos=max(3, n // rng.randint(3000, 9000)),
                 decades=rng.choice([2.0, 3.0]))
    if rng.random() < 0.3 and kind != "train":
        c.update(my=m + rng.randint(0, 5), mz=m + rng.randint(0, 9))
    if kind == "step":
        c.update(dt=0.002 if clustered else 0.05)
    elif kind == "train":
        c.update(steps=rng.randint(2, 10), dt=0.05, eps=0.1)
    elif kind == "vjp":
        c.update(eps=rng.choice([0.05, 0.1]))
    if form == "species":
        c.update(masses=1, soft=rng.randint(0, 1), eps=0.05)
    elif form == "open":
        c.update(open=1, deconv=0, masses=rng.randint(0, 1), eps=0.05)
    elif form == "host":
        c.update(host=1)
    elif form == "fp64":
        c.update(fp64=1)
    elif form == "active":
        c.update(active=round(math.exp(rng.uniform(math.log(0.01), math.log(0.5))), 4))
    elif form == "adaptive":
        c.update(adaptive=1, eps=0.01)
    return c


# ---- inputs -----------------------------------------------------------------

def _box(c):
    h = c["box"] / c["mx"]
    return (c["box"], h * c["my"], h * c["mz"])


def _spacing(c):
    b = _box(c)
    return (b[0] * b[1] * b[2] / c["n"]) ** (1 / 3)


def _displacements(side, rms, gen):
    """Zel'dovich displacements of a side^3 lattice in lattice spacings, P(k) ~ k^-2."""
    dk = torch.fft.rfftn(torch.randn((side,) * 3, generator=gen, device="cuda", dtype=F64))
    k = torch.fft.fftfreq(side, device="cuda", dtype=F64) * side
    kz = torch.fft.rfftfreq(side, device="cuda", dtype=F64) * side
    k2 = k[:, None, None] ** 2 + k[None, :, None] ** 2 + kz[None, None, :] ** 2
    k2[0, 0, 0] = 1.0
    dk = dk / k2.sqrt() / k2
    dk[0, 0, 0] = 0.0
    psi = torch.stack([torch.fft.irfftn(1j * a * dk, s=(side,) * 3).reshape(-1)
                       for a in (k[:, None, None], k[None, :, None], kz[None, None, :])])
    return psi * (rms / psi.square().sum(0).mean().sqrt())


def _wrap(v, length):
    w = torch.remainder(v, length)
    return torch.where(w >= length, torch.zeros_like(w), w)


def _particles(c, seed):
    """x (3, n) in the box, v (3, n), mass (n), previous acceleration (3, n)."""
    gen = torch.Generator(device="cuda").manual_seed(1000003 * seed + 17)

    def rand(*shape):
        return torch.rand(*shape, generator=gen, device="cuda", dtype=F64)

    n, box = c["n"], torch.tensor(_box(c), device="cuda", dtype=F64)[:, None]
    halos = c["halos"] if c["halo_fraction"] > 0 else 0
    side = int(((1.0 - c["halo_fraction"]) * n) ** (1 / 3) + 1e-6)
    rest = n - side ** 3
    g = (torch.arange(side, device="cuda", dtype=F64) + 0.5) / side
    q = torch.stack([a.reshape(-1) for a in torch.meshgrid(g, g, g, indexing="ij")])
    psi = _displacements(side, c["rms"], gen) * (box / side)
    x, v = q * box + psi, psi
    if rest and halos:
        w = 10.0 ** (rand(halos) * c["decades"])
        of = torch.searchsorted(torch.cumsum(w, 0) / w.sum(), rand(rest)).clamp_(max=halos - 1)
        count = torch.bincount(of, minlength=halos).to(F64)
        r_vir = (3.0 * count / (4.0 * math.pi * 200.0 * n / box.prod())) ** (1 / 3)
        conc = (4.0 + 8.0 * rand(halos))[of]
        # radius by bisection of the NFW mass profile ln(1 + s) - s / (1 + s)
        want = rand(rest) * (torch.log1p(conc) - conc / (1.0 + conc))
        lo, hi = torch.zeros_like(conc), conc.clone()
        for _ in range(40):
            mid = 0.5 * (lo + hi)
            below = torch.log1p(mid) - mid / (1.0 + mid) < want
            lo, hi = torch.where(below, mid, lo), torch.where(below, hi, mid)
        r = 0.5 * (lo + hi) / conc * r_vir[of]
        mu, phi = 2.0 * rand(rest) - 1.0, 2.0 * math.pi * rand(rest)
        s = (1.0 - mu * mu).clamp(min=0).sqrt()
        d = torch.stack([r * s * torch.cos(phi), r * s * torch.sin(phi), r * mu])
        x = torch.cat([x, (rand(3, halos) * box)[:, of] + d], 1)
        v = torch.cat([v, torch.zeros_like(d)], 1)
    elif rest:
        x = torch.cat([x, rand(3, rest) * box], 1)
        v = torch.cat([v, torch.zeros(3, rest, device="cuda", dtype=F64)], 1)
    perm = torch.randperm(n, generator=gen, device="cuda")  # row order carries no spatial information
    x, v = x[:, perm], v[:, perm].contiguous()
    # open boundaries: a few particles drift out of the mesh
    x = x * 1.02 - 0.01 * box if c["open"] else torch.stack([_wrap(x[a], float(box[a])) for a in range(3)])
    m = torch.full((n,), _spacing(c) ** 3, device="cuda", dtype=F64)  # mean density 1
    if c["masses"]:
        m = m * 8.0 ** (rand(n) - 0.5)
    return x.contiguous(), v, m, v * (4.0 * math.pi / 3.0)


def _config(c, **kw):
    b, abi = _box(c), ct._abi
    k = dict(pm_grid_nx=c["mx"], pm_grid_ny=c["my"], pm_grid_nz=c["mz"], box_x=b[0], box_y=b[1], box_z=b[2],
             asmth_cells=ASMTH, rcut_cells=RCUT, opening_theta=c["theta"], max_leaf_size=c["leaf"],
             assignment_scheme=abi.TSC if c["tsc"] else abi.CIC, window_deconvolution=c["deconv"],
             softening=c["eps"] * _spacing(c), precision=abi.FP64 if c["fp64"] else abi.MIXED,
             boundary_condition=abi.BOUNDARY_ISOLATED_OPEN if c["open"] else abi.BOUNDARY_PERIODIC)
    return ct.TreePmConfig(**dict(k, **kw))


def _softening(c, seed):
    """Per-particle epsilons: half the particles of a finer species."""
    gen = torch.Generator(device="cuda").manual_seed(77 * seed + 5)
    fine = torch.rand(c["n"], generator=gen, device="cuda", dtype=F64) < 0.5
    e = c["eps"] * _spacing(c)
    return torch.where(fine, torch.full_like(fine, 0.4 * e, dtype=F64), torch.full_like(fine, e, dtype=F64))


def _active(c, seed):
    gen = torch.Generator(device="cuda").manual_seed(91 * seed + 3)
    return torch.randperm(c["n"], generator=gen, device="cuda")[:max(1, int(c["n"] * c["active"]))].contiguous()


def _cotangent(c, seed):
    gen = torch.Generator(device="cuda").manual_seed(13 * seed + 7)
    return torch.randn(3, c["n"], generator=gen, device="cuda", dtype=F64)


def _train_inputs(c, seed):
    """Lattice sites, displacements and the displacements of the target box."""
    side = round(c["n"] ** (1 / 3))
    h = c["box"] / side
    g = (torch.arange(side, device="cuda", dtype=F64) + 0.5) * h
    q = torch.stack([a.reshape(-1) for a in torch.meshgrid(g, g, g, indexing="ij")])
    psi = [_displacements(side, c["rms"], torch.Generator(device="cuda").manual_seed(1000003 * seed + k)) * h for k in (1, 2)]
    return q, psi[0], psi[1], torch.full((c["n"],), h ** 3, device="cuda", dtype=F64)


def _coarse(a):
    """|a| to 4 bits of mantissa: a history that rounding in the last step does not change."""
    m, e = torch.frexp(a)
    return torch.ldexp(torch.round(m * 16.0) / 16.0, e)


def prepare(case, seed):
    c = dict(_DEFAULT, **case)
    if c["kind"] == "train":
        q, psi, other, m = _train_inputs(c, seed)
        solver, dens = ct.TreePmCoordinator(_config(c)), ct.TreePmCoordinator(_config(c))
        side = round(c["n"] ** (1 / 3))
        target = dens.assign_density(*(q + other), m).reshape(c["mx"], c["my"], c["mz"])
        return dict(c=c, solver=solver, dens=dens, q=q, psi=psi, m=m, target=target, side=side)
    x, v, m, a = _particles(c, seed)
    s = dict(c=c, x=x, m=m)
    if c["kind"] == "step":
        s.update(v=v, a=a, factors=ct.kdk_factors_static(c["dt"]))
    elif c["kind"] == "vjp":
        s.update(cot=_cotangent(c, seed))
    s["kw"] = kw = {}
    if c["soft"]:
        kw["softening"] = _softening(c, seed)
    if c["host"]:
        s["x"], s["m"] = x.cpu().numpy(), m.cpu().numpy()
        kw.update({k: t.cpu().numpy() for k, t in kw.items()})
    if c["adaptive"]:
        with ct.TreePmCoordinator(_config(c)) as strict:
            r = strict.solve_active_set(*x, m)
        kw["previous_acceleration"] = _coarse(torch.sqrt(r["ax"] ** 2 + r["ay"] ** 2 + r["az"] ** 2))
        abi = ct._abi
        s["solver"] = ct.TreePmCoordinator(_config(
            c, acceptance_policy=abi.POLICY_ADAPTIVE, adaptive_error_estimator=abi.ESTIMATOR_RELATIVE_MONOPOLE,
            cutoff_node_policy=abi.CUTOFF_COM_DISTANCE, relative_force_tolerance=0.0025, adaptive_maximum_opening_angle=1.0))
    else:
        s["solver"] = ct.TreePmCoordinator(_config(c))
    if c["active"] < 1.0:
        kw["active"] = _active(c, seed).to(torch.int32)
        s["solver"].solve_active_set(*x, m)  # the full step before, whose PM field the subset reuses
    return s


def run(s):
    c, solver = s["c"], s["solver"]
    if c["kind"] == "train":
        psi = [t.clone().requires_grad_() for t in s["psi"]]
        xn = adjoint.kdk(solver, *[s["q"][k] + psi[k] for k in range(3)], *psi, s["m"], c["steps"], c["dt"])
        rho = adjoint.cic_density(s["dens"], xn[0], xn[1], xn[2], s["m"])
        loss = ((rho - s["target"]) ** 2).mean()
        loss.backward()
        return [rho.detach(), loss.detach()] + [t.grad for t in psi]
    if c["kind"] == "vjp":
        return list(solver.force_vjp(*s["x"], s["m"], *s["cot"]))
    if c["kind"] == "step":
        x, v = s["x"].clone(), s["v"].clone()
        d, k1, k2, g1, g2 = s["factors"]
        solver.kick(*v, *s["a"], k1, g1)
        solver.drift(*x, *v, d)
        r = solver.solve_active_set(*x, s["m"])
        solver.kick(*v, r["ax"], r["ay"], r["az"], k2, g2)
        return [x, v, r["ax"], r["ay"], r["az"]]
    r = solver.solve_active_set_with_pm_cadence(*s["x"], s["m"], c["active"] >= 1.0, **s["kw"])
    return [r["ax"], r["ay"], r["az"]]


# ---- what a pass cannot do without ------------------------------------------

def _pairs(c):
    """Ordered pairs inside r_cut: the mean density's, plus those inside the halos
    (masses log-uniform over the decades; the share of a halo's mass within
    r_cut of a member taken as the smaller of 1 and r_cut / (0.7 r_vir))."""
    n, b = c["n"], _box(c)
    vol, cut = b[0] * b[1] * b[2], RCUT * c["box"] / c["mx"]
    p = n * n * min(1.0, 4.0 / 3.0 * math.pi * cut ** 3 / vol)
    if c["halo_fraction"] > 0 and c["halos"]:
        k = 64
        w = [10.0 ** (c["decades"] * (i + 0.5) / k) for i in range(k)]
        for x in w:
            in_halo = c["halo_fraction"] * n * x * k / (sum(w) * c["halos"])
            r_vir = (3.0 * in_halo * vol / (4.0 * math.pi * 200.0 * n)) ** (1 / 3)
            p += c["halos"] / k * in_halo ** 2 * min(1.0, cut / (0.7 * r_vir))
    return p * min(1.0, c["active"])


def work(case):
    c = dict(_DEFAULT, **case)
    cells = c["mx"] * c["my"] * c["mz"] * (8 if c["open"] else 1)
    real = 8 if c["fp64"] else 4
    fft = 2.5 * cells * math.log2(cells)
    # positions and mass in, accelerations out; one transform of the density and
    # three of the force; 28 operations per pair (3 differences, r^2, the kernel,
    # 3 accumulations), 60 with its derivative
    force = {"bytes": c["n"] * 32.0 + c["n"] * c["active"] * 24.0 + cells * real * 4.0 * (1 if c["active"] >= 1.0 else 0.75),
             "flops": 28.0 * _pairs(c) + (4.0 * fft if c["active"] >= 1.0 else 0.0) + 100.0 * c["n"]}
    vjp = {"bytes": c["n"] * 80.0 + cells * real * 8.0, "flops": 60.0 * _pairs(c) + 8.0 * fft + 200.0 * c["n"]}
    if c["kind"] == "vjp":
        return vjp
    if c["kind"] == "step":  # two kicks and a drift: x, v and a in, x and v out
        return {"bytes": force["bytes"] + c["n"] * 120.0, "flops": force["flops"] + 18.0 * c["n"]}
    if c["kind"] == "train":
        k = c["steps"] + 1
        return {"bytes": k * (force["bytes"] + vjp["bytes"] + c["n"] * 240.0), "flops": k * (force["flops"] + vjp["flops"])}
    return force


def tolerance(case):
    # about four times the largest distance from `exact` that was measured for the kind
    c = dict(_DEFAULT, **case)
    if c["fp64"]:
        # FP64 sums of FP64 pair forces (1.2e-14 measured)
        return {"rel": 1.0e-13}
    if c["adaptive"]:
        # the acceptance criterion's own error (2.7e-4): a node may be taken as a
        # multipole or as the pairs it stands for
        return {"rel": 1.0e-3}
    if c["kind"] == "train":
        # up to ten steps of FP32 forces, and their gradient (1.4e-4)
        return {"rel": 6.0e-4}
    if c["active"] < 1.0:
        # sparse targets: pair offsets are rounded over wide groups of targets (2.6e-5)
        return {"rel": 1.0e-4}
    # FP32 pair forces and mesh; a near-lattice's forces are small differences of
    # the mesh's (7.8e-6)
    return {"rel": 3.0e-5}


# ---- the same values in FP64, by direct sums --------------------------------

def _stencil(gp, tsc):
    if not tsc:
        base = torch.floor(gp.detach())
        t = gp - base
        return base.long(), (1.0 - t, t)
    near = torch.floor(gp.detach() + 0.5)
    d = gp - near
    return near.long() - 1, (0.5 * (0.5 - d) ** 2, 0.75 - d * d, 0.5 * (0.5 + d) ** 2)


def _cells(c, x):
    """(flat cell, weight) of every stencil point; open: points off the mesh at weight 0."""
    mesh, b = (c["mx"], c["my"], c["mz"]), _box(c)
    st, ok = [], True
    for a in range(3):
        w = x[a] if c["open"] else torch.remainder(x[a], b[a])
        st.append(_stencil(w * (mesh[a] / b[a]), c["tsc"]))
        if c["open"]:
            ok = ok & (x[a] >= 0) & (x[a] < b[a])
    t = len(st[0][1])
    for i in range(t):
        for j in range(t):
            for k in range(t):
                cell, w = [st[0][0] + i, st[1][0] + j, st[2][0] + k], st[0][1][i] * st[1][1][j] * st[2][1][k]
                if c["open"]:
                    inside = ok
                    for a in range(3):
                        inside = inside & (cell[a] >= 0) & (cell[a] < mesh[a])
                    w = torch.where(inside, w, torch.zeros_like(w))
                    cell = [cell[a].clamp(0, mesh[a] - 1) for a in range(3)]
                else:
                    cell = [torch.remainder(cell[a], mesh[a]) for a in range(3)]
                yield (cell[0] * mesh[1] + cell[1]) * mesh[2] + cell[2], w


def _density(c, x, m):
    mesh, b = (c["mx"], c["my"], c["mz"]), _box(c)
    rho = torch.zeros(mesh[0] * mesh[1] * mesh[2], device="cuda", dtype=F64)
    for cell, w in _cells(c, x):
        rho = rho.index_add(0, cell, m * w)
    return (rho * (mesh[0] * mesh[1] * mesh[2] / (b[0] * b[1] * b[2]))).reshape(mesh)


def _mesh_force(c, rho):
    mesh, b = (c["mx"], c["my"], c["mz"]), _box(c)
    h = c["box"] / c["mx"]
    rs = ASMTH * h
    if c["open"]:
        d = []
        for a in range(3):
            i = torch.arange(2 * mesh[a], device="cuda")
            d.append(torch.where(i <= mesh[a], i, i - 2 * mesh[a]).to(F64) * h)
        r = (d[0][:, None, None] ** 2 + d[1][None, :, None] ** 2 + d[2][None, None, :] ** 2).sqrt()
        green = torch.where(r > 0, -torch.erf(0.5 * r / rs) / r.clamp(min=1e-300), torch.full_like(r, -1.0 / (math.sqrt(math.pi) * rs)))
        s = [2 * k for k in mesh]
        phi = torch.fft.irfftn(torch.fft.rfftn(rho, s=s) * torch.fft.rfftn(green), s=s)[:mesh[0], :mesh[1], :mesh[2]] * h ** 3
        return [-torch.gradient(phi, spacing=h, dim=a, edge_order=2)[0] for a in range(3)]
    k, g, w = [], [], []
    for a in range(3):
        i = torch.arange(mesh[a] // 2 + 1 if a == 2 else mesh[a], device="cuda")
        kk = torch.where(i <= mesh[a] // 2, i, i - mesh[a]).to(F64) * (2.0 * math.pi / b[a])
        gg = kk.clone()
        if mesh[a] % 2 == 0:
            gg[mesh[a] // 2] = 0.0  # the derivative has no Nyquist mode
        shape = [1, 1, 1]
        shape[a] = -1
        k.append(kk.reshape(shape))
        g.append(gg.reshape(shape))
        w.append(torch.sinc(kk * (b[a] / mesh[a] / (2.0 * math.pi))).reshape(shape) ** (3 if c["tsc"] else 2))
    k2 = k[0] ** 2 + k[1] ** 2 + k[2] ** 2
    op = -4.0 * math.pi * torch.exp(-k2 * rs * rs) / torch.where(k2 > 0, k2, torch.ones_like(k2))
    if c["deconv"]:
        op = op / ((w[0] * w[1] * w[2]) ** 2).clamp(min=1e-12)
    op[0, 0, 0] = 0.0
    psi = torch.fft.rfftn(rho) * op
    return [torch.fft.irfftn(-1j * g[a] * psi, s=mesh) for a in range(3)]


def _mesh_acceleration(c, field_x, x, m):
    """Mesh force at x of the density of the particles at field_x."""
    f = [t.reshape(-1) for t in _mesh_force(c, _density(c, field_x, m))]
    out = [0.0, 0.0, 0.0]
    for cell, w in _cells(c, x):
        out = [out[a] + w * f[a][cell] for a in range(3)]
    return torch.stack(out)


def _kernel(r2, eps2, rs, derivative):
    """K = (r^2 + eps^2)^-3/2 - H(t) / (8 r_s^3), t = r^2 / (4 r_s^2), H(t) = [erf(q) - 2 q e^-t / sqrt(pi)] / q^3,
    q = sqrt(t) (its series where the difference would cancel), and with derivative (dK/dr) / r."""
    t = r2 / (4.0 * rs * rs)
    q, e, pi = t.sqrt(), torch.exp(-t), 1.0 / math.sqrt(math.pi)
    small = t < 0.5
    ts = torch.where(small, t, torch.zeros_like(t))
    series, slope, term = torch.zeros_like(t), torch.zeros_like(t), torch.full_like(t, 4.0 * pi)
    for k in range(16):
        series = series + term / (2 * k + 3)
        if derivative:
            slope = slope - term / (2 * k + 5)
        term = term * (-ts) / (k + 1)
    tl = torch.where(small, torch.ones_like(t), t)
    h = torch.where(small, series, (torch.erf(q) - 2.0 * pi * q * e) / (tl * tl.sqrt()))
    d = r2 + eps2
    soft = 1.0 / (d * d.sqrt())
    kern = soft - h / (8.0 * rs ** 3)
    if not derivative:
        return kern, None
    hp = torch.where(small, slope, (2.0 * pi * e - 1.5 * h) / tl)
    return kern, -3.0 * soft / d - hp / (16.0 * rs ** 5)


def _pair_sums(c, x, m, eps, targets=None, cot=None):
    """Direct sums over the pairs inside r_cut: the short-range acceleration of the targets, or with cot the force's
    transposed Jacobian applied to it. Targets cell by cell against the 27 cells around, with ghost copies of the
    particles around a periodic box."""
    b, cut, rs = _box(c), RCUT * c["box"] / c["mx"], ASMTH * c["box"] / c["mx"]
    lo, length, src = [0.0] * 3, list(b), x
    rows = torch.arange(x.shape[1], device="cuda")
    if c["open"]:
        lo = [float(x[a].min()) for a in range(3)]
        length = [max(float(x[a].max()) - lo[a], cut) * (1.0 + 1e-12) for a in range(3)]
    nc = [max(1, min(160, int(length[a] / cut))) for a in range(3)]
    w = [length[a] / nc[a] for a in range(3)]
    if not c["open"]:
        src = torch.stack([torch.remainder(x[a], b[a]) for a in range(3)])
        for a in range(3):
            up, down = src[a] < w[a], src[a] >= b[a] - w[a]
            parts, at = [src], [rows]
            for side, shift in ((up, b[a]), (down, -b[a])):
                ghost = src[:, side].clone()
                ghost[a] += shift
                parts.append(ghost)
                at.append(rows[side])
            src, rows = torch.cat(parts, 1), torch.cat(at)
    dims = [k + 2 for k in nc]
    idx = [torch.floor((src[a] - lo[a]) / w[a]).long().clamp(-1, nc[a]) + 1 for a in range(3)]
    order = torch.argsort((idx[0] * dims[1] + idx[1]) * dims[2] + idx[2])
    src, rows = src[:, order].contiguous(), rows[order]
    cell = ((idx[0] * dims[1] + idx[1]) * dims[2] + idx[2])[order]
    start = torch.searchsorted(cell, torch.arange(dims[0] * dims[1] * dims[2] + 1, device="cuda")).tolist()
    home = torch.zeros(x.shape[1], device="cuda", dtype=torch.bool)
    home[rows if targets is None else targets] = True
    out = torch.zeros(3, x.shape[1], device="cuda", dtype=F64)
    ms, es = m[rows], eps[rows]
    cs = cot[:, rows] if cot is not None else None
    for i in range(1, nc[0] + 1):
        for j in range(1, nc[1] + 1):
            for k in range(1, nc[2] + 1):
                at = (i * dims[1] + j) * dims[2] + k
                if start[at] == start[at + 1]:
                    continue
                t = torch.arange(start[at], start[at + 1], device="cuda")
                if targets is not None:
                    t = t[home[rows[t]]]
                    if t.numel() == 0:
                        continue
                near = []
                for di in (-1, 0, 1):
                    for dj in (-1, 0, 1):
                        row = ((i + di) * dims[1] + j + dj) * dims[2] + k
                        near.append((start[row - 1], start[row + 2]))
                near = [p for p in near if p[1] > p[0]]
                sx, sm, se = (torch.cat([v[..., p:q] for p, q in near], -1) for v in (src, ms, es))
                sc = torch.cat([cs[:, p:q] for p, q in near], -1) if cot is not None else None
                per = max(1, 12_000_000 // sm.numel())
                for tt in t.split(per):
                    d = [sx[a][None, :] - src[a][tt][:, None] for a in range(3)]
                    r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
                    use = (r2 <= cut * cut) & (r2 > 0)
                    r2 = torch.where(use, r2, torch.full_like(r2, cut * cut))
                    e = torch.maximum(se[None, :], es[tt][:, None])
                    kern, slope = _kernel(r2, e * e, rs, cot is not None)
                    if cot is None:
                        f = torch.where(use, kern, torch.zeros_like(kern)) * sm
                        out[:, rows[tt]] = torch.stack([(f * d[a]).sum(1) for a in range(3)])
                        continue
                    z = torch.zeros_like(kern)
                    kern, slope = torch.where(use, kern, z), torch.where(use, slope, z)
                    mt, ctt = ms[tt][:, None], cs[:, tt]
                    p = [mt * sc[a][None, :] - sm[None, :] * ctt[a][:, None] for a in range(3)]
                    dc = (d[0] * p[0] + d[1] * p[1] + d[2] * p[2]) * slope
                    out[:, rows[tt]] = torch.stack([(kern * p[a] + dc * d[a]).sum(1) for a in range(3)])
    return out


def _force(c, x, m, eps=None, targets=None):
    if eps is None:
        eps = torch.full_like(m, c["eps"] * _spacing(c))
    near = _pair_sums(c, x, m, eps, targets)
    at = x if targets is None else x[:, targets]
    return _mesh_acceleration(c, x, at, m) + (near if targets is None else near[:, targets])


def _force_vjp(c, x, m, cot):
    near = _pair_sums(c, x, m, torch.full_like(m, c["eps"] * _spacing(c)), None, cot)
    with torch.enable_grad():
        p = x.detach().clone().requires_grad_()
        (far,) = torch.autograd.grad((_mesh_acceleration(c, p, p, m) * cot).sum(), p)
    return near + far


def exact(case, seed):
    c = dict(_DEFAULT, **case)
    if _pairs(c) > 6.0e10:
        return None
    with torch.no_grad():
        if c["kind"] == "train":
            return _exact_train(c, seed)
        x, v, m, a = _particles(c, seed)
        if c["kind"] == "vjp":
            return list(_force_vjp(c, x, m, _cotangent(c, seed)))
        if c["kind"] == "step":
            v = v + 0.5 * c["dt"] * a
            x = x + c["dt"] * v
            x = torch.stack([_wrap(x[k], _box(c)[k]) for k in range(3)])
            a = _force(c, x, m)
            return [x, v + 0.5 * c["dt"] * a, *a]
        out = _force(c, x, m, _softening(c, seed) if c["soft"] else None, _active(c, seed) if c["active"] < 1.0 else None)
        return [t.cpu().numpy() for t in out] if c["host"] else list(out)


def _exact_train(c, seed):
    q, psi, other, m = _train_inputs(c, seed)
    target, dt = _density(c, q + other, m), c["dt"]
    x, v = q + psi, psi.clone()
    path, a = [x], _force(c, x, m)
    for _ in range(c["steps"]):
        v = v + 0.5 * dt * a
        x = torch.stack([_wrap(t, c["box"]) for t in x + dt * v])
        a = _force(c, x, m)
        v = v + 0.5 * dt * a
        path.append(x)
    with torch.enable_grad():
        p = x.detach().clone().requires_grad_()
        rho = _density(c, p, m)
        loss = ((rho - target) ** 2).mean()
        (xb,) = torch.autograd.grad(loss, p)
    vb, ab = torch.zeros_like(xb), torch.zeros_like(xb)
    for k in range(c["steps"] - 1, -1, -1):
        xb = xb + _force_vjp(c, path[k + 1], m, ab)
        vb = vb + dt * xb
        ab = 0.5 * dt * vb + (0.0 if k == 0 else 0.5 * dt * vb)
    xb = xb + _force_vjp(c, path[0], m, ab)
    return [rho.detach(), loss.detach()] + list(xb + vb)
