"""The strict policy's production walk where its groups, images and batches can
go wrong: fewer targets than a warp, remainders, meshes so coarse that a pair's
other image is in reach, boxes whose leaves are wider than their shortest side,
targets spread over the box, coincident particles with and without softening,
explicit targets, softening lanes, and the sizes around the walk's choice of
lanes per target -- against the FP64 oracle, each target's error on the scale
of its own pairs (the accelerations of dense blobs hide a sparse target's)."""
import math

import numpy as np
import pytest

import oracle

torch = pytest.importorskip("torch")

import chui_treepm as ct  # noqa: E402

pytestmark = pytest.mark.gpu

BOX = (10.0, 9.0, 11.0)


@pytest.fixture(autouse=True)
def cuda_ok():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def particles(n, seed):
    """A third uniform, the rest in blobs, one of them across the box corner;
    two coincident particles."""
    rng = np.random.default_rng(seed)
    L = np.array(BOX)
    x = rng.uniform(0.0, 1.0, (n, 3)) * L
    for k, c in enumerate(([0.02, 0.97, 0.01], [0.4, 0.5, 0.6])):
        rows = np.arange(n) % 3 == k + 1
        x[rows] = np.array(c) * L + rng.normal(0.0, 0.25, (int(rows.sum()), 3))
    x = np.mod(x, L)
    if n > 4:
        x[n // 2] = x[n // 3]
    m = rng.uniform(0.5, 2.0, n)
    return x[:, 0].copy(), x[:, 1].copy(), x[:, 2].copy(), m


def config(mesh, precision, **kw):
    return ct.TreePmConfig(pm_grid_nx=mesh, pm_grid_ny=mesh, pm_grid_nz=mesh, opening_theta=0.6, max_leaf_size=16,
                           precision=precision,
                           **dict(dict(box_x=BOX[0], box_y=BOX[1], box_z=BOX[2], softening=0.05), **kw))


def reference(p, mesh, active=None, quadrupole=1, eps=0.05, **kw):
    o = oracle.treepm_solve(*p, oracle.make_params(box=BOX, mesh=(mesh,) * 3, theta=0.6, eps=eps, leaf=16,
                                                   quadrupole=quadrupole, **kw), active=active)
    return np.stack([o["ax"], o["ay"], o["az"]])


def cell(mesh):
    return (BOX[0] * BOX[1] * BOX[2]) ** (1 / 3) / mesh


# FP32 pairs: the long-range polynomial is within 5e-5 of its part of each pair
# and most accelerations are sums of pairs of their own size
MIXED = 1.0e-4


def apart(got, ref):
    """The largest difference of a row's vector, on the scale of its length or
    of the median row's."""
    size = torch.linalg.norm(ref, dim=0)
    return float((torch.linalg.norm(got - ref, dim=0) / (size + size.median())).max())


def pair_sums(p, box, rs, rcut, eps, rows):
    """Over the sources j within rcut of each target row: the short-range
    acceleration sum m K d of the pairs, and the sums m d K_long, m d K_soft and
    m (r^2 + eps^2)^(-3/2) of the pairs' parts (FP64)."""
    x, m, L = np.stack(p[:3], 1), p[3], np.array(box)
    acc, lng, soft, slope = np.zeros((len(rows), 3)), np.zeros(len(rows)), np.zeros(len(rows)), np.zeros(len(rows))
    for i, row in enumerate(rows):
        d = x - x[row]
        d -= L * np.rint(d / L)
        r2 = (d * d).sum(1)
        use = (r2 <= rcut * rcut) & (r2 > 0.0)
        d, r2, mj = d[use], r2[use], m[use]
        r = np.sqrt(r2)
        q = r / (2.0 * rs)
        k_soft = (r2 + eps * eps) ** -1.5
        k_long = np.where(q < 0.02, 0.752252778 / (8.0 * rs ** 3),
                          (np.array([math.erf(v) for v in q]) - 2.0 / math.sqrt(math.pi) * q * np.exp(-q * q)) / r ** 3)
        acc[i] = ((mj * (k_soft - k_long))[:, None] * d).sum(0)
        lng[i], soft[i], slope[i] = (mj * r * k_long).sum(), (mj * r * k_soft).sum(), (mj * k_soft).sum()
    return acc, lng, soft, slope


def beyond(r, ref, p, box, h, eps, fp64, rows=None, reach=None, ratio=6.25):
    """The largest error of a target, each against its own allowance: the sums
    of its own pairs times what each part of a pair is rounded to, and the
    mesh's rounding (h: mesh cell, ratio: r_cut in cells). A lost pair of a
    sparse target is far above it, whatever the accelerations elsewhere in the
    box.
      mixed: the long-range polynomial is within 5e-5 of its part of a pair,
      FP32 products within 1e-6; offsets of up to reach (3 r_cut) are rounded to
      24 bits, the kernel's slope is at most 2 (r^2 + eps^2)^(-3/2); the FP32
      mesh is within 1e-5 of the rms mesh force.
      FP64: 1e-12 of the parts, offsets to 53 bits of a box length, and the
      mesh within 1e-11."""
    rows = np.arange(len(p[0])) if rows is None else rows
    rs, rcut = 1.25 * h, ratio * h
    reach = 3.0 * rcut if reach is None else reach
    acc, lng, soft, slope = pair_sums(p, box, rs, rcut, eps, rows)
    mesh = np.sqrt(((ref.T - acc) ** 2).sum(1).mean())
    got = np.stack([np.asarray(r[k]) for k in ("ax", "ay", "az")])
    assert np.isfinite(got).all()
    if fp64:
        allow = 1e-12 * (lng + soft) + 2.0 * slope * 4.4e-16 * max(box) + 1e-11 * mesh
    else:
        allow = 5e-5 * lng + 1e-6 * soft + 2.0 * slope * 2.4e-7 * reach + 1e-5 * mesh
    return (np.sqrt(((got - ref) ** 2).sum(0)) / allow).max()



@pytest.mark.parametrize("eps", [0.05, 0.0])
@pytest.mark.parametrize("n", [1, 2, 31, 33, 257, 3000])
@pytest.mark.parametrize("mesh", [14, 20, 48])
def test_small_boxes_and_remainders(n, mesh, eps):
    p = particles(n, n + mesh)
    with ct.TreePmCoordinator(config(mesh, ct._abi.MIXED, softening=eps)) as s:
        r = s.solve_active_set(*p)
    if n == 1:
        # no pairs: the mesh's own force, zero up to its FP32 rounding (about
        # 1e-7 of the deposited particle's force scale m / r_s^2)
        rs = 1.25 * cell(mesh)
        assert max(abs(r[k][0]) for k in ("ax", "ay", "az")) <= 1e-6 * p[3][0] / rs ** 2
        return
    assert beyond(r, reference(p, mesh, eps=eps), p, BOX, cell(mesh), eps, False) <= 1.0
    # monopole order 0: nothing is accepted, every pair is summed
    with ct.TreePmCoordinator(config(mesh, ct._abi.FP64, multipole_order=0, softening=eps)) as s:
        r = s.solve_active_set(*p)
    assert beyond(r, reference(p, mesh, quadrupole=0, eps=eps), p, BOX, cell(mesh), eps, True) <= 1.0


@pytest.mark.parametrize("eps", [0.05, 0.0])
@pytest.mark.parametrize("count", [1, 5, 40, 333])
@pytest.mark.parametrize("mesh", [16, 40])
def test_sparse_and_explicit_targets(count, mesh, eps):
    p = particles(2500, 7)
    act = np.random.default_rng(count).permutation(2500)[:count].astype(np.uint32)
    # a run of 32 sparse targets may share an origin up to half a box away
    scale = dict(p=p, box=BOX, h=cell(mesh), eps=eps, rows=act, reach=0.6 * max(BOX))
    ref = reference(p, mesh, active=act, eps=eps)
    with ct.TreePmCoordinator(config(mesh, ct._abi.MIXED, softening=eps)) as s:
        assert beyond(s.solve_active_set(*p, active=act), ref, fp64=False, **scale) <= 1.0
        # the same targets given by position, a box length away on two axes
        t = (p[0][act] + BOX[0], p[1][act], p[2][act] - BOX[2])
        assert beyond(s.solve_active_set(*p, active=act, targets=t), ref, fp64=False, **scale) <= 1.0
    with ct.TreePmCoordinator(config(mesh, ct._abi.FP64, multipole_order=0, softening=eps)) as s:
        ref = reference(p, mesh, active=act, quadrupole=0, eps=eps)
        assert beyond(s.solve_active_set(*p, active=act), ref, fp64=True, **scale) <= 1.0
        if eps > 0.0:  # (moved by a box length, a coincident particle is an ulp away)
            assert beyond(s.solve_active_set(*p, active=act, targets=t), ref, fp64=True, **scale) <= 1.0


@pytest.mark.parametrize("explicit", [False, True])
@pytest.mark.parametrize("n", [300, 5000])
@pytest.mark.parametrize("mesh", [16, 48])
def test_softening_lanes(n, mesh, explicit):
    """Per-particle softening, none for a fifth of the particles, and targets with
    lanes of their own: mixed against the FP64 per-node walk."""
    p, rng = particles(n, 31 + n), np.random.default_rng(n)
    lane = np.where(rng.random(n) < 0.2, 0.0, 0.01 * 8.0 ** rng.random(n))
    if n > 4:
        lane[n // 2] = lane[n // 3] = 0.0  # the coincident pair, unsoftened
    act = rng.permutation(n)[:n // 3].astype(np.uint32)
    kw = dict(softening=lane)
    if explicit:
        kw.update(active=act, targets=tuple(p[k][act] for k in range(3)), target_softening=lane[act])
    out = {}
    for prec in (ct._abi.MIXED, ct._abi.FP64):
        with ct.TreePmCoordinator(config(mesh, prec)) as s:
            r = s.solve_active_set(*p, **kw)
            out[prec] = torch.stack([torch.as_tensor(np.asarray(r[k])) for k in ("ax", "ay", "az")])
    assert bool(torch.isfinite(out[ct._abi.MIXED]).all())
    assert apart(out[ct._abi.MIXED], out[ct._abi.FP64]) <= MIXED


@pytest.mark.parametrize("isolated", [False, True])
@pytest.mark.parametrize("n", [4735, 4736, 32001, 64005, 128031])
def test_lanes_per_target(n, isolated):
    """The sizes on both sides of each change of the lanes sharing a target:
    mixed against the FP64 walk (itself against the oracle above)."""
    p = particles(n, n)
    t = [torch.tensor(v, device="cuda") for v in p]
    kw = dict(boundary_condition=ct._abi.BOUNDARY_ISOLATED_OPEN) if isolated else {}
    if isolated:  # the isolated mesh has cubic cells
        kw.update(box_x=11.0, box_y=11.0, box_z=11.0)
    out = {}
    for prec in (ct._abi.MIXED, ct._abi.FP64):
        with ct.TreePmCoordinator(config(48, prec, **kw)) as s:
            r = s.solve_active_set(*t)
            out[prec] = torch.stack([r[k] for k in ("ax", "ay", "az")])
    assert apart(out[ct._abi.MIXED], out[ct._abi.FP64]) <= MIXED


@pytest.mark.parametrize("r_cut", [6.25, 9.0, 14.0])
def test_fp64_long_range_coefficient(r_cut):
    """r_cut / r_s of 5, 7.2 and 11.2: the polynomial and the closed form of the
    FP64 pairs."""
    p = particles(600, 3)
    with ct.TreePmCoordinator(config(48, ct._abi.FP64, multipole_order=0, rcut_cells=r_cut)) as s:
        r = s.solve_active_set(*p)
    assert beyond(r, reference(p, 48, quadrupole=0, rcut=r_cut), p, BOX, cell(48), 0.05, True, ratio=r_cut) <= 1.0


@pytest.mark.parametrize("equal", [True, False])
@pytest.mark.parametrize("mesh", [14, 48])
@pytest.mark.parametrize("n", [2, 33, 257, 5000])
def test_force_vjp_groups(n, mesh, equal):
    """The mixed adjoint walk (the same groups and images, equal masses as one
    value) against the FP64 adjoint; the bar is the forward walk's."""
    p = [torch.tensor(v, device="cuda") for v in particles(n, n + mesh)]
    if equal:
        p[3] = torch.full_like(p[3], 1.25)
    g = torch.Generator(device="cpu").manual_seed(n)
    cot = [torch.randn(n, generator=g, dtype=torch.float64).to("cuda") for _ in range(3)]
    out = {}
    for prec in (ct._abi.MIXED, ct._abi.FP64):
        with ct.TreePmCoordinator(config(mesh, prec)) as s:
            out[prec] = torch.stack(s.force_vjp(*p, *cot))
    d = torch.linalg.norm(out[ct._abi.MIXED] - out[ct._abi.FP64]) / torch.linalg.norm(out[ct._abi.FP64])
    assert float(d) <= MIXED
    if n > 2:  # (two particles: the smaller gradient is the difference of larger terms)
        assert apart(out[ct._abi.MIXED], out[ct._abi.FP64]) <= MIXED


# sides in units of 16 mesh cells; r_cut is 0.39 of the shortest
ELONGATED = [((6, 1, 1), 100, False), ((8, 1, 1), 100, False), ((10, 1, 1), 64, False), ((1, 16, 1), 400, False),
             ((12, 1, 1), 2000, True), ((6, 1, 6), 1500, True)]


def slab(sides, n, blob, seed):
    rng = np.random.default_rng(seed)
    x = rng.uniform(0.0, 1.0, (n, 3)) * np.array(sides)
    if blob:  # nine tenths in a blob across a corner of the box: the void's leaves are wide
        k = n - n // 10
        x[:k] = rng.normal(0.0, 0.08, (k, 3))
        x = np.mod(x, np.array(sides, dtype=float))
    return x[:, 0].copy(), x[:, 1].copy(), x[:, 2].copy(), rng.uniform(0.5, 2.0, n)


def slab_config(sides, precision, **kw):
    return ct.TreePmConfig(pm_grid_nx=16 * sides[0], pm_grid_ny=16 * sides[1], pm_grid_nz=16 * sides[2],
                           box_x=float(sides[0]), box_y=float(sides[1]), box_z=float(sides[2]), opening_theta=0.6,
                           max_leaf_size=16, softening=0.005, precision=precision, **kw)


@pytest.mark.parametrize("sides,n,blob", ELONGATED)
def test_elongated_boxes(sides, n, blob):
    """Leaves whose cubes span several short sides of the box: their sources are
    found at every image, for all targets and for a few."""
    p = slab(sides, n, blob, n)
    box, act = [float(v) for v in sides], np.arange(0, n, 7, dtype=np.uint32)
    for prec, quad in ((ct._abi.MIXED, 1), (ct._abi.FP64, 0)):
        o = oracle.treepm_solve(*p, oracle.make_params(box=box, mesh=tuple(16 * v for v in sides), theta=0.6, eps=0.005,
                                                       leaf=16, quadrupole=quad))
        ref = np.stack([o["ax"], o["ay"], o["az"]])
        with ct.TreePmCoordinator(slab_config(sides, prec, multipole_order=2 * quad)) as s:
            fp64 = prec == ct._abi.FP64
            assert beyond(s.solve_active_set(*p), ref, p, box, 1 / 16, 0.005, fp64) <= 1.0
            assert beyond(s.solve_active_set(*p, active=act), ref[:, act], p, box, 1 / 16, 0.005, fp64, act,
                          reach=max(box)) <= 1.0
    # the adaptive walk with a tolerance that accepts nothing: the same pairs
    prev = np.linalg.norm(ref, axis=0)
    with ct.TreePmCoordinator(slab_config(sides, ct._abi.MIXED, acceptance_policy=ct._abi.POLICY_ADAPTIVE,
                                          adaptive_error_estimator=ct._abi.ESTIMATOR_RELATIVE_MONOPOLE,
                                          relative_force_tolerance=1e-30)) as s:
        r = s.solve_active_set(*p, previous_acceleration=prev)
        assert beyond(r, ref, p, box, 1 / 16, 0.005, False, reach=max(box)) <= 1.0


@pytest.mark.parametrize("sides,n,blob", ELONGATED)
def test_force_vjp_elongated(sides, n, blob):
    """The mixed adjoint walk in the same boxes against the FP64 adjoint, each
    particle's gradient on the scale of the median one."""
    p = [torch.tensor(v, device="cuda") for v in slab(sides, n, blob, n)]
    g = torch.Generator(device="cpu").manual_seed(n)
    cot = [torch.randn(n, generator=g, dtype=torch.float64).to("cuda") for _ in range(3)]
    out = {}
    for prec in (ct._abi.MIXED, ct._abi.FP64):
        with ct.TreePmCoordinator(slab_config(sides, prec)) as s:
            out[prec] = torch.stack(s.force_vjp(*p, *cot))
    assert apart(out[ct._abi.MIXED], out[ct._abi.FP64]) <= MIXED


@pytest.mark.parametrize("equal", [False, True])
@pytest.mark.parametrize("eps", [1e-10, 1e-13])
def test_tiny_softening_and_heavy_masses(eps, equal):
    """m / eps^3 beyond FP32 with a softening that is only a guard: a target's
    own entry and a coincident particle still add nothing (full, active and
    explicit targets)."""
    n = 4000
    p = list(particles(n, 11))
    p[3] = np.full(n, 3.0e9) if equal else 10.0 ** np.random.default_rng(1).uniform(0.0, 10.0, n)
    act = np.arange(3, n, 11, dtype=np.uint32)
    t = (p[0][act] + BOX[0], p[1][act], p[2][act])
    cfg = dict(softening=eps)
    with ct.TreePmCoordinator(config(48, ct._abi.FP64, **cfg)) as s:
        r = s.solve_active_set(*p)
    ref = np.stack([np.asarray(r[k]) for k in ("ax", "ay", "az")])
    with ct.TreePmCoordinator(config(48, ct._abi.MIXED, **cfg)) as s:
        assert beyond(s.solve_active_set(*p), ref, p, BOX, cell(48), eps, False) <= 1.0
        assert beyond(s.solve_active_set(*p, active=act), ref[:, act], p, BOX, cell(48), eps, False, act) <= 1.0
        assert beyond(s.solve_active_set(*p, active=act, targets=t), ref[:, act], p, BOX, cell(48), eps, False, act) <= 1.0


def test_softening_in_small_units():
    """A softening below 1e-12 in a box of 1e-9 is a softening like any other:
    a blob of its size against the FP64 walk."""
    n, unit, eps = 4000, 1e-10, 9e-13
    p = list(particles(n, 5))
    rng = np.random.default_rng(2)
    for k in range(3):
        p[k][:500] = 0.6 * BOX[k] + rng.normal(0.0, 0.02, 500)
        p[k] *= unit
    cfg = dict(softening=eps, box_x=BOX[0] * unit, box_y=BOX[1] * unit, box_z=BOX[2] * unit)
    out = {}
    for prec in (ct._abi.MIXED, ct._abi.FP64):
        with ct.TreePmCoordinator(config(48, prec, **cfg)) as s:
            r = s.solve_active_set(*p)
            out[prec] = np.stack([np.asarray(r[k]) for k in ("ax", "ay", "az")])
    size = np.linalg.norm(out[ct._abi.FP64], axis=0)
    d = np.linalg.norm(out[ct._abi.MIXED] - out[ct._abi.FP64], axis=0)
    assert (d / (size + np.median(size))).max() <= MIXED


@pytest.mark.parametrize("away", [0, 1])
def test_fp64_coincident_and_close_pairs(away):
    """FP64 without softening: particles that coincide add nothing to each other,
    and pairs a few hundred ulps of the box length apart keep their separation,
    on either side of the tree frame's seam (the positions it moves by a box
    length are rounded there); away: every coordinate outside the box."""
    n = 4000
    p = list(particles(n, 17))
    rng = np.random.default_rng(4)
    at = rng.permutation(n)[:1200]
    for k in range(3):
        p[k][at[600:]] = p[k][at[:600]]  # 600 pairs, coincident
    far = at[900:]  # the last 300 of them 0.02 .. 0.5 * 2^-40 apart on each axis
    for k in range(3):
        p[k][far] = np.mod(p[k][far] + rng.uniform(0.02, 0.5, 300) * 2.0 ** -40, BOX[k])
        p[k] += away * (1, -2, 3)[k] * BOX[k]
    o = oracle.treepm_solve(*p, oracle.make_params(box=BOX, mesh=(48,) * 3, theta=0.6, eps=0.0, leaf=16, quadrupole=0))
    ref = np.stack([o["ax"], o["ay"], o["az"]])
    with ct.TreePmCoordinator(config(48, ct._abi.FP64, multipole_order=0, softening=0.0)) as s:
        for rows in (np.arange(n), at.astype(np.uint32)):
            r = s.solve_active_set(*p) if len(rows) == n else s.solve_active_set(*p, active=rows)
            got = np.stack([np.asarray(r[k]) for k in ("ax", "ay", "az")])
            assert np.isfinite(got).all()
            size = np.linalg.norm(ref[:, rows], axis=0)
            # a close pair's separation is exact up to 2^-53 of the offsets it is the
            # difference of (below 4 box-lengths / 10): 1e-3 of 2^-45 and more
            assert (np.linalg.norm(got - ref[:, rows], axis=0) <= 1e-3 * size + 1e-11 * np.median(size)).all()
            alone = ~np.isin(rows, at[300:600]) & ~np.isin(rows, far)
            scale = size[alone] + np.median(size)
            assert (np.linalg.norm(got - ref[:, rows], axis=0)[alone] / scale).max() <= 1e-11


def long_double_pairs(p, box, rs, rcut, eps):
    """Short-range accelerations in long double, and the sums of m d K_soft and
    m K_soft over each target's pairs."""
    x, m, L = np.stack(p[:3], 1).astype(np.longdouble), p[3], np.array(box, np.longdouble)
    acc, soft, slope = np.zeros(x.shape, np.longdouble), np.zeros(len(m)), np.zeros(len(m))
    for i in range(len(m)):
        d = x - x[i]
        d -= L * np.rint(d / L)
        r2 = (d * d).sum(1)
        use = (r2 <= np.longdouble(rcut) ** 2) & (r2 > 0)
        d, r2, mj = d[use], r2[use], m[use]
        t = r2 / (4 * np.longdouble(rs) ** 2)
        h, term = np.zeros_like(t), np.full_like(t, 1 / np.longdouble(3))
        for k in range(1, 120):  # H(t) = (4/sqrt(pi)) e^-t sum_k (2t)^k / (3 5 ... (2k+3))
            h, term = h + term, term * 2 * t / (2 * k + 3)
        h *= 4 / np.sqrt(np.longdouble("3.14159265358979323846264338327950288")) * np.exp(-t)
        k_soft = (r2 + np.longdouble(eps) ** 2) ** np.longdouble(-1.5)
        acc[i] = ((mj * (k_soft - h / (8 * np.longdouble(rs) ** 3)))[:, None] * d).sum(0)
        soft[i], slope[i] = float((mj * k_soft * np.sqrt(r2)).sum()), float((mj * k_soft).sum())
    return acc.T, soft, slope


def test_fp64_pairs_to_the_last_digits():
    """The FP64 pairs alone, against long double: every pair within 4e-16 of its
    K_soft part, offsets of up to 3 r_cut within 2^-53, sums of up to 2000 pairs.
    set_config changes the polynomial with the cutoff."""
    p = particles(2000, 23)
    p[0][0] = p[0][1] + 1e-6  # one close pair
    with ct.TreePmCoordinator(config(48, ct._abi.FP64, multipole_order=0, softening=0.002, short_range_only=1)) as s:
        for cells in (6.25, 4.5):
            s.set_config(config(48, ct._abi.FP64, multipole_order=0, softening=0.002, short_range_only=1, rcut_cells=cells))
            r = s.solve_active_set(*p)
            ref, soft, slope = long_double_pairs(p, BOX, 1.25 * cell(48), cells * cell(48), 0.002)
            d = np.sqrt(((np.stack([np.asarray(r[k]) for k in ("ax", "ay", "az")]) - ref) ** 2).sum(0)).astype(float)
            allow = 1.2e-15 * soft + 2.0 * slope * 3.0 * cells * cell(48) * 2.0 ** -53
            assert (d <= allow).all(), (d / allow).max()
