"""The periodic unwrap's anchors (the value after the largest circular gap of
each axis) at the sizes around the change from one block per axis to the
launches over all buckets, against sorted coordinates."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import chui_treepm as ct  # noqa: E402

pytestmark = pytest.mark.gpu

BOX = (10.0, 9.0, 11.0)


def anchor_of(x, box):
    v = x - box * np.floor(x / box)
    v[v >= box] = 0.0
    v = np.sort(v)
    after = np.append(v[1:], v[0])
    gap = np.append(v[1:], v[0] + box) - v
    return after[gap == gap.max()].min()


@pytest.mark.parametrize("n", [1, 2, 9, 1000, 8200, 262136, 262152])
@pytest.mark.parametrize("holes", [False, True])
def test_anchors(n, holes):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(n)
    p = [rng.uniform(-0.3, 1.3, n) * L for L in BOX]
    if holes:  # a wide empty band: its edge is the anchor
        p = [np.where((v % L > 0.4 * L) & (v % L < 0.55 * L), v + 0.2 * L, v) for v, L in zip(p, BOX)]
    cfg = ct.TreePmConfig(pm_grid_nx=32, pm_grid_ny=32, pm_grid_nz=32, box_x=BOX[0], box_y=BOX[1], box_z=BOX[2],
                          softening=0.05)
    with ct.TreePmCoordinator(cfg) as s:
        s.solve_active_set(*p, np.ones(n), active=np.zeros(1, dtype=np.uint32))
        d = s.dump_tree(n)
    for a, (v, L) in enumerate(zip(p, BOX)):
        want = anchor_of(v, L)
        assert d["anchors"][a] == want
        u = d["ux uy uz".split()[a]]
        assert u.min() >= want and u.max() <= want + L
