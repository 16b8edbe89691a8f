"""Kernel variants that are chosen by size or input range, at the edges of
those ranges, against the FP64 oracle."""
import numpy as np
import pytest

from miluphpc_b200 import ics
from miluphpc_b200.miluphpc import Miluphpc
from oracle import oracle as O
from tests.helpers import gravity_cfg, rel_err

pytestmark = pytest.mark.gpu


# ---------------------------------------------------------------- v2 walk
# 8 warps per group up to 296 groups, 4 up to 4736, then 2; a group is 32 particles
@pytest.mark.parametrize("n", [31, 33, 1000, 9472, 9473, 30_001, 151_552, 151_553])
def test_v2_walk_sizes(n, cuda):
    """Accelerations equal the oracle's warp-voted walk to rounding (the accept
    decisions are the same; sums of ~1000 terms in another order: 1e-9 as in
    the other v2 tests)."""
    P = ics.plummer(n, seed=5)
    sim = Miluphpc(gravity_cfg(sfc=1, theta=0.5, smoothing=1e-4), P)
    sim.rhs(0)
    bb = O.bbox(P["x"], P["y"], P["z"])
    T = O.Tree(P["x"], P["y"], P["z"], P["mass"], bb)
    _, perm = O.sort(O.keys(P["x"], P["y"], P["z"], bb, 1))
    o = O.gravity_v2(T, perm, 0.5 * (bb[1] - bb[0]), 0.5, 1e-4)
    g = [sim.numpy(f) for f in ("g_ax", "g_ay", "g_az")]
    big = np.sqrt(sum(c ** 2 for c in o)).max()
    assert max(np.abs(a - b).max() for a, b in zip(g, o)) <= 1e-9 * big
    sim.close()


@pytest.mark.parametrize("n", [3000, 12_000, 160_000])
def test_v2_walk_shared_keys(n, cuda):
    """Runs of identical positions (buckets longer than a block's step) with an
    opening parameter that accepts no cell: the direct sum over all particles."""
    P = ics.plummer(n, seed=8)
    for k in ("x", "y", "z"):
        P[k][100:800] = P[k][7]
        P[k][1500:1533] = P[k][900]
    sim = Miluphpc(gravity_cfg(sfc=0, theta=1e-6, smoothing=1e-4), P)
    sim.rhs(0)
    tg = np.unique(np.concatenate([[7, 100, 799, 900, 1500], np.arange(0, n, 97)])).astype(np.int32)
    o = O.direct(P["x"], P["y"], P["z"], P["mass"], tg, 1e-4)[:3]
    g = [sim.numpy(f)[tg] for f in ("g_ax", "g_ay", "g_az")]
    assert rel_err(*g, *o).max() < 1e-9
    sim.close()
