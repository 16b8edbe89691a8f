"""Kernel variants that are chosen by size or input range, at the edges of
those ranges, against the FP64 oracle."""
import ctypes

import numpy as np
import pytest
import torch

from miluphpc_b200 import _lib, ics
from miluphpc_b200.miluphpc import Miluphpc, material
from oracle import oracle as O
from tests.helpers import gravity_cfg, rel_err, sph_cfg

pytestmark = pytest.mark.gpu


def dptr(t):
    return ctypes.c_void_p(t.data_ptr())


def sedov_state(nside, seed=4):
    """Sedov lattice with a random velocity field (some pairs approach)."""
    S = ics.sedov(nside=nside, seed=seed)
    rng = np.random.default_rng(seed)
    for f in ("vx", "vy", "vz"):
        S[f] = 0.1 * rng.standard_normal(len(S["x"]))
    S["p"] = (S["gamma"] - 1.0) * S["e"]
    S["cs"] = np.sqrt(S["gamma"] * (S["gamma"] - 1.0) * S["e"])
    return S


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
    opening parameter that accepts only cells of a few 1e-5 (the buckets
    themselves): the direct sum over all particles.  A bucket of 700 acts on
    its own members through the rounding of its centre of mass, at most
    700 * 2^-53 |x| M / eps^3 = 2e-11 |g| here."""
    P = ics.plummer(n, seed=8)
    for k in ("x", "y", "z"):
        P[k][100:800] = P[k][7]
        P[k][1500:1533] = P[k][900]
    sim = Miluphpc(gravity_cfg(sfc=0, theta=1e-6, smoothing=1e-2), P)
    sim.rhs(0)
    tg = np.unique(np.concatenate([[7, 100, 799, 900, 1500], np.arange(0, n, 97)])).astype(np.int32)
    o = O.direct(P["x"], P["y"], P["z"], P["mass"], tg, 1e-2)[:3]
    g = [sim.numpy(f)[tg] for f in ("g_ax", "g_ay", "g_az")]
    assert rel_err(*g, *o).max() < 1e-9
    sim.close()


@pytest.mark.parametrize("k", [-90, -76, -73, -70, -66, -56, -40, 40, 66, 90])
def test_v2_walk_scales(k, cuda):
    """A system scaled by 2^k (every product of the walk scales exactly in FP64)
    has the same interactions, and its accelerations scale by 2^-2k: the cells
    that FP32 decides, and those it must leave to the vote because squares of
    their distances are below or above FP32's normal range."""
    n, s = 20_000, 2.0 ** k
    P = ics.plummer(n, seed=5)
    out = []
    for f in (1.0, s):
        sim = Miluphpc(gravity_cfg(sfc=1, theta=0.5, smoothing=1e-4 * f * f), {**P, **{c: P[c] * f for c in "xyz"}})
        sim.rhs(0)
        out.append((sim.stats()["gravity_interactions"], [sim.numpy(c) * f * f for c in ("g_ax", "g_ay", "g_az")]))
        sim.close()
    assert out[0][0] == out[1][0]
    assert rel_err(*out[1][1], *out[0][1]).max() < 1e-12


# two warps per group take a stack of 1536 entries below theta 0.3, else of 768
@pytest.mark.parametrize("theta", [1e-6, 0.02, 0.29, 0.3])
@pytest.mark.parametrize("n", [12_000, 151_553])
def test_v2_walk_small_theta(n, theta, cuda):
    """Opening parameters at which most cells open, so that the stack stays full:
    the oracle's interactions and accelerations (theta 1e-6: the direct sum)."""
    P = ics.plummer(n, seed=5)
    sim = Miluphpc(gravity_cfg(sfc=1, theta=theta, smoothing=1e-4), P)
    sim.rhs(0)
    g = [sim.numpy(f) for f in ("g_ax", "g_ay", "g_az")]
    if theta < 1e-3:
        tg = np.arange(0, n, n // 300).astype(np.int32)
        o = O.direct(P["x"], P["y"], P["z"], P["mass"], tg, 1e-4)[:3]
        g = [c[tg] for c in g]
    else:
        bb = O.bbox(P["x"], P["y"], P["z"])
        T = O.Tree(P["x"], P["y"], P["z"], P["mass"], bb)
        _, perm = O.sort(O.keys(P["x"], P["y"], P["z"], bb, 1))
        o = O.gravity_v2(T, perm, 0.5 * (bb[1] - bb[0]), theta, 1e-4)
    big = np.sqrt(sum(c ** 2 for c in o)).max()
    assert max(np.abs(a - b).max() for a, b in zip(g, o)) <= 1e-9 * big
    sim.close()


def test_v2_walk_time_small_theta(cuda):
    """Time per interaction at theta 0.05 within 1.5 times that at 0.5 (300,000
    particles; 2.2 times it when the stack of 768 entries held the steps back)."""
    P = ics.plummer(300_000, seed=3)
    per = []
    for theta in (0.5, 0.05):
        sim = Miluphpc(gravity_cfg(sfc=1, theta=theta, smoothing=1e-4), P)
        sim.rhs(0)
        t = []
        for _ in range(4):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            _lib.check(sim.L.mhpc_gravity(sim.ctx, ctypes.byref(sim.soa), 0), "gravity")
            b.record()
            torch.cuda.synchronize()
            t.append(a.elapsed_time(b))
        sim.rhs(0)
        per.append(min(t) / sim.stats()["gravity_interactions"])
        sim.close()
    assert per[1] < 1.5 * per[0], per


# -------------------------------------------------------------------- keys
def box_keys(x, y, z, lo, hi, curve):
    dev = torch.device("cuda:0")
    t = [torch.as_tensor(np.ascontiguousarray(a), device=dev) for a in (x, y, z)]
    bb = torch.tensor([lo, hi] * 3, dtype=torch.float64, device=dev)
    keys = torch.zeros(len(x), dtype=torch.int64, device=dev)
    _lib.check(_lib.load().mhpc_keys(*(dptr(a) for a in t), len(x), dptr(bb), curve, dptr(keys),
                                     ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "keys")
    return keys.cpu().numpy().view(np.uint64)


@pytest.mark.parametrize("curve", [0, 1])
@pytest.mark.parametrize("lo,hi", [(-1.0, 1.0), (-3.7, 11.3), (0.0, 1.0), (-1e-3, 0.0), (1e6, 1e6 + 1.0),
                                   (-1e9 - 1e-3, -1e9 + 1e-3), (-1e-290, 1e-290), (0.0, 5e-324 * 1e6),
                                   (-1e307, 1.2e308), (-1e200, 1e210), (2.0, 2.0)])
def test_keys_near_grid_points(lo, hi, curve, cuda):
    """Keys bit-equal to the oracle's bisection for coordinates on, next to (1 to
    3 ulp) and far from the 2^21 grid points of boxes around, beside and far
    from the origin, tiny, huge and empty boxes, and coordinates outside."""
    rng = np.random.default_rng(5)
    n = 60_000
    f = rng.integers(0, 2 ** 21 + 1, n) / 2.0 ** 21
    f[::3] = rng.uniform(0.0, 1.0, len(f[::3]))
    f[::50] = np.round(f[::50] * 64) / 64
    f[:4] = (0.0, 1.0, -0.01, 1.01)
    with np.errstate(over="ignore", invalid="ignore"):
        v = lo * (1.0 - f) + hi * f
        for k in range(3):
            m = rng.integers(0, 4, n) > k
            v = np.where(m, np.nextafter(v, rng.choice([lo - 1.0, hi + 1.0], n)), v)
    v = np.where(np.isfinite(v), v, lo)
    x, y, z = v[: n // 3], v[n // 3: 2 * (n // 3)], v[2 * (n // 3): 3 * (n // 3)]
    assert np.array_equal(box_keys(x, y, z, lo, hi, curve), O.keys(x, y, z, np.array([lo, hi] * 3), curve))


# -------------------------------------------------------------------- sort
def gpu_sort(keys, vals=None, in_place=False):
    dev = torch.device("cuda:0")
    n, L = len(keys), _lib.load()
    kin = torch.as_tensor(keys.view(np.int64), device=dev)
    vin = torch.as_tensor(vals, device=dev) if vals is not None else None
    kout = kin if in_place else torch.zeros(n, dtype=torch.int64, device=dev)
    vout = vin if in_place else torch.zeros(n, dtype=torch.int32, device=dev)
    nb = L.mhpc_sort_scratch_bytes(n)
    scratch = torch.zeros(nb, dtype=torch.uint8, device=dev)
    _lib.check(L.mhpc_sort_pairs(dptr(kin), dptr(vin) if vin is not None else None, dptr(kout), dptr(vout), n,
                                 dptr(scratch), nb, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "sort")
    assert int(scratch[nb - 256:nb - 252].view(torch.int32).item()) == 0
    return kout.cpu().numpy().view(np.uint64), vout.cpu().numpy()


# one block up to 1024 and 4096 keys, look-back with tiles of 1024 up to 200,000 and
# of 4096 up to 600,000, counted tiles of 2048 up to 6,000,000 and of 3072 above
@pytest.mark.parametrize("n", [1, 2, 33, 1023, 1024, 1025, 4095, 4096, 4097, 5121, 199_999, 200_000, 200_001, 600_000,
                               600_001, 1_000_003, 6_000_001])
def test_sort_sizes(n, cuda):
    """Stable ascending order over all 64 key bits, with and without values:
    random keys, few distinct keys, keys equal to the largest, descending."""
    rng = np.random.default_rng(n)
    kinds = [rng.integers(0, 2 ** 64 - 1, n, dtype=np.uint64, endpoint=True),
             rng.integers(0, 5, n).astype(np.uint64) << np.uint64(61),
             np.where(rng.random(n) < 0.5, np.uint64(2 ** 64 - 1), rng.integers(0, 2 ** 63, n).astype(np.uint64)),
             np.arange(n, 0, -1).astype(np.uint64) * np.uint64(3)]
    for i, keys in enumerate(kinds):
        vals = rng.permutation(n).astype(np.int32) if i % 2 else None
        order = np.argsort(keys, kind="stable")
        ks, vs = gpu_sort(keys, vals)
        assert np.array_equal(ks, keys[order])
        assert np.array_equal(vs, order.astype(np.int32) if vals is None else vals[order])


@pytest.mark.parametrize("n", [1, 33, 1000, 1024, 1025, 3000, 4096, 4097, 200_001, 600_001])
def test_sort_in_place(n, cuda):
    """Keys and values sorted in the arrays they came in, by every form of the
    sort (a value must be read before its place is written)."""
    for seed in range(5):
        rng = np.random.default_rng(seed)
        keys = rng.integers(0, 2 ** 64 - 1, n, dtype=np.uint64, endpoint=True)
        vals = rng.permutation(n).astype(np.int32)
        order = np.argsort(keys, kind="stable")
        ks, vs = gpu_sort(keys, vals, in_place=True)
        assert np.array_equal(ks, keys[order])
        assert np.array_equal(vs, vals[order])


def test_sort_scratch_serves_smaller_n(cuda):
    """Scratch made for n keys is large enough for every smaller number."""
    L = _lib.load()
    sizes = sorted({1, 1000, 4096, 4097, 199_999, 200_000, 200_001, 300_000, 599_999, 600_000, 600_001, 1 << 20, 6_000_000,
                    6_000_001, 1 << 24, 2_000_000_000})
    b = [L.mhpc_sort_scratch_bytes(n) for n in sizes]
    assert b == sorted(b)


# ------------------------------------------------------------- upward pass
# 4 positions per thread up to 8,192, 1 up to 65,536, 2 up to 200,000, 4 up to 454,656, 8 up to
# 909,312, 4 up to 1,060,864, then 8; with walk records (precision 1) eight lanes per cell up
# to 200,000, and no mask of leaf slots above 1,060,864; nodes are counted in one block up
# to 16,384
@pytest.mark.parametrize("n", [1, 2, 5, 8192, 8193, 16_384, 16_385, 65_536, 65_537, 200_000, 200_001, 454_656, 454_657,
                               909_312, 909_313, 1_060_864, 1_060_865, 2_000_001])
@pytest.mark.parametrize("precision", [0, 1])
def test_upward_pass_sizes(n, precision, cuda):
    """The cells' masses and centres of mass are bit-equal to the oracle's
    (Lebesgue order: the same sums; compared as sorted lists, the numbering
    differs), whatever the block sizes."""
    P = ics.plummer(n, seed=12) if n > 1 else {k: np.array([0.5]) for k in ("x", "y", "z", "mass", "vx", "vy", "vz")}
    sim = Miluphpc(gravity_cfg(sfc=0, precision=precision, theta_mixed=0.3), P)
    sim.rhs(0)
    bb = O.bbox(P["x"], P["y"], P["z"])
    T = O.Tree(P["x"], P["y"], P["z"], P["mass"], bb)
    tr = sim.export_tree(T.num_nodes)
    c = tr["cells"]
    assert c == T.nodes - n
    for k in ("m", "x", "y", "z"):
        assert np.array_equal(np.sort(tr[k][n:n + c]), np.sort(getattr(T, k)[n:n + c])), k
    sim.close()


# a block's range is 1024 sorted particles up to 8,192 and from 200,001 to 454,656, 2048
# up to 909,312 and from 1,060,865 on; its queue of hand-offs holds 1024
@pytest.mark.parametrize("n", [8_000, 20_000, 300_001, 500_001, 2_000_001])
@pytest.mark.parametrize("precision", [0, 1])
def test_upward_pass_runs_longer_than_a_block(n, precision, cuda):
    """Runs of identical positions longer than a block's range: a block inside one
    hands off every particle of its range, more than its queue holds.  Masses are
    equal powers of two and coordinates multiples of 2^-26, so the sums over a
    cell's particles (those with its prefix) are exact: masses equal, centres of
    mass within the roundings of a bucket's 2600 sums, 2600 * 2^-53 * 16 = 5e-12."""
    P = ics.plummer(n, seed=31)
    P["mass"] = np.full(n, 2.0 ** -22)
    for k in "xyz":
        P[k] = np.round(P[k] * 2.0 ** 26) * 2.0 ** -26
        for a, src in ((200, 100), (3000, 7000)):
            P[k][a:a + 2600] = P[k][src]
    sim = Miluphpc(gravity_cfg(sfc=0, precision=precision, theta_mixed=0.3), P)
    sp = ctypes.byref(sim.soa)
    _lib.check(sim.L.mhpc_stage_tree(sim.ctx, sp), "stage_tree")
    _lib.check(sim.L.mhpc_ctx_status(sim.ctx), "status")
    keys, perm = sim.export_sorted()
    tr = sim.export_tree()
    child = tr["child"].reshape(-1, 8)
    sums = {k: np.concatenate([[0.0], np.cumsum(P[k][perm])]) for k in "xyz"}
    node, pre = np.zeros(1, dtype=np.int64), np.zeros(1, dtype=np.uint64)
    cells = longest = 0
    for level in range(1, 22):
        ch = child[node].astype(np.int64)
        r, c = np.nonzero(ch >= n)
        node, pre = ch[r, c], (pre[r] << np.uint64(3)) | c.astype(np.uint64)
        if not len(node):
            break
        sh = np.uint64(3 * (21 - level))
        lo = np.searchsorted(keys, pre << sh, side="left")
        hi = np.searchsorted(keys, (pre << sh) | np.uint64((1 << (3 * (21 - level))) - 1), side="right")
        assert np.array_equal(tr["m"][node], (hi - lo) * 2.0 ** -22)
        for k in "xyz":
            assert np.abs(tr[k][node] - (sums[k][hi] - sums[k][lo]) / (hi - lo)).max() < 5e-12
        cells += len(node)
        if level == 21:
            longest = (hi - lo).max()
    assert cells == tr["cells"] and longest >= 2600
    sim.close()


# ------------------------------------------------------------------ list walk
# teams of four warps up to 340,992 particles (geometric rule with theta from 0.1 to 0.3:
# 606,208, relative rule: 1,060,864), then one warp a group; above 1,060,864 the
# records have no mask of leaf slots
@pytest.mark.parametrize("n,mac,theta,eps2", [(340_992, 0, 0.5, 1e-4), (340_993, 0, 0.5, 1e-4),
                                              (606_208, 0, 0.28, 1e-4), (606_209, 0, 0.28, 1e-4),
                                              (606_209, 0, 0.28, 0.0), (1_060_864, 1, 0.28, 1e-4),
                                              (1_060_865, 1, 0.28, 1e-4), (1_060_865, 1, 0.28, 0.0),
                                              (2_000_001, 0, 0.28, 1e-4), (2_000_001, 1, 0.28, 1e-4)])
def test_list_walk_sizes(n, mac, theta, eps2, cuda):
    """The list walk on either side of its lines, relative and geometric rule,
    guarded (eps2 = 0) or not: p99 <= 1e-3 of the direct sum (theta 0.28), and (eps2 > 0)
    close to the FP64 statement of the same rule with the same interactions;
    bars as for 131,072 particles in the parity tests."""
    P = ics.plummer(n, seed=1)
    sim = Miluphpc(gravity_cfg(sfc=1, precision=1, theta_mixed=theta, smoothing=eps2, gravity_mac=mac, mac_alpha=3e-3), P)
    sim.rhs(0)
    prev = np.sqrt(sum(sim.numpy(f) ** 2 for f in ("g_ax", "g_ay", "g_az")))
    if mac:
        sim.rhs(1)
    g = [sim.numpy(f) for f in ("g_ax", "g_ay", "g_az")]
    tg = np.random.default_rng(7).choice(n, 512, replace=False).astype(np.int32)
    d = O.direct(P["x"], P["y"], P["z"], P["mass"], tg, eps2)[:3]
    assert theta > 0.3 or np.percentile(rel_err(*(c[tg] for c in g), *d), 99) <= 1e-3
    if eps2 > 0:
        bb = O.bbox(P["x"], P["y"], P["z"])
        T = O.Tree(P["x"], P["y"], P["z"], P["mass"], bb)
        q = O.quad(T)
        _, perm = O.sort(O.keys(P["x"], P["y"], P["z"], bb, 1))
        radius = 0.5 * (bb[1] - bb[0])
        if mac:
            *o, cnt, nq = O.gravity_boxes_rel(T, perm, radius, 1.0, eps2, q, prev, 3e-3, 3)
        else:
            *o, cnt, nq = O.gravity_boxes(T, perm, radius, theta, eps2, q, gsize=64, nsub=8)
        assert np.percentile(rel_err(*g, *o), 99) < 2e-4
        st = sim.stats()
        assert abs(st["gravity_interactions"] / cnt.sum() - 1.0) < (3e-3 if mac else 1e-3)
        assert abs(st["gravity_quad_interactions"] / nq.sum() - 1.0) < (1e-2 if mac else 1e-3)
    sim.close()


@pytest.mark.parametrize("n", [606_208, 606_209])
def test_potential_walk_sizes(n, cuda):
    """Potentials of both forms of the list walk against the direct sum."""
    P = ics.plummer(n, seed=11)
    sim = Miluphpc(gravity_cfg(sfc=1, precision=1, theta_mixed=0.3, smoothing=1e-4), P)
    w, pot = sim.potential(per_particle=True)
    pot = pot.cpu().numpy()
    tg = np.arange(0, n, n // 512).astype(np.int32)
    ref = O.direct(P["x"], P["y"], P["z"], P["mass"], tg, 1e-4)[3]
    assert np.percentile(np.abs(pot[tg] / ref - 1.0), 99) < 1e-3
    assert abs(w - 0.5 * np.sum(P["mass"] * pot)) <= 1e-12 * abs(w)
    sim.close()


# ---------------------------------------------------------- gather by records
# fields of 192 MiB and more go through records of 4, 8 or 12 doubles: 6,291,456
# particles of 4 fields, 3,145,728 of 8, 2,097,152 of 12
@pytest.mark.parametrize("n", [6_291_455, 6_291_456])
def test_gather_gravity_fields(n, cuda):
    """x, y, z and mass (4 fields): masses and centres of mass of all cells
    bit-equal to the oracle's tree, masses all different."""
    P = ics.plummer(n, seed=12)
    P["mass"] = np.random.default_rng(1).uniform(0.5, 1.5, n) / n
    sim = Miluphpc(gravity_cfg(sfc=0), P)
    _lib.check(sim.L.mhpc_stage_tree(sim.ctx, ctypes.byref(sim.soa)), "stage_tree")
    _lib.check(sim.L.mhpc_ctx_status(sim.ctx), "status")
    bb = O.bbox(P["x"], P["y"], P["z"])
    T = O.Tree(P["x"], P["y"], P["z"], P["mass"], bb)
    tr = sim.export_tree(T.num_nodes)
    c = tr["cells"]
    assert c == T.nodes - n
    for k in ("m", "x", "y", "z"):
        assert np.array_equal(np.sort(tr[k][n:n + c]), np.sort(getattr(T, k)[n:n + c])), k
    sim.close()


@pytest.mark.parametrize("fields,nside", [(8, 146), (8, 147), (12, 127), (12, 128)])
def test_gather_sph_fields(fields, nside, cuda):
    """x, y, z, mass, h and v (8 fields), and with them e, rho, p and c_s (12
    fields, two materials by id): every field in its particle's place.  Material
    1 of the 12 has an equation of state without rules, so its p and c_s come
    back as they went in; material 0's follow from its e, rho and previous p.
    Forces of the shuffled lattice within 1e-10 of the oracle's."""
    n = nside ** 3
    rng = np.random.default_rng(nside)
    S = ics.sedov(nside=nside, seed=4, jitter=0.2)
    order = rng.permutation(n)
    S = {k: v[order] for k, v in S.items() if isinstance(v, np.ndarray)}
    S["sml"] = rng.uniform(1.1, 1.3, n) / nside
    S["mass"] = rng.uniform(0.5, 1.5, n) / n
    for k in ("vx", "vy", "vz"):
        S[k] = 0.1 * rng.standard_normal(n)
    for k in ("e", "rho", "p", "cs"):
        S[k] = rng.uniform(0.5, 1.5, n)
    mats = [material(interactions=60, eos_type=3)]
    if fields == 12:
        mats = [material(interactions=60, eos_type=9, gamma=1.5), material(interactions=60, eos_type=7)]
        S["material_id"] = rng.integers(0, 2, n).astype(np.int32)
    sim = Miluphpc(sph_cfg(integrate_density=int(fields == 12), max_num_interactions=40), S, materials=mats)
    sim.rhs(0)
    rho, p, cs = (sim.numpy(k) for k in ("rho", "p", "cs"))
    off, nbr = O.frnn(S["x"], S["y"], S["z"], S["sml"])
    assert np.array_equal(sim.numpy("noi"), np.diff(off))
    if fields == 12:
        m0 = S["material_id"] == 0
        assert np.array_equal(rho, S["rho"])
        assert np.array_equal(p[~m0], S["p"][~m0]) and np.array_equal(cs[~m0], S["cs"][~m0])
        np.testing.assert_allclose(p[m0], 0.5 * S["rho"][m0] * S["e"][m0], rtol=1e-15)
        np.testing.assert_allclose(cs[m0], np.sqrt(1.5 * S["p"][m0] / S["rho"][m0]), rtol=1e-15)
    else:
        want = O.density(S["x"], S["y"], S["z"], S["mass"], S["sml"], off, nbr)
        np.testing.assert_allclose(rho, want, rtol=1e-12)
    f = O.forces(S["x"], S["y"], S["z"], S["vx"], S["vy"], S["vz"], S["mass"], S["sml"], rho, p, cs, off, nbr, 1.0, 2.0)
    for got, want in zip(("ax", "ay", "az", "drhodt", "dedt"), f):
        assert np.abs(sim.numpy(got) - want).max() <= 1e-10 * np.abs(want).max(), got
    sim.close()


# --------------------------------------------------------------- pair sums
# 4 lanes per particle up to 65,536, then 2 (FP32 density: 1 above 500,000)
@pytest.mark.parametrize("nside", [9, 40, 41])
def test_pair_sums_lanes(nside, cuda):
    """FP64 density and forces of a jittered lattice with random velocities
    against the oracle over its brute-force lists (density 1e-12, forces
    1e-10 of the largest, as in the other parity tests)."""
    S = sedov_state(nside)
    n = nside ** 3
    sim = Miluphpc(sph_cfg(), S, materials=[material(interactions=60)])
    sim.rhs(0)
    off, nbr = O.frnn(S["x"], S["y"], S["z"], S["sml"])
    rho = O.density(S["x"], S["y"], S["z"], S["mass"], S["sml"], off, nbr)
    np.testing.assert_allclose(sim.numpy("rho"), rho, rtol=1e-12)
    p, cs = sim.numpy("p"), sim.numpy("cs")
    f = O.forces(S["x"], S["y"], S["z"], S["vx"], S["vy"], S["vz"], S["mass"], S["sml"], rho, p, cs, off, nbr, 1.0, 2.0)
    for got, want in zip(("ax", "ay", "az"), f[:3]):
        assert np.abs(sim.numpy(got) - want).max() <= 1e-10 * np.abs(want).max()
    assert len(rho) == n
    sim.close()


def test_pair_sums_fp32_large(cuda):
    """FP32 pair sums with one lane per particle in the density pass against the
    FP64 sums of the same state: rho within 2e-6, a within 2e-5 of its largest."""
    S = sedov_state(80)
    out = []
    for precision in (0, 1):
        sim = Miluphpc(sph_cfg(precision=precision), S, materials=[material(interactions=60)])
        sim.rhs(0)
        out.append([sim.numpy(f) for f in ("rho", "ax", "ay", "az", "drhodt", "dedt")])
        sim.close()
    assert np.abs(out[1][0] / out[0][0] - 1.0).max() < 2e-6
    for a, b in zip(out[0][1:], out[1][1:]):
        assert np.abs(a - b).max() <= 2e-5 * np.abs(a).max()


def test_sph_context_memory(cuda):
    """Device memory of an SPH context of 4,000,000 particles with lists of 8:
    610 bytes a particle before the pair sums had records (96 bytes in place of
    56), which the arrays of the band repair share.  5 bytes a particle of slack
    for the allocator's 2 MB pages."""
    n = 4_000_000
    cfg = sph_cfg(max_num_interactions=8)
    mat, ctx = material(), ctypes.c_void_p()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    _lib.check(_lib.load().mhpc_ctx_create(ctypes.byref(ctx), n, ctypes.byref(cfg), ctypes.byref(mat), 1), "create")
    used = before - torch.cuda.mem_get_info()[0]
    _lib.check(_lib.load().mhpc_ctx_destroy(ctx), "destroy")
    assert used <= 615 * n, used / n


# ------------------------------------------------------------ neighbour lists
@pytest.mark.parametrize("avg_h", [0, 1])
@pytest.mark.parametrize("scale,offset", [(1.0, 0.0), (1e-20, 0.0), (1e-14, 3e-15), (1e20, 0.0), (1.0, 1e6), (1.0, -3e3)])
def test_neighbour_lists_scales(scale, offset, avg_h, cuda):
    """Every list equals the brute-force set at scales where the FP32 form of the
    pair test holds and where it does not, far from the origin, with particles
    far outside (groups much wider than h) and distances that equal h."""
    rng = np.random.default_rng(17)
    C = ics.rotating_cloud(4000, seed=6)
    n = 4096
    pos = {k: np.concatenate([C[k], np.zeros(96)]) for k in ("x", "y", "z")}
    g = np.arange(64)
    pos["x"][4000:4064], pos["y"][4000:4064], pos["z"][4000:4064] = 3.0 + 0.25 * (g & 3), 0.25 * ((g >> 2) & 3), 0.25 * (g >> 4)
    for k in ("x", "y", "z"):
        pos[k][4064:] = rng.uniform(-1e3, 1e3, 32)
        pos[k] = pos[k] * scale + offset
    h = np.full(n, C["sml"][0])
    if avg_h:
        h = h * rng.uniform(0.6, 1.4, n)
    h[4000:4064] = 0.25  # lattice neighbours at exactly h: no pair
    h[4064:] = 40.0 if avg_h else h[0]
    S = dict(pos, sml=h * scale, mass=np.full(n, 1.0 / n), e=np.ones(n), rho=np.ones(n), p=np.ones(n), cs=np.ones(n),
             **{f: np.zeros(n) for f in ("vx", "vy", "vz")})
    sim = Miluphpc(sph_cfg(integrate_sml=avg_h, integrate_energy=0, max_num_interactions=400), S,
                   materials=[material(interactions=60, eos_type=0, K=1.0, gamma=1.0)], want_nnl=True)
    sim.rhs(0)
    off, nbr = O.frnn(S["x"], S["y"], S["z"], S["sml"])
    noi = sim.numpy("noi")
    assert np.array_equal(noi, np.diff(off))
    nnl = sim.t["nnl"].cpu().numpy().reshape(n, 400)
    for i in range(n):
        assert np.array_equal(np.sort(nnl[i, :noi[i]]), nbr[off[i]:off[i + 1]]), i
    sim.close()


def sparse_state(nside, spacings, jitter=0.3, seed=3):
    """Jittered lattice with h of `spacings` lattice spacings, for EOS 0."""
    S = ics.sedov(nside=nside, seed=seed, jitter=jitter)
    n = nside ** 3
    return dict({k: S[k] for k in ("x", "y", "z")}, sml=np.full(n, spacings / nside), mass=np.full(n, 1.0 / n),
                e=np.ones(n), rho=np.ones(n), p=np.ones(n), cs=np.ones(n), **{f: np.zeros(n) for f in ("vx", "vy", "vz")})


@pytest.mark.parametrize("nside,spacings", [(16, 0.0)] + [(k, f) for k in (16, 33, 41) for f in (0.3, 0.8, 1.2)])
def test_neighbour_lists_sparse(nside, spacings, cuda):
    """Lists where h is about the spacing or less (every gap between consecutive
    particles is longer than the cut in h; groups of 8, 16 and 32) equal the
    brute-force sets."""
    S, n = sparse_state(nside, spacings), nside ** 3
    if spacings == 0.0:
        S["sml"][:] = 1e-300
    sim = Miluphpc(sph_cfg(integrate_energy=0, max_num_interactions=64), S,
                   materials=[material(interactions=60, eos_type=0, K=1.0, gamma=1.0)], want_nnl=True)
    sp = ctypes.byref(sim.soa)
    for f in ("tree_build", "com"):
        _lib.check(getattr(sim.L, "mhpc_" + f)(sim.ctx, sp), f)
    _lib.check(sim.L.mhpc_frnn(sim.ctx, sp, 0, 0), "frnn")
    _lib.check(sim.L.mhpc_forces(sim.ctx, sp), "forces")
    off, nbr = O.frnn(S["x"], S["y"], S["z"], S["sml"])
    noi = sim.numpy("noi")
    assert np.array_equal(noi, np.diff(off))
    nnl = np.sort(np.where(np.arange(64) < noi[:, None], sim.t["nnl"].cpu().numpy().reshape(n, 64), n), axis=1)
    want = np.full((n, 64), n)
    want[np.arange(64) < noi[:, None]] = nbr
    assert np.array_equal(nnl, want)
    sim.close()


def test_neighbour_walk_sparse_time(cuda):
    """The walk of a lattice whose h is below its spacing costs no more than
    twice the one whose h reaches the next neighbours (a group cut at every
    particle walks 32 times: 6.6 times the cost)."""
    us = []
    for spacings in (0.4, 1.0):
        sim = Miluphpc(sph_cfg(integrate_energy=0, max_num_interactions=64), sparse_state(64, spacings, jitter=1e-3),
                       materials=[material(interactions=60, eos_type=0, K=1.0, gamma=1.0)])
        sp = ctypes.byref(sim.soa)
        for f in ("tree_build", "com"):
            _lib.check(getattr(sim.L, "mhpc_" + f)(sim.ctx, sp), f)
        t = []
        for _ in range(8):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            _lib.check(sim.L.mhpc_frnn(sim.ctx, sp, 0, 0), "frnn")
            b.record()
            torch.cuda.synchronize()
            t.append(a.elapsed_time(b) * 1e3)
        us.append(min(t[2:]))
        sim.close()
    assert us[0] < 2.0 * us[1], us


# 8 particles per warp up to 25,000, 16 up to 65,000, then 32
@pytest.mark.parametrize("n", [25_000, 25_001, 65_000, 65_001])
def test_neighbour_counts_group_sizes(n, cuda):
    """Counts of the neighbour walk and of the variable-h walk (same start h, one
    sweep decides nothing: tolerance above every count) are the brute-force
    counts at the edges of the group sizes."""
    C = ics.rotating_cloud(n, seed=8)
    rng = np.random.default_rng(n)
    S = dict({k: C[k] for k in ("x", "y", "z")}, sml=C["sml"] * rng.uniform(0.7, 1.2, n), mass=np.full(n, 1.0 / n),
             e=np.ones(n), rho=np.ones(n), p=np.ones(n), cs=np.ones(n), **{f: np.zeros(n) for f in ("vx", "vy", "vz")})
    off, _ = O.frnn(S["x"], S["y"], S["z"], S["sml"])
    for kw in (dict(integrate_sml=1), dict(variable_sml=1, nb_tolerance=1000)):
        sim = Miluphpc(sph_cfg(integrate_energy=0, max_num_interactions=400, **kw), S,
                       materials=[material(interactions=60, eos_type=0, K=1.0, gamma=1.0)])
        sim.rhs(0)
        assert np.array_equal(sim.numpy("sml"), S["sml"])
        assert np.array_equal(sim.numpy("noi"), np.diff(off))
        sim.close()


# lists with appended entries are sorted with 2 entries per lane up to 64, 8 up
# to 256, by one lane above
@pytest.mark.parametrize("target", [55, 200, 270])
@pytest.mark.parametrize("rounds", [0, 4])
def test_appended_lists(target, rounds, cuda):
    """Lists of a variable-h cloud equal the brute-force sets of its final h,
    whatever length the appended lists are sorted at."""
    n = 3000
    C = ics.rotating_cloud(n, seed=9)
    rng = np.random.default_rng(target)
    h = C["sml"] * (target / 60.0) ** (1.0 / 3.0) * rng.uniform(0.8, 1.2, n)
    S = dict({k: C[k] for k in ("x", "y", "z")}, sml=h, mass=np.full(n, 1.0 / n),
             e=np.ones(n), rho=np.ones(n), p=np.ones(n), cs=np.ones(n), **{f: np.zeros(n) for f in ("vx", "vy", "vz")})
    sim = Miluphpc(sph_cfg(variable_sml=1, integrate_energy=0, max_num_interactions=700, sml_band_rounds=rounds), S,
                   materials=[material(interactions=target, eos_type=0, K=1.0, gamma=1.0)], want_nnl=True)
    sim.rhs(0)
    off, nbr = O.frnn(S["x"], S["y"], S["z"], sim.numpy("sml"))
    noi = sim.numpy("noi")
    assert np.array_equal(noi, np.diff(off))
    nnl = sim.t["nnl"].cpu().numpy().reshape(n, 700)
    for i in range(n):
        assert np.array_equal(np.sort(nnl[i, :noi[i]]), nbr[off[i]:off[i + 1]]), i
    sim.close()


def test_neighbour_walk_wide_bucket(cuda):
    """A shared-key bucket of more than 65,536 particles, which the walks stage as
    one range: 80,000 particles on a line shorter than a grid cell, 2.5 spacings
    of h, so each has its two neighbours on either side."""
    n, d = 80_000, 5e-13
    x = np.concatenate([0.3 + d * np.arange(n), [0.0, 1.0]])
    y, z = np.full(n + 2, 0.3), np.full(n + 2, 0.3)
    y[n:] = z[n:] = [0.0, 1.0]
    h = np.full(n + 2, 2.5 * d)
    S = dict(x=x, y=y, z=z, sml=h, mass=np.full(n + 2, 1.0 / n), e=np.ones(n + 2), rho=np.ones(n + 2),
             p=np.ones(n + 2), cs=np.ones(n + 2), **{f: np.zeros(n + 2) for f in ("vx", "vy", "vz")})
    want = np.array([np.sum(np.abs(x[max(0, i - 4):min(n, i + 5)] - x[i]) < h[i]) - 1 for i in range(n)])
    sim = Miluphpc(sph_cfg(integrate_energy=0, max_num_interactions=64), S,
                   materials=[material(interactions=60, eos_type=0, K=1.0, gamma=1.0)])
    sim.rhs(0)
    noi = sim.numpy("noi")
    assert np.array_equal(noi[:n], want) and (noi[n:] == 0).all()
    sim.close()
