"""Timed cases of the framework's public entry points.

Each case is a piece of work that a simulation run on this library does step
after step: an integration step of a self-gravitating sphere (plain FP64 or
mixed precision), of a Sedov blast (SPH, predictor-corrector), of a rotating
self-gravitating gas cloud with variable smoothing lengths, a step on state
that lives in host memory, and the stateless ordering of particles along the
space-filling curve.  Sizes run from 1,000 particles, where a step is a chain
of short launches, to 2^24.

    listed()            the named cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) inputs and the context (made from the seed alone)
    run(state)          one pass through the public entry points
    work(case)          bytes and operations one pass cannot do without
    tolerance(case)     how far another correct implementation may be off
    exact(case, seed)   what run() returns, in plain FP64 torch
"""
import ctypes
import math

import torch

from miluphpc_b200 import _lib
from miluphpc_b200.miluphpc import Miluphpc, material

DEV = "cuda:0"
EPS2 = 1e-4          # Plummer softening^2
GAMMA = 5.0 / 3.0
# opening parameters of the mixed walk at p99 force error < 1e-3
THETA_MIXED, MAC_ALPHA, MAC_QUAD = 0.28, 1.8e-3, 3e-4
CLOUD_CS2 = 0.26 * (3.0 / 5.0) / 1.5
# direct sums and neighbour sums in FP64 torch stay within seconds up to these sizes
EXACT_GRAVITY_N = 300_000
EXACT_SPH_N = 3_000_000


def listed():
    return [
        # a test particle set or a star cluster: every step is a chain of short launches
        dict(name="plummer_1k_fp64", kind="plummer", n=1000, precision=0, sfc=0, dt=0.005, mac=0, v1=0, host=0),
        # the reference's own single-GPU case (Lebesgue order, theta 0.5, leapfrog dt 0.025)
        dict(name="plummer_131k_fp64", kind="plummer", n=131072, precision=0, sfc=0, dt=0.025, mac=0, v1=0, host=0),
        # a globular-cluster sized run in mixed precision, no round size
        dict(name="plummer_100k_mixed", kind="plummer", n=100003, precision=1, sfc=1, dt=0.01, mac=1, v1=0, host=0),
        # a program that keeps its state in (pinned) host memory and hands it in every step
        dict(name="plummer_1m_host", kind="plummer", n=1000003, precision=1, sfc=1, dt=0.01, mac=1, v1=0, host=1),
        # one galaxy component; its tree is larger than L2
        dict(name="plummer_2m_mixed", kind="plummer", n=1 << 21, precision=1, sfc=1, dt=0.01, mac=1, v1=0, host=0),
        # the headline workload
        dict(name="plummer_16m_mixed", kind="plummer", n=1 << 24, precision=1, sfc=1, dt=0.01, mac=1, v1=0, host=0),
        # Sedov blast, the reference's SPH test case, plain FP64 (two right-hand sides a step)
        dict(name="sedov_262k_fp64", kind="sedov", nside=64, precision=0, sfc=0, balsara=0),
        # the same at the scale of a production run, FP32 pair sums
        dict(name="sedov_2m_mixed", kind="sedov", nside=128, precision=1, sfc=0, balsara=0),
        # a small collapse run with the reference's semantics throughout (odd size)
        dict(name="cloud_20k_fp64", kind="cloud", n=20011, precision=0, sfc=1, dt=0.001, rounds=0),
        # collapse runs: gravity + SPH + variable h with the neighbour-band repair
        dict(name="cloud_1m_mixed", kind="cloud", n=1 << 20, precision=1, sfc=1, dt=0.002, rounds=8),
        dict(name="cloud_8m_mixed", kind="cloud", n=1 << 23, precision=1, sfc=1, dt=0.002, rounds=8),
        # ordering particles along the curve with the stateless calls (a code that has its own tree)
        dict(name="sfc_order_3m", kind="order", n=3000017, sfc=1),
    ]


def _log_int(rng, lo, hi):
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return min(hi, max(lo, v))


def draw(rng):
    kind = rng.choice(["plummer", "plummer", "sedov", "cloud", "order"])
    if kind == "plummer":
        precision = rng.choice([0, 1, 1])
        n = _log_int(rng, 1000, 1 << 20) if precision == 0 else _log_int(rng, 1000, 1 << 23)
        host = int(precision == 1 and n < 1 << 21 and rng.random() < 0.2)
        return dict(kind=kind, n=n, precision=precision, sfc=rng.choice([0, 1]), dt=0.005 if n < 50000 else 0.01,
                    mac=int(precision == 1 and rng.random() < 0.7), v1=int(precision == 0 and rng.random() < 0.2),
                    host=host)
    if kind == "sedov":
        return dict(kind=kind, nside=_log_int(rng, 16, 120), precision=rng.choice([0, 1]), sfc=rng.choice([0, 1]),
                    balsara=int(rng.random() < 0.25))
    if kind == "cloud":
        n = _log_int(rng, 5000, 3 << 20)
        return dict(kind=kind, n=n, precision=rng.choice([0, 1, 1]) if n < 1 << 20 else 1, sfc=rng.choice([0, 1]),
                    dt=0.001 if n < 1 << 19 else 0.002, rounds=rng.choice([0, 8]))
    return dict(kind=kind, n=_log_int(rng, 1000, 1 << 24), sfc=rng.choice([0, 1]))


# ------------------------------------------------------------------ inputs
def _rng(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _uniform(g, n, lo=0.0, hi=1.0):
    return torch.rand(n, generator=g, device=DEV, dtype=torch.float64) * (hi - lo) + lo


def _directions(g, n, r):
    ct, ph = _uniform(g, n, -1.0, 1.0), _uniform(g, n, 0.0, 2.0 * math.pi)
    st = torch.sqrt(1.0 - ct * ct)
    return r * st * torch.cos(ph), r * st * torch.sin(ph), r * ct


def _plummer(n, seed):
    """Plummer sphere, G = M = a = 1, cut at 10 a, isotropic equilibrium velocities."""
    g = _rng(seed)
    mmax = 1000.0 / 101.0 ** 1.5  # mass inside r = 10
    m = torch.clamp(_uniform(g, n) * mmax, min=1e-12)
    r = 1.0 / torch.sqrt(m ** (-2.0 / 3.0) - 1.0)
    x, y, z = _directions(g, n, r)
    q = torch.empty(n, dtype=torch.float64, device=DEV)
    todo = torch.arange(n, device=DEV)
    while todo.numel():
        q0, g0 = _uniform(g, todo.numel()), _uniform(g, todo.numel(), 0.0, 0.1)
        ok = g0 < q0 * q0 * (1.0 - q0 * q0) ** 3.5
        q[todo[ok]] = q0[ok]
        todo = todo[~ok]
    vx, vy, vz = _directions(g, n, q * math.sqrt(2.0) * (1.0 + r * r) ** -0.25)
    s = dict(x=x, y=y, z=z, vx=vx, vy=vy, vz=vz)
    for f in s:
        s[f] -= s[f].mean()
    s["mass"] = torch.full((n,), 1.0 / n, dtype=torch.float64, device=DEV)
    return s


def _cubic(r, h):
    """Cubic spline with support h: W and dW/dr."""
    q = r / h
    f = 8.0 / math.pi / h ** 3
    a = 1.0 - q
    w = torch.where(q > 0.5, 2.0 * f * a ** 3, f * (6.0 * q ** 3 - 6.0 * q * q + 1.0))
    d = torch.where(q > 0.5, -6.0 * f / h * a * a, 6.0 * f / h * (3.0 * q * q - 2.0 * q))
    inside = q <= 1.0
    return torch.where(inside, w, 0.0), torch.where(inside, d, 0.0)


def _sedov(nside, seed):
    """Sedov blast: jittered lattice in [-0.5, 0.5]^3, rho = 1, energy 1 spread over
    r < 2h, h = 2.5 lattice steps, a subsonic velocity field on top."""
    g = _rng(seed)
    n, dx = nside ** 3, 1.0 / nside
    c = -0.5 + (torch.arange(nside, device=DEV, dtype=torch.float64) + 0.5) * dx
    z, y, x = (t.reshape(-1) + _uniform(g, n, -1e-3, 1e-3) * dx for t in torch.meshgrid(c, c, c, indexing="ij"))
    h = 2.5 * dx
    w, _ = _cubic(torch.sqrt(x * x + y * y + z * z), 2.0 * h)
    mass = torch.full((n,), 1.0 / n, dtype=torch.float64, device=DEV)
    e = 1e-6 + w / w.sum() * n
    s = dict(x=x, y=y, z=z, mass=mass, e=e)
    for f in ("vx", "vy", "vz"):
        s[f] = 1e-3 * torch.randn(n, generator=g, device=DEV, dtype=torch.float64)
    s["sml"] = torch.full_like(mass, h)
    s["rho"] = torch.ones_like(mass)
    s["p"] = (GAMMA - 1.0) * e
    s["cs"] = torch.sqrt(GAMMA * (GAMMA - 1.0) * e)
    return s


def _cloud(n, seed):
    """Uniform sphere with a 10 % m = 2 density perturbation, solid-body rotation
    (E_rot / |E_grav| = 0.16), isothermal (E_th / |E_grav| = 0.26), G = M = R = 1."""
    g = _rng(seed)
    parts, got = [], 0
    while got < n:
        k = int((n - got) * 2.2) + 1024
        p = _uniform(g, 3 * k, -1.0, 1.0).reshape(k, 3)
        u = _uniform(g, k, 0.0, 1.1)
        keep = ((p * p).sum(1) < 1.0) & (u < 1.0 + 0.1 * torch.cos(2.0 * torch.atan2(p[:, 1], p[:, 0])))
        p = p[keep][: n - got]
        parts.append(p)
        got += p.shape[0]
    p = torch.cat(parts)
    x, y, z = (p[:, d].contiguous() for d in range(3))
    omega = math.sqrt(2.0 * 0.16 * 0.6 / 0.4)
    full = lambda v: torch.full((n,), v, dtype=torch.float64, device=DEV)  # noqa: E731
    return dict(x=x, y=y, z=z, vx=-omega * y, vy=omega * x, vz=full(0.0), mass=full(1.0 / n),
                sml=full((60.0 / n) ** (1.0 / 3.0)), e=full(CLOUD_CS2), rho=full(3.0 / (4.0 * math.pi)))


def _inputs(case, seed):
    if case["kind"] == "sedov":
        return _sedov(case["nside"], seed)
    return _cloud(case["n"], seed) if case["kind"] == "cloud" else _plummer(case["n"], seed)


# --------------------------------------------------------- context and calls
SEDOV_DT = 1e-6


def _config(case):
    if case["kind"] == "plummer":
        return _lib.default_config(gravity=1, sph=0, integrator=2, time_step=case["dt"], smoothing=EPS2,
                                   sfc=case["sfc"], theta=0.5, theta_mixed=THETA_MIXED, precision=case["precision"],
                                   gravity_mac=case["mac"], mac_alpha=MAC_ALPHA, mac_quad_alpha=MAC_QUAD,
                                   gravity_force_version=2 if case["v1"] else 0)
    if case["kind"] == "sedov":
        return _lib.default_config(gravity=0, sph=1, integrator=1, max_time_step=SEDOV_DT, time_end=1e30,
                                   smoothing_kernel=1, integrate_energy=1, integrate_density=0, sfc=case["sfc"],
                                   precision=case["precision"], balsara=case["balsara"])
    return _lib.default_config(gravity=1, sph=1, integrator=0, time_step=case["dt"], smoothing=0.0,
                               softening_mode=1, softening_h_factor=0.5, sfc=case["sfc"], variable_sml=1,
                               smoothing_kernel=1, integrate_energy=0, precision=case["precision"], theta=0.5,
                               theta_mixed=0.25, gravity_mac=int(case["precision"] == 1), mac_alpha=1.5e-3,
                               mac_quad_alpha=0.0, sml_band_rounds=case["rounds"])


def _materials(case):
    if case["kind"] == "cloud":
        return [material(interactions=60, alpha=1.0, beta=2.0, eos_type=0, K=CLOUD_CS2, gamma=1.0)]
    return [material(interactions=60, alpha=1.0, beta=2.0, eos_type=9, gamma=GAMMA)]


OUT = {
    "plummer": ["x", "y", "z", "vx", "vy", "vz", "g_ax", "g_ay", "g_az"],
    "sedov": ["x", "y", "z", "vx", "vy", "vz", "e", "rho", "p", "cs", "ax", "ay", "az", "drhodt", "dedt", "noi"],
    "cloud": ["x", "y", "z", "vx", "vy", "vz", "g_ax", "g_ay", "g_az", "sml", "rho", "p", "cs", "ax", "ay", "az",
              "drhodt", "noi"],
}


def prepare(case, seed):
    s = _inputs(case, seed)
    n = int(s["x"].numel())
    if case["kind"] == "order":
        L = _lib.load()
        nbytes = int(L.mhpc_sort_scratch_bytes(n))
        state = dict(case=case, L=L, n=n, x=s["x"], y=s["y"], z=s["z"], nbytes=nbytes,
                     bbox=torch.zeros(6, dtype=torch.float64, device=DEV),
                     keys=torch.zeros(n, dtype=torch.int64, device=DEV),
                     skeys=torch.zeros(n, dtype=torch.int64, device=DEV),
                     perm=torch.zeros(n, dtype=torch.int32, device=DEV),
                     scratch=torch.empty(nbytes, dtype=torch.uint8, device=DEV))
        return state
    if case.get("host"):
        # the particles in pinned host memory; the context's own device copy is made inside the step
        sim = Miluphpc(_config(case), {"x": [0.0]}, materials=_materials(case), capacity=n, device=DEV)
        host, soa = {}, _lib.Particles()
        soa.n = soa.num_nodes = n
        for f in ("x", "y", "z", "mass", "vx", "vy", "vz", "g_ax", "g_ay", "g_az"):
            host[f] = torch.zeros(n, dtype=torch.float64, pin_memory=True)
            if f in s:
                host[f].copy_(s[f])
            setattr(soa, f, ctypes.cast(ctypes.c_void_p(host[f].data_ptr()), _lib.P_d))
        return dict(case=case, sim=sim, host=host, soa=soa, step=0)
    sim = Miluphpc(_config(case), {"x": torch.zeros(n, dtype=torch.float64).numpy()}, materials=_materials(case),
                   device=DEV)
    for f, v in s.items():
        sim.t[f][:n].copy_(v)
    return dict(case=case, sim=sim, step=0)


def run(state):
    case = state["case"]
    if case["kind"] == "order":
        L, n = state["L"], state["n"]
        p = lambda t: ctypes.c_void_p(state[t].data_ptr())  # noqa: E731
        stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        _lib.check(L.mhpc_bbox(p("x"), p("y"), p("z"), n, p("bbox"), stream), "bbox")
        _lib.check(L.mhpc_keys(p("x"), p("y"), p("z"), n, p("bbox"), case["sfc"], p("keys"), stream), "keys")
        _lib.check(L.mhpc_sort_pairs(p("keys"), None, p("skeys"), p("perm"), n, p("scratch"), state["nbytes"],
                                     stream), "sort_pairs")
        return dict(bbox=state["bbox"], keys=state["keys"], skeys=state["skeys"], perm=state["perm"])
    sim, step = state["sim"], state["step"]
    state["step"] = step + 1
    if case.get("host"):
        dt = ctypes.c_double(0)
        _lib.check(sim.L.mhpc_integrate_host(sim.ctx, ctypes.byref(state["soa"]), step, ctypes.byref(dt)),
                   "integrate_host")
        return {f: state["host"][f] for f in OUT["plummer"]}
    sim.integrate(step)
    return {f: sim.t[f] for f in OUT[case["kind"]]}


# ------------------------------------------------------------ work and errors
def _count(case):
    return case["nside"] ** 3 if case["kind"] == "sedov" else case["n"]


def work(case):
    n = _count(case)
    if case["kind"] == "order":
        # positions read, keys, sorted keys and permutation written; 21 bisections of 3 axes
        return {"bytes": n * (24 + 8 + 8 + 4.0), "flops": n * 63 * 3.0}
    # accepted nodes of the tree walk: 19 flop each, 34 more for a quadrupole
    if case["precision"]:
        nodes = min(n, 1550.0)
        gravity = nodes * (45.5 if case["kind"] == "cloud" else 29.0)
    else:
        gravity = min(n, 63.0 * math.log2(n)) * 19.0
    if case["kind"] == "plummer":
        # state in (x, m, v, g), state out (x, v, g, g_old)
        return {"bytes": n * 8.0 * (10 + 12), "flops": n * gravity}
    if case["kind"] == "sedov":
        # two right-hand sides: state in, rates out; 77 pairs of density and force terms
        return {"bytes": 2 * n * 8.0 * (10 + 9), "flops": 2 * n * 77 * 110.0}
    return {"bytes": n * 8.0 * (8 + 18), "flops": n * (gravity + 60 * 110.0)}


def tolerance(case):
    if case["kind"] == "order":
        return "exact"
    if case["kind"] == "plummer":
        # FP64: sums in another order.  Mixed: the tree's own truncation error (FP32 sums
        # are far below it): the walk is 2.9e-4 off the direct sum
        return {"rel": 1.2e-3, "max": 5e-2} if case["precision"] else {"rel": 1e-11}
    if case["kind"] == "sedov":
        # FP32 pair terms on FP64 sums: 2.4e-7 off; FP64: 9e-16 off
        return {"rel": 1e-6, "max": 1e-4} if case["precision"] else {"rel": 1e-12}
    # gravity as above; a pair at the edge of the support may be in or out by the last
    # bit, and then a few particles converge to another h of the same band
    if case["precision"]:
        return {"rel": 1.5e-3, "max": 0.5, "differ": 1e-3}
    return {"rel": 1e-6, "max": 0.1, "differ": 1e-3}


# ----------------------------------------------------------- plain FP64 torch
def _direct(x, y, z, m, eps2):
    """Accelerations by direct summation, softened with the target's eps2 (number or tensor)."""
    n = x.numel()
    out = [torch.empty_like(x) for _ in range(3)]
    rows = max(1, (1 << 27) // n)
    for a in range(0, n, rows):
        b = min(n, a + rows)
        d = [c[None, :] - c[a:b, None] for c in (x, y, z)]
        r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
        r2 += eps2[a:b, None] if torch.is_tensor(eps2) else eps2
        w = m[None, :] * r2 ** -1.5
        for k in range(3):
            out[k][a:b] = (w * d[k]).sum(1)
    return out


def _pairs(x, y, z, h):
    """All (i, j), i != j, closer than h (one number), from cells of edge >= h."""
    pos = torch.stack([x, y, z], 1)
    lo = pos.min(0).values
    nc = int(max(1, math.floor(float((pos.max(0).values - lo).max()) / h)))
    edge = float((pos.max(0).values - lo).max()) / nc * (1.0 + 1e-12)
    c = torch.clamp(((pos - lo) / edge).long(), max=nc - 1)
    cid = (c[:, 0] * nc + c[:, 1]) * nc + c[:, 2]
    order = torch.argsort(cid)
    start = torch.searchsorted(cid[order].contiguous(), torch.arange(nc ** 3 + 1, device=DEV))
    ii, jj = [], []
    for dx in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dz in (-1, 0, 1):
                q = c + torch.tensor([dx, dy, dz], device=DEV)
                i = torch.nonzero(((q >= 0) & (q < nc)).all(1))[:, 0]
                k = (q[i, 0] * nc + q[i, 1]) * nc + q[i, 2]
                cnt = start[k + 1] - start[k]
                end = torch.cumsum(cnt, 0)
                i2 = torch.repeat_interleave(i, cnt)
                off = torch.arange(i2.numel(), device=DEV) - torch.repeat_interleave(end - cnt, cnt)
                j2 = order[torch.repeat_interleave(start[k], cnt) + off]
                d2 = (x[i2] - x[j2]) ** 2 + (y[i2] - y[j2]) ** 2 + (z[i2] - z[j2]) ** 2
                keep = (d2 < h * h) & (i2 != j2)
                ii.append(i2[keep])
                jj.append(j2[keep])
    return torch.cat(ii), torch.cat(jj)


def _sph_rhs(s):
    """Density, sound speed (from the previous pressure), pressure and the pair forces
    of an ideal gas with one fixed h, cubic spline, Monaghan viscosity (1, 2)."""
    n, h = s["x"].numel(), float(s["sml"][0])
    i, j = _pairs(s["x"], s["y"], s["z"], h)
    add = lambda v: torch.zeros(n, dtype=torch.float64, device=DEV).index_add_(0, i, v)  # noqa: E731
    d = [s[f][i] - s[f][j] for f in ("x", "y", "z")]
    r2 = d[0] ** 2 + d[1] ** 2 + d[2] ** 2
    w, dw = _cubic(torch.sqrt(r2), h)
    m = s["mass"]
    rho = m * (8.0 / math.pi / h ** 3) + add(m[j] * w)
    del w
    cs = torch.sqrt(GAMMA * s["p"] / rho)
    p = (GAMMA - 1.0) * rho * s["e"]
    g = dw / torch.sqrt(r2)
    del dw
    dv = [s[f][i] - s[f][j] for f in ("vx", "vy", "vz")]
    vr = dv[0] * d[0] + dv[1] * d[1] + dv[2] * d[2]
    mu = h * vr / (r2 + 0.01 * h * h)
    pij = torch.where(vr < 0, (2.0 * mu - 0.5 * (cs[i] + cs[j])) * mu / (0.5 * (rho[i] + rho[j])), 0.0)
    del mu, r2
    pf = p / (rho * rho)
    pf = pf[i] + pf[j]
    mj = m[j]
    out = dict(rho=rho, cs=cs, p=p, noi=None)
    for k, f in enumerate(("ax", "ay", "az")):
        out[f] = add(-mj * (pf + pij) * g * d[k])
    out["drhodt"] = rho * add(mj / rho[j] * vr * g)
    out["dedt"] = add(0.5 * mj * (pf + pij) * vr * g)
    return out


def exact(case, seed):
    if case["kind"] == "order":
        return None
    n = _count(case)
    if case["kind"] == "sedov":
        if n > EXACT_SPH_N or case["balsara"]:
            return None
        s = _inputs(case, seed)
        a, dt = _sph_rhs(s), SEDOV_DT
        q = dict(s, p=a["p"], e=torch.clamp(s["e"] + dt * a["dedt"], min=1e-6))
        for x, v, f in (("x", "vx", "ax"), ("y", "vy", "ay"), ("z", "vz", "az")):
            q[x], q[v] = s[x] + dt * s[v], s[v] + dt * a[f]
        b = _sph_rhs(q)
        o = dict(rho=a["rho"], p=a["p"], cs=a["cs"], drhodt=a["drhodt"], noi=None)
        for x, v, f in (("x", "vx", "ax"), ("y", "vy", "ay"), ("z", "vz", "az")):
            o[f] = 0.5 * (a[f] + b[f])
            o[x], o[v] = s[x] + 0.5 * dt * (q[v] + s[v]), s[v] + 0.5 * dt * (a[f] + b[f])
        o["dedt"] = 0.5 * (a["dedt"] + b["dedt"])
        o["e"] = torch.clamp(s["e"] + dt * o["dedt"], min=1e-6)
        return {f: o[f] for f in OUT["sedov"]}
    if n > EXACT_GRAVITY_N:
        return None
    s = _inputs(case, seed)
    names = ("g_ax", "g_ay", "g_az")
    if case["kind"] == "cloud":
        # the walk softens with the h that the step starts from; h and the gas forces
        # come out of an iteration on neighbour counts
        o = dict.fromkeys(OUT["cloud"])
        o.update(zip(names, _direct(s["x"], s["y"], s["z"], s["mass"], (0.5 * s["sml"]) ** 2)))
        return o
    dt, o = case["dt"], {}
    g0 = _direct(s["x"], s["y"], s["z"], s["mass"], EPS2)
    for k, (x, v) in enumerate((("x", "vx"), ("y", "vy"), ("z", "vz"))):
        o[x] = s[x] + dt * (s[v] + 0.5 * dt * g0[k])
    g1 = _direct(o["x"], o["y"], o["z"], s["mass"], EPS2)
    for k, v in enumerate(("vx", "vy", "vz")):
        o[v] = s[v] + 0.5 * dt * (g0[k] + g1[k])
        o[names[k]] = g1[k]
    return {f: o[f] for f in OUT["plummer"]}
