"""Performance cases: the work that users of this library have it do.

A case is one pass through the library's public entry points, from the smallest calls (one
planetary system, a direct sum of a thousand bodies), where launches and latency count, to a
galaxy collision of a million particles:

* ``accel``    -- ``acceleration()`` on host arrays (grav_sim's acceleration entry point);
* ``sim``      -- the device-resident simulation (``gsgpu_sim_*``): some steps, then the
                  positions and velocities brought to the host, as a program does between two
                  pictures or two checkpoints;
* ``launch``   -- ``launch_simulation`` on host arrays, the call grav_sim's Python package makes;
* ``ensemble`` -- batched planetary systems (``Ensemble``): some steps, then a download;
* ``cosmo``    -- ``launch_cosmological_simulation``: the particle-mesh leapfrog.

``exact`` restates each in FP64 with torch or numpy (a direct sum in place of a tree).
"""
from __future__ import annotations

import ctypes
import importlib.util
import math
import sys
from pathlib import Path

import numpy as np
import torch

PKG = Path(__file__).resolve().parents[1] / "gravity-simulator_gb300"


def _module(name):
    key = f"gsgpu_{name}"
    if key not in sys.modules:
        spec = importlib.util.spec_from_file_location(key, PKG / f"{name}.py")
        mod = importlib.util.module_from_spec(spec)
        sys.modules[key] = mod
        spec.loader.exec_module(mod)
    return sys.modules[key]


g = _module("gsgpu")
wl = _module("workloads")
_lib = None

EPS = 0.01          # Plummer softening of the star systems
DT = 1e-3           # their leapfrog step
COSMO = dict(h=0.7, omega_m=0.3, omega_lambda=0.7, box_width=50.0, a_begin=0.125, da=1.0 / 256)


def lib():
    global _lib
    if _lib is None:
        _lib = g.load_c_lib()
        vp = ctypes.c_void_p
        dp = ctypes.POINTER(ctypes.c_double)
        _lib.gsgpu_sim_create.argtypes = [
            ctypes.POINTER(vp), ctypes.c_int, ctypes.c_double,
            ctypes.POINTER(g.AccelerationParam), ctypes.c_int, ctypes.c_double, vp]
        _lib.gsgpu_sim_upload.argtypes = [vp, dp, dp, dp]
        _lib.gsgpu_sim_run.argtypes = [vp, ctypes.c_int64]
        _lib.gsgpu_sim_download.argtypes = [vp, dp, dp]
        _lib.gsgpu_sim_destroy.argtypes = [vp]
        _lib.gsgpu_sim_destroy.restype = None
    return _lib


def listed():
    return [
        # a script that asks for the forces on a star cluster once per frame or per analysis
        # step: a small, ragged direct sum with host arrays in and out, bound by latency
        dict(name="accel_pairwise_1500", kind="accel", ic="plummer", n=1500, method=101),
        # the reference's own CPU-sized run, FP64 in the reference's summation order
        dict(name="leapfrog_fp64_1024", kind="sim", ic="plummer", n=1024, method=111, steps=20),
        # an open cluster evolved by the compensated direct sum, not a whole number of tiles
        dict(name="leapfrog_direct_12000", kind="sim", ic="plummer", n=12000, method=101,
             steps=20),
        # the largest direct sums that are still run for their accuracy
        dict(name="leapfrog_direct_100000", kind="sim", ic="plummer", n=100000, method=101,
             steps=4),
        # the solar system: grav_sim's first example, thousands of tiny steps
        dict(name="solar_whfast", kind="launch", ic="belt", n=9, integrator=10, method=102,
             dt=1.0, steps=400, eps=0.0),
        # the same by the adaptive high-order integrator, forces in the reference's order
        dict(name="solar_ias15", kind="launch", ic="belt", n=9, integrator=9, method=111,
             tf=100.0, eps=0.0),
        # an asteroid belt: Sun, planets and massless asteroids
        dict(name="belt_leapfrog_50009", kind="launch", ic="belt", n=50009, integrator=4,
             method=102, dt=1.0, steps=50, eps=0.0),
        # a galaxy collision of the size of the reference's Gadget-2 example file
        dict(name="galaxy_group_60000", kind="sim", ic="galaxy", n=60000, method=106, theta=0.5,
             steps=10),
        # the large galaxy collision by the fast Barnes-Hut walk
        dict(name="galaxy_group_1048576", kind="sim", ic="galaxy", n=1048576, method=106,
             theta=0.5, steps=8),
        # the reference's own Barnes-Hut decisions (one particle per leaf, monopole cells)
        dict(name="galaxy_plain_150000", kind="sim", ic="galaxy", n=150000, method=103,
             theta=0.5, steps=4),
        # a batch of planetary systems of uneven size
        dict(name="ensemble_whfast_512", kind="ensemble", systems=512, max_test=4096,
             integrator=10, method=102, dt=1.0, steps=10),
        # a cosmological particle-mesh run
        dict(name="cosmo_pm_128", kind="cosmo", side=128, grid=128, steps=8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["accel", "direct", "fp64", "small", "belt", "group", "plain", "ensemble",
                       "cosmo"])
    if kind == "accel":
        return dict(kind="accel", ic="plummer", n=_log(rng, 200, 20000),
                    method=rng.choice([101, 101, 111]), eps=rng.choice([EPS, 0.0]))
    if kind == "direct":
        n = _log(rng, 1000, 100000)
        return dict(kind="sim", ic="plummer", n=n, method=101,
                    steps=max(2, min(20, int(4 * (1e5 / n) ** 2))))
    if kind == "fp64":
        return dict(kind="sim", ic="plummer", n=_log(rng, 64, 4096), method=111,
                    steps=rng.randint(5, 20))
    if kind == "small":
        integ = rng.choice([4, 6, 9, 10])
        c = dict(kind="launch", ic="belt", n=rng.randint(3, 40), integrator=integ,
                 method=rng.choice([102, 111]) if integ != 10 else 102, eps=0.0)
        return dict(c, dt=1.0, steps=rng.randint(100, 400)) if integ in (4, 10) else \
            dict(c, tf=float(rng.randint(30, 100)))
    if kind == "belt":
        return dict(kind="launch", ic="belt", n=9 + _log(rng, 500, 100000),
                    integrator=rng.choice([3, 4]), method=102, dt=1.0,
                    steps=rng.randint(10, 40), eps=0.0)
    if kind == "group":
        return dict(kind="sim", ic="galaxy", n=_log(rng, 8000, 1000000),
                    method=rng.choice([106, 106, 107]), theta=rng.choice([0.5, 0.65, 0.75]),
                    steps=rng.randint(3, 8))
    if kind == "plain":
        return dict(kind="sim", ic="galaxy", n=_log(rng, 8000, 150000),
                    method=rng.choice([103, 105]), theta=rng.choice([0.5, 0.75]),
                    steps=rng.randint(2, 4))
    if kind == "ensemble":
        return dict(kind="ensemble", systems=_log(rng, 8, 512), max_test=4096,
                    integrator=rng.choice([10, 10, 4]), method=102, dt=1.0,
                    steps=rng.randint(5, 10))
    return dict(kind="cosmo", side=_log(rng, 24, 128), grid=rng.choice([32, 48, 60, 75, 96, 128]),
                steps=rng.randint(4, 8))


# ---- inputs ---------------------------------------------------------------
def _planets_and_asteroids(rng, light):
    """Sun + 8 planets (log-spaced, near-circular) + ``light`` massless asteroids, per system:
    the distributions of workloads.planetary_ensemble.  light: asteroids of each system."""
    S = len(light)
    G = wl.G_AU_MSUN_DAY
    a_pl = np.tile(np.exp(np.linspace(math.log(0.39), math.log(30.0), 8)), S)
    ang = rng.uniform(0.0, 2.0 * math.pi, (3, 8 * S))
    xp, vp = wl.kepler_to_cartesian(a_pl, rng.uniform(0.0, 0.1, 8 * S),
                                    np.radians(rng.uniform(0.0, 3.0, 8 * S)), ang[0], ang[1],
                                    ang[2], G * (1.0 + np.tile(wl.PLANET_MASSES, S)))
    L = int(sum(light))
    ang = rng.uniform(0.0, 2.0 * math.pi, (3, L))
    xt, vt = wl.kepler_to_cartesian(rng.uniform(2.0, 3.5, L), rng.uniform(0.0, 0.1, L),
                                    np.radians(rng.uniform(0.0, 5.0, L)), ang[0], ang[1], ang[2],
                                    np.full(L, G))
    counts = np.array([9 + q for q in light], dtype=np.int32)
    off = np.concatenate([[0], np.cumsum(counts)])
    n = int(off[-1])
    x, v, m = np.zeros((n, 3)), np.zeros((n, 3)), np.zeros(n)
    k = 0
    for s in range(S):
        o, e = off[s], off[s + 1]
        x[o + 1:o + 9], v[o + 1:o + 9] = xp[8 * s:8 * s + 8], vp[8 * s:8 * s + 8]
        m[o], m[o + 1:o + 9] = 1.0, wl.PLANET_MASSES
        x[o + 9:e], v[o + 9:e] = xt[k:k + light[s]], vt[k:k + light[s]]
        k += light[s]
        M = m[o:o + 9]
        x[o:e] -= (M[:, None] * x[o:o + 9]).sum(0) / M.sum()
        v[o:e] -= (M[:, None] * v[o:o + 9]).sum(0) / M.sum()
    ids = np.concatenate([np.arange(c, dtype=np.int32) for c in counts])
    return counts, ids, x, v, m


def _inputs(case, seed):
    """(x, v, m) on the host, and for planetary systems (counts, ids) before them."""
    rng = np.random.default_rng(seed)
    if case["kind"] == "ensemble":
        # log-uniform sizes, the same for every seed of a case
        u = np.random.default_rng(case["systems"]).uniform(0.0, math.log(case["max_test"] + 1),
                                                           case["systems"])
        light = [int(q) - 1 for q in np.exp(u)]
        return _planets_and_asteroids(rng, light)
    if case["kind"] == "cosmo":
        side, bw = case["side"], COSMO["box_width"]
        lattice = np.indices((side, side, side)).reshape(3, -1).T.astype(np.float64)
        x = -bw + (lattice + 0.5 + rng.uniform(-0.3, 0.3, lattice.shape)) * (2.0 * bw / side)
        return np.ascontiguousarray(x), rng.normal(0.0, 5.0, x.shape), np.ones(side ** 3)
    if case["ic"] == "belt":
        n = case["n"]
        if n >= 9:
            return _planets_and_asteroids(rng, [n - 9])
        c, ids, x, v, m = _planets_and_asteroids(rng, [0])   # a Sun with fewer planets
        return np.array([n], dtype=np.int32), ids[:n].copy(), x[:n].copy(), v[:n].copy(), m[:n].copy()
    return (wl.plummer if case["ic"] == "plummer" else wl.galaxy_pair)(case["n"], seed)


class Sim:
    """A device-resident leapfrog simulation and the host arrays it is read into."""

    def __init__(self, case, x, v, m):
        n = case["n"]
        h = ctypes.c_void_p()
        p = g.AccelerationParam(case["method"], case.get("theta", 1.0), case.get("eps", EPS), -1)
        if lib().gsgpu_sim_create(ctypes.byref(h), n, 1.0, ctypes.byref(p), 4, DT, None):
            raise RuntimeError("gsgpu_sim_create failed")
        self.handle = h
        if lib().gsgpu_sim_upload(h, g._dp(x), g._dp(v), g._dp(m)):
            raise RuntimeError("gsgpu_sim_upload failed")
        self.keep = (x, v, m)
        self.x, self.v = np.zeros((n, 3)), np.zeros((n, 3))

    def __del__(self):
        if getattr(self, "handle", None):
            lib().gsgpu_sim_destroy(self.handle)
            self.handle = None


def prepare(case, seed):
    lib()
    data = _inputs(case, seed)
    kind = case["kind"]
    if kind == "accel":
        return dict(case=case, x=data[0], m=data[2])
    if kind == "sim":
        return dict(case=case, sim=Sim(case, *data))
    if kind == "ensemble":
        counts, ids, x, v, m = data
        e = g.Ensemble(lib(), counts, wl.G_AU_MSUN_DAY, integrator=case["integrator"],
                       method=case["method"], dt=case["dt"])
        e.upload(ids, x, v, m)
        return dict(case=case, ens=e)
    if kind == "cosmo":
        return dict(case=case, x=data[0], v=data[1], m=data[2])
    return dict(case=case, ids=data[1], x=data[2], v=data[3], m=data[4])


# ---- one pass ---------------------------------------------------------------
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "accel":
        return g.acceleration(lib(), state["x"], state["m"], 1.0, case["method"],
                              softening_length=case.get("eps", EPS))
    if kind == "sim":
        s = state["sim"]
        if lib().gsgpu_sim_run(s.handle, case["steps"]) or \
                lib().gsgpu_sim_download(s.handle, g._dp(s.x), g._dp(s.v)):
            raise RuntimeError("simulation failed")
        return s.x, s.v
    if kind == "ensemble":
        state["ens"].run(case["steps"])
        return state["ens"].download()
    if kind == "cosmo":
        g.launch_cosmological_simulation(
            lib(), state["x"], state["v"], state["m"], h=COSMO["h"], omega_m=COSMO["omega_m"],
            omega_lambda=COSMO["omega_lambda"], box_center=(0.0, 0.0, 0.0),
            box_width=COSMO["box_width"], dt=COSMO["da"], a_begin=COSMO["a_begin"],
            a_final=COSMO["a_begin"] + case["steps"] * COSMO["da"], pm_grid_size=case["grid"])
        return state["x"]
    adaptive = case["integrator"] in (6, 9)
    return g.launch_simulation(
        lib(), state["x"], state["v"], state["m"], wl.G_AU_MSUN_DAY,
        integrator=case["integrator"], dt=-1.0 if adaptive else case["dt"],
        tf=case["tf"] if adaptive else case["dt"] * case["steps"], method=case["method"],
        softening_length=case["eps"], tolerance=1e-9 if adaptive else -1.0, ids=state["ids"])


def _counts(case):
    """(particles, massive bodies per particle's sum, force evaluations) of a pass."""
    if case["kind"] == "ensemble":
        L = (case["max_test"] - 1) / math.log(case["max_test"]) - 1   # mean of exp(U) - 1
        return case["systems"] * (9 + L), 9, case["steps"]
    if case["kind"] == "cosmo":
        return case["side"] ** 3, 1, case["steps"] + 1
    n = case["n"]
    if case["kind"] == "accel":
        return n, n, 1
    if case["kind"] == "sim":
        return n, n, case["steps"]
    if case["integrator"] in (6, 9):
        return n, min(n, 9), 4 * case["tf"]
    return n, min(n, 9), case["steps"] * (4 if case["integrator"] == 3 else 1)


def work(case):
    """State in and out once; 20 operations per pair term (a tree: about 150 log2 N terms per
    particle at an opening angle of 0.5, fewer as its inverse square; the mesh: its two
    transforms and 120 operations per particle)."""
    n, sources, evals = _counts(case)
    moved = 8.0 * n * (7 if case["kind"] == "accel" else 13)
    if case["kind"] == "cosmo":
        g3 = case["grid"] ** 3
        return dict(bytes=moved, flops=evals * (5.0 * g3 * math.log2(g3) + 120.0 * n))
    if "theta" in case:
        return dict(bytes=moved, flops=evals * 20.0 * n * 150 * math.log2(n)
                    * (0.5 / case["theta"]) ** 2)
    return dict(bytes=moved, flops=evals * 20.0 * n * sources)


# ---- the same in FP64 with torch and numpy ----------------------------------------------------
def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _sum_over(x, xs, ms, G, eps):
    """Accelerations of x from the bodies (xs, ms), by rows of about 2^26 pairs."""
    out = torch.empty_like(x)
    rows = max(1, (1 << 26) // xs.shape[0])
    for i in range(0, x.shape[0], rows):
        d = xs[None, :, :] - x[i:i + rows, None, :]
        r2 = (d * d).sum(-1) + eps * eps
        w = torch.where(r2 > 0, ms * r2.rsqrt() / r2, torch.zeros_like(r2))
        out[i:i + rows] = G * (w[:, :, None] * d).sum(1)
    return out


def _leapfrog(x, v, force, dt, steps):
    a = force(x)
    v = v + a * (0.5 * dt)
    for _ in range(steps):
        x = x + v * dt
        a = force(x)
        v = v + a * dt
    return x, v - a * (0.5 * dt)


def _rk4(x, v, force, dt, steps):
    for _ in range(steps):
        k1x, k1v = v, force(x)
        k2x, k2v = v + 0.5 * dt * k1v, force(x + 0.5 * dt * k1x)
        k3x, k3v = v + 0.5 * dt * k2v, force(x + 0.5 * dt * k2x)
        k4x, k4v = v + dt * k3v, force(x + dt * k3x)
        x = x + dt / 6.0 * (k1x + 2 * k2x + 2 * k3x + k4x)
        v = v + dt / 6.0 * (k1v + 2 * k2v + 2 * k3v + k4v)
    return x, v


def _bulirsch_stoer(x, v, force, tf):
    """Extrapolated Stoermer steps (Gragg's modified midpoint, n = 2, 4, ..., 16) of one day."""
    y = np.stack([x, v])

    def f(s):
        return np.stack([s[1], force(s[0])])
    steps = max(1, int(math.ceil(tf)))
    H = tf / steps
    for _ in range(steps):
        rows = []
        for k in range(8):
            nsub = 2 * (k + 1)
            h = H / nsub
            z0, z1 = y, y + h * f(y)
            for _ in range(nsub - 1):
                z0, z1 = z1, z0 + 2 * h * f(z1)
            row = [0.5 * (z0 + z1 + h * f(z1))]
            for j in range(k):
                q = ((k + 1) / (k - j)) ** 2
                row.append(row[j] + (row[j] - rows[k - 1][j]) / (q - 1.0))
            rows.append(row)
        y = rows[-1][-1]
    return y[0], y[1]


def _stumpff(z):
    q = torch.zeros_like(z)
    big = z.abs() > 0.1
    while bool(big.any()):
        z = torch.where(big, z / 4.0, z)
        q = q + big
        big = z.abs() > 0.1
    c2, c3 = torch.zeros_like(z), torch.zeros_like(z)
    for k in range(9, -1, -1):   # c2 = sum (-z)^k / (2k+2)!, c3 = sum (-z)^k / (2k+3)!
        c2 = 1.0 / math.factorial(2 * k + 2) - z * c2
        c3 = 1.0 / math.factorial(2 * k + 3) - z * c3
    c1, c0 = 1.0 - z * c3, 1.0 - z * c2
    for k in range(int(q.max())):
        up = q > k
        n3, n2 = (c2 + c0 * c3) / 4.0, c1 * c1 / 2.0
        n1, n0 = c0 * c1, 2.0 * c0 * c0 - 1.0
        c0, c1, c2, c3 = (torch.where(up, p, o) for p, o in ((n0, c0), (n1, c1), (n2, c2), (n3, c3)))
    return c0, c1, c2, c3


def _whfast(counts, ids, x, v, m, G, dt, steps):
    """Wisdom-Holman steps in Jacobi coordinates of several systems at once: order by distance
    to the primary, Kepler drift, interaction kick.  Every system has the same number of massive
    bodies; sums over interior bodies are sums over those.  Positions and velocities are the
    Cartesian ones of the last drift."""
    dev = _dev()
    S = len(counts)
    sys_of = torch.repeat_interleave(torch.arange(S, device=dev),
                                     torch.as_tensor(counts, device=dev).long())
    start = torch.as_tensor(np.concatenate([[0], np.cumsum(counts)[:-1]]), device=dev)
    ids, x, v, m = (torch.as_tensor(q, device=dev) for q in (ids, x, v, m))

    def order(p, vel, ids, m):
        primary = p[(ids == 0).nonzero()[:, 0]][sys_of]
        o = torch.argsort((p - primary).norm(dim=1), stable=True)
        o = o[torch.argsort(sys_of[o], stable=True)]
        return p[o], vel[o], ids[o], m[o]

    def massive(m):
        return (m != 0).nonzero()[:, 0].reshape(S, -1)   # by system, then by distance

    def before(at, B):   # [particle, body]: the body is nearer than the particle
        return B[sys_of] < at[:, None]

    at = torch.arange(x.shape[0], device=dev)
    first = start[sys_of]

    def etas(m, B):
        mb = m[B][sys_of]
        inner = (mb * before(at, B)).sum(1)
        return inner + m, inner, mb

    def accel(x, jx, m, B, eta, inner, mb):
        is_m, isf = m != 0, at == first
        xb = x[B]                                          # [S, M, 3]
        near, far = B[sys_of] < at[:, None], B[sys_of] > at[:, None]
        x0 = xb[:, 0][sys_of]
        t = x - x0
        inn = torch.where(isf, torch.ones_like(inner), inner)
        ratio = torch.where(is_m, eta / inn, torch.ones_like(inn))
        m0 = m[B[:, 0]][sys_of]
        a = (G * m0 * ratio)[:, None] * (jx / jx.norm(dim=1, keepdim=True) ** 3
                                         - t / t.norm(dim=1, keepdim=True) ** 3)
        M = B.shape[1]
        for j in range(1, M):
            d = x - xb[:, j][sys_of]
            r3 = d.norm(dim=1) ** 3
            w = G * mb[:, j] / torch.where(r3 > 0, r3, torch.ones_like(r3))
            a = a - (w * (near[:, j] * ratio + far[:, j]))[:, None] * d
        for j in range(M):
            for k in range(j + 1, M):
                d = xb[:, k] - xb[:, j]
                f = (G * m[B[:, j]] * m[B[:, k]] / d.norm(dim=1) ** 3)[:, None] * d
                a = a - (near[:, j] & far[:, k])[:, None] * f[sys_of] / inn[:, None]
        return torch.where(isf[:, None], torch.zeros_like(a), a)

    x, v, ids, m = order(x, v, ids, m)
    B = massive(m)
    eta, inner, mb = etas(m, B)
    isf = at == first
    inn = torch.where(isf, torch.ones_like(inner), inner)
    total = m[B].sum(1)

    def com(y):
        w = (mb * before(at, B))[:, :, None] * y[B][sys_of]
        whole = (m[B][:, :, None] * y[B]).sum(1) / total[:, None]
        return torch.where(isf[:, None], whole[sys_of], y - w.sum(1) / inn[:, None])
    jx, jv = com(x), com(v)
    jv = jv + 0.5 * dt * accel(x, jx, m, B, eta, inner, mb)
    for _ in range(steps):
        jx, jv, ids, m = order(jx, jv, ids, m)
        B = massive(m)
        eta, inner, mb = etas(m, B)
        inn = torch.where(isf, torch.ones_like(inner), inner)
        gm = G * m[B[:, 0]][sys_of] * eta / inn
        r0 = torch.where(isf, torch.ones_like(gm), jx.norm(dim=1))   # the primary does not drift
        rv = (jx * jv).sum(1) / r0
        alpha = torch.where(isf, torch.zeros_like(gm), 2.0 * gm / r0 - (jv * jv).sum(1))
        s = dt / r0
        for _ in range(12):
            c0, c1, c2, c3 = _stumpff(alpha * s * s)
            F = r0 * s * c1 + r0 * rv * s * s * c2 + gm * s ** 3 * c3 - dt
            s = s - F / (r0 * c0 + r0 * rv * s * c1 + gm * s * s * c2)
        c0, c1, c2, c3 = _stumpff(alpha * s * s)
        r = r0 * c0 + r0 * rv * s * c1 + gm * s * s * c2
        f, gg = 1.0 - gm * s * s * c2 / r0, dt - gm * s ** 3 * c3
        df, dg = -gm * s * c1 / (r * r0), 1.0 - gm * s * s * c2 / r
        nx, nv = f[:, None] * jx + gg[:, None] * jv, df[:, None] * jx + dg[:, None] * jv
        jx = torch.where(isf[:, None], jx, nx)
        jv = torch.where(isf[:, None], jv, nv)

        def cart(j):   # x_i = j_i + (centre of all) - sum of m_b j_b / eta_b over b at i or beyond
            w = (m[B] / eta[B])[:, :, None] * j[B]
            keep = (B[sys_of] >= torch.where(isf, at + 1, at)[:, None])
            c = j[start][sys_of] - (keep[:, :, None] * w[sys_of]).sum(1)
            return torch.where(isf[:, None], c, j + c)
        x, v = cart(jx), cart(jv)
        jv = jv + dt * accel(x, jx, m, B, eta, inner, mb)
    return [q.cpu().numpy() for q in (ids, x, v, m)]


def _mesh_accel(x, m, grid, scale, mean):
    """Cloud-in-cell particle-mesh accelerations (FFT, -1/k^2, fourth-order differences)."""
    bw = COSMO["box_width"]
    length = 2.0 * bw
    cell = length / grid
    u = (x + bw) / cell
    i0 = u.floor().long()
    w1 = u - i0
    idx = [i0 % grid, (i0 + 1) % grid]
    w = [1.0 - w1, w1]
    corners = [(a, b, c) for a in (0, 1) for b in (0, 1) for c in (0, 1)]
    rho = torch.zeros(grid ** 3, dtype=torch.float64, device=x.device)
    flat = []
    for a, b, c in corners:
        q = (idx[a][:, 0] * grid + idx[b][:, 1]) * grid + idx[c][:, 2]
        flat.append((q, w[a][:, 0] * w[b][:, 1] * w[c][:, 2]))
        rho.index_add_(0, q, m * flat[-1][1])
    delta = (rho / (cell ** 3 * mean) - 1.0).reshape(grid, grid, grid)
    k = torch.arange(grid, device=x.device)
    half = grid // 2 + 1
    k = torch.where(k < half, k, k - grid).double()
    kz = torch.arange(half, device=x.device).double()
    k2 = (k[:, None, None] ** 2 + k[None, :, None] ** 2 + kz ** 2) * (2.0 * math.pi / length) ** 2
    green = torch.where(k2 > 0, -1.0 / torch.where(k2 > 0, k2, torch.ones_like(k2)),
                        torch.zeros_like(k2))
    phi = torch.fft.irfftn(torch.fft.rfftn(delta) * green, s=(grid,) * 3)
    phi = phi * (1.5 * COSMO["omega_m"] * (COSMO["h"] * 100.0) ** 2 / scale)
    out = torch.zeros_like(x)
    for d in range(3):
        gr = (phi.roll(2, d) - 8.0 * phi.roll(1, d) + 8.0 * phi.roll(-1, d) - phi.roll(-2, d))
        gr = (gr / (12.0 * cell)).reshape(-1)
        for q, ww in flat:
            out[:, d] += gr[q] * ww
    return out


def _cosmo(case, x, v, m):
    H0, bw, da, a0 = COSMO["h"] * 100.0, COSMO["box_width"], COSMO["da"], COSMO["a_begin"]
    mean = float(m.sum()) / (2.0 * bw) ** 3

    def rate(a):
        om, ol = COSMO["omega_m"], COSMO["omega_lambda"]
        return H0 * a * math.sqrt(ol + om / a ** 3 + (1.0 - om - ol) / a ** 2)
    x, v, m = (torch.as_tensor(q, device=_dev()) for q in (x, v, m))
    p = a0 * a0 * v
    acc = _mesh_accel(x, m, case["grid"], a0, mean)
    for k in range(case["steps"]):
        t = a0 + k * da
        p = p - 0.5 * da * acc / rate(t)
        t += 0.5 * da
        x = x + da * p / (t * t * rate(t))
        x = torch.where(x > bw, x - 2.0 * bw, torch.where(x < -bw, x + 2.0 * bw, x))
        acc = _mesh_accel(x, m, case["grid"], t, mean)
        p = p - 0.5 * da * acc / rate(t)
    return x.cpu().numpy()


def exact(case, seed):
    data = _inputs(case, seed)
    kind = case["kind"]
    if kind == "cosmo":
        return _cosmo(case, *data)
    if kind == "ensemble":
        counts, ids, x, v, m = data
        G = wl.G_AU_MSUN_DAY
        if case["integrator"] == 10:
            ids, x, v, m = _whfast(counts, ids, x, v, m, G, case["dt"], case["steps"])
            return counts, ids, x, v, m
        S = len(counts)
        sys_of = np.repeat(np.arange(S), counts)
        start = np.concatenate([[0], np.cumsum(counts)[:-1]])
        sys_of, heavy, mt = (torch.as_tensor(q, device=_dev())
                             for q in (sys_of, start[:, None] + np.arange(9), m))

        def force(y):
            a = torch.zeros_like(y)
            for j in range(9):
                d = y[heavy[:, j]][sys_of] - y
                r2 = (d * d).sum(1, keepdim=True)
                r2 = torch.where(r2 > 0, r2, torch.ones_like(r2))
                a += mt[heavy[:, j]][sys_of][:, None] * d * (G / (r2 * r2.sqrt()))
            return a
        xt, vt = _leapfrog(torch.as_tensor(x, device=_dev()), torch.as_tensor(v, device=_dev()),
                           force, case["dt"], case["steps"])
        return counts, ids, xt.cpu().numpy(), vt.cpu().numpy(), m
    if kind == "launch":
        counts, ids, x, v, m = data
        G = wl.G_AU_MSUN_DAY
        if case["integrator"] == 10:
            return _whfast(counts, ids, x, v, m, G, case["dt"], case["steps"])
        b = m != 0
        if case["integrator"] in (6, 9):
            def few(y):
                d = y[b][None] - y[:, None]
                r2 = (d * d).sum(-1)
                r2[r2 == 0] = np.inf
                return (G * m[b] / (r2 * np.sqrt(r2)))[:, :, None].__mul__(d).sum(1)
            return (ids, *_bulirsch_stoer(x, v, few, case["tf"]), m)
        bt, mt = torch.as_tensor(b, device=_dev()), torch.as_tensor(m, device=_dev())
        step = _rk4 if case["integrator"] == 3 else _leapfrog
        xt, vt = step(torch.as_tensor(x, device=_dev()), torch.as_tensor(v, device=_dev()),
                      lambda y: _sum_over(y, y[bt], mt[bt], G, 0.0), case["dt"], case["steps"])
        return ids, xt.cpu().numpy(), vt.cpu().numpy(), m
    x, v, m = (torch.as_tensor(q, device=_dev()) for q in data)
    eps = case.get("eps", EPS)
    if kind == "accel":
        return _sum_over(x, x, m, 1.0, eps).cpu().numpy()
    if float(case["n"]) ** 2 * (case["steps"] + 1) > 1.2e11:
        return None   # over about 20 seconds
    xt, vt = _leapfrog(x, v, lambda y: _sum_over(y, y, m, 1.0, eps), DT, case["steps"])
    return xt.cpu().numpy(), vt.cpu().numpy()
