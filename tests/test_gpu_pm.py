"""Particle-mesh gravity and the cosmological leapfrog on the GPU.

acceleration_PM runs its cloud-in-cell deposit, Green's function, gradient
and interpolation as GPU kernels that repeat the reference's FP64
expressions (src/acceleration_PM.c), with the 3-D transforms through cuFFT.
The reference's transforms are FFTW's; the golden vectors were made with the
oracle's direct DFT standing in, and the deposit here adds with atomics in
no fixed order, so the comparison is to a tolerance: every component within
1e-10 of the largest acceleration (FP64 transforms of 16^3-64^3 meshes agree
to ~1e-14 of their largest term).
"""
import json

import numpy as np
import pytest

from conftest import cases, golden

pytestmark = pytest.mark.gpu

REL = 1e-10


def _close(a, ref, rel=REL):
    scale = np.abs(ref).max()
    err = np.abs(a - ref).max()
    assert err <= rel * scale, (err, scale)


def test_acceleration_pm_golden(lib, g):
    d = golden("pm")
    c, bw = d["box_center"], float(d["box_width"])
    H0, om, sf = float(d["H0"]), float(d["omega_m"]), float(d["scale_factor"])
    for name, cs in cases(d).items():
        if name == "cosmo":
            continue
        rho = cs["m"].sum() / ((bw * 2) ** 3)
        a = g.acceleration_pm(lib, cs["x"], cs["m"], c, bw, H0, om, rho, int(cs["grid"]), sf)
        _close(a, cs["a"])


def test_acceleration_pm_oracle_g64(lib, g, orc):
    """A 64^3 mesh with 200,000 clustered particles against the oracle."""
    rng = np.random.default_rng(5)
    c, bw = np.array([0.0, 0.0, 0.0]), 10.0
    n = 200_000
    x = np.clip(rng.standard_normal((n, 3)) * 2.5, -bw, bw)
    m = rng.uniform(0.5, 1.5, n)
    rho = m.sum() / ((bw * 2) ** 3)
    a = g.acceleration_pm(lib, x, m, c, bw, 70.0, 0.3, rho, 64, 0.25)
    a_ref = orc.acceleration_pm(x, m, c, bw, 70.0, 0.3, rho, 64, 0.25)
    _close(a, a_ref)


def mesh_reference(x, m, c, bw, H0, om, rho, grid, sf):
    """The same quantity with numpy's transforms."""
    cell = 2.0 * bw / grid
    u = (x - c + bw) / cell
    i0 = np.floor(u).astype(int)
    idx, w = (i0 % grid, (i0 + 1) % grid), (1.0 - (u - i0), u - i0)
    mesh, flat = np.zeros(grid ** 3), []
    for e in np.ndindex(2, 2, 2):
        q = (idx[e[0]][:, 0] * grid + idx[e[1]][:, 1]) * grid + idx[e[2]][:, 2]
        flat.append((q, w[e[0]][:, 0] * w[e[1]][:, 1] * w[e[2]][:, 2]))
        mesh += np.bincount(q, m * flat[-1][1], grid ** 3)
    delta = (mesh / (cell ** 3 * rho) - 1.0).reshape(grid, grid, grid)
    k = np.minimum(np.arange(grid), grid - np.arange(grid))
    k2 = (k[:, None, None] ** 2 + k[:, None] ** 2 + k[:grid // 2 + 1] ** 2) * (np.pi / bw) ** 2
    k2[0, 0, 0] = np.inf
    phi = np.fft.irfftn(np.fft.rfftn(delta) / -k2, (grid,) * 3, (0, 1, 2)) * 1.5 * om * H0 ** 2 / sf
    a = np.zeros_like(x)
    for d in range(3):
        gr = np.roll(phi, 2, d) - 8 * np.roll(phi, 1, d) + 8 * np.roll(phi, -1, d) - np.roll(phi, -2, d)
        for q, ww in flat:
            a[:, d] += (gr / (12.0 * cell)).reshape(-1)[q] * ww
    return a


@pytest.mark.parametrize("grid", [16, 31, 32, 40, 48, 60, 64, 66, 72, 75, 80, 96, 100, 120, 128, 144,
                                  160, 192, 256])
def test_acceleration_pm_mesh_sizes(lib, g, grid):
    """Every size of the own transforms and, around them, the library's (16, 31, 66, 75)."""
    rng = np.random.default_rng(grid)
    c, bw = np.array([1.0, -2.0, 3.0]), 7.0
    x = c + np.clip(rng.standard_normal((20000, 3)) * 2.0, -0.999 * bw, 0.999 * bw)
    m = rng.uniform(0.5, 1.5, len(x))
    args = (c, bw, 70.0, 0.3, m.sum() / (2 * bw) ** 3, grid, 0.25)
    _close(g.acceleration_pm(lib, x, m, *args), mesh_reference(x, m, *args))


def test_acceleration_pm_momentum_and_determinism(lib, g):
    """Size-independent properties at 128^3 and 2M particles: the mesh force
    of a periodic box sums to zero (Newton's third law on the mesh, to the
    rounding of the transforms), and two calls agree to the atomic-order
    rounding of the deposit."""
    rng = np.random.default_rng(9)
    c, bw = np.array([5.0, 5.0, 5.0]), 5.0
    n = 2_000_000
    x = c + rng.uniform(-bw, bw, (n, 3))
    m = np.full(n, 1.0)
    rho = m.sum() / ((bw * 2) ** 3)
    a1 = g.acceleration_pm(lib, x, m, c, bw, 70.0, 0.3, rho, 128, 1.0)
    a2 = g.acceleration_pm(lib, x, m, c, bw, 70.0, 0.3, rho, 128, 1.0)
    scale = np.abs(a1).max()
    assert np.isfinite(a1).all() and scale > 0
    assert np.abs(a1 - a2).max() <= 1e-12 * scale
    assert np.abs((m[:, None] * a1).sum(0)).max() <= 1e-8 * scale * m.sum()


def test_cosmological_simulation_golden(lib, g):
    cs = cases(golden("pm"))["cosmo"]
    kw = json.loads(bytes(cs["args.json"]).decode())
    x = cs["x0"].copy()
    v = cs["v0"].copy()
    st = g.launch_cosmological_simulation(lib, x, v, cs["m"], **kw)
    assert st.num_steps == int(cs["steps"]) and st.t == float(cs["t"])
    assert np.array_equal(v, cs["v0"])             # the reference leaves v alone
    assert np.abs(x - cs["x"]).max() <= 1e-9 * kw["box_width"]
    lo = np.array(kw["box_center"]) - kw["box_width"]
    hi = np.array(kw["box_center"]) + kw["box_width"]
    assert ((x >= lo) & (x <= hi)).all()


@pytest.mark.parametrize("grid", [32, 30])
@pytest.mark.parametrize("centre", [1e6, -3e9])
def test_acceleration_pm_box_far_from_origin(lib, g, grid, centre):
    """A box far from the origin gives the accelerations of the same box at the origin: the
    positions are multiples of 2^-20, so x - centre is exact, and nothing else may depend on the
    centre (its half width of 1/3 is no such multiple)."""
    rng = np.random.default_rng(grid)
    bw = 1.0 / 3.0
    x = np.round(np.clip(rng.standard_normal((5000, 3)) * 0.1, -0.3, 0.3) * 2.0 ** 20) / 2.0 ** 20
    m = rng.uniform(0.5, 1.5, len(x))
    c = np.array([centre, 0.0, -centre])
    rest = (bw, 70.0, 0.3, m.sum() / (2 * bw) ** 3, grid, 0.25)
    _close(g.acceleration_pm(lib, x + c, m, c, *rest),
           g.acceleration_pm(lib, x, m, np.zeros(3), *rest), 1e-12)


@pytest.mark.parametrize("grid", [32, 30])
def test_acceleration_pm_light_deposits(lib, g, grid):
    """Deposits far below the mean density add up: 200,000 particles in a blob, each less than
    half of the last bit of a contrast of -1 (5e-17 of the mean).  The accelerations are those
    of the usual mean over the ratio of the means, to the contrast's own rounding (1e-16 of
    1e-13 a cell, and the transforms' of a mesh near -1): within 5 % of the largest."""
    rng = np.random.default_rng(grid)
    bw, n = 1.0, 200_000
    x = np.clip(rng.standard_normal((n, 3)) * 0.05, -0.9, 0.9)
    m = np.ones(n)
    c = np.zeros(3)
    cell = (2 * bw / grid) ** 3
    usual, high = n / (2 * bw) ** 3, 1.0 / (cell * 5e-17)
    a = g.acceleration_pm(lib, x, m, c, bw, 70.0, 0.3, usual, grid, 0.25)
    b = g.acceleration_pm(lib, x, m, c, bw, 70.0, 0.3, high, grid, 0.25)
    _close(b * (high / usual), a, 0.05)


@pytest.mark.parametrize("grid", [32, 30])
def test_acceleration_pm_huge_box(lib, g, grid):
    """A box so wide that its squared wave numbers underflow has no potential: zeros."""
    rng = np.random.default_rng(grid)
    x = rng.uniform(-1.0, 1.0, (100, 3)) * 1e165
    a = g.acceleration_pm(lib, x, np.ones(100), np.zeros(3), 1e165, 70.0, 0.3, 1.0, grid, 0.25)
    assert (a == 0.0).all()
