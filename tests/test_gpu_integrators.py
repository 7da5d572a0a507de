"""Integrator loops on the GPU through launch_simulation_python.

With the FP64 reference-order direct sum (111) the whole run -- force,
compensated kicks and drifts, dt clamp, final velocity synchronisation --
must equal grav_sim's run bit for bit (FP64 integrator steps, tolerance 0).
With the compensated-FP32 force (101) the final state agrees to the
accuracy of the force, and the energy drift matches the reference's.
"""
import ctypes
import threading
import time

import numpy as np
import pytest

from conftest import golden

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("integ", [1, 2, 3, 4])
def test_fixed_step_bitexact_golden(lib, g, integ):
    d = golden("integrators")
    x, v = d["x"].copy(), d["v"].copy()
    _, xo, vo, _ = g.launch_simulation(lib, x, v, d["m"].copy(), 1.0, integrator=integ, dt=1e-3,
                                       tf=0.0995, method=g.METHOD_GPU_PAIRWISE_FP64,
                                       softening_length=0.01)
    assert np.array_equal(xo, d[f"int{integ}/x"])
    assert np.array_equal(vo, d[f"int{integ}/v"])


def test_leapfrog_plummer1024_1000_steps_bitexact(lib, g):
    d = golden("leapfrog_plummer1024")
    x, v = d["x0"].copy(), d["v0"].copy()
    _, xo, vo, _ = g.launch_simulation(lib, x, v, d["m"].copy(), 1.0, integrator=4, dt=1e-3,
                                       tf=1.0, method=g.METHOD_GPU_PAIRWISE_FP64,
                                       softening_length=0.01)
    assert np.array_equal(xo, d["x"]) and np.array_equal(vo, d["v"])


def test_leapfrog_plummer1024_fp32_force(lib, g, orc):
    d = golden("leapfrog_plummer1024")
    x, v = d["x0"].copy(), d["v0"].copy()
    _, xo, vo, _ = g.launch_simulation(lib, x, v, d["m"].copy(), 1.0, integrator=4, dt=1e-3,
                                       tf=1.0, method=g.METHOD_GPU_PAIRWISE,
                                       softening_length=0.01)
    dx = np.linalg.norm(xo - d["x"], axis=1)
    assert np.median(dx) < 1e-6 and dx.max() < 1e-3
    e0, e_ref = float(d["e0"]), float(d["e1"])
    e_gpu = orc.energy(xo, vo, d["m"], 1.0)
    drift_ref = abs(e_ref - e0) / abs(e0)
    drift_gpu = abs(e_gpu - e0) / abs(e0)
    print(f"relative energy drift: gpu {drift_gpu:.3g} reference {drift_ref:.3g}")
    assert drift_gpu < 5 * drift_ref + 1e-7


@pytest.mark.parametrize("integ", [1, 2, 3, 4])
def test_oracle_random_tf_clamp(lib, g, orc, wl, integ):
    """tf not a multiple of dt: the last step is clamped (all but rk4)."""
    x, v, m = wl.plummer(300, 90 + integ)
    _, xo, vo, _ = g.launch_simulation(lib, x.copy(), v.copy(), m, 1.0, integrator=integ,
                                       dt=2e-3, tf=0.0371, method=g.METHOD_GPU_PAIRWISE_FP64,
                                       softening_length=0.02)
    xr, vr = orc.fixed_step_run(integ, 1, x, v, m, 1.0, 0.02, 2e-3, 0.0371)
    assert np.array_equal(xo, xr) and np.array_equal(vo, vr)


def test_is_exit_stops_after_one_step(lib, g, orc, wl):
    x, v, m = wl.plummer(200, 5)
    flag = ctypes.c_bool(True)
    _, xo, vo, _ = g.launch_simulation(lib, x.copy(), v.copy(), m, 1.0, integrator=4, dt=1e-3,
                                       tf=1.0, method=g.METHOD_GPU_PAIRWISE_FP64,
                                       softening_length=0.01, is_exit=flag)
    xr, vr = orc.fixed_step_run(4, 1, x, v, m, 1.0, 0.01, 1e-3, 1e-3)
    assert np.array_equal(xo, xr) and np.array_equal(vo, vr)


def test_energy_diagnostics(lib, g, orc):
    d = golden("energy")
    n = d["m"].size
    state = np.ascontiguousarray(np.concatenate([d["m"][:, None], d["x"], d["v"]], 1))
    e = np.empty(1)
    dp = ctypes.POINTER(ctypes.c_double)
    lib.compute_energy_python(e.ctypes.data_as(dp), ctypes.c_double(float(d["G"])),
                              state.ctypes.data_as(dp), ctypes.c_int32(1), ctypes.c_int32(n))
    assert abs(e[0] - float(d["e"])) <= 1e-13 * abs(float(d["e"]))
    p = np.empty(1)
    lib.compute_linear_momentum_python(p.ctypes.data_as(dp), state.ctypes.data_as(dp),
                                       ctypes.c_int32(1), ctypes.c_int32(n))
    assert abs(p[0] - orc.linear_momentum(d["v"], d["m"])) <= 1e-13
    L = np.empty(1)
    lib.compute_angular_momentum_python(L.ctypes.data_as(dp), state.ctypes.data_as(dp),
                                        ctypes.c_int32(1), ctypes.c_int32(n))
    Lr = orc.angular_momentum(d["x"], d["v"], d["m"])
    assert abs(L[0] - Lr) <= 1e-12 * max(1.0, abs(Lr))


@pytest.mark.parametrize("integ", [5, 6, 7, 8])
def test_rk_embedded_bitexact_golden(lib, g, integ):
    """RKF45 / DOPRI / DVERK / RKF78: the GPU stages and combine with the
    host-side error sum and step control reproduce the reference's adaptive
    run bit for bit, with the reference's initial-step estimate and with a
    given initial dt."""
    d = golden("rk_embedded")
    for tag in ("auto", "given"):
        c = f"int{integ}_{tag}"
        x, v = d["x"].copy(), d["v"].copy()
        _, xo, vo, _ = g.launch_simulation(lib, x, v, d["m"].copy(), 1.0, integrator=integ,
                                           dt=1e-3, tf=0.5, method=g.METHOD_GPU_PAIRWISE_FP64,
                                           softening_length=0.01, tolerance=float(d[f"{c}/tol"]),
                                           initial_dt=float(d[f"{c}/initial_dt"]))
        assert np.array_equal(xo, d[f"{c}/x"]), c
        assert np.array_equal(vo, d[f"{c}/v"]), c


def test_rk_embedded_massless_golden(lib, g):
    d = golden("rk_embedded")
    x, v = d["massless_x0"].copy(), d["massless_v0"].copy()
    _, xo, vo, _ = g.launch_simulation(lib, x, v, d["massless_m"].copy(), float(d["massless_G"]),
                                       integrator=6, dt=1.0, tf=200.0,
                                       method=g.METHOD_GPU_MASSLESS, tolerance=1e-9)
    assert np.array_equal(xo, d["massless_x"]) and np.array_equal(vo, d["massless_v"])


def test_rk_embedded_oracle_random(lib, g, orc, wl):
    """A fresh system against the oracle's restatement (DOPRI, tf not reached
    by whole steps)."""
    x, v, m = wl.plummer(200, 777)
    xo_ref, vo_ref, *_ = orc.rk_embedded_run(6, 1, x, v, m, 1.0, 0.02, 1e-7, 0.3)
    _, xo, vo, _ = g.launch_simulation(lib, x.copy(), v.copy(), m, 1.0, integrator=6, dt=1e-3,
                                       tf=0.3, method=g.METHOD_GPU_PAIRWISE_FP64,
                                       softening_length=0.02, tolerance=1e-7)
    assert np.array_equal(xo, xo_ref) and np.array_equal(vo, vo_ref)


@pytest.mark.parametrize("n, method, integ, tf", [(2048, "METHOD_GPU_PAIRWISE_FP64", 6, 0.3),
                                                  (1048576, "METHOD_GPU_MASSLESS", 5, 0.02)])
def test_rk_embedded_device_error_sum(lib, g, wl, n, method, integ, tf):
    """The device-side error sum (gsgpu_set_rk_error_sum(1)) gives the run of
    the reference's host-side order to within the last bits of the step sizes
    (positions and velocities within 1e-12), without the 6N-term copy and host
    loop per attempt.  The second case is a million test particles around
    eight massive bodies, where the force is cheap and that loop is most of an
    attempt (both wall times printed)."""
    import time
    lib.gsgpu_set_rk_error_sum.argtypes = [ctypes.c_int]
    if n <= 4096:
        x, v, m = wl.plummer(n, 4242)
    else:
        x, v, m = wl.plummer(n, 4243)
        m = np.zeros(n)
        m[:8] = 1.0 / 8
    kw = dict(integrator=integ, dt=1e-3, tf=tf, method=getattr(g, method),
              softening_length=0.01, tolerance=1e-6)
    out, wall = {}, {}
    try:
        for mode in (0, 1, 0, 1):   # each mode twice: the second run is timed warm
            assert lib.gsgpu_set_rk_error_sum(mode) == 0
            xs, vs = x.copy(), v.copy()
            t0 = time.perf_counter()
            g.launch_simulation(lib, xs, vs, m, 1.0, **kw)
            wall[mode] = time.perf_counter() - t0
            out[mode] = (xs, vs)
    finally:
        lib.gsgpu_set_rk_error_sum(0)
    (x0, v0), (x1, v1) = out[0], out[1]
    print(f"N={n}: host-order sum {wall[0]:.3f} s, device sum {wall[1]:.3f} s")
    assert np.abs(x1 - x0).max() <= 1e-12 * np.abs(x0).max()
    assert np.abs(v1 - v0).max() <= 1e-12 * np.abs(v0).max()


def test_ias15_bitexact_golden(lib, g):
    """IAS15: the GPU predictor / corrector kernels with the host-side
    convergence test and step control reproduce the reference's run bit for
    bit, with its initial-step estimate and with a given initial dt."""
    d = golden("ias15")
    for tag in ("auto", "given"):
        x, v = d["x"].copy(), d["v"].copy()
        _, xo, vo, _ = g.launch_simulation(lib, x, v, d["m"].copy(), 1.0, integrator=9, dt=1e-3,
                                           tf=0.5, method=g.METHOD_GPU_PAIRWISE_FP64,
                                           softening_length=0.01, tolerance=float(d[f"{tag}/tol"]),
                                           initial_dt=float(d[f"{tag}/initial_dt"]))
        assert np.array_equal(xo, d[f"{tag}/x"]), tag
        assert np.array_equal(vo, d[f"{tag}/v"]), tag


def test_ias15_massless_golden(lib, g):
    d = golden("ias15")
    x, v = d["massless_x0"].copy(), d["massless_v0"].copy()
    _, xo, vo, _ = g.launch_simulation(lib, x, v, d["massless_m"].copy(), float(d["massless_G"]),
                                       integrator=9, dt=1.0, tf=200.0,
                                       method=g.METHOD_GPU_MASSLESS, tolerance=1e-9)
    assert np.array_equal(xo, d["massless_x"]) and np.array_equal(vo, d["massless_v"])


def test_ias15_oracle_random(lib, g, orc, wl):
    x, v, m = wl.plummer(300, 778)
    xo_ref, vo_ref, *_ = orc.ias15_run(1, x, v, m, 1.0, 0.02, 1e-8, 0.2)
    _, xo, vo, _ = g.launch_simulation(lib, x.copy(), v.copy(), m, 1.0, integrator=9, dt=1e-3,
                                       tf=0.2, method=g.METHOD_GPU_PAIRWISE_FP64,
                                       softening_length=0.02, tolerance=1e-8)
    assert np.array_equal(xo, xo_ref) and np.array_equal(vo, vo_ref)


def _softened_energy(x, v, m, G, eps):
    ke = 0.5 * np.sum(m * np.sum(v * v, axis=1))
    pe = 0.0
    for i0 in range(0, len(m), 512):
        d = x[i0:i0 + 512, None, :] - x[None, :, :]
        w = m[i0:i0 + 512, None] * m[None, :] / np.sqrt(np.sum(d * d, axis=2) + eps * eps)
        idx = np.arange(i0, min(i0 + 512, len(m)))
        w[idx - i0, idx] = 0.0
        pe += w.sum()
    return ke - 0.5 * G * pe


def test_energy_drift_against_reference_barnes_hut(lib, g, orc, wl):
    """Relative drift of the softened energy over 200 leapfrog steps of a
    galaxy pair (N = 2,048, eps = 0.01, dt = 1e-3): the group walk (106,
    theta 0.5, quadrupole cells) against the same run with grav_sim's
    Barnes-Hut as the oracle restates it (theta 0.5, true leaf multipoles,
    monopole cells).  The GPU run may not drift more than the reference's
    (with a floor for round-off)."""
    x, v, m = wl.galaxy_pair(2048, 13)
    G, eps, dt, tf = 1.0, 0.01, 1e-3, 0.2
    e0 = _softened_energy(x, v, m, G, eps)
    xg, vg = x.copy(), v.copy()
    g.launch_simulation(lib, xg, vg, m.copy(), G, integrator=4, dt=dt, tf=tf,
                        method=g.METHOD_GPU_BARNES_HUT_GROUP, opening_angle=0.5,
                        softening_length=eps, max_num_particles_per_leaf=16)
    xr, vr = orc.fixed_step_run(4, 3, x, v, m, G, eps, dt, tf, bh=(0.5, 1, 0))
    drift_gpu = abs(_softened_energy(xg, vg, m, G, eps) - e0) / abs(e0)
    drift_ref = abs(_softened_energy(xr, vr, m, G, eps) - e0) / abs(e0)
    print(f"relative energy drift over 200 steps: GPU group walk {drift_gpu:.3g}, "
          f"reference Barnes-Hut {drift_ref:.3g}")
    assert drift_gpu <= max(drift_ref, 1e-7)


@pytest.mark.parametrize("massless", [False, True])
@pytest.mark.parametrize("n", [2, 3, 9, 23, 24, 32, 33, 40, 41, 43, 48, 49])
@pytest.mark.parametrize("integ", [1, 2, 3, 4, 5, 8, 9])
def test_small_systems_bitexact(lib, g, orc, wl, integ, n, massless):
    """Systems of at most 48 bodies, which one block steps (under the pairwise force up to 256
    pairs for the fixed steps, 512 for Runge-Kutta and 800 for IAS15: 23 and 24, 32 and 33, 40 and
    41 bodies are on either side), with massive and massless
    bodies interleaved, more than a batch of 32 steps and a clamped last one.  Bit for bit
    against the oracle."""
    x, v, m = wl.plummer(n, 60 + n)
    if massless:
        m = np.where(np.arange(n) % 3 == 1, 0.0, m)
    method, code = (g.METHOD_GPU_MASSLESS, 2) if massless else (g.METHOD_GPU_PAIRWISE_FP64, 1)
    kw = dict(method=method, softening_length=0.05)
    if integ <= 4:
        ref = orc.fixed_step_run(integ, code, x, v, m, 1.0, 0.05, 4e-3, 0.2791)
        kw.update(dt=4e-3, tf=0.2791)
    elif integ <= 8:
        ref = orc.rk_embedded_run(integ, code, x, v, m, 1.0, 0.05, 1e-9, 0.4)
        kw.update(dt=1e-3, tf=0.4, tolerance=1e-9)
    else:
        ref = orc.ias15_run(code, x, v, m, 1.0, 0.05, 1e-9, 0.4)
        kw.update(dt=1e-3, tf=0.4, tolerance=1e-9)
    _, xo, vo, _ = g.launch_simulation(lib, x.copy(), v.copy(), m, 1.0, integrator=integ, **kw)
    assert xo.tobytes() == ref[0].tobytes() and vo.tobytes() == ref[1].tobytes()


def test_small_system_is_exit_and_single_body(lib, g, orc, wl):
    """A set exit flag ends a small system's run after one step; one body alone drifts."""
    x, v, m = wl.plummer(12, 5)
    _, xo, vo, _ = g.launch_simulation(lib, x.copy(), v.copy(), m, 1.0, integrator=4, dt=1e-3,
                                       tf=1.0, method=g.METHOD_GPU_PAIRWISE_FP64,
                                       softening_length=0.01, is_exit=ctypes.c_bool(True))
    xr, vr = orc.fixed_step_run(4, 1, x, v, m, 1.0, 0.01, 1e-3, 1e-3)
    assert np.array_equal(xo, xr) and np.array_equal(vo, vr)
    x1, v1, m1 = x[:1].copy(), v[:1].copy(), m[:1].copy()
    xr, vr = orc.fixed_step_run(4, 1, x1, v1, m1, 1.0, 0.0, 1e-3, 0.05)
    _, xo, vo, _ = g.launch_simulation(lib, x1, v1, m1, 1.0, integrator=4, dt=1e-3, tf=0.05,
                                       method=g.METHOD_GPU_PAIRWISE_FP64)
    assert np.array_equal(xo, xr) and np.array_equal(vo, vr)


@pytest.mark.parametrize("n", [9, 60])
def test_run_of_no_steps_changes_nothing(lib, g, wl, n):
    """gsgpu_sim_run(0) after a run whose last step was clamped leaves the state, and the
    velocities a download synchronises with the last step, as they are; a system of one block and
    one of several launches."""
    x, v, m = wl.plummer(n, 70)
    dp = ctypes.POINTER(ctypes.c_double)
    lib.gsgpu_sim_create.argtypes = [
        ctypes.POINTER(ctypes.c_void_p), ctypes.c_int, ctypes.c_double,
        ctypes.POINTER(g.AccelerationParam), ctypes.c_int, ctypes.c_double, ctypes.c_void_p]
    lib.gsgpu_sim_upload.argtypes = [ctypes.c_void_p, dp, dp, dp]
    lib.gsgpu_sim_run.argtypes = [ctypes.c_void_p, ctypes.c_int64]
    lib.gsgpu_sim_run_until.argtypes = [ctypes.c_void_p, ctypes.c_double]
    lib.gsgpu_sim_download.argtypes = [ctypes.c_void_p, dp, dp]
    lib.gsgpu_sim_destroy.argtypes = [ctypes.c_void_p]
    lib.gsgpu_sim_destroy.restype = None
    p = g.AccelerationParam(g.METHOD_GPU_PAIRWISE_FP64, 1.0, 0.05, 1)
    sim = ctypes.c_void_p()
    assert lib.gsgpu_sim_create(ctypes.byref(sim), n, 1.0, ctypes.byref(p), 4, 4e-3, None) == 0
    state = [np.empty((n, 3)) for _ in range(4)]
    try:
        assert lib.gsgpu_sim_upload(sim, *[a.ctypes.data_as(dp) for a in (x, v, m)]) == 0
        assert lib.gsgpu_sim_run_until(sim, 0.0101) == 0
        assert lib.gsgpu_sim_download(sim, *[a.ctypes.data_as(dp) for a in state[:2]]) == 0
        assert lib.gsgpu_sim_run(sim, 0) == 0
        assert lib.gsgpu_sim_download(sim, *[a.ctypes.data_as(dp) for a in state[2:]]) == 0
    finally:
        lib.gsgpu_sim_destroy(sim)
    assert np.array_equal(state[0], state[2]) and np.array_equal(state[1], state[3])


class IntegratorParam(ctypes.Structure):
    _fields_ = [("integrator", ctypes.c_int), ("dt", ctypes.c_double),
                ("tolerance", ctypes.c_double), ("initial_dt", ctypes.c_double),
                ("whfast_remove_invalid_particles", ctypes.c_bool)]


@pytest.mark.parametrize("integ", [4, 10])
def test_exit_flag_set_during_a_small_systems_run(lib, g, wl, integ):
    """A flag that another thread sets while a system of one block runs (up to 32 steps a
    launch) ends the run within a second, at a step that num_steps, t and the state agree on: the
    same as a run of num_steps steps."""
    G, dt = wl.G_AU_MSUN_DAY, 1.0
    x, v, m = (a[:9].copy() for a in next(s for s in wl.planetary_ensemble(8, 3) if s[2].size >= 9))

    def run(tf, after):
        xs, vs, ms = x.copy(), v.copy(), m.copy()
        system, keep = g.make_system(xs, ms, G, vs)
        flag = ctypes.c_bool(False)
        status = g.SimulationStatus(0.0, 0.0, 0)
        settings = g.Settings(0, False, ctypes.pointer(flag))
        ip = IntegratorParam(integ, dt, -1.0, -1.0, True)
        ap = g.AccelerationParam(g.METHOD_GPU_MASSLESS, 1.0, 0.0, 1)
        op = g.OutputParam(g.OUTPUT_METHOD_DISABLED, None, False, 0.0, 2, 2, 2, 0)
        lib.launch_simulation.restype = g.ErrorStatus
        timer = threading.Timer(after, setattr, (flag, "value", True))
        if after > 0:
            timer.start()
        t0 = time.perf_counter()
        st = lib.launch_simulation(ctypes.byref(system), ctypes.byref(ip), ctypes.byref(ap),
                                   ctypes.byref(op), ctypes.byref(status), ctypes.byref(settings),
                                   ctypes.c_double(tf))
        wall = time.perf_counter() - t0
        assert st.return_code == 0, g.take_traceback(lib, st)
        assert system.num_particles == 9
        return status, xs, vs, wall

    run(64 * dt, 0.0)   # the library is loaded and the GPU awake
    status, xs, vs, wall = run(1e9 * dt, 0.2)
    assert 32 < status.num_steps < 1e9 and status.t == status.num_steps * dt and wall < 1.2
    again, xr, vr, _ = run(status.num_steps * dt, 0.0)
    assert again.num_steps == status.num_steps
    assert xs.tobytes() == xr.tobytes() and vs.tobytes() == vr.tobytes()
