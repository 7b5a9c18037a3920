"""GPU parity of the kernels for E zero with B a dipole, and for uniform fields.

FP32C results in the dipole equal those of the two-particles-per-thread
kernels, which run the general functions.  The float64 results equal the oracle's operation order; tolerance 1e-13 as in
test_gpu_parity.py (bitwise equality is expected).  The ensembles hold what the
segment loops and the shared reciprocals can get wrong: step counts and save
intervals around the segment length, lanes that end inside a segment, particle
counts off the warp size, zero coordinates, radii at which the general path
takes over, the Taylor branch of the Multistep rotation, NaN.
"""
import math

import numpy as np
import pytest

from test_gpu_parity import _both, _check_same_layout, _rel

pytestmark = pytest.mark.gpu

MOMENT = (0.0, 0.0, -8.0e22)


def _dipole_case(tp, n=77, seed=1):
    """(u0, dt): protons between 1.5 and 7 Earth radii; step angles from 1e-5 to 0.3 rad."""
    rng = np.random.RandomState(seed)
    r = tp.Re * rng.uniform(1.5, 7.0, n)
    d = rng.normal(size=(3, n))
    x = r * d / np.linalg.norm(d, axis=0)
    x[2, : n // 4] = 0.0          # equatorial plane, some with no velocity along z
    v = rng.normal(size=(3, n)) * 10 ** rng.uniform(5.0, 7.0, n)
    v[2, : n // 8] = 0.0
    gyro = 2 * math.pi / (tp.qi / tp.mi * 1.0e-7 * 8.0e22 / r**3)
    return np.concatenate([x, v]), gyro * 10 ** rng.uniform(-5.5, -1.3, n)


@pytest.mark.parametrize("nt,ssi", [(1, 1), (63, 1000), (64, 64), (65, 64), (200, 1), (200, 7), (1000, 129)])
@pytest.mark.parametrize("alg", ["boris", "ms2", "ms4", "ms6"])
def test_dipole_fixed_step(tp, orc, alg, nt, ssi):
    a = {"boris": tp.Boris(), "ms2": tp.MultistepBoris2(1), "ms4": tp.MultistepBoris4(2), "ms6": tp.MultistepBoris6(3)}[alg]
    u0, dt = _dipole_case(tp)
    steps = np.maximum(1, nt - np.arange(dt.size) % 5)  # uneven ends
    for stop in (None, tp.TerminateShell(1.6 * tp.Re, 6.5 * tp.Re)):
        prob = tp.TraceProblem(u0, (0.0, float((steps * dt).max())), tp.prepare(tp.ZeroField(), tp.DipoleField(MOMENT)))
        sols, ref = _both(tp, orc, prob, a, dt=dt, tend=steps * dt, savestepinterval=ssi, isoutside=stop, trajectories=dt.size)
        _check_same_layout(sols, ref)
        assert np.array_equal(sols.t_all, ref.t)
        assert _rel(sols.u_all, ref.u) <= 1e-13


@pytest.mark.parametrize("center", [(0.0, 0.0, 0.0), (1.0e6, -2.0e6, 3.0e5)])
def test_dipole_out_of_range_states(tp, orc, center):
    """Radii outside the reciprocals' range, the origin and NaN take the general functions."""
    u0, dt = _dipole_case(tp, 40, 2)
    u0[:3, 0] = center                       # r = 0: NaN from the first step
    u0[:3, 1] = np.array(center) + 1.0e-17   # below 2^-50 from an origin centre
    u0[:3, 2] = 1.0e16
    u0[:3, 3] = 1.0e200                      # |r|^2 overflows
    u0[3, 4] = np.nan
    u0[3, 5] = 1.0e300
    prob = tp.TraceProblem(u0, (0.0, 1.0), tp.prepare(tp.ZeroField(), tp.DipoleField(MOMENT, center)))
    for alg in (tp.Boris(), tp.MultistepBoris4(2)):
        sols, ref = _both(tp, orc, prob, alg, dt=dt, tend=70 * dt, savestepinterval=30, trajectories=40)
        _check_same_layout(sols, ref)
        assert np.array_equal(np.isnan(sols.u_all), np.isnan(ref.u))
        fine = np.isfinite(ref.u).all(axis=1)
        assert np.array_equal(fine, np.isfinite(sols.u_all).all(axis=1))
        assert _rel(sols.u_all[fine], ref.u[fine]) <= 1e-13


@pytest.mark.parametrize("E", [None, (3.0e-4, -1.0e-4, 2.0e-4)])
@pytest.mark.parametrize("B", [None, (1.0e-8, -2.0e-8, 3.0e-8)])
@pytest.mark.parametrize("alg", ["boris", "ms2", "ms4", "ms6"])
def test_uniform_fixed_step(tp, orc, alg, E, B):
    a = {"boris": tp.Boris(), "ms2": tp.MultistepBoris2(1), "ms4": tp.MultistepBoris4(2), "ms6": tp.MultistepBoris6(3)}[alg]
    rng = np.random.RandomState(3)
    u0 = np.concatenate([rng.normal(size=(3, 37)), 1.0e5 * rng.normal(size=(3, 37))])
    dt = 10 ** rng.uniform(-7.0, -1.5, 37)
    field = lambda f: tp.ZeroField() if f is None else tp.UniformField(f)  # noqa: E731
    prob = tp.TraceProblem(u0, (0.0, 1.0), tp.prepare(field(E), field(B)))
    for nt, ssi in ((1, 1), (130, 1), (130, 64), (257, 300)):
        sols, ref = _both(tp, orc, prob, a, dt=dt, tend=nt * dt, savestepinterval=ssi, trajectories=37)
        _check_same_layout(sols, ref)
        assert np.array_equal(sols.t_all, ref.t)
        assert _rel(sols.u_all, ref.u) <= 1e-13


def test_shell_edges(tp, orc):
    """Squared-radius thresholds decide as the square roots do, to the last bit."""
    rmin, rmax = 1.1 * tp.Re, 3.3 * tp.Re
    r = np.concatenate([rmin * (1 + np.arange(-8, 9) * 2.0**-53), rmax * (1 + np.arange(-8, 9) * 2.0**-53)])
    n = r.size
    for axis in range(3):
        u0 = np.zeros((6, n))
        u0[axis] = r
        u0[(axis + 1) % 3] = 1.0e-9 * r * (np.arange(n) % 3)
        for E, B in ((tp.ZeroField(), tp.DipoleField(MOMENT)), (tp.ZeroField(), tp.UniformField((0.0, 0.0, 1.0e-9)))):
            for lo, hi in ((rmin, rmax), (-1.0, rmax), (rmin, math.inf), (0.0, 0.0)):
                prob = tp.TraceProblem(u0, (0.0, 3.0e-3), tp.prepare(E, B))
                sols, ref = _both(tp, orc, prob, tp.Boris(), dt=1.0e-3, isoutside=tp.TerminateShell(lo, hi), trajectories=n)
                _check_same_layout(sols, ref)
                assert _rel(sols.u_all, ref.u) <= 1e-13


@pytest.mark.parametrize("ssi,every", [(1000, False), (1, True), (7, True), (64, True)])
@pytest.mark.parametrize("cap", [0, 1, 64, 65, 300])
def test_dipole_adaptive(tp, orc, cap, ssi, every):
    u0, dt = _dipole_case(tp, 77, 4)
    u0[:3, 3] = 1.0e16  # refused by the fast functions at every step
    B0 = np.linalg.norm(tp.workloads.dipole_B(u0[:3].T), axis=1)
    tend = 0.1 * 2 * math.pi / (tp.qi / tp.mi * B0) * np.linspace(0.3, 200.0, dt.size)
    for stop in (None, tp.TerminateShell(1.6 * tp.Re, 6.5 * tp.Re)):
        prob = tp.TraceProblem(u0, (0.0, float(tend.max())), tp.prepare(tp.ZeroField(), tp.DipoleField(MOMENT)))
        sols, ref = _both(tp, orc, prob, tp.AdaptiveBoris(0.1), tend=tend, savestepinterval=ssi, save_everystep=every,
                          isoutside=stop, step_cap=cap, trajectories=dt.size)
        _check_same_layout(sols, ref)
        assert _rel(sols.t_all, ref.t) <= 1e-13
        assert _rel(sols.u_all, ref.u) <= 1e-13


@pytest.mark.parametrize("alg", ["boris", "ms2", "ms4", "ms6"])
def test_dipole_fp32c_equals_two_per_thread(tp, alg):
    a = {"boris": tp.Boris(), "ms2": tp.MultistepBoris2(1), "ms4": tp.MultistepBoris4(2), "ms6": tp.MultistepBoris6(3)}[alg]
    u0, dt = _dipole_case(tp, 77, 5)
    for nt, ssi, stop in ((1, 1, None), (130, 1, None), (200, 64, tp.TerminateShell(1.6 * tp.Re, 6.5 * tp.Re))):
        prob = tp.TraceProblem(u0, (0.0, float(nt * dt.max())), tp.prepare(tp.ZeroField(), tp.DipoleField(MOMENT)))
        one, two = (tp.solve(prob, a, tp.EnsembleB200(precision="fp32c", particles_per_thread=k), dt=dt, tend=nt * dt,
                             savestepinterval=ssi, isoutside=stop, trajectories=77) for k in (1, 2))
        for x in ("nsaved", "nsteps", "retcodes", "t_all", "u_all"):
            assert np.array_equal(getattr(one, x), getattr(two, x))


@pytest.mark.parametrize("cap,ssi", [(1, 1), (64, 64), (65, 7), (300, 1000)])
def test_dipole_adaptive_fp32c_schedules(tp, cap, ssi):
    u0, _ = _dipole_case(tp, 77, 6)
    prob = tp.TraceProblem(u0, (0.0, 1.0e9), tp.prepare(tp.ZeroField(), tp.DipoleField(MOMENT)))
    one, two = (tp.solve(prob, tp.AdaptiveBoris(0.1), tp.EnsembleB200(precision="fp32c", schedule=s, block=b),
                         savestepinterval=ssi, step_cap=cap, trajectories=77) for s, b in (("static", 32), ("queue", 128)))
    for x in ("nsaved", "nsteps", "retcodes", "t_all", "u_all"):
        assert np.array_equal(getattr(one, x), getattr(two, x))


@pytest.mark.parametrize("alg", ["boris", "ms2", "ms4", "ms6"])
@pytest.mark.parametrize("E", [None, (3.0e-4, -1.0e-4, 2.0e-4)])
def test_uniform_fp32c_error(tp, orc, alg, E):
    """Float rotation factors misplace the phase by at most 2^-22 of a step's angle
    (< 1 rad) per step and a position increment is rounded to float, so after N
    steps the position is within N 2^-22 of the path length."""
    a = {"boris": tp.Boris(), "ms2": tp.MultistepBoris2(1), "ms4": tp.MultistepBoris4(2), "ms6": tp.MultistepBoris6(3)}[alg]
    rng = np.random.RandomState(7)
    u0 = np.concatenate([rng.normal(size=(3, 37)), 1.0e5 * rng.normal(size=(3, 37))])
    dt = 10 ** rng.uniform(-4.0, -1.5, 37)
    field = tp.ZeroField() if E is None else tp.UniformField(E)
    prob = tp.TraceProblem(u0, (0.0, 1.0), tp.prepare(field, tp.UniformField((1.0e-8, -2.0e-8, 3.0e-8))))
    for nt, ssi in ((1, 1), (130, 1), (257, 64)):
        sols, ref = _both(tp, orc, prob, a, tp.EnsembleB200(precision="fp32c"), dt=dt, tend=nt * dt, savestepinterval=ssi,
                          trajectories=37)
        _check_same_layout(sols, ref)
        assert np.array_equal(sols.t_all, ref.t)
        off = np.linalg.norm(sols.u_all[:, :3] - ref.u[:, :3], axis=1)
        speed = np.linalg.norm(ref.u[:, 3:], axis=1) + 2.0e4  # E x B drift below 2e4 m/s
        assert np.all(off <= nt * 2.0**-22 * speed * np.maximum(ref.t, np.repeat(dt, ref.nsaved)))
