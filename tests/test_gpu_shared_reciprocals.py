"""Quotients and roots that share a reciprocal equal `/` and sqrt to the last bit.

The float64 dipole kernels (full orbits and guiding centres) divide with fdiv64.cuh.  The same
runs through the general kernels, which use the operators, must give the same bits: two
particles per thread, and a uniform E of zero instead of no E (it adds +0 everywhere).
"""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MOMENT = (0.0, 0.0, -8.0e22)
N = 20_000


def _orbits(tp):
    rng = np.random.RandomState(17)
    r = tp.Re * rng.uniform(1.2, 10.0, N)
    d = rng.normal(size=(3, N))
    x = r * d / np.linalg.norm(d, axis=0)
    v = rng.normal(size=(3, N)) * 10 ** rng.uniform(4.0, 7.3, N)
    gyro = 2 * math.pi / (tp.qi / tp.mi * 1.0e-7 * 8.0e22 / r**3)
    return np.concatenate([x, v]), gyro * 10 ** rng.uniform(-5.0, -1.0, N)


def _same(a, b):
    for x in ("nsaved", "nsteps", "retcodes", "t_all"):
        assert np.array_equal(getattr(a, x), getattr(b, x)), x
    assert np.array_equal(a.u_all, b.u_all, equal_nan=True)


@pytest.mark.parametrize("moment", [MOMENT, (3.0e22, -2.0e22, 7.0e22)])
@pytest.mark.parametrize("alg", ["boris", "ms2", "ms4", "ms6"])
def test_fixed_steps(tp, alg, moment):
    a = {"boris": tp.Boris(), "ms2": tp.MultistepBoris2(1), "ms4": tp.MultistepBoris4(2), "ms6": tp.MultistepBoris6(3)}[alg]
    u0, dt = _orbits(tp)
    prob = tp.TraceProblem(u0, (0.0, 1.0), tp.prepare(tp.ZeroField(), tp.DipoleField(moment, (1.0e5, -2.0e5, 0.0))))
    _same(*[tp.solve(prob, a, tp.EnsembleB200(particles_per_thread=k), dt=dt, tend=100 * dt, savestepinterval=33, trajectories=N)
            for k in (1, 2)])


def test_adaptive_steps(tp):
    u0, dt = _orbits(tp)
    sols = []
    for E in (tp.ZeroField(), tp.UniformField((0.0, 0.0, 0.0))):
        prob = tp.TraceProblem(u0, (0.0, 1.0e9), tp.prepare(E, tp.DipoleField(MOMENT)))
        sols.append(tp.solve(prob, tp.AdaptiveBoris(0.1), tp.EnsembleB200(), savestepinterval=33, step_cap=100, trajectories=N))
    _same(*sols)


@pytest.mark.parametrize("moment", [MOMENT, (3.0e22, -2.0e22, 7.0e22)])
@pytest.mark.parametrize("alg", ["rk4", "rk45"])
def test_guiding_centres(tp, alg, moment):
    rng = np.random.RandomState(19)
    r, phi, z = tp.Re * rng.uniform(2.0, 8.0, N), rng.uniform(0, 2 * math.pi, N), rng.uniform(-0.5, 0.5, N)
    x = np.array([r * np.cos(phi), r * np.sin(phi), r * z])
    y0 = np.concatenate([x, 10 ** rng.uniform(4.0, 6.0, (1, N))])
    mu = 10 ** rng.uniform(-11.0, -9.0, N)
    kw = dict(alg=alg, trajectories=N, savestepinterval=7)
    if alg == "rk4":
        kw["dt"] = 0.3
    sols = []
    for E in (tp.ZeroField(), tp.UniformField((0.0, 0.0, 0.0))):
        prob = tp.TraceGCProblem(y0, (0.0, 15.0), (np.full(N, tp.qi), np.full(N, tp.qi / tp.mi), mu, E, tp.DipoleField(moment)))
        sols.append(tp.solve(prob, tp.EnsembleB200(), **kw))
    _same(*sols)
