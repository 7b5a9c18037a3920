"""GPU parity of the dipole guiding-centre kernels (float64): the oracle's operations,
1e-13 for RK4 and 1e-10 for RK45, the bars of test_gpu_parity.py.

The ensemble holds what sends a step to the general right-hand side (radii and q/m
outside the range of the shared reciprocals, the dipole's centre, NaN) beside
ordinary lanes, and the zeros that an axial moment leaves out.
"""
import numpy as np
import pytest

from test_gpu_parity import _check_same_layout, _rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("alg", ["rk4", "rk45"])
@pytest.mark.parametrize("moment,center", [((0.0, 0.0, -8.0e22), (0.0, 0.0, 0.0)), ((0.0, 0.0, 5.0e22), (1.0e5, -3.0e5, 2.0e6)),
                                           ((1.0e22, -2.0e22, 7.0e22), (0.0, 0.0, 0.0)), ((3.0e22, 0.0, 0.0), (0.0, 5.0e5, 0.0))])
@pytest.mark.parametrize("odd", [False, True])
def test_gc_dipole(tp, orc, alg, moment, center, odd):
    w = tp.workloads.config4(70)
    y0, q2m = w.y0.copy(), w.q2m.copy()
    y0[2, ::3] = 0.2 * y0[0, ::3]
    y0[3, 5] = 0.0
    if odd:
        y0[:3, 0] = center
        y0[:3, 1] = 1.0e16
        y0[0, 2] = np.nan
        y0[3, 3] = np.nan
        q2m[4] = 1.0e-40
        q2m[6] = -1.0e40
    prob = tp.TraceGCProblem(y0, (0.0, float(w.tau_b.max())), (w.q, q2m, w.mu, tp.ZeroField(), tp.DipoleField(moment, center)))
    stop = tp.TerminateShell(1.5 * tp.Re, 9.0 * tp.Re) | tp.TerminateNaN()
    for kw in (dict(dt=w.tau_b / 200, tend=w.tau_b * 0.15, savestepinterval=7), dict(dt=w.tau_b / 200, tend=w.tau_b * 0.15, isoutside=stop)):
        if alg == "rk45":
            kw.update(reltol=1.0e-6, abstol=1.0e-9, maxiters=40)
        sols = tp.solve(prob, alg=alg, **kw)
        plan = tp.plan_gc(prob, alg=alg, **kw)
        ref = orc.gc_run(plan.desc, plan.E, plan.B, plan.y0, plan.q_i, plan.q2m_i, plan.mu_i, dt_i=plan.dt_i, tend_i=plan.tend_i)
        _check_same_layout(sols, ref)
        fine = np.isfinite(ref.u).all(axis=1)
        assert np.array_equal(np.isnan(sols.u_all), np.isnan(ref.u))
        bar = 1e-13 if alg == "rk4" else 1e-10
        assert _rel(sols.t_all, ref.t) <= bar
        assert _rel(sols.u_all[fine], ref.u[fine]) <= bar
