"""Host-to-host solves of one chunk: around the size at which there are two, with device inputs."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _plan(tp, n, **kw):
    w = tp.workloads.config3(n, nt=60, ssi=7)
    prob = tp.TraceProblem(w.u0, w.tspan, tp.prepare(w.E, w.B, species=w.species))
    return tp.plan_boris(prob, tp.Boris(), tp.EnsembleB200(), dt=w.dt, tend=w.tend * (0.3 + 0.7 * (np.arange(n) % 11) / 10),
                         savestepinterval=7, isoutside=w.isoutside, **kw)


def _same(a, b):
    for name in ("nsaved", "retcode", "nsteps", "t", "u"):
        assert np.array_equal(getattr(a, name), getattr(b, name)), name


@pytest.mark.parametrize("n", [1, 33, 65535, 65536, 65537])
@pytest.mark.parametrize("extra", [False, True])
def test_one_and_two_chunks(tp, n, extra):
    p = _plan(tp, n, save_fields=extra, save_work=extra)
    ctx = tp.Context.get(0)
    args = (p.desc, p.E, p.B, p.u0, p.dt_i, p.tend_i)
    _same(ctx.boris_run(*args, pipelined=True), ctx.boris_run(*args, pipelined=False))


def test_device_inputs(tp):
    import torch

    n = 500
    p = _plan(tp, n)
    ctx = tp.Context.get(0)
    ref = ctx.boris_run(p.desc, p.E, p.B, p.u0, p.dt_i, p.tend_i)
    u0 = torch.from_numpy(p.u0).cuda()
    torch.cuda.synchronize()
    rows = int(ref.nsaved.sum())
    out = [np.zeros(n, np.int32), np.zeros(n, np.int8), np.zeros(n, np.int64), np.zeros(rows), np.zeros((rows, 6))]
    total, ms = C.c_int64(), C.c_double()
    # dt and tspan are checked on the host, so they are host arrays
    ins = [u0.data_ptr(), p.dt_i.ctypes.data, p.tend_i.ctypes.data]
    code = ctx.lib.tp_boris_run_host(ctx.handle, C.byref(p.desc), ctx.field(p.E), ctx.field(p.B), *[C.c_void_p(x) for x in ins],
                                     n, rows, *[a.ctypes.data_as(C.c_void_p) for a in out], C.byref(total), C.byref(ms))
    assert code == 0 and total.value == rows
    for got, name in zip(out, ("nsaved", "retcode", "nsteps", "t", "u")):
        assert np.array_equal(got, getattr(ref, name)), name


@pytest.mark.parametrize("n,bad", [(1, 0), (70000, 0), (70000, 69999), (70000, 35000)])
def test_guiding_centres_with_a_backward_step(tp, n, bad):
    """One dt of the wrong sign is refused wherever it is in the table."""
    y0 = np.tile(np.array([[4 * tp.Re], [0.0], [0.0], [1.0e5]]), n)
    dt = np.full(n, 0.1)
    dt[bad] = -0.1
    prob = tp.TraceGCProblem(y0, (0.0, 1.0), (tp.qi, tp.qi / tp.mi, 1.0e-10, tp.ZeroField(), tp.DipoleField((0.0, 0.0, -8.0e22))))
    with pytest.raises(tp.ArgumentError):
        tp.solve(prob, tp.EnsembleB200(), alg="rk4", dt=dt, trajectories=n)
