"""The node tables that a run reads belong to the fields of that run.

E and B grids on one geometry are read through a table that holds both.  After
field_update a solve has to use the new values, as a solve with a new field does.
"""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DX = 1.0e5
N3 = (9, 8, 10)
DT = 0.25


def _data(seed, scale=1.0):
    rng = np.random.RandomState(seed)
    X = np.meshgrid(*[2 * math.pi * np.arange(m) / m for m in N3], indexing="ij")
    wave = lambda: sum(rng.uniform(-1, 1) * np.cos(c + rng.uniform(0, 6)) for c in X)  # noqa: E731
    return (scale * np.array([1.0e-9 * wave(), 1.0e-9 * wave(), 5.0e-9 + 1.0e-9 * wave()])).astype(np.float32)


def _field(tp, data, order):
    return tp.build_interpolator(data, *[np.arange(m) * DX for m in N3], order, tp.WrapExtrap())


def _u0(n=100):
    rng = np.random.RandomState(3)
    return np.concatenate([DX * np.array(N3)[:, None] * rng.uniform(0, 1, (3, n)), 2.0e5 * rng.normal(size=(3, n))])


def _solve(tp, E, B, precision="fp32c", adaptive=False):
    prob = tp.TraceProblem(_u0(), (0.0, 60 * DT), tp.prepare(E, B))
    if adaptive:
        return tp.solve(prob, tp.AdaptiveBoris(0.1), tp.EnsembleB200(precision=precision), savestepinterval=10, trajectories=100)
    return tp.solve(prob, tp.Boris(), tp.EnsembleB200(precision=precision), dt=DT, savestepinterval=20, trajectories=100)


@pytest.mark.parametrize("order", [1, 3])
@pytest.mark.parametrize("which", ["E", "B"])
@pytest.mark.parametrize("precision,adaptive", [("fp32c", False), ("fp32c", True), ("fp64", False)])
def test_solve_after_update(tp, order, which, precision, adaptive):
    ctx = tp.Context.get(0)
    E, B = _field(tp, _data(1, 4.0e5), order), _field(tp, _data(2), order)
    old = _solve(tp, E, B, precision, adaptive)
    new = _data(7, 4.0e5 if which == "E" else 1.0)
    ctx.field_update(E if which == "E" else B, new)
    got = _solve(tp, E, B, precision, adaptive)
    fresh = _solve(tp, *[_field(tp, f.data, order) for f in (E, B)], precision, adaptive)
    assert not np.array_equal(got.u_all, old.u_all)
    assert np.array_equal(got.t_all, fresh.t_all)
    assert np.array_equal(got.u_all, fresh.u_all)


def _churn(tp, B, order):
    """Give B another partner and let new fields and tapes take what was released."""
    for seed in (21, 22):
        _solve(tp, _field(tp, _data(seed, 4.0e5), order), B)
    for seed in (23, 24, 25):
        _solve(tp, _field(tp, _data(seed, 4.0e5), order), _field(tp, _data(seed + 5), order))


def test_tape_keeps_its_table(tp):
    """A tape of (E1, B) is run backward after solves of (E2, B)."""
    ctx = tp.Context.get(0)
    E, B = _field(tp, _data(1, 4.0e5), 1), _field(tp, _data(2), 1)
    prob = tp.TraceProblem(_u0(), (0.0, 60 * DT), tp.prepare(E, B))
    grad = np.random.RandomState(5).normal(size=(100, 6))
    out = []
    for churn in (False, True):
        p = tp.plan_adjoint(prob, dt=DT, trajectories=100)
        _, tape = ctx.adjoint_forward(p.desc, p.E, p.B, p.u0)
        if churn:
            _churn(tp, B, 1)
        out.append(tape.backward(grad))
        tape.close()
    assert np.array_equal(out[0].u0, out[1].u0)
    # node gradients are summed by atomics: float32 sums of at most 60 steps x 100 orbits
    for a, b in ((out[0].E, out[1].E), (out[0].B, out[1].B)):
        assert np.abs(a - b).max() <= 6000 * 2.0**-24 * np.abs(a).max()


@pytest.mark.parametrize("order", [1, 3])
def test_graph_keeps_its_table_and_sees_updates(tp, order):
    import torch

    ctx = tp.Context.get(0)
    E, B = _field(tp, _data(1, 4.0e5), order), _field(tp, _data(2), order)
    prob = tp.TraceProblem(_u0(), (0.0, 60 * DT), tp.prepare(E, B))
    plan = tp.plan_boris(prob, tp.Boris(), tp.EnsembleB200(precision="fp32c"), dt=DT, savestepinterval=20, trajectories=100)
    n, slots = 100, ctx.slots(plan.desc, 100)
    u0 = torch.from_numpy(plan.u0).cuda()
    out = [torch.zeros((slots, n), dtype=torch.float64, device="cuda"), torch.zeros((slots, 6, n), dtype=torch.float64, device="cuda"),
           torch.zeros(n, dtype=torch.int32, device="cuda"), torch.zeros(n, dtype=torch.int8, device="cuda"),
           torch.zeros(n, dtype=torch.int64, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")]
    args = (plan.desc, plan.E, plan.B, u0.data_ptr(), None, None, n, slots, *[x.data_ptr() for x in out])
    stream = torch.cuda.current_stream().cuda_stream

    def states():
        torch.cuda.synchronize()
        u = out[1].clone()
        out[1].zero_()
        return u

    ctx.boris_run_device(*args, stream)
    ref = states()
    graph = ctx.boris_graph(*args)
    _churn(tp, B, order)
    graph.launch(stream)
    assert torch.equal(states(), ref)
    for f, d in ((E, _data(31, 4.0e5)), (B, _data(32))):
        ctx.field_update(f, d)
        graph.launch(stream)
        got = states()
        assert not torch.equal(got, ref)
        ctx.boris_run_device(*args, stream)
        ref = states()
        assert torch.equal(got, ref)
    graph.close()
