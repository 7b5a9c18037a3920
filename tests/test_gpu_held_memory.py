"""Fields and tapes give their device memory back.

The library keeps at most 2 GB of what released fields and tapes held, whatever their
number; other allocators in the process and other processes get the rest.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KEEP = 2 << 30
SLACK = 256 << 20  # driver structures, other pools' granularity


def _free():
    import torch

    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_tapes_return_their_memory(tp):
    ctx = tp.Context.get(0)
    n, steps = 200_000, 200
    rng = np.random.RandomState(0)
    u0 = np.concatenate([rng.normal(size=(3, n)), 1.0e5 * rng.normal(size=(3, n))])
    prob = tp.TraceProblem(u0, (0.0, steps * 1.0e-2), tp.prepare(tp.ZeroField(), tp.UniformField((0.0, 0.0, 1.0e-8))))
    plan = tp.plan_adjoint(prob, dt=1.0e-2, trajectories=n, checkpoint_every=2)
    ctx.adjoint_forward(plan.desc, plan.E, plan.B, plan.u0)[1].close()  # library and module loading
    before = _free()
    tapes = [ctx.adjoint_forward(plan.desc, plan.E, plan.B, plan.u0)[1] for _ in range(5)]
    held = sum(t.info()[0] for t in tapes)
    assert held > KEEP + 4 * SLACK and before - _free() > held - KEEP - SLACK
    for t in tapes:
        t.close()
    assert before - _free() <= KEEP + SLACK


def test_fields_return_their_memory(tp):
    import gc

    ctx = tp.Context.get(0)
    before = _free()
    nodes = np.zeros((3, 200, 200, 200))  # float64: raw, two node tables: 8e6 x 72 bytes
    axes = [np.arange(200.0)] * 3
    fields = [tp.build_interpolator(nodes, *axes, 1, tp.FillExtrap()) for _ in range(6)]
    for f in fields:
        ctx.field(f)
    assert before - _free() > 6 * 8_000_000 * 72 - KEEP - SLACK
    del fields, f
    gc.collect()
    assert before - _free() <= KEEP + SLACK
