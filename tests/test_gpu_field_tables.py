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
