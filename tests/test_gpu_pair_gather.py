"""GPU parity of the gridded pushes whose stencils pairs of lanes gather together.

Float64 results equal the oracle's operation order (1e-13, as test_gpu_parity.py).
FP32C rounds fields, rotations and increments to float: over the 40 steps here the
positions stay within 40 x 2^-22 of the path length (about 1e-5), as derived in
test_gpu_segments.py, the fields being smooth on the scale of that error.  Particle
counts are off the warp size, so pairs and warps are incomplete, and grids have as
few as two nodes per axis, so neighbours wrap onto the same line or node.
"""
import math

import numpy as np
import pytest

from test_gpu_parity import _both, _check_same_layout, _rel

pytestmark = pytest.mark.gpu

DX = 1.0e5


def _grid(tp, n, bc, dtype, seed):
    rng = np.random.RandomState(seed)
    x = [2 * math.pi * np.arange(m) / m for m in n]
    X = np.meshgrid(*x, indexing="ij")
    wave = lambda: sum(rng.uniform(-1, 1) * np.cos(c + rng.uniform(0, 6)) for c in X)  # noqa: E731
    B = np.array([1.0e-9 * wave(), 1.0e-9 * wave(), 5.0e-9 + 1.0e-9 * wave()]).astype(dtype)
    E = np.array([1.0e-4 * wave() for _ in range(3)]).astype(dtype)
    axes = [np.arange(m) * DX for m in n]
    return [tp.build_interpolator(a, *axes, 1, bc) for a in (E, B)]


@pytest.mark.parametrize("n", [(2, 2, 2), (3, 5, 2), (7, 4, 9), (33, 32, 31)])
@pytest.mark.parametrize("bc", ["wrap", "clamp", "fill"])
@pytest.mark.parametrize("count", [1, 33, 70])
def test_grid_push(tp, orc, n, bc, count):
    edge = {"wrap": tp.WrapExtrap(), "clamp": tp.ClampExtrap(), "fill": tp.FillExtrap()}[bc]
    E, B = _grid(tp, n, edge, np.float32, 3)
    rng = np.random.RandomState(count)
    size = np.array(n) - (0 if bc == "wrap" else 1)
    u0 = np.concatenate([DX * size[:, None] * rng.uniform(0.2, 0.8, (3, count)), 2.0e5 * rng.normal(size=(3, count))])
    if count > 3:
        u0[:3, 1] = 0.0                      # a node
        u0[:3, 2] = DX * (size - 1)          # the last node, or the last cell of a periodic axis
        if bc != "fill":
            u0[:3, 3] = -2.3 * DX * size     # outside
    else:
        u0[3:] *= 0.1
    steps = np.maximum(1, 40 - np.arange(count) % 3)
    dt = 2 * math.pi / (tp.qi / tp.mi * 5.0e-9) / 100
    if bc == "fill":  # stay inside: NaN fields are compared in test_grid_push_outside
        u0[:3] = np.clip(u0[:3], 0.45 * DX * size[:, None], 0.55 * DX * size[:, None])
        u0[3:] *= 1.0e-4
        E.data *= 1.0e-6
    prob = tp.TraceProblem(u0, (0.0, 40 * dt), tp.prepare(E, B))
    for alg in (tp.Boris(), tp.MultistepBoris4(2)):
        for ssi in (1, 17):
            kw = dict(dt=dt, tend=steps * dt, savestepinterval=ssi, trajectories=count)
            sols, ref = _both(tp, orc, prob, alg, **kw)
            _check_same_layout(sols, ref)
            assert np.array_equal(sols.t_all, ref.t)
            assert _rel(sols.u_all, ref.u) <= 1e-13
            got = tp.solve(prob, alg, tp.EnsembleB200(precision="fp32c"), **kw)
            _check_same_layout(got, ref)
            off = np.linalg.norm(got.u_all[:, :3] - ref.u[:, :3], axis=1)
            path = np.linalg.norm(u0[3:], axis=0).repeat(ref.nsaved) * ref.t + 1.0e6 * dt
            assert np.all(off <= 40 * 2.0**-22 * path)


@pytest.mark.parametrize("precision", ["fp64", "fp32c"])
def test_grid_push_outside(tp, orc, precision):
    """Outside a FillExtrap(NaN) grid, and at NaN and infinite positions, lanes end in NaN without disturbing their partners."""
    E, B = _grid(tp, (9, 8, 7), tp.FillExtrap(), np.float32, 4)
    rng = np.random.RandomState(9)
    u0 = np.concatenate([DX * rng.uniform(2.0, 4.0, (3, 66)), 1.0e3 * rng.normal(size=(3, 66))])
    u0[:3, 5::7] = -3.0 * DX
    u0[0, 6] = np.nan
    u0[1, 9] = np.inf
    u0[2, 12] = -np.inf
    dt = 1.0e-3
    prob = tp.TraceProblem(u0, (0.0, 20 * dt), tp.prepare(E, B))
    sols, ref = _both(tp, orc, prob, tp.Boris(), tp.EnsembleB200(precision=precision), dt=dt, savestepinterval=10,
                      trajectories=66)
    _check_same_layout(sols, ref)
    assert np.array_equal(np.isnan(sols.u_all), np.isnan(ref.u))
    E, B = _grid(tp, (9, 8, 7), tp.ClampExtrap(), np.float32, 4)
    prob = tp.TraceProblem(u0, (0.0, 20 * dt), tp.prepare(E, B))
    got = tp.solve(prob, tp.Boris(), tp.EnsembleB200(precision=precision), dt=dt, savestepinterval=10, trajectories=66)
    fine = np.isfinite(u0).all(axis=0)
    one = tp.solve(prob.remake(u0=u0[:, fine]), tp.Boris(), tp.EnsembleB200(precision=precision), dt=dt, savestepinterval=10,
                   trajectories=int(fine.sum()))
    keep = np.repeat(fine, got.nsaved)
    assert np.array_equal(got.u_all[keep], one.u_all)


def test_interleaved_table_of_a_large_odd_grid(tp, orc):
    """The transposed table of a grid whose sides are off the tile size, through save_fields."""
    E, B = _grid(tp, (65, 3, 70), tp.WrapExtrap(), np.float32, 6)
    rng = np.random.RandomState(1)
    u0 = np.concatenate([DX * np.array([[65], [3], [70]]) * rng.uniform(0, 1, (3, 101)), np.zeros((3, 101))])
    prob = tp.TraceProblem(u0, (0.0, 1.0e-3), tp.prepare(E, B))
    sols, ref = _both(tp, orc, prob, tp.Boris(), dt=1.0e-3, save_fields=True, trajectories=101)
    assert _rel(sols.u_all, ref.u) <= 1e-13


@pytest.mark.parametrize("n", [(2, 2, 2), (3, 5, 2), (33, 34, 65)])
@pytest.mark.parametrize("bc", ["wrap", "clamp", "fill"])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_grid_push_b_alone(tp, orc, n, bc, dtype):
    """E zero and B on a grid, float64: the oracle's operation order in every order of the update; lanes that start
    outside a filled grid or at NaN stay NaN."""
    edge = {"wrap": tp.WrapExtrap(), "clamp": tp.ClampExtrap(), "fill": tp.FillExtrap()}[bc]
    B = _grid(tp, n, edge, dtype, 6)[1]
    count = 70
    rng = np.random.RandomState(count)
    size = np.array(n) - (0 if bc == "wrap" else 1)
    u0 = np.concatenate([DX * size[:, None] * rng.uniform(0.4, 0.6, (3, count)), 20.0 * rng.normal(size=(3, count))])
    u0[:3, 1] = 0.0                  # a node
    u0[:3, 2] = -2.3 * DX * size     # outside
    u0[2, 3] = np.nan
    if bc != "fill":
        u0[3:, 4:] *= 1.0e4
        u0[:3, 5] = DX * (size - 1)
    steps = 40 - np.arange(count) % 3
    dt = 2 * math.pi / (tp.qi / tp.mi * 5.0e-9) / 100
    prob = tp.TraceProblem(u0, (0.0, 40 * dt), tp.prepare(tp.ZeroField(), B))
    for alg in (tp.Boris(), tp.MultistepBoris2(), tp.MultistepBoris4(2), tp.MultistepBoris6(3)):
        for ssi in (1, 17):
            sols, ref = _both(tp, orc, prob, alg, dt=dt, tend=steps * dt, savestepinterval=ssi, trajectories=count)
            _check_same_layout(sols, ref)
            assert np.array_equal(sols.t_all, ref.t)
            assert np.array_equal(np.isnan(sols.u_all), np.isnan(ref.u))
            assert _rel(np.nan_to_num(sols.u_all), np.nan_to_num(ref.u)) <= 1e-13


@pytest.mark.parametrize("bc", ["wrap", "clamp", "fill"])
@pytest.mark.parametrize("count", [1, 33, 150])
def test_adjoint_forward(tp, bc, count):
    """The recorded forward gathers as the FP32C push does: its final states stay within the same 40 x 2^-22 of the path."""
    import torch
    from testparticle_b200.autograd import GridTensor, boris_final_state

    edge = {"wrap": tp.WrapExtrap(), "clamp": tp.ClampExtrap(), "fill": tp.FillExtrap()}[bc]
    n = (7, 4, 9)
    E, B = _grid(tp, n, edge, np.float32, 5)
    rng = np.random.RandomState(count)
    size = np.array(n) - 1
    u0 = np.concatenate([DX * size[:, None] * rng.uniform(0.4, 0.6, (3, count)), 2.0e4 * rng.normal(size=(3, count))])
    if bc != "fill" and count > 1:
        u0[:3, 1] = -2.3 * DX * size
    dt = 2 * math.pi / (tp.qi / tp.mi * 5.0e-9) / 100
    E.data *= 0.1
    want = tp.solve(tp.TraceProblem(u0, (0.0, 40 * dt), tp.prepare(E, B)), tp.Boris(), tp.EnsembleB200(precision="fp32c"),
                    dt=dt, save_everystep=False, save_start=False, trajectories=count).u_all
    grids = [GridTensor(torch.from_numpy(np.ascontiguousarray(f.data.T)).cuda().permute(3, 2, 1, 0), (0.0,) * 3, (DX,) * 3, edge)
             for f in (E, B)]
    got = boris_final_state(torch.from_numpy(np.ascontiguousarray(u0.T)).cuda(), *grids, q2m=tp.qi / tp.mi, dt=dt,
                            tspan=(0.0, 40 * dt)).cpu().numpy()
    path = 40 * dt * (np.linalg.norm(u0[3:], axis=0) + 1.0e5)
    fine = np.isfinite(want).all(axis=1)  # a particle that leaves a filled grid ends in NaN
    assert np.array_equal(np.isnan(got), np.isnan(want))
    want, got, path = want[fine], got[fine], path[fine]
    assert np.all(np.linalg.norm(got[:, :3] - want[:, :3], axis=1) <= 40 * 2.0**-22 * path)
    assert np.all(np.linalg.norm(got[:, 3:] - want[:, 3:], axis=1) <= 40 * 2.0**-22 * path / (40 * dt))
