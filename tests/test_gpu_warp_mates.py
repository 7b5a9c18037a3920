"""An orbit does not depend on the particles that share its warp.

The segment kernels take saves, first half steps and ends in a pass in which the other
lanes of the warp step too, so a step runs through different code depending on the
neighbours; and which kernel or processing order a gridded solve takes depends on the
particle count.  Every orbit of a solve with uneven ends has to equal, bit for bit, the
one of a solve of every third particle alone.
"""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MOMENT = (0.0, 0.0, -8.0e22)
DX = 1.0e5


def _grid(tp, n, dtype, bc, seed=4, scale=1.0, order=1):
    rng = np.random.RandomState(seed)
    X = np.meshgrid(*[2 * math.pi * np.arange(m) / m for m in n], indexing="ij")
    wave = lambda: sum(rng.uniform(-1, 1) * np.cos(c + rng.uniform(0, 6)) for c in X)  # noqa: E731
    A = scale * np.array([1.0e-9 * wave(), 1.0e-9 * wave(), 5.0e-9 + 1.0e-9 * wave()])
    return tp.build_interpolator(A.astype(dtype), *[np.arange(m) * DX for m in n], order, bc)


def _setup(tp, field, n):
    """(E, B, u0, per-particle dt)."""
    rng = np.random.RandomState(11)
    if field == "dipole":
        r = tp.Re * rng.uniform(2.0, 6.0, n)
        d = rng.normal(size=(3, n))
        x = r * d / np.linalg.norm(d, axis=0)
        dt = 2 * math.pi / (tp.qi / tp.mi * 1.0e-7 * 8.0e22 / r**3) * 10 ** rng.uniform(-3.0, -1.3, n)
        return tp.ZeroField(), tp.DipoleField(MOMENT), np.concatenate([x, 1.0e7 * rng.normal(size=(3, n))]), dt
    dt = np.full(n, 2 * math.pi / (tp.qi / tp.mi * 5.0e-9) / 60)
    if field == "uniform":
        u0 = np.concatenate([rng.normal(size=(3, n)), 1.0e5 * rng.normal(size=(3, n))])
        return tp.UniformField((1.0e-4, 0.0, 2.0e-5)), tp.UniformField((1.0e-9, 2.0e-9, 5.0e-9)), u0, dt
    shape = (13, 11, 17)
    u0 = np.concatenate([DX * np.array(shape)[:, None] * rng.uniform(0.1, 0.9, (3, n)), 2.0e5 * rng.normal(size=(3, n))])
    if field == "b64":
        return tp.ZeroField(), _grid(tp, shape, np.float64, tp.FillExtrap()), u0, dt
    kind, order = np.float32 if field.startswith("eb32") else np.float64, 3 if field == "cubic64" else 1
    bc = {"eb32clamp": tp.ClampExtrap(), "eb32fill": tp.FillExtrap()}.get(field, tp.WrapExtrap())
    return [_grid(tp, shape, kind, bc, s, scale, order) for s, scale in ((5, 4.0e5), (4, 1.0))] + [u0, dt]


@pytest.mark.parametrize("precision", ["fp64", "fp32c"])
@pytest.mark.parametrize("alg", ["boris", "ms4"])
@pytest.mark.parametrize("field,n,every", [("uniform", 3000, 3), ("dipole", 3000, 3), ("dipole", 200000, 1), ("eb32", 3000, 40),
                                           ("eb32", 70000, 2), ("eb32", 70000, 20), ("eb32clamp", 200000, 20),
                                           ("eb32clamp", 70000, 2), ("eb32fill", 70000, 2), ("b64", 3000, 3), ("eb64", 70000, 20), ("cubic64", 70000, 20)])
def test_orbits_alone_and_together(tp, field, n, every, alg, precision):
    E, B, u0, dt = _setup(tp, field, n)
    a = {"boris": tp.Boris(), "ms4": tp.MultistepBoris4(2)}[alg]
    steps = 1 + (np.arange(n) * 7919) % 61
    idx = np.arange(0, n, 3)
    stop = tp.TerminateShell(1.5 * tp.Re, 7.0 * tp.Re) if field == "dipole" else None
    sols = []
    for k in (slice(None), idx):
        prob = tp.TraceProblem(np.ascontiguousarray(u0[:, k]), (0.0, float((steps * dt).max())), tp.prepare(E, B))
        sols.append(tp.solve(prob, a, tp.EnsembleB200(precision=precision, schedule="queue"), dt=dt[k], tend=(steps * dt)[k],
                             savestepinterval=every, isoutside=stop, trajectories=u0[0, k].size))
    full, sub = sols
    for x in ("nsaved", "nsteps", "retcodes"):
        assert np.array_equal(getattr(full, x)[idx], getattr(sub, x))
    first = np.concatenate([[0], np.cumsum(full.nsaved)])
    rows = np.concatenate([np.arange(first[i], first[i + 1]) for i in idx])
    assert np.array_equal(full.t_all[rows], sub.t_all)
    assert np.array_equal(full.u_all[rows], sub.u_all, equal_nan=True)
