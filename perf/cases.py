"""The performance cases: what a program that uses this package has it do, through its public entry points.

Three kinds of call cover the package's paths:

  solve    solve() on host tables, the reference's entry point: full orbits and guiding centres
  push     Context.boris_run_device on device tables, the same full-orbit solve for programs that keep
           their particles on the GPU (what bench.py times)
  adjoint  boris_final_state and its backward pass on CUDA tensors

The fields, particle distributions and step sizes are those of the benchmark workloads
(testparticle.jl_b200/workloads.py): protons in a uniform field, the Earth-dipole ensemble, a turbulent
periodic grid, dipole guiding centres.  Step counts stay where an orbit's final state still depends
smoothly on its start (one or a few save intervals): longer runs repeat the same step.

`exact` restates each solve in float64 torch; it shares no code with the package.
"""
import importlib.util
import math
import sys
from pathlib import Path

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

RE = 6371.0e3
QI, MI, ME = 1.602176634e-19, 1.67262192369e-27, 9.1093837015e-31
LIGHT = 299792458.0
Q2M = QI / MI
COEF = 1.25663706212e-6 / (4.0 * math.pi)
MOMENT = (0.0, 0.0, -8.0e22)


def _package():
    """This directory's package under its import name."""
    name = "testparticle_b200"
    if name not in sys.modules:
        root = Path(__file__).resolve().parent.parent / "testparticle.jl_b200"
        spec = importlib.util.spec_from_file_location(name, root / "__init__.py", submodule_search_locations=[str(root)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


# ------------------------------------------------------------------ the cases
def _case(kind, **kw):
    """Every key of a case, with the values that most kinds share."""
    d = {"kind": kind, "field": "dipole", "alg": "boris", "precision": "fp64", "n": 1, "steps": 1, "save_every": 1,
         "nx": 0, "ny": 0, "nz": 0, "order": 1}
    d.update(kw)
    return d


def listed():
    return [
        # one orbit traced in crossed uniform fields, every step saved: the first thing a user runs
        _case("solve", name="one_orbit", field="uniform", n=1, steps=200),
        # the plain-Boris workload: 1000 protons, uniform B, 1e4 steps, saves every 100
        _case("solve", name="uniform_1k", field="uniform", n=1000, steps=10000, save_every=100),
        # the headline ensemble on the device, float32 push: 1e6 dipole protons to the first save
        _case("push", name="dipole_fp32c", alg="multistep", precision="fp32c", n=1000000, steps=1000, save_every=500),
        # the same ensemble in the drop-in precision, from host tables to host results
        _case("solve", name="dipole_solve_fp64", alg="multistep", n=250000, steps=2000, save_every=500),
        # adaptive steps in the dipole: uneven lifetimes, work queue
        _case("push", name="dipole_adaptive", alg="adaptive", n=300001, steps=1000),
        # 1e6 protons in the 128^3 turbulent field, float32 push
        _case("push", name="grid_fp32c", field="turbulence", precision="fp32c", n=1000000, steps=250, save_every=125,
              nx=128, ny=128, nz=128),
        # the drop-in precision on a ragged grid and an odd particle count
        _case("push", name="grid_fp64", field="turbulence", n=400009, steps=250, save_every=100, nx=120, ny=100, nz=91),
        # cubic interpolation of the same kind of field
        _case("push", name="grid_cubic", field="turbulence", precision="fp32c", n=200000, steps=200, save_every=100,
              nx=96, ny=96, nz=96, order=3),
        # magnetic field only, float64 nodes from a simulation box: particles end at its walls
        _case("push", name="box_b_only", field="box", n=200003, steps=250, save_every=50, nx=61, ny=53, nz=47),
        # guiding centres over one bounce period, half electrons and half protons
        _case("solve", name="gc_rk4", alg="rk4", n=262144, steps=200),
        _case("solve", name="gc_rk45", alg="rk45", n=262144),
        # forward and gradient of the final states with respect to starts and field nodes
        _case("adjoint", name="adjoint_grid", field="turbulence", precision="fp32c", n=131072, steps=128, nx=128, ny=128,
              nz=128),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    def steps(lo, hi):
        s = _log(rng, lo, hi)
        every = max(1, s // rng.randint(1, 10))
        return {"steps": s, "save_every": every}

    def grid(lo, hi):
        return {k: rng.randint(lo, hi) for k in ("nx", "ny", "nz")}

    prec = rng.choice(["fp64", "fp32c"])
    what = rng.randrange(9)
    if what == 0:
        n = _log(rng, 1, 2000)
        return _case("solve", field="uniform", precision=prec, n=n, **steps(50, 5000 if n < 500 else 1000))
    if what == 1:
        return _case("push", alg="multistep", precision=prec, n=_log(rng, 1000, 500000), **steps(100, 1000))
    if what == 2:
        return _case("solve", alg=rng.choice(["boris", "multistep"]), precision=prec, n=_log(rng, 1000, 200000),
                     **steps(100, 1000))
    if what == 3:
        return _case("push", alg="adaptive", precision=prec, n=_log(rng, 1000, 300000), steps=_log(rng, 100, 1000))
    if what == 4:
        return _case("push", field="turbulence", alg=rng.choice(["boris", "boris", "multistep"]), precision=prec,
                     n=_log(rng, 1000, 700000), **steps(50, 250), **grid(24, 128))
    if what == 5:
        return _case("push", field="turbulence", precision="fp32c", n=_log(rng, 1000, 200000), order=3, **steps(50, 200),
                     **grid(24, 100))
    if what == 6:
        return _case("push", field="box", precision=prec, n=_log(rng, 100, 300000), **steps(50, 250), **grid(20, 80))
    if what == 7:
        alg = rng.choice(["rk4", "rk45"])
        return _case("solve", alg=alg, precision=prec if alg == "rk4" else "fp64", n=_log(rng, 500, 200000),
                     steps=_log(rng, 50, 400) if alg == "rk4" else 1)
    return _case("adjoint", field="turbulence", precision="fp32c", n=_log(rng, 500, 100000), steps=_log(rng, 20, 128),
                 **grid(24, 128))


# ------------------------------------------------------------------ inputs
def _rng(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _uniform(g, n, lo, hi):
    return lo + (hi - lo) * torch.rand(n, generator=g, device="cuda", dtype=torch.float64)


def _normal(g, shape, sigma):
    return sigma * torch.randn(shape, generator=g, device="cuda", dtype=torch.float64)


def _dipole(r):
    """Dipole field at rows of r, float64."""
    m = torch.tensor(MOMENT, dtype=torch.float64, device=r.device)
    d = r.norm(dim=1, keepdim=True)
    rh = r / d
    return COEF * (3 * (rh @ m)[:, None] * rh - m) / d**3


def _turbulence(seed, nx, ny, nz, dx=1.0e5, b0=5.0e-9, modes=48):
    """E = -u x B and B = B0 z + divergence-free periodic waves (rms 0.3 B0): (3, nx, ny, nz) float64."""
    r = np.random.RandomState(seed % (1 << 31))
    n = (nx, ny, nz)
    ax = [torch.arange(m, dtype=torch.float64, device="cuda") * (2 * math.pi / m) for m in n]
    B = torch.zeros((3,) + n, dtype=torch.float64, device="cuda")
    for kmag in np.exp(np.linspace(0.0, math.log(8.0), modes)):
        while True:
            d = r.standard_normal(3)
            k = np.rint(kmag * d / np.linalg.norm(d)).astype(int)
            if k.any():
                break
        kv = k / (np.array(n) * dx)
        e = np.cross(kv, r.standard_normal(3))
        e *= np.linalg.norm(k) ** (-1.0 / 3.0) / np.linalg.norm(e)
        wave = torch.cos((int(k[0]) * ax[0])[:, None, None] + (int(k[1]) * ax[1])[None, :, None]
                         + (int(k[2]) * ax[2])[None, None, :] + r.uniform(0.0, 2 * math.pi))
        for c in range(3):
            B[c].add_(wave, alpha=float(e[c]))
    B *= 0.3 * b0 / float(B.square().sum(0).mean().sqrt())
    B[2] += b0
    E = torch.zeros_like(B)
    E[1], E[2] = 4.0e5 * B[2], -4.0e5 * B[1]  # u = (4e5, 0, 0) m/s
    return E, B


def _box_field(seed, nx, ny, nz):
    """A smooth non-periodic B on [0, 1e7 m]^3: (3, nx, ny, nz) float64."""
    r = np.random.RandomState(seed % (1 << 31))
    x, y, z = torch.meshgrid(*[torch.linspace(0.0, 1.0, m, dtype=torch.float64, device="cuda") for m in (nx, ny, nz)],
                             indexing="ij")
    a = r.uniform(0.5, 2.5, 9)
    p = r.uniform(0.0, 6.0, 3)
    return 5.0e-9 * torch.stack([0.3 * torch.sin(a[0] * x + a[1] * y + a[2] * z + p[0]),
                                 0.3 * torch.sin(a[3] * x + a[4] * y + a[5] * z + p[1]),
                                 1.0 + 0.3 * torch.sin(a[6] * x + a[7] * y + a[8] * z + p[2])])


def _inputs(case, seed):
    """The case's tables in float64 on the GPU: plain values and tensors, no package objects."""
    g, n, f = _rng(seed), case["n"], case["field"]
    s = {"t0": 0.0, "dt": None, "tend": None}
    if f == "uniform":  # 1e-8 T along z, Maxwellian protons, dt = T_gyro / 100
        s["E"], s["B"] = (1.0e-5, 0.0, 0.0), (0.0, 0.0, 1.0e-8)
        s["u0"] = torch.cat([_uniform(g, (n, 3), -1.0, 1.0), _normal(g, (n, 3), 1.0e5 / math.sqrt(2))], 1)
        s["dt"] = 2 * math.pi / (Q2M * 1.0e-8) / 100
        s["t1"] = case["steps"] * s["dt"]
    elif f == "dipole" and case["alg"] in ("rk4", "rk45"):
        half = n // 2
        first = torch.arange(n, device="cuda") < half  # electrons, then protons
        mass = torch.where(first, ME, MI).double()
        q = torch.where(first, -QI, QI).double()
        ek = torch.exp(_uniform(g, n, math.log(1.0e3), math.log(1.0e6)))
        v = LIGHT * torch.sqrt(1 - 1 / (1 + ek * QI / (mass * LIGHT**2)) ** 2)
        alpha = _uniform(g, n, math.radians(10.0), math.radians(90.0))
        shell, phi = _uniform(g, n, 2.0, 8.0), _uniform(g, n, 0.0, 2 * math.pi)
        x = RE * shell[:, None] * torch.stack([torch.cos(phi), torch.sin(phi), torch.zeros_like(phi)], 1)
        s["u0"] = torch.cat([x, (v * torch.cos(alpha))[:, None]], 1)
        s["q"], s["q2m"] = q, q / mass
        s["mu"] = mass * (v * torch.sin(alpha)) ** 2 / (2 * _dipole(x).norm(dim=1))
        bounce = 4 * shell * RE / v * (1.30 - 0.56 * torch.sin(alpha))
        s["tend"] = bounce
        if case["alg"] == "rk4":
            s["dt"] = bounce / case["steps"]
        s["t1"] = float(bounce.max())
    elif f == "dipole":
        # solve() packs what was saved: its ensemble stays below the energies that the dipole loses
        ek = torch.exp(_uniform(g, n, math.log(1.0e4), math.log(1.0e7 if case["kind"] == "push" else 1.0e6)))
        v = torch.sqrt(2 * ek * QI / MI)
        shell, phi = _uniform(g, n, 3.0, 7.0), _uniform(g, n, 0.0, 2 * math.pi)
        r = RE * shell[:, None] * torch.stack([torch.cos(phi), torch.sin(phi), torch.zeros_like(phi)], 1)
        # trapped: equatorial pitch angles of 45 to 135 degrees about the field (here along z)
        cos, psi = _uniform(g, n, -0.7, 0.7), _uniform(g, n, 0.0, 2 * math.pi)
        sin = torch.sqrt(1 - cos**2)
        s["u0"] = torch.cat([r, v[:, None] * torch.stack([sin * torch.cos(psi), sin * torch.sin(psi), cos], 1)], 1)
        gyro = 2 * math.pi / (Q2M * _dipole(r).norm(dim=1))
        if case["alg"] == "adaptive":
            s["tend"] = 0.05 * case["steps"] * gyro
        else:
            s["dt"] = 0.02 * gyro
            s["tend"] = case["steps"] * s["dt"]
        s["t1"] = float(s["tend"].max())
        s["shell"] = (RE, 15 * RE)
    elif f == "turbulence":
        dx = 1.0e5
        n3 = (case["nx"], case["ny"], case["nz"])
        E, B = _turbulence(seed, *n3, dx=dx)
        s["E"], s["B"] = E.float(), B.float()
        s["spacing"] = (dx, dx, dx)
        L = torch.tensor([m * dx for m in n3], dtype=torch.float64, device="cuda")
        s["u0"] = torch.cat([L * _uniform(g, (n, 3), 0.0, 1.0), _normal(g, (n, 3), 2.0e5 / math.sqrt(2))], 1)
        s["dt"] = 2 * math.pi / (Q2M * 5.0e-9) / 50
        s["t1"] = case["steps"] * s["dt"]
        if case["kind"] == "adjoint":
            s["grad"] = torch.cat([_normal(g, (n, 3), 1.0), _normal(g, (n, 3), 10.0)], 1)
    else:  # box
        n3 = (case["nx"], case["ny"], case["nz"])
        s["B"] = _box_field(seed, *n3)
        s["spacing"] = tuple(1.0e7 / (m - 1) for m in n3)
        s["walls"] = (2.0e5, 9.8e6)
        s["u0"] = torch.cat([_uniform(g, (n, 3), 1.0e6, 9.0e6), _normal(g, (n, 3), 3.0e5 / math.sqrt(2))], 1)
        s["dt"] = 2 * math.pi / (Q2M * 5.0e-9) / 50
        s["t1"] = case["steps"] * s["dt"]
    return s


def _host(v):
    if not torch.is_tensor(v):
        return v
    if v.dim() == 4:  # node values, in the memory order the package stores them
        return v.permute(3, 2, 1, 0).contiguous().cpu().numpy().T
    return v.cpu().numpy()


def prepare(case, seed):
    tp = _package()
    s = _inputs(case, seed)
    ens = tp.EnsembleB200(precision=case["precision"])
    if case["kind"] == "adjoint":
        from testparticle_b200.autograd import GridTensor

        grids = [GridTensor(s[k].requires_grad_(True), (0.0, 0.0, 0.0), s["spacing"], tp.WrapExtrap()) for k in "EB"]
        return {"kind": "adjoint", "u0": s["u0"].requires_grad_(True), "E": grids[0], "B": grids[1], "grad": s["grad"],
                "dt": s["dt"], "tspan": (0.0, s["t1"])}
    stop = None
    if case["field"] == "uniform":
        E, B = tp.UniformField(s["E"]), tp.UniformField(s["B"])
    elif case["field"] == "dipole":
        E, B = tp.ZeroField(), tp.DipoleField(MOMENT)
        if "shell" in s:
            stop = tp.TerminateShell(*s["shell"])
    else:
        axes = [np.arange(case[k]) * s["spacing"][c] for c, k in enumerate(("nx", "ny", "nz"))]
        bc = tp.WrapExtrap() if case["field"] == "turbulence" else tp.FillExtrap()
        B = tp.build_interpolator(_host(s["B"]), *axes, case["order"], bc)
        E = tp.build_interpolator(_host(s["E"]), *axes, case["order"], bc) if "E" in s else tp.ZeroField()
        if "walls" in s:
            stop = tp.TerminateBox((s["walls"][0],) * 3, (s["walls"][1],) * 3)
    u0 = np.ascontiguousarray(_host(s["u0"]).T)
    kw = {"trajectories": case["n"], "isoutside": stop, "dt": _host(s["dt"]), "tend": _host(s["tend"])}
    if case["alg"] in ("rk4", "rk45"):
        prob = tp.TraceGCProblem(u0, (0.0, s["t1"]), (_host(s["q"]), _host(s["q2m"]), _host(s["mu"]), E, B))
        kw.update(alg=case["alg"], save_everystep=False)
        if case["alg"] == "rk45":
            kw.update(reltol=1.0e-6, abstol=1.0e-9)
        return {"kind": "solve", "prob": prob, "args": (ens,), "kw": kw}
    alg = {"boris": tp.Boris(), "multistep": tp.MultistepBoris4(2), "adaptive": tp.AdaptiveBoris(0.1)}[case["alg"]]
    kw.update(savestepinterval=case["save_every"])
    if case["alg"] == "adaptive":
        kw.update(save_everystep=False, step_cap=case["steps"])
    prob = tp.TraceProblem(u0, (0.0, s["t1"]), tp.prepare(E, B))
    if case["kind"] == "solve":
        return {"kind": "solve", "prob": prob, "args": (alg, ens), "kw": kw}
    plan = tp.plan_boris(prob, alg, ens, **kw)
    ctx = tp.Context.get(0)
    ctx.field(plan.E), ctx.field(plan.B)
    slots = ctx.slots(plan.desc, case["n"], plan.dt_i, plan.tend_i)
    n, f64 = case["n"], torch.float64
    to = lambda a: None if a is None else torch.from_numpy(a).cuda()  # noqa: E731
    return {"kind": "push", "ctx": ctx, "plan": plan, "n": n, "slots": slots,
            "in": [to(plan.u0), to(plan.dt_i), to(plan.tend_i)],
            # a slot that a lost particle never reaches keeps its zero
            "t": torch.zeros((slots, n), dtype=f64, device="cuda"),
            "u": torch.zeros((slots, 6, n), dtype=f64, device="cuda"),
            "nsaved": torch.zeros(n, dtype=torch.int32, device="cuda"),
            "retcode": torch.zeros(n, dtype=torch.int8, device="cuda"),
            "nsteps": torch.zeros(n, dtype=torch.int64, device="cuda"),
            "status": torch.zeros(1, dtype=torch.int32, device="cuda")}


# ------------------------------------------------------------------ one pass
def run(state):
    if state["kind"] == "solve":
        sol = _package().solve(state["prob"], *state["args"], **state["kw"])
        return {"t": sol.t_all, "u": sol.u_all, "nsaved": sol.nsaved, "retcode": sol.retcodes, "nsteps": sol.nsteps}
    if state["kind"] == "push":
        s, plan = state, state["plan"]
        ptr = lambda x: None if x is None else x.data_ptr()  # noqa: E731
        s["ctx"].boris_run_device(plan.desc, plan.E, plan.B, *[ptr(x) for x in s["in"]], s["n"], s["slots"], ptr(s["t"]),
                                  ptr(s["u"]), ptr(s["nsaved"]), ptr(s["retcode"]), ptr(s["nsteps"]), ptr(s["status"]),
                                  stream=torch.cuda.current_stream().cuda_stream)
        return {k: s[k] for k in ("t", "u", "nsaved", "retcode", "nsteps", "status")}
    from testparticle_b200.autograd import boris_final_state

    x = boris_final_state(state["u0"], state["E"], state["B"], q2m=Q2M, dt=state["dt"], tspan=state["tspan"])
    gu, ge, gb = torch.autograd.grad(x, [state["u0"], state["E"].data, state["B"].data], state["grad"])
    return {"x": x.detach(), "grad_u0": gu, "grad_E": ge, "grad_B": gb}


# ------------------------------------------------------------------ work
def work(case):
    n, steps = case["n"], case["steps"]
    nodes = case["nx"] * case["ny"] * case["nz"]
    if case["kind"] == "adjoint":
        # starts, cotangents and final states, start gradients; two float32 grids and their gradients
        return {"bytes": n * 4 * 48 + nodes * 4 * 12, "flops": n * steps * (190 + 190 + 420)}
    if case["alg"] in ("rk4", "rk45"):
        evals = 4 * steps if case["alg"] == "rk4" else 7 * 40
        return {"bytes": n * (9 * 8 + 2 * 40 + 13), "flops": n * evals * 180}
    saves = 2 if case["alg"] == "adaptive" else 1 + -(-steps // case["save_every"])
    per = {"uniform": 50, "dipole": 150, "box": 120, "turbulence": 190}[case["field"]]
    if case["order"] == 3:
        per = 64 * 14 + 100
    if case["alg"] == "adaptive":
        per, steps = 250, steps * 3 // 4
    tables = nodes * (24 if case["field"] != "uniform" else 0)
    return {"bytes": n * (48 + (16 if case["field"] == "dipole" else 0) + saves * 56 + 13) + tables, "flops": n * steps * per}


# ------------------------------------------------------------------ the same in 64 bits
def _cross(a, b):
    return torch.linalg.cross(a, b, dim=1)


def _dot(a, b):
    return (a * b).sum(1, keepdim=True)


def _stencil(r, s, shape, periodic):
    """Cell indices, wrapped neighbours and fractions of the trilinear interpolant."""
    i0, i1, f = [], [], []
    for c in range(3):
        u = r[:, c] / s[c]
        fl = torch.floor(u.detach())
        if not periodic:
            fl = fl.clamp(0, shape[c] - 2)
        f.append(u - fl)
        i = fl.long()
        i0.append(i % shape[c] if periodic else i)
        i1.append((i + 1) % shape[c] if periodic else i + 1)
    return i0, i1, f


def _gather_field(tables, shape, r, s, periodic):
    """Trilinear values of node tables (nx * ny * nz, 3) at rows of r."""
    i0, i1, f = _stencil(r, s, shape, periodic)
    out = [0.0] * len(tables)
    for cx in (0, 1):
        for cy in (0, 1):
            for cz in (0, 1):
                w = ((f[0] if cx else 1 - f[0]) * (f[1] if cy else 1 - f[1]) * (f[2] if cz else 1 - f[2]))[:, None]
                at = (((i1 if cx else i0)[0] * shape[1] + (i1 if cy else i0)[1]) * shape[2] + (i1 if cz else i0)[2])
                out = [o + w * t.index_select(0, at) for o, t in zip(out, tables)]
    return out


def _cubic_field(tables, shape, r, s):
    """Periodic Catmull-Rom values of node tables (nx * ny * nz, 3) at rows of r."""
    i0, _, f = _stencil(r, s, shape, True)
    w = [[-t / 2 + t**2 - t**3 / 2, 1 - 2.5 * t**2 + 1.5 * t**3, t / 2 + 2 * t**2 - 1.5 * t**3, -t**2 / 2 + t**3 / 2] for t in f]
    out = [0.0] * len(tables)
    for a in range(4):
        for b in range(4):
            for c in range(4):
                at = (((i0[0] + a - 1) % shape[0]) * shape[1] + (i0[1] + b - 1) % shape[1]) * shape[2] + (i0[2] + c - 1) % shape[2]
                ww = (w[0][a] * w[1][b] * w[2][c])[:, None]
                out = [o + ww * t.index_select(0, at) for o, t in zip(out, tables)]
    return out


def _nodes(a):
    return a.permute(1, 2, 3, 0).reshape(-1, 3)


def _fields(case, s):
    """r -> (E, B) in float64; E None where it is zero."""
    if case["field"] == "uniform":
        E, B = (torch.tensor([s[k]], dtype=torch.float64, device="cuda") for k in "EB")
        return lambda r: (E.expand_as(r), B.expand_as(r))
    if case["field"] == "dipole":
        return lambda r: (None, _dipole(r))
    shape = s["B"].shape[1:]
    B = _nodes(s["B"].double())
    if "E" not in s:
        return lambda r: (None, _gather_field([B], shape, r, s["spacing"], False)[0])
    E = _nodes(s["E"].double())
    if case["order"] == 3:
        return lambda r: tuple(_cubic_field([E, B], shape, r, s["spacing"]))
    return lambda r: tuple(_gather_field([E, B], shape, r, s["spacing"], True))


def _kick(case, v, E, B, dt):
    """The velocity update of length dt (dt: number or a column)."""
    if case["alg"] == "multistep":  # gyrophase-corrected fourth order, two substeps
        n = 2
        t, e = Q2M * dt / (2 * n) * B, 0.0 if E is None else Q2M * dt / (2 * n) * E
        fn = 1 + _dot(t, t) / 3
        if E is not None:
            e = fn * e - _dot(e, t) / 3 * t
        t = fn * t
        tt = _dot(t, t)
        m = tt.sqrt()
        a = 2 * n * torch.atan(m)
        c2, c3 = torch.sin(a) / m, (1 - torch.cos(a)) / tt
        out = torch.cos(a) * v + c2 * _cross(v, t) + c3 * _dot(v, t) * t
        if E is not None:
            out = out + c2 * e + c3 * _cross(e, t) + (2 * n - c2) / tt * _dot(e, t) * t
        return out
    h = Q2M * dt / 2
    t = h * B
    vm = v if E is None else v + h * E
    vp = vm + _cross(vm + _cross(vm, t), 2 * t / (1 + _dot(t, t)))
    return vp if E is None else vp + h * E


def _outside(s, r):
    if "shell" in s:
        d = r.norm(dim=1)
        return (d < s["shell"][0]) | (d > s["shell"][1])
    if "walls" in s:
        return ((r < s["walls"][0]) | (r > s["walls"][1])).any(1)
    return None


def _fixed(case, s):
    """(t, u, nsaved) slot-major of a fixed-step solve that saves its start, every save_every steps and its end."""
    n, steps, every = case["n"], case["steps"], case["save_every"]
    f, r, v = _fields(case, s), s["u0"][:, :3].clone(), s["u0"][:, 3:].clone()
    dt = s["dt"][:, None] if torch.is_tensor(s["dt"]) else s["dt"]
    col = dt[:, 0] if torch.is_tensor(dt) else torch.full((n,), dt, dtype=torch.float64, device="cuda")
    slots = 1 + -(-steps // every)
    T = torch.zeros((slots, n), dtype=torch.float64, device="cuda")
    U = torch.zeros((slots, n, 6), dtype=torch.float64, device="cuda")
    U[0] = s["u0"]
    saved = torch.ones(n, dtype=torch.long, device="cuda")
    alive = torch.ones(n, dtype=torch.bool, device="cuda")
    ended = torch.full((n,), steps, dtype=torch.long, device="cuda")
    E, B = f(r)
    v = _kick(case, v, E, B, -0.5 * dt)
    for it in range(1, steps + 1):
        E, B = f(r)
        if it > 1 and (it - 1) % every == 0:
            keep = (r, _kick(case, v, E, B, 0.5 * dt))
        vn = _kick(case, v, E, B, dt)
        rn = r + vn * dt
        out = _outside(s, rn)
        if out is not None:
            now = alive & out
            ended = torch.where(now, it - 1, ended)
            alive = alive & ~out
        if it > 1 and (it - 1) % every == 0:
            k = (it - 1) // every
            U[k] = torch.where(alive[:, None], torch.cat(keep, 1), U[k])
            T[k] = torch.where(alive, (it - 1) * col, T[k])
            saved += alive
        r, v = torch.where(alive[:, None], rn, r), torch.where(alive[:, None], vn, v)
    E, B = f(r)
    last = torch.cat([r, _kick(case, v, E, B, 0.5 * dt)], 1)
    new = (ended > (saved - 1) * every) & (saved < slots)
    who = torch.nonzero(new)[:, 0]
    U[saved[who], who] = last[who]
    T[saved[who], who] = (ended * col)[who]
    return T, U, saved + new


def _adaptive(case, s):
    f, r, v = _fields(case, s), s["u0"][:, :3].clone(), s["u0"][:, 3:].clone()
    C = 0.1 * 2 * math.pi / Q2M
    n, tend = case["n"], s["tend"]
    t = torch.zeros(n, dtype=torch.float64, device="cuda")
    alive = t < tend
    E, B = f(r)
    dt = C / B.norm(dim=1)
    v = _kick(case, v, E, B, -0.5 * dt[:, None])
    for _ in range(case["steps"]):
        alive = alive & (t < tend)
        clip = alive & (t + dt > tend)
        short = tend - t
        vc = _kick(case, _kick(case, v, E, B, 0.5 * dt[:, None]), E, B, -0.5 * short[:, None])
        v, dt = torch.where(clip[:, None], vc, v), torch.where(clip, short, dt)
        vn = _kick(case, v, E, B, dt[:, None])
        rn = r + vn * dt[:, None]
        alive = alive & ~_outside(s, rn)
        En, Bn = f(rn)
        dn = C / Bn.norm(dim=1)
        vn = _kick(case, _kick(case, vn, En, Bn, 0.5 * dt[:, None]), En, Bn, -0.5 * dn[:, None])
        a = alive[:, None]
        t = torch.where(alive, t + dt, t)
        r, v, B, dt = torch.where(a, rn, r), torch.where(a, vn, v), torch.where(a, Bn, B), torch.where(alive, dn, dt)
    U = torch.stack([s["u0"], torch.cat([r, _kick(case, v, E, B, 0.5 * dt[:, None])], 1)])
    T = torch.stack([torch.zeros_like(t), t])
    gone = t == 0  # lost in its first step: the start is its only save
    U[1], T[1] = torch.where(gone[:, None], 0.0, U[1]), torch.where(gone, 0.0, T[1])
    return T, U, 2 - gone.long()


def _drift(y, q, q2m, mu):
    """Guiding-centre right-hand side in the dipole."""
    x, u = y[:, :3], y[:, 3:]
    m = torch.tensor(MOMENT, dtype=torch.float64, device="cuda")
    r2 = _dot(x, x)
    r5 = r2 * r2 * r2.sqrt()
    md = (x @ m)[:, None]
    B = COEF * (3 * md * x - m * r2) / r5
    eye = torch.eye(3, dtype=torch.float64, device="cuda")
    J = COEF * (3 * (x[:, :, None] * m + md[:, :, None] * eye + m[:, None] * x[:, None, :]) / r5[:, :, None]
                - 15 * (md / (r5 * r2))[:, :, None] * x[:, :, None] * x[:, None, :])
    size = B.norm(dim=1, keepdim=True)
    b = B / size
    g = (J * b[:, :, None]).sum(1)  # gradient of |B|; the curl of a dipole is zero
    star = B + u / q2m[:, None] * _cross(b, g) / size
    force = -(mu / q)[:, None] * g
    par = _dot(b, star)
    return torch.cat([(u * star + _cross(force, b)) / par, q2m[:, None] * _dot(star, force) / par], 1)


_A = [[1 / 5], [3 / 40, 9 / 40], [44 / 45, -56 / 15, 32 / 9], [19372 / 6561, -25360 / 2187, 64448 / 6561, -212 / 729],
      [9017 / 3168, -355 / 33, 46732 / 5247, 49 / 176, -5103 / 18656], [35 / 384, 0.0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84]]
_ERR = [71 / 57600, 0.0, -71 / 16695, 71 / 1920, -17253 / 339200, 22 / 525, -1 / 40]


def _centres(case, s):
    y, par = s["u0"].clone(), (s["q"], s["q2m"], s["mu"])
    tend = s["tend"]
    if case["alg"] == "rk4":
        h = s["dt"][:, None]
        for _ in range(case["steps"]):
            k1 = _drift(y, *par)
            k2 = _drift(y + h / 2 * k1, *par)
            k3 = _drift(y + h / 2 * k2, *par)
            y = y + h / 6 * (k1 + 2 * k2 + 2 * k3 + _drift(y + h * k3, *par))
    else:
        t = torch.zeros_like(tend)
        dt = math.pi / (s["q2m"].abs() * _dipole(y[:, :3]).norm(dim=1))
        for _ in range(10000):
            on = t < tend
            if not bool(on.any()):
                break
            last = t + dt > tend
            dt = torch.where(last, tend - t, dt)
            h, k = dt[:, None], [_drift(y, *par)]
            for row in _A:
                yn = y + h * sum(a * b for a, b in zip(row, k))
                k.append(_drift(yn, *par))
            err = h * sum(a * b for a, b in zip(_ERR, k))
            ratio = (err / (1.0e-9 + 1.0e-6 * torch.maximum(y.abs(), yn.abs()))).norm(dim=1) / 2
            ok = on & ~(ratio > 1)
            y = torch.where(ok[:, None], yn, y)
            t = torch.where(ok, torch.where(last, tend, t + dt), t)
            dt = torch.where(on, dt * (0.9 * ratio**-0.2).clamp(0.2, 5.0), dt)
    return torch.stack([torch.zeros_like(tend), tend]), torch.stack([s["u0"], y]), torch.full_like(tend, 2).long()


def _gradient(case, s):
    grids = [s[k].double().requires_grad_(True) for k in "EB"]
    u0 = s["u0"].clone().requires_grad_(True)
    dt = s["dt"]

    def kick(r, v, tables, h):
        return _kick(case, v, *_gather_field(tables, s["B"].shape[1:], r, s["spacing"], True), h)

    def steps(r, v, E, B, count):
        tables = [_nodes(E), _nodes(B)]
        for _ in range(count):
            v = kick(r, v, tables, dt)
            r = r + v * dt
        return r, v

    def half(r, v, E, B, h):
        return kick(r, v, [_nodes(E), _nodes(B)], h)

    r, v = u0[:, :3], half(u0[:, :3], u0[:, 3:], *grids, -0.5 * dt)
    for k in range(0, case["steps"], 8):
        r, v = checkpoint(steps, r, v, *grids, min(8, case["steps"] - k), use_reentrant=False)
    x = torch.cat([r, half(r, v, *grids, 0.5 * dt)], 1)
    gu, ge, gb = torch.autograd.grad(x, [u0, *grids], s["grad"])
    return {"x": x.detach(), "grad_u0": gu, "grad_E": ge.float(), "grad_B": gb.float()}


def exact(case, seed):
    s = _inputs(case, seed)
    if case["kind"] == "adjoint":
        return _gradient(case, s)
    if case["alg"] in ("rk4", "rk45"):
        T, U, saved = _centres(case, s)
    else:
        T, U, saved = (_adaptive if case["alg"] == "adaptive" else _fixed)(case, s)
    if case["kind"] == "push":
        return {"t": T, "u": U.transpose(1, 2).contiguous()}
    there = (torch.arange(T.shape[0], device="cuda")[:, None] < saved).T
    return {"t": T.T[there].cpu().numpy(), "u": U.transpose(0, 1)[there].cpu().numpy()}
