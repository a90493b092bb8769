"""Measured cases: the work a user of the framework has it do, through its public entry points.

Four kinds of pass ("op"):
  step      one time step of a model: `Nyles(param)`, then `model.forward(t, dt)`
            (with `auto_dt`, `compute_dt()` before it, as `Nyles.run` does)
  rhs       one right-hand side through the C ABI (`nyles_rhs_f64/_f32`), as a host code that
            keeps its own time loop calls it; any extents, odd ones among them
  solve     one pressure solve of the stand-alone multigrid (`multigrid.MG`) from x = 0
  ensemble  one batch of a serving bucket: admit the runs, project them, advance them k steps

`exact` restates each pass in plain 64-bit torch: the WENO right-hand side with its
array-end closures, the time-scheme updates, the multigrid V-cycles with their stop rule,
projection and diagnostics.
"""
import ctypes
import math

import numpy as np
import torch

from nyles_gb300 import _native as nat
from nyles_gb300 import parameters, serving
from nyles_gb300.multigrid import MG
from nyles_gb300.nyles import Nyles

TWO_PI = 6.283185307179586
DEFAULTS = {"op": "step", "precision": "fp64", "geometry": "closed", "nx": 64, "ny": 64, "nz": 64, "flow": "lock",
            "scheme": "RK3_SSP", "model": "LES", "tol": 1e-6, "maxite": 20, "dt": 1e-3, "auto_dt": False,
            "tracers": 0, "viscous": False, "runs": 1, "steps": 1}


def listed():
    return [
        # the lock-exchange configuration's grid: a small closed tank, bound by launches and latency
        dict(name="step lock 64x32x32 fp64", op="step", precision="fp64", geometry="closed", nx=64, ny=32, nz=32,
             flow="lock", scheme="RK3_SSP", dt=2e-3),
        # one run of the serving ensemble's 3*2^n size by itself, mixed precision
        dict(name="step lock 48 mixed", op="step", precision="mixed", geometry="closed", nx=48, ny=48, nz=48,
             flow="lock", scheme="RK3_SSP", dt=2e-3),
        # the parameter defaults (LFAM3, adaptive dt, FP64) with a tracer and viscosity in a
        # periodic channel: an ordinary experiment script
        dict(name="step shear 128x64x64 fp64 lfam3", op="step", precision="fp64", geometry="perio_xy", nx=128, ny=64,
             nz=64, flow="shear", scheme="LFAM3", auto_dt=True, tracers=1, viscous=True),
        # Taylor-Green 128^3, triply periodic, relative residual 1e-10
        dict(name="step tgv 128 fp64 tight", op="step", precision="fp64", geometry="perio_xyz", nx=128, ny=128,
             nz=128, flow="tgv", scheme="RK3_SSP", dt=5e-3, tol=1e-20, maxite=40),
        # the headline benchmark: Rayleigh-Taylor 256^3, relative residual 1e-10, both precisions
        dict(name="step rt 256 fp64 tight", op="step", precision="fp64", geometry="perio_xy", nx=256, ny=256, nz=256,
             flow="rt", scheme="RK3_SSP", dt=1e-3, tol=1e-20, maxite=40),
        dict(name="step rt 256 mixed tight", op="step", precision="mixed", geometry="perio_xy", nx=256, ny=256,
             nz=256, flow="rt", scheme="RK3_SSP", dt=1e-3, tol=1e-20, maxite=40),
        # the stratified shear configuration's grid with a tracer and adaptive dt, mixed: the largest
        dict(name="step shear 512x256x256 mixed", op="step", precision="mixed", geometry="perio_xy", nx=512, ny=256,
             nz=256, flow="shear", scheme="RK3_SSP", auto_dt=True, tracers=1),
        # right-hand sides on extents that are no multiple of anything, with every term
        dict(name="rhs 109x75x53 closed fp64", op="rhs", precision="fp64", geometry="closed", nx=109, ny=75, nz=53,
             tracers=1, viscous=True),
        dict(name="rhs 301x203x97 perio_xy mixed", op="rhs", precision="mixed", geometry="perio_xy", nx=301, ny=203,
             nz=97),
        # the stand-alone pressure solver at its default tolerance
        dict(name="solve 128 closed fp64", op="solve", precision="fp64", geometry="closed", nx=128, ny=128, nz=128),
        dict(name="solve 256x256x128 perio_xy mixed", op="solve", precision="mixed", geometry="perio_xy", nx=256,
             ny=256, nz=128),
        # a full serving bucket of 64^3 runs: eight lock exchanges in one batched launch
        dict(name="ensemble 8x64 lock mixed", op="ensemble", precision="mixed", nx=64, ny=64, nz=64, flow="lock",
             runs=8, steps=10),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _even_grid(rng, lo, hi, cells):
    """extents [3*]2^n (what the parameters accept) with z even on every multigrid level
    above the coarsest, at most `cells` cells"""
    sizes = [n for n in (16, 24, 32, 48, 64, 96, 128, 192, 256, 384, 512) if lo <= n <= hi]
    while True:
        nx, ny, nz = (rng.choice(sizes) for _ in range(3))
        x, y, z, ok = nx, ny, nz, max(nx, ny, nz) <= 4 * min(nx, ny, nz) and nx * ny * nz <= cells
        while x > 2 and y > 2 and x % 2 == 0 and y % 2 == 0:
            ok = ok and z % 2 == 0
            x, y, z = x // 2, y // 2, z // 2
        if ok and z >= 1:
            return nx, ny, nz


def draw(rng):
    op = rng.choice(["step", "step", "step", "rhs", "rhs", "solve", "solve", "ensemble"])
    prec = rng.choice(["fp64", "mixed"])
    if op == "rhs":
        cells = 3e6 if prec == "fp64" else 2e7
        while True:
            nx, ny, nz = (_log_int(rng, 12, 400) for _ in range(3))
            if nx * ny * nz <= cells:
                break
        return dict(op=op, precision=prec, geometry=rng.choice(["closed", "perio_xy", "perio_xyz", "perio_x"]),
                    nx=nx, ny=ny, nz=nz, tracers=rng.choice([0, 0, 1, 2]), viscous=rng.random() < 0.3,
                    model=rng.choice(["LES", "LES", "LES", "linear"]))
    if op == "solve":
        nx, ny, nz = _even_grid(rng, 16, 512, 3e6 if prec == "fp64" else 2e7)
        return dict(op=op, precision=prec, geometry=rng.choice(["closed", "perio_xy", "perio_xyz"]), nx=nx, ny=ny,
                    nz=nz)
    if op == "ensemble":
        n = rng.choice([32, 48, 64, 96])
        return dict(op=op, precision="mixed", nx=n, ny=n, nz=n, flow=rng.choice(["lock", "tgv"]),
                    runs=rng.randint(2, serving.auto_capacity(n, 8)), steps=rng.randint(4, 10))
    nx, ny, nz = _even_grid(rng, 16, 512, 3e6 if prec == "fp64" else 2e7)
    flow = rng.choice(["lock", "tgv", "rt", "shear"])
    tight = rng.random() < 0.3
    case = dict(op=op, precision=prec, geometry={"lock": "closed", "tgv": "perio_xyz"}.get(flow, "perio_xy"),
                nx=nx, ny=ny, nz=nz, flow=flow, scheme=rng.choice(["RK3_SSP", "RK3_SSP", "LFAM3"]),
                tol=1e-20 if tight else 1e-6, maxite=40 if tight else 20, tracers=rng.choice([0, 0, 1]),
                viscous=rng.random() < 0.2)
    if flow == "shear":
        case["auto_dt"] = True
    else:
        case["dt"] = 1e-3
    return case


# ---------------------------------------------------------------- inputs
def _full(case):
    c = dict(DEFAULTS, **case)
    if c["op"] == "ensemble":
        c["geometry"] = serving.CASES[c["flow"]]["geometry"]
    return c


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _params(c):
    # cubic cells: with them the projection removes the divergence and the flow is stable
    h = (TWO_PI if c["flow"] == "tgv" else 1.0) / c["nz"]
    parameters.InextensibleDict.unfreeze()
    p = parameters.UserParameters()
    p.model["modelname"] = c["model"]
    p.model["geometry"] = c["geometry"]
    p.model["Lx"], p.model["Ly"], p.model["Lz"] = c["nx"] * h, c["ny"] * h, c["nz"] * h
    p.model["n_tracers"] = c["tracers"]
    p.time["timestepping"] = c["scheme"]
    p.time["auto_dt"] = c["auto_dt"]
    p.time["dt"] = c["dt"]
    p.time["cfl"] = 0.5
    p.time["dt_max"] = 1e-2
    p.physics["diff_coef"] = {"u": 1e-4} if c["viscous"] else {}
    p.discretization["global_nx"], p.discretization["global_ny"], p.discretization["global_nz"] = (c["nx"], c["ny"],
                                                                                                   c["nz"])
    p.gpu["precision"] = c["precision"]
    p.gpu["mg_tol"] = c["tol"]
    p.gpu["mg_maxite"] = c["maxite"]
    p.gpu["history"] = False
    return p


def _initial(c, grid, seed):
    """seeded initial state of a flow on the (z, y, x) arrays (float64, on the GPU)"""
    gen = _generator(seed)
    ax = [torch.from_numpy(np.asarray(a)).cuda() for a in (grid.z_b_1D, grid.y_b_1D, grid.x_b_1D)]
    z, y, x = ax[0][:, None, None], ax[1][None, :, None], ax[2][None, None, :]
    shape = (len(ax[0]), len(ax[1]), len(ax[2]))
    h = grid.dx
    noise = lambda: torch.randn(shape, generator=gen, device="cuda", dtype=torch.float64)  # noqa: E731
    zero = torch.zeros(shape, device="cuda", dtype=torch.float64)
    f = {"b": zero, "u_i": zero, "u_j": zero, "u_k": zero}
    zz = (z / grid.Lz).expand(shape)
    if c["flow"] == "lock":
        # a dam front that is not parallel to the walls: all three velocity components count
        ph = torch.rand(1, generator=gen, device="cuda", dtype=torch.float64) * TWO_PI
        front = grid.Lx * (0.5 + 0.1 * torch.cos(TWO_PI * y / grid.Ly + ph))
        f["b"] = torch.where(x < front, -0.5, 0.5) + 1e-3 * noise()
    elif c["flow"] == "rt":      # an interface perturbed by random Fourier modes
        eta = torch.zeros(shape[1:], device="cuda", dtype=torch.float64)
        amp = torch.randn((4, 4, 2), generator=gen, device="cuda", dtype=torch.float64).cpu()
        for kx in range(4):
            for ky in range(4):
                ph = TWO_PI * (kx * x[0] / grid.Lx + ky * y[0] / grid.Ly)
                eta = eta + amp[kx, ky, 0] * torch.cos(ph) + amp[kx, ky, 1] * torch.sin(ph)
        f["b"] = torch.where(zz > 0.5 + 0.01 * eta / 4, 0.5, -0.5)
    elif c["flow"] == "tgv":
        k = [TWO_PI / s for s in (grid.Lx, grid.Ly, grid.Lz)]
        s = 0.5 * h
        f["u_i"] = (torch.sin(k[0] * (x + s)) * torch.cos(k[1] * y) * torch.cos(k[2] * z) + 1e-4 * noise()) * h
        f["u_j"] = (-torch.cos(k[0] * x) * torch.sin(k[1] * (y + s)) * torch.cos(k[2] * z) + 1e-4 * noise()) * h
        f["u_k"] = 1e-4 * noise() * h
        f["b"] = 0.3 * torch.sin(k[0] * x) * torch.cos(k[2] * z) + zero
    else:                        # stratified shear
        f["u_i"] = (0.1 * torch.tanh((zz - 0.5) / 0.05) + 1e-3 * noise()) * h
        f["u_j"] = 1e-3 * noise() * h
        f["u_k"] = 1e-3 * noise() * h
        f["b"] = zz.clone()
    for t in range(c["tracers"]):
        f["t%d" % t] = torch.tanh((zz - 0.4 - 0.1 * t) / 0.1) + 1e-3 * noise()
    for name, axis, key in (("u_i", 2, "x"), ("u_j", 1, "y"), ("u_k", 0, "z")):
        if key not in c["geometry"]:          # walls at rest
            v = f[name].clone()
            v.select(axis, shape[axis] - 1).zero_()
            f[name] = v
    return f


def _line_extents(c):
    """array extents (z, y, x): a halo of 3 on both sides of periodic directions"""
    per = [int(a in c["geometry"].replace("perio", "")) for a in "zyx"] if c["geometry"] != "closed" else [0, 0, 0]
    n = [c["nz"], c["ny"], c["nx"]]
    return per, n, [m + 6 * p for m, p in zip(n, per)]


def _smooth(shape, gen, amp):
    """a smooth random field with a flat patch and a little noise"""
    ax = [torch.linspace(0, 1, m, device="cuda", dtype=torch.float64) for m in shape]
    v = torch.zeros(shape, device="cuda", dtype=torch.float64)
    for k in range(1, 4):
        ph = torch.rand(3, generator=gen, device="cuda", dtype=torch.float64) * TWO_PI
        a = torch.randn(1, generator=gen, device="cuda", dtype=torch.float64) / k
        v += a * (torch.cos(TWO_PI * k * ax[0] + ph[0])[:, None, None] * torch.cos(TWO_PI * k * ax[1] + ph[1])[:, None]
                  * torch.cos(TWO_PI * k * ax[2] + ph[2]))
    v += 1e-2 * torch.randn(shape, generator=gen, device="cuda", dtype=torch.float64)
    v[: shape[0] // 4, : shape[1] // 4] = 0.25
    return amp * v


FIELDS = ["b", "p", "ke", "div", "u_i", "u_j", "u_k", "U_i", "U_j", "U_k", "vor_i", "vor_j", "vor_k", "work"]


def _rhs_desc(c):
    d = nat.NylesDesc()
    per, n, _ = _line_extents(c)
    h = 1.0 / c["nz"]
    d.nx, d.ny, d.nz, d.nh = c["nx"], c["ny"], c["nz"], 3
    d.periodic_z, d.periodic_y, d.periodic_x = per
    d.n_tracers = c["tracers"]
    d.model = nat.MODEL[c["model"]]
    d.dx = d.dy = d.dz = h
    d.idx2 = d.idy2 = d.idz2 = 1 / h ** 2
    d.dx2 = h ** 2
    if c["viscous"]:
        d.add_viscosity, d.viscosity = 1, 1e-4
    return d


def _rhs_fields(c, seed):
    gen = _generator(seed)
    _, _, shape = _line_extents(c)
    h = 1.0 / c["nz"]
    amp = {"b": 0.5, "ke": 0.5, "u": h, "U": 1 / h, "vor": h}
    names = FIELDS + ["t%d" % t for t in range(c["tracers"])]
    return {k: _smooth(tuple(shape), gen, amp.get(k, amp.get(k.split("_")[0], 1.0))) for k in names}


def _solve_rhs(c, seed):
    """divergence of a seeded smooth-plus-noise field, mean removed"""
    gen = _generator(seed)
    v = _smooth((c["nz"], c["ny"], c["nx"]), gen, 1.0)
    return v - v.mean()


def prepare(case, seed):
    c = _full(case)
    if c["op"] == "rhs":
        dt = torch.float64 if c["precision"] == "fp64" else torch.float32
        vals = _rhs_fields(c, seed)
        fields = {k: v.to(dt).contiguous() for k, v in vals.items()}
        out = [torch.zeros_like(fields["b"]) for _ in range(4 + c["tracers"])]
        desc = _rhs_desc(c)
        return dict(c=c, desc=desc, fields=fields, out=out,
                    fp=nat.ptr_array([t.data_ptr() for t in fields.values()]),
                    op=nat.ptr_array([t.data_ptr() for t in out]))
    if c["op"] == "solve":
        mg = MG(c["nx"], c["ny"], c["nz"], topology=c["geometry"], precision=c["precision"])
        mg.set_params(c["tol"], c["maxite"], 0.9)
        mg.set(1, 2, _solve_rhs(c, seed))
        return dict(c=c, mg=mg, x0=mg.level_tensor(1, 1))
    if c["op"] == "ensemble":
        reqs = [serving.Request(r, c["flow"], c["nx"], seed * 64 + r, c["steps"], 0.0) for r in range(c["runs"])]
        bucket = serving.Bucket((c["flow"], c["nx"], c["steps"]), "mixed", c["tol"],
                                torch.device("cuda", torch.cuda.current_device()), c["runs"])
        grid = serving.case_grid(c["flow"], c["nx"])
        staged = [{k: v.float().cpu().pin_memory() for k, v in _initial(c, grid, r.seed).items()} for r in reqs]
        return dict(c=c, bucket=bucket, reqs=reqs, staged=staged)
    nyl = Nyles(_params(c))
    for k, v in _initial(c, nyl.grid, seed).items():
        nyl.model.state.get(k).view("i").copy_(v)
    nyl.model.diagnose_var(nyl.model.state)
    return dict(c=c, nyl=nyl, t=0.0)


def run(state):
    c = state["c"]
    if c["op"] == "rhs":
        fn = nat.lib().nyles_rhs_f64 if c["precision"] == "fp64" else nat.lib().nyles_rhs_f32
        nat.check(fn(ctypes.byref(state["desc"]), state["fp"], state["op"], 1, nat.stream_ptr()))
        return state["out"]
    if c["op"] == "solve":
        state["x0"].zero_()
        x, stats = state["mg"].solve()
        return [x, stats["nite"]]
    if c["op"] == "ensemble":
        b = state["bucket"]
        for slot, req, staged in zip(b.slots, state["reqs"], state["staged"]):
            b.admit(slot, req, 0.0, staged=staged)
        b.launch()
        b.poll()
        for slot in b.slots:
            b.release(slot)
        return [slot.nyl.model.state.get(k).view("i") for slot in b.slots for k in ("b", "u_i", "u_j", "u_k", "p")]
    nyl = state["nyl"]
    dt = nyl.compute_dt()
    nyl.model.forward(state["t"], dt)
    state["t"] += dt
    return {k: nyl.model.state.get(k).view("i") for k in nyl.model.state.get_prognostic_scalars() + ["p"]}


STAGES = {"RK3_SSP": 3, "LFAM3": 2, "EF": 1}


def work(case):
    """each input read once and each output written once; arithmetic of the WENO
    reconstructions (9 per cell and right-hand side, 3 per tracer, about 75 operations each)
    and of the V-cycles (about 60 operations per cell and cycle)"""
    c = _full(case)
    w = 8 if c["precision"] == "fp64" else 4
    cells = c["nx"] * c["ny"] * c["nz"]
    ntr = c["tracers"]
    recon = (9 if c["model"] != "linear" else 3) + 3 * ntr
    if c["op"] == "rhs":
        _, _, shape = _line_extents(c)
        cells = shape[0] * shape[1] * shape[2]
        words = 8 + ntr + (3 if c["viscous"] else 0) + 4 + ntr
        return {"bytes": words * w * cells, "flops": (75 * recon + 50) * cells}
    cycles = 18 if c["tol"] < 1e-12 else 6
    if c["op"] == "solve":
        return {"bytes": 2 * 8 * cells, "flops": 60 * cycles * cells}
    n = c["runs"] * c["steps"]
    stage = 75 * recon + 50 + 60 * cycles + 60
    return {"bytes": n * (2 * (4 + ntr) + 1) * w * cells, "flops": n * STAGES[c["scheme"]] * stage * cells}


# ---------------------------------------------------------------- 64-bit restatement
# REAL(4) literals of the scheme, widened
_F = {k: float(np.float32(v)) for k, v in
      dict(c13=np.float32(1) / np.float32(3), c76=np.float32(7) / np.float32(6), c116=np.float32(11) / np.float32(6),
           c16=np.float32(1) / np.float32(6), c56=np.float32(5) / np.float32(6), k1=np.float32(13) / np.float32(12),
           eps5=1e-16, eps3=1e-14).items()}


def _weno3(qm, q0, qp):
    b1, b2 = (q0 - qm) ** 2, (qp - q0) ** 2
    tau = (b2 - b1).abs()
    w1, w2 = 1 + tau / (b1 + _F["eps3"]), 2 * (1 + tau / (b2 + _F["eps3"]))
    return (w1 * ((3 * q0 - qm) * 0.5) + w2 * ((q0 + qp) * 0.5)) / (w1 + w2)


def _weno5(a, b, c, d, e):
    q1 = _F["c13"] * a - _F["c76"] * b + _F["c116"] * c
    q2 = -_F["c16"] * b + _F["c56"] * c + _F["c13"] * d
    q3 = _F["c13"] * c + _F["c56"] * d - _F["c16"] * e
    b1 = _F["k1"] * (a - 2 * b + c) ** 2 + 0.25 * (a - 4 * b + 3 * c) ** 2
    b2 = _F["k1"] * (b - 2 * c + d) ** 2 + 0.25 * (b - d) ** 2
    b3 = _F["k1"] * (c - 2 * d + e) ** 2 + 0.25 * (3 * c - 4 * d + e) ** 2
    tau = (b1 - b3).abs().float().double()
    w1 = 1 + tau / (b1 + _F["eps5"])
    w2 = 6 * (1 + tau / (b2 + _F["eps5"]))
    w3 = 3 * (1 + tau / (b3 + _F["eps5"]))
    return (w1 * q1 + w2 * q2 + w3 * q3) / (w1 + w2 + w3)


def _flux(u, q):
    """upwind flux along the last axis: interior WENO5, closures at the ends"""
    n = u.shape[-1]
    f = torch.zeros_like(u)
    S = lambda k, lo, hi: q[..., lo + k:hi + k + 1]  # noqa: E731
    lo, hi = 2, n - 4
    if hi >= lo:
        v = [S(k, lo, hi) for k in (-2, -1, 0, 1, 2, 3)]
        pos = u[..., lo:hi + 1] > 0
        sel = [torch.where(pos, v[k], v[5 - k]) for k in range(5)]
        f[..., lo:hi + 1] = u[..., lo:hi + 1] * _weno5(*sel)

    def put(i, plus, minus):
        f[..., i] = torch.where(u[..., i] > 0, u[..., i] * plus, u[..., i] * minus)

    g = [q[..., k] for k in range(n)] if n <= 8 else None
    at = (lambda k: g[k]) if g else (lambda k: q[..., k])
    put(0, at(0), _weno3(at(2), at(1), at(0)))
    put(1, _weno3(at(0), at(1), at(2)), _weno5(at(4), at(3), at(2), at(1), at(0)))
    put(n - 3, _weno5(*[at(n - 5 + k) for k in range(5)]), _weno3(at(n - 1), at(n - 2), at(n - 3)))
    put(n - 2, _weno3(at(n - 3), at(n - 2), at(n - 1)), at(n - 1))
    return f


def _shift(a, axis, k):
    """a at index + k along axis, 0 beyond the array"""
    r = torch.zeros_like(a)
    n = a.shape[axis]
    if k > 0:
        r.narrow(axis, 0, n - k).copy_(a.narrow(axis, k, n - k))
    else:
        r.narrow(axis, -k, n + k).copy_(a.narrow(axis, 0, n + k))
    return r


def _not_last(a, axis):
    r = a.clone()
    r.select(axis, a.shape[axis] - 1).zero_()
    return r


def _line_flux(u, q, axis):
    return _flux(u.transpose(axis, 2).contiguous(), q.transpose(axis, 2).contiguous()).transpose(axis, 2).contiguous()


def _lap(u, axis):
    return _not_last(_shift(u, axis, 1) - u, axis) - _shift(_not_last(_shift(u, axis, 1) - u, axis), axis, -1)


AXES = {"i": 2, "j": 1, "k": 0}


def _ref_rhs(s, c, h, last):
    """tendencies of b, u and the tracers on the whole arrays; s: fields by name"""
    out = {}
    for q in ["b"] + ["t%d" % t for t in range(c["tracers"])]:
        acc = 0
        for d in "ijk":
            F = _line_flux(s["U_" + d], s[q], AXES[d])
            acc = acc + _shift(F, AXES[d], -1) - F
        out[q] = acc
    du = {d: torch.zeros_like(s["b"]) for d in "ijk"}
    if c["model"] != "linear":
        # u_t -= or += U^f w_v: the velocity averaged along t, then along the flux direction f
        for t, f, v, sg in (("j", "i", "k", -1), ("i", "j", "k", 1), ("k", "j", "i", -1), ("j", "k", "i", 1),
                            ("i", "k", "j", -1), ("k", "i", "j", 1)):
            U = s["U_" + f]
            m = 0.5 * (U + _shift(U, AXES[t], 1))
            u1 = 0.5 * (m + _shift(m, AXES[f], -1))
            fl = _line_flux(u1, _shift(s["vor_" + v], AXES[f], -1), AXES[f])
            du[t] = du[t] + sg * _not_last(fl, AXES[t])
    for d in "ijk":
        du[d] = du[d] - _not_last(_shift(s["ke"], AXES[d], 1) - s["ke"], AXES[d])
    du["k"] = du["k"] + _not_last(0.5 * h * (_shift(s["b"], 0, 1) + s["b"]), 0)
    if last and c["viscous"]:
        for e in "ijk":
            for d in "ijk":
                du[d] = du[d] + 1e-4 / h ** 2 * _lap(s["u_" + d], AXES[e])
    out.update({"u_" + d: du[d] for d in "ijk"})
    return out


def _nb(a, axis, k, per):
    """neighbour at index + k along axis: the periodic image, or 0 across a wall"""
    return torch.roll(a, -k, axis) if per else _shift(a, axis, k)


def _wet(shape, axis, k, per):
    r = torch.ones(shape[axis], device="cuda", dtype=torch.float64)
    if not per:
        r[-1 if k > 0 else 0] = 0
    return r.reshape([-1 if a == axis else 1 for a in range(3)])


class _RefMG:
    def __init__(self, n, per, omega=0.9):
        self.per, self.omega, self.x = per, omega, None
        z, y, x = n
        self.levels = [(z, y, x)]
        while x != 2 and y != 2 and x % 2 == 0 and y % 2 == 0 and x >= 4 and y >= 4:
            z, y, x = z // 2, y // 2, x // 2
            self.levels.append((z, y, x))
        self.diag = [sum(_wet(s, a, k, per[a]) for a in range(3) for k in (-1, 1)) for s in self.levels]
        self.diag = [d.expand(s) for d, s in zip(self.diag, self.levels)]

    def nsum(self, x):
        return sum(_nb(x, a, k, self.per[a]) for a in (2, 1, 0) for k in (-1, 1))

    def resid(self, l, x, b):
        return b + self.diag[l] * x - self.nsum(x)

    def smooth(self, l, x, b):
        for _ in range(2):
            x = x - self.omega / self.diag[l] * self.resid(l, x, b)
        return x

    def vcycle(self, l, x, b):
        x = self.smooth(l, x, b)
        if l + 1 == len(self.levels):
            return x
        r = self.resid(l, x, b)
        z, y, w = self.levels[l + 1]
        rc = 0.5 * r.reshape(z, 2, y, 2, w, 2).sum((1, 3, 5))
        e = self.vcycle(l + 1, torch.zeros_like(rc), rc)
        for a in range(3):      # one direction after the other: (3 own + neighbour) / (3 + wet)
            lo = (3 * e + _nb(e, a, -1, self.per[a])) / (3 + _wet(e.shape, a, -1, self.per[a]))
            hi = (3 * e + _nb(e, a, 1, self.per[a])) / (3 + _wet(e.shape, a, 1, self.per[a]))
            e = torch.stack((lo, hi), a + 1).flatten(a, a + 1)
        return self.smooth(l, x + e, b)

    def solve(self, b, tol, maxite):
        x = torch.zeros_like(b) if self.x is None else self.x
        normb = float((b * b).sum())
        nite = 0
        while normb > 0:
            r = self.resid(0, x, b)
            if float((r * r).sum()) / normb < tol or nite >= maxite:
                break
            x = self.vcycle(0, x, b)
            nite += 1
        self.x = x
        return x, nite


class _RefModel:
    def __init__(self, c, h, fields):
        self.c, self.h, self.s = c, h, dict(fields)
        self.per, self.n, self.N = _line_extents(c)
        self.mg = _RefMG(self.n, self.per)
        self.box = tuple(slice(3, 3 + m) if p else slice(0, m) for p, m in zip(self.per, self.n))
        self.prog = ["b", "u_i", "u_j", "u_k"] + ["t%d" % t for t in range(c["tracers"])]

    def fill(self, inner):
        for a in range(3):
            if self.per[a]:
                n = inner.shape[a]
                inner = torch.cat((inner.narrow(a, n - 3, 3), inner, inner.narrow(a, 0, 3)), a)
        return inner

    def refill(self, name):
        self.s[name] = self.fill(self.s[name][self.box])

    def diagnose(self):
        s, h = self.s, self.h
        i2 = 1 / h ** 2
        for k in ("b", "u_i", "u_j", "u_k"):
            self.refill(k)
        div = sum(i2 * (s["u_" + d] - _shift(s["u_" + d], AXES[d], -1)) for d in "ijk")
        x, _ = self.mg.solve(div[self.box].contiguous(), self.c["tol"], self.c["maxite"])
        s["p"] = self.fill(x * h ** 2)
        for d in "ijk":
            s["u_" + d] = s["u_" + d] - _not_last(_shift(s["p"], AXES[d], 1) - s["p"], AXES[d])
            self.refill("u_" + d)
        u = {d: s["u_" + d] for d in "ijk"}
        for d in "ijk":
            s["U_" + d] = i2 * u[d]
        for v, p, q in (("i", "j", "k"), ("j", "k", "i"), ("k", "i", "j")):
            w = (_shift(u[q], AXES[p], 1) - u[q]) - (_shift(u[p], AXES[q], 1) - u[p])
            s["vor_" + v] = self.fill(_not_last(_not_last(w, AXES[p]), AXES[q])[self.box])
        ke = 0
        for d in "ijk":
            m = _shift(u[d], AXES[d], -1)
            e = 0.25 * i2 * (u[d] ** 2 + m ** 2)
            e.select(AXES[d], 0).zero_()
            ke = ke + e
        s["ke"] = self.fill(ke[self.box])

    def add(self, terms):
        for k in self.prog:
            self.s[k] = self.s[k] + sum(w * d[k] for w, d in terms)

    def forward(self, dt):
        c, h = self.c, self.h
        r0 = _ref_rhs(self.s, c, h, c["scheme"] == "EF")
        self.add([(dt, r0)])
        self.diagnose()          # LFAM3's first step is an Euler step
        if c["scheme"] != "RK3_SSP":
            return
        r1 = _ref_rhs(self.s, c, h, False)
        self.add([(dt / 4, r1), (-3 * dt / 4, r0)])
        self.diagnose()
        r2 = _ref_rhs(self.s, c, h, True)
        self.add([(8 * dt / 12, r2), (-dt / 12, r0), (-dt / 12, r1)])
        self.diagnose()


def exact(case, seed):
    c = _full(case)
    if c["op"] == "rhs":
        s = _rhs_fields(c, seed)
        if c["precision"] != "fp64":
            s = {k: v.float().double() for k, v in s.items()}
        d = _ref_rhs(s, c, 1.0 / c["nz"], True)
        return [d[k] for k in ["b", "u_i", "u_j", "u_k"] + ["t%d" % t for t in range(c["tracers"])]]
    if c["op"] == "solve":
        per, n, _ = _line_extents(c)
        x, _ = _RefMG(n, per).solve(_solve_rhs(c, seed), c["tol"], c["maxite"])
        return [x, None]
    if c["op"] == "ensemble":
        dt = serving.CASES[c["flow"]]["dt"]
        grid = serving.case_grid(c["flow"], c["nx"])
        out = []
        for r in range(c["runs"]):
            f = _initial(c, grid, seed * 64 + r)
            m = _RefModel(c, grid.dx, {k: v.float().double() for k, v in f.items()})
            m.diagnose()
            for _ in range(c["steps"]):
                m.forward(dt)
            out += [m.s[k] for k in ("b", "u_i", "u_j", "u_k", "p")]
        return out
    from nyles_gb300.grid import Grid
    from nyles_gb300.nyles import prepare_parameters
    grid = Grid(prepare_parameters(_params(c)))
    f = _initial(c, grid, seed)
    if c["precision"] != "fp64":
        f = {k: v.float().double() for k, v in f.items()}
    m = _RefModel(c, grid.dx, f)
    m.diagnose()
    dt = c["dt"]
    if c["auto_dt"]:
        u2 = float(sum(m.s["U_" + d] ** 2 for d in "ijk").max())
        dt = min(0.5 / math.sqrt(u2), 1e-2) if u2 > 0 else 1e-2
    m.forward(dt)
    out = {k: m.s[k] for k in m.prog + ["p"]}
    if c["precision"] == "mixed" and c["tol"] <= 1e-16:
        out["p"] = None      # the Krylov solve leaves the pressure's constant elsewhere
    return out
