"""Performance cases of the per-step particle path, through the package's public entry points.

The simulation cases are what a run does between two outputs, started from a saved state:
the state is set from page-locked host arrays (positions, velocities, pressure and the
unclamped pressure solutions the warm starts read), a few steps run, and the result is read
back.  The workloads are the package's own configurations (polymps_gb300/cases.py): the 2D
incompressible dam break with particle walls, the 3D weakly compressible and incompressible
dam breaks with polygon walls, and the tank with the box obstacle and shifting.  The other
cases are the entry points that are called on their own: one operator, the neighbour lists,
the learned warm start's network (inference and gradient) and the allocation-free PCG.

The mixed FP32/FP64 solves run to 1e-10 (the plain FP64 ones to the default 1e-8): they stop
on an FP64 residual, and one at 1e-8 leaves the last digits of the pressure to the rounding
of its FP32 iterations.
"""
import ctypes as C
import math
import os

import numpy as np
import torch

import polymps_gb300
from polymps_gb300 import abi, cases, mps

WEIGHTS = os.path.join(os.path.dirname(polymps_gb300.__file__), "mlp_warmstart.npz")


def _sim(name, work, tier, nx, ny, nz, l0, steps, **more):
    """A simulation case: fluid of nx x ny x nz particles (nz unused in 2D)."""
    return dict(name=name, kind="sim", work=work, tier=tier, nx=nx, ny=ny, nz=nz, l0=l0, steps=steps, **more)


def listed():
    return [
        # the smallest run: the 2D dam break of configuration 1 (1250 fluid particles and three
        # layers of wall particles), FP64; launches and latencies count
        _sim("dam2d_fp64", "dam2d", "fp64", 25, 50, 0, 0.01, 10),
        # the 3D incompressible dam break coarsened five times (6,912 particles), FP64: quick
        # parameter studies, the size of the smoke test
        _sim("inc_7k_fp64", "inc", "fp64", 24, 24, 12, 0.025, 10),
        # configuration 2: weakly compressible, diffusive PND, position shifting, FP64
        _sim("wc_108k_fp64", "wc", "fp64", 60, 60, 30, 0.01, 4),
        # configuration 4: incompressible at l0 = 0.01, float-float tier, learned warm start
        _sim("inc_108k_learned", "inc", "learned", 60, 60, 30, 0.01, 4),
        # configuration 3, the headline workload, float-float tier and mixed solver from the
        # quadratic extrapolation
        _sim("inc_864k_df32", "inc", "df32", 120, 120, 60, 0.005, 4),
        # the same in the FP64 tier with the plain FP64 solver (the drop-in, the default)
        _sim("inc_864k_fp64", "inc", "fp64", 120, 120, 60, 0.005, 2),
        # configuration 5 at 1.5 times its spacing (2.79 M particles): obstacle and shifting;
        # its mixed solve is above the size whose vectors fit in shared memory
        _sim("obstacle_2m8_df32", "obstacle", "df32", 200, 167, 83, 0.006, 2),
        # one operator called as a class method of the reference: bucket update and viscosity
        # at an odd size, FP64
        dict(name="viscosity_fp64", kind="visc", nx=73, ny=59, nz=31, l0=0.01, tier="fp64"),
        # neighbour lists of the current positions on the host
        dict(name="neighbors_108k", kind="nbr", nx=60, ny=60, nz=30, l0=0.01, tier="fp64"),
        # inference of the learned start's network for the rows of an 864k system
        dict(name="mlp_forward_864k", kind="mlp", rows=864000),
        # gradient of one training batch (forward and backward)
        dict(name="mlp_gradient_8k", kind="grad", rows=8192),
        # allocation-free PCG on a pressure system of 108k rows held by the caller
        dict(name="pcg_static_108k", kind="pcg", nx=60, ny=60, nz=30, tol=1e-8),
    ]


def _log(rng, a, b):
    return math.exp(rng.uniform(math.log(a), math.log(b)))


def _box(rng, lo, hi):
    """Odd and even fluid extents of about the workloads' 2 : 2 : 1 proportions."""
    n = _log(rng, lo, hi)
    f = rng.uniform(0.7, 1.4)
    nz = max(7, round((n / 4.0) ** (1.0 / 3.0)))
    nx = max(9, round(2 * nz * f))
    ny = max(9, round(n / (nx * nz)))
    return nx, ny, nz


def draw(rng):
    kind = rng.choice(["dam2d", "wc", "inc", "inc", "inc", "obstacle", "visc", "nbr", "mlp", "grad", "pcg", "pcg"])
    if kind == "dam2d":
        nx = round(_log(rng, 17, 120))
        return dict(kind="sim", work="dam2d", tier=rng.choice(["fp64", "df32"]), nx=nx, ny=2 * nx + rng.randrange(3), nz=0,
                    l0=round(0.25 / nx, 5), steps=rng.choice([3, 5, 10]))
    if kind in ("wc", "inc", "obstacle"):
        tier = rng.choice(["fp64", "df32"]) if kind != "inc" else rng.choice(["fp64", "df32", "learned"])
        nx, ny, nz = _box(rng, 5000, 700000)
        steps = rng.choice([2, 3, 4]) if nx * ny * nz > 50000 else rng.choice([4, 7, 10])
        return dict(kind="sim", work=kind, tier=tier, nx=nx, ny=ny, nz=nz, l0=round(0.3 / nz, 5), steps=steps)
    if kind in ("visc", "nbr"):
        nx, ny, nz = _box(rng, 5000, 300000)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, l0=round(0.3 / nz, 5), tier=rng.choice(["fp64", "df32"]))
    if kind == "mlp":
        return dict(kind="mlp", rows=round(_log(rng, 1000, 864000)))
    if kind == "grad":
        return dict(kind="grad", rows=64 * math.ceil(_log(rng, 0.5, 4096)))
    nx, ny, nz = _box(rng, 2000, abi.STATIC_MAX_ROWS * 0.9)
    while nx * ny * nz > abi.STATIC_MAX_ROWS:
        ny -= 1
    return dict(kind="pcg", nx=nx, ny=ny, nz=nz, tol=rng.choice([1e-8, 1e-10, 1e-12]))


# ------------------------------------------------------------------ inputs
def _generated(case, seed):
    """The generated workload with jittered fluid, and its fluid extent."""
    l0, nx, ny, nz = case["l0"], case["nx"], case["ny"], case["nz"]
    if case.get("work") == "dam2d":
        size = (nx * l0, ny * l0)
        c = cases.dam2d_particle_walls(l0=l0, width=size[0], height=size[1], tank=(4 * size[0], 1.2 * size[1]),
                                       jitter=0.03, seed=seed, dt=0.05 * l0)
        return c, size
    size = (nx * l0, ny * l0, nz * l0)
    tank = (2.683 * size[0], size[1], 2.0 * size[2])
    if case.get("work") == "wc":
        return cases.dam3d_polygon(l0=l0, fluid=size, tank=tank, mode="wc", jitter=0.03, seed=seed, dt=0.01 * l0), size
    obstacle = None
    if case.get("work") == "obstacle":
        obstacle = ((2.0 * size[0], 0.42 * size[1], 0.0), (0.13 * size[0], 0.16 * size[1], 0.8 * size[2]))
    c = cases.dam3d_polygon(l0=l0, fluid=size, tank=tank, mode="inc", jitter=0.03, seed=seed, dt=0.05 * l0,
                            obstacle=obstacle)
    if obstacle is not None:
        c.params.update(shiftingType=2)
    return c, size


def _velocity(c, size, rng):
    """A collapsing column's smooth velocities with particle noise on the fluid."""
    fluid = c.type == cases.FLUID
    h = 1 if len(size) == 2 else 2
    a = rng.uniform(0.1, 0.4)
    x, z = c.pos[:, 0] / size[0], c.pos[:, h] / size[-1]
    v = np.zeros_like(c.pos)
    v[:, 0] = a * x * x * (1.2 - z)
    v[:, h] = -a * x * z
    noise = rng.normal(scale=0.003, size=v.shape)
    if h == 1:
        noise[:, 2] = 0.0
    return np.where(fluid[:, None], v + noise, 0.0)


def _pressure(c, size, rng):
    """Hydrostatic pressure of the column, as a clamped field and three unclamped solutions."""
    h = 1 if len(size) == 2 else 2
    p = 1000.0 * 9.81 * np.maximum(size[-1] - c.pos[:, h], 0.0) * (1.0 - 0.3 * np.clip(c.pos[:, 0] / size[0], 0, 1))
    noise = rng.normal(scale=0.01, size=p.shape)
    return [p * (1.0 + noise), p * (1.0 + noise) * 0.99, p * (1.0 + noise) * 0.98]


def _pinned(a):
    t = torch.empty(a.size, dtype=torch.float64).pin_memory()
    v = t.numpy().reshape(a.shape)
    v[...] = a
    return v


def _handle(c, tier):
    kw = dict(precision=abi.PRECISION_FP64 if tier == "fp64" else abi.PRECISION_DF32)
    g = mps.MpsGpu(c, **kw)
    if tier == "learned":
        w = np.load(WEIGHTS)
        g.mlp_set_weights(w["params"], w["norm"])
        g.set_solver(abi.SOLVER_MIXED, abi.WARM_MLP, tol=1e-10)
    elif tier == "df32":
        g.set_solver(abi.SOLVER_MIXED, abi.WARM_EXTRAP2, tol=1e-10)
    return g


def _mlp_inputs(case, seed):
    rng = np.random.default_rng(seed)
    n = case["rows"]
    feat = rng.normal(size=(n, abi.MLP_NFEAT)).astype(np.float32)
    target = rng.normal(size=n).astype(np.float32)
    w = np.load(WEIGHTS)
    norm = w["norm"].astype(np.float32)
    # features and targets in their raw units: the normalisation brings them back to unit spread
    return ((feat / norm[16:32] + norm[:16]).astype(np.float32), (target / norm[33] + norm[32]).astype(np.float32),
            w["params"].astype(np.float32), norm)


def _pcg_system(case, seed):
    """Pressure matrix of a jittered lattice (weights re/r - 1 within 2.1 spacings), its free
    surface rows and right-hand side, as CSR on the GPU."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    jit = (torch.rand((nx, ny, nz, 3), generator=gen, device="cuda", dtype=torch.float64) - 0.5) * 0.06
    idx = torch.arange(nx * ny * nz, device="cuda").reshape(nx, ny, nz)
    free = torch.zeros((nx, ny, nz), dtype=torch.bool, device="cuda")
    free[:, :, -1] = True
    free[-1] = True
    offs = [(a, b, c) for a in range(-2, 3) for b in range(-2, 3) for c in range(-2, 3)
            if 0 < a * a + b * b + c * c <= 4]
    rows, cols, vals = [], [], []
    diag = torch.full((nx, ny, nz), 1e-3, device="cuda", dtype=torch.float64)
    for o in offs:
        src = tuple(slice(max(0, -d), n - max(0, d)) for d, n in zip(o, (nx, ny, nz)))
        dst = tuple(slice(max(0, d), n - max(0, -d)) for d, n in zip(o, (nx, ny, nz)))
        r = (torch.tensor(o, device="cuda", dtype=torch.float64) + jit[dst] - jit[src]).norm(dim=-1)
        w = (2.1 / r - 1.0).clamp_min(0.0)
        diag[src] += w
        keep = ~free[src] & ~free[dst]
        rows.append(idx[src][keep]), cols.append(idx[dst][keep]), vals.append(-w[keep])
    diag[free] = 1.0
    rows.append(idx.reshape(-1)), cols.append(idx.reshape(-1)), vals.append(diag.reshape(-1))
    rows, cols, vals = torch.cat(rows), torch.cat(cols), torch.cat(vals)
    n = nx * ny * nz
    order = torch.argsort(rows * n + cols)
    rows, cols, vals = rows[order], cols[order], vals[order]
    ptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    ptr[1:] = torch.cumsum(torch.bincount(rows, minlength=n), 0)
    b = torch.randn(n, generator=gen, device="cuda", dtype=torch.float64)
    z = (torch.arange(n, device="cuda") % nz).double() / nz
    b = torch.where(free.reshape(-1), torch.zeros_like(b), 0.3 * b + torch.cos(3.0 * z))
    x0 = 10.0 * (1.0 - z) * (~free.reshape(-1))
    return ptr.int(), cols.int(), vals, b, x0.contiguous()


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "sim":
        c, size = _generated(case, seed)
        rng = np.random.default_rng(seed + 1)
        vel, press = _velocity(c, size, rng), _pressure(c, size, rng)
        g = _handle(c, case["tier"])
        g.initialize()
        s["in"] = [(abi.F_POS, _pinned(c.pos)), (abi.F_VEL, _pinned(vel)), (abi.F_PRESS, _pinned(press[0]))]
        if c.params["mpsType"] == 2:   # the solutions the warm starts read
            s["in"] += [(f, _pinned(p)) for f, p in zip((abi.F_PRESSPPE, abi.F_PRESSPPE_PREV, abi.F_PRESSPPE_PREV2), press)]
        else:                          # the diffusive PND is carried from step to step
            s["in"].append((abi.F_PNDI, _pinned(g.get(abi.F_PNDI))))
        s["out"] = {f: _pinned(np.zeros_like(a)) for f, a in s["in"][:4]}
        s["g"] = g
    elif kind in ("visc", "nbr"):
        c, size = _generated(case, seed)
        s["vel"] = _pinned(_velocity(c, size, np.random.default_rng(seed + 1)))
        s["pos"] = _pinned(c.pos)
        s["out"] = _pinned(np.zeros_like(c.pos))
        s["g"] = _handle(c, case["tier"])
        s["g"].initialize()
    elif kind in ("mlp", "grad"):
        feat, target, params, norm = _mlp_inputs(case, seed)
        s["g"] = mps.MpsGpu(cases.config(3, scale=8.0))
        s["g"].mlp_set_weights(params, norm)
        s["feat"], s["target"] = feat, target
    else:
        s["sys"] = _pcg_system(case, seed)
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "sim":
        g = s["g"]
        for f, a in s["in"]:
            g.set(f, a)
        g.run(case["steps"])
        return {abi.FIELD_NAMES[f]: g.get(f, out=a) for f, a in s["out"].items()}
    if kind == "visc":
        g = s["g"]
        g.set(abi.F_POS, s["pos"])
        g.set(abi.F_VEL, s["vel"])
        g.run_op("UPDATE_BUCKETS")
        g.run_op("VISCOSITY")
        return g.get(abi.F_ACC, out=s["out"])
    if kind == "nbr":
        g = s["g"]
        g.set(abi.F_POS, s["pos"])
        g.run_op("UPDATE_BUCKETS")
        return list(g.neighbors())
    if kind == "mlp":
        return s["g"].mlp_forward(s["feat"])
    if kind == "grad":
        return list(s["g"].mlp_gradient(s["feat"], s["target"]))
    ptr, col, val, b, x0 = s["sys"]
    x = x0.clone()
    it, res = C.c_int(), C.c_double()
    code = mps.lib().mpsgpu_pcg_solve_static(
        len(b), ptr.data_ptr(), col.data_ptr(), val.data_ptr(), b.data_ptr(), x.data_ptr(), case["tol"], 10000,
        torch.cuda.current_stream().cuda_stream, C.byref(it), C.byref(res))
    if code:
        raise mps.MpsError("mpsgpu_pcg_solve_static", code)
    return x


# ------------------------------------------------------------------ work and exact values
def work(case):
    kind = case["kind"]
    if kind == "sim":
        two = case["work"] == "dam2d"
        n = case["nx"] * case["ny"] * max(case["nz"], 1) + (3 * (4 * case["nx"] + 3 * case["ny"]) if two else 0)
        pairs = n * (13 if two else 32)
        # per step: the particle state read and written, each pair in about seven sums of twenty
        # operations; the pressure matrix (value and column) once for each of about 15 iterations
        solve = 0 if case["work"] == "wc" else 15
        return {"bytes": case["steps"] * (n * 128.0 + pairs * 8.0 * solve) + n * 144.0,
                "flops": case["steps"] * pairs * (140.0 + 2.0 * solve)}
    if kind in ("visc", "nbr"):
        n = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": n * (72.0 if kind == "visc" else 24.0 + 4 + 4 * 30), "flops": n * 30 * (20.0 if kind == "visc" else 8.0)}
    if kind in ("mlp", "grad"):
        macs = 16 * 64 + 2 * 64 * 64 + 64
        return {"bytes": case["rows"] * 68.0 + 4.0 * abi.MLP_NPARAM, "flops": case["rows"] * 2.0 * macs * (3 if kind == "grad" else 1)}
    n = case["nx"] * case["ny"] * case["nz"]
    its = 20 + 2 * (abs(math.log10(case["tol"])) - 8)
    return {"bytes": its * n * (30 * 12.0 + 8 * 8), "flops": its * n * 30 * 2.0}


def _pairs(pos, r, cells):
    """All ordered pairs closer than r: a jittered lattice of `cells` points, x-major."""
    p = torch.from_numpy(np.ascontiguousarray(pos)).cuda().reshape(*cells, 3)
    idx = torch.arange(p.shape[0] * p.shape[1] * p.shape[2], device="cuda").reshape(cells)
    for o in [(a, b, c) for a in range(-2, 3) for b in range(-2, 3) for c in range(-2, 3) if (a, b, c) != (0, 0, 0)]:
        src = tuple(slice(max(0, -d), n - max(0, d)) for d, n in zip(o, cells))
        dst = tuple(slice(max(0, d), n - max(0, -d)) for d, n in zip(o, cells))
        d2 = ((p[dst] - p[src]) ** 2).sum(-1)
        keep = d2 < r * r
        yield idx[src][keep], idx[dst][keep], d2[keep]


def _exact_viscosity(case, seed):
    c, size = _generated(case, seed)
    vel = torch.from_numpy(_velocity(c, size, np.random.default_rng(seed + 1))).cuda()
    l0 = case["l0"]
    re = 2.1 * l0
    # lattice constants: n0 and lambda of the particle at the centre of a full neighbourhood
    o = np.stack(np.meshgrid(*[np.arange(-4, 5)] * 3, indexing="ij"), -1).reshape(-1, 3) * l0
    r2 = (o ** 2).sum(-1)
    r2 = r2[(r2 > 0) & (r2 < re * re)]
    w = re / np.sqrt(r2) - 1.0
    coef = 2.0 * 3.0 / (w.sum() * ((r2 * w).sum() / w.sum()))
    acc = torch.zeros_like(vel)
    for i, j, d2 in _pairs(c.pos, re, (case["nx"], case["ny"], case["nz"])):
        acc.index_add_(0, i, (vel[j] - vel[i]) * ((re / d2.sqrt() - 1.0) * 1e-6)[:, None])
    return (coef * acc).cpu().numpy()


def _gelu(z):
    return 0.5 * z * (1.0 + torch.tanh(0.7978845608028654 * (z + 0.044715 * z ** 3)))


def _exact_mlp(case, seed):
    feat, target, params, norm = (torch.from_numpy(a).cuda().double() for a in _mlp_inputs(case, seed))
    params.requires_grad_(case["kind"] == "grad")
    sizes = [(64, 16), (64,), (64, 64), (64,), (64, 64), (64,), (1, 64), (1,)]
    W = [t.reshape(z) for t, z in zip(torch.split(params, [math.prod(z) for z in sizes]), sizes)]
    h = (feat - norm[:16]) * norm[16:32]
    for k in range(3):
        h = _gelu(h @ W[2 * k].T + W[2 * k + 1])
    out = (h @ W[6].T + W[7])[:, 0]
    if case["kind"] == "mlp":
        return out.cpu().numpy()
    loss = ((out - (target - norm[32]) * norm[33]) ** 2).mean()
    loss.backward()
    return [params.grad.cpu().numpy(), float(loss)]


def _exact_pcg(case, seed):
    ptr, col, val, b, x = _pcg_system(case, seed)
    A = torch.sparse_csr_tensor(ptr.long(), col.long(), val, size=(len(b), len(b)))
    rows = torch.repeat_interleave(torch.arange(len(b), device="cuda"), ptr.long().diff())
    dinv = torch.empty_like(b)
    dinv[rows[rows == col]] = 1.0 / val[rows == col]
    mul = lambda v: (A @ v[:, None])[:, 0]  # noqa: E731
    for _ in range(3):   # restarted, so that the residual is the true one
        r = b - mul(x)
        z = r * dinv
        p, rz = z, r @ z
        for _ in range(120):
            if float(r.norm()) <= 1e-15 * float(b.norm()):
                break
            q = mul(p)
            a = rz / (p @ q)
            x, r = x + a * p, r - a * q
            z = r * dinv
            rz, old = r @ z, rz
            p = z + (rz / old) * p
    return x


def exact(case, seed):
    kind = case["kind"]
    if kind == "visc":
        return _exact_viscosity(case, seed)
    if kind in ("mlp", "grad"):
        return _exact_mlp(case, seed)
    if kind == "pcg":
        return _exact_pcg(case, seed)
    return None
