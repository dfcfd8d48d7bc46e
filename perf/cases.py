"""The work a user of this framework has it do, as cases that can be timed.

Every case goes through the package's public entry points (Solver, FluidSolverGPU,
FluidSolverGaussSeidel, Batch, PinnedArray, learned.Net) the way a program that uses them
does. Kinds:

  step      one device-resident step of one grid (fs_step), the fields staying on the GPU
  frame     one frame of the device-resident simulation driver: a point source of density
            and velocity, a step, the sources cleared (fs_add_*_source, fs_update), the
            frame finished before the next one begins
  host      the drop-in call on host grids, fluid_solver_gpu::solve (fs_solve_host):
            pageable arrays as the reference's std::vector grids, or page-locked ones
  residual  one step whose projections run to a residual target under a sweep cap, from
            the previous step's pressure
  gs        one step of the host solver's Gauss-Seidel method, square grids
  batch     a few steps of many uneven grids, then their fields read back
  learned   one step whose projections meet a residual target with network corrections
  train     one training step of that network: forward, loss, backward, Adam

Fields are sums of Gaussian-core vortices (velocity) and low-frequency noise (density), the
family the repository's benchmark workloads draw from, with the grid's size setting the
cores' radii. exact() evaluates a case in float64 with torch alone.
"""
import math
import pathlib

import numpy as np
import torch

import __graft_entry__

fluid = __graft_entry__.load_package()

ROOT = pathlib.Path(__file__).resolve().parents[1]
PARAMS = ROOT / "tests" / "golden" / "warmstart_params.npy"
DEV = "cuda"


def listed():
    return [
        # the smallest calls: the 130^2 grid with point sources, a frame loop's latency
        {"name": "frame_130", "kind": "frame", "rows": 130, "cols": 130, "kd": 20, "kp": 20, "rate": 1e-4,
         "visc": 1e-4, "dt": 0.1},
        # an odd, non-square grid at the reference's own sweep counts
        {"name": "step_771x1283", "kind": "step", "rows": 771, "cols": 1283, "kd": 15, "kp": 20, "rate": 1e-5,
         "visc": 1e-5, "dt": 0.05},
        # the benchmark's headline grid and sweep counts
        {"name": "step_2050", "kind": "step", "rows": 2050, "cols": 2050, "kd": 40, "kp": 40, "rate": 1e-5,
         "visc": 1e-5, "dt": 0.05},
        # the largest grid of the benchmark's workloads
        {"name": "step_8194", "kind": "step", "rows": 8194, "cols": 8194, "kd": 15, "kp": 20, "rate": 1e-5,
         "visc": 1e-5, "dt": 0.05},
        # the reference application's own grid, rates and time step, through the drop-in call
        {"name": "host_800", "kind": "host", "rows": 800, "cols": 800, "kd": 15, "kp": 20, "rate": 0.5,
         "visc": 1e-6, "dt": 0.02, "pinned": False},
        # the drop-in call on the headline grid, page-locked host grids
        {"name": "host_2050_pinned", "kind": "host", "rows": 2050, "cols": 2050, "kd": 40, "kp": 40, "rate": 1e-5,
         "visc": 1e-5, "dt": 0.05, "pinned": True},
        # projections to a residual target that the sweep cap ends, previous-pressure start
        {"name": "residual_1026", "kind": "residual", "rows": 1026, "cols": 1026, "kd": 20, "cap": 200, "tol": 1e-4,
         "rate": 1e-5, "visc": 1e-5, "dt": 0.05},
        # uneven grids advanced together, fields read back every few steps
        {"name": "batch_24", "kind": "batch", "count": 24, "smallest": 64, "largest": 512, "kd": 30, "kp": 30,
         "steps": 8, "rate": 1e-5, "visc": 1e-5, "dt": 0.05},
        # the host solver's method on the small benchmark grid (one SM's shared memory holds it)
        {"name": "gs_130", "kind": "gs", "n": 130, "kd": 20, "kp": 20, "rate": 1e-4, "visc": 1e-4, "dt": 0.02},
        # the host solver's method at the reference application's size
        {"name": "gs_800", "kind": "gs", "n": 800, "kd": 20, "kp": 20, "rate": 0.5, "visc": 1e-6, "dt": 0.02},
        # learned corrections to a residual target, the committed network
        {"name": "learned_514", "kind": "learned", "n": 514, "kd": 20, "tol": 1e-2, "cap": 20000, "rate": 1e-5,
         "visc": 1e-5, "dt": 0.05},
        # one training step of the network on a batch of coarse grids
        {"name": "train_64", "kind": "train", "grids": 64},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "frame", "host", "host", "residual", "batch", "gs", "gs", "learned",
                       "train"])
    rate = rng.choice([1e-6, 1e-5, 1e-4])
    dt = rng.choice([0.02, 0.05])
    if kind == "step":
        rows, cols = _log(rng, 100, 6000), _log(rng, 100, 6000)
        return {"kind": kind, "rows": rows, "cols": cols, "kd": rng.randint(10, 24), "kp": rng.randint(10, 30),
                "rate": rate, "visc": rate, "dt": dt}
    if kind == "frame":
        return {"kind": kind, "rows": _log(rng, 66, 900), "cols": _log(rng, 66, 900), "kd": rng.choice([15, 20]),
                "kp": rng.choice([20, 30]), "rate": rate, "visc": rate, "dt": dt}
    if kind == "host":
        return {"kind": kind, "rows": _log(rng, 130, 2050), "cols": _log(rng, 130, 2050), "kd": rng.randint(15, 40),
                "kp": rng.randint(15, 40), "rate": rate, "visc": rate, "dt": dt, "pinned": rng.random() < 0.5}
    if kind == "residual":
        return {"kind": kind, "rows": _log(rng, 200, 2050), "cols": _log(rng, 200, 2050), "kd": 20,
                "cap": 8 * rng.randint(8, 40), "tol": 1e-4, "rate": rate, "visc": rate, "dt": dt}
    if kind == "batch":
        lo = rng.randint(40, 120)
        return {"kind": kind, "count": rng.randint(6, 32), "smallest": lo, "largest": rng.randint(2 * lo, 512),
                "kd": rng.randint(15, 30), "kp": rng.randint(15, 30), "steps": rng.randint(4, 8), "rate": rate,
                "visc": rate, "dt": dt}
    if kind == "gs":
        return {"kind": kind, "n": _log(rng, 66, 900), "kd": 20, "kp": 20, "rate": rate, "visc": rate, "dt": 0.02}
    if kind == "learned":
        return {"kind": kind, "n": 2 + 32 * rng.randint(8, 24), "kd": 20, "tol": rng.choice([1e-1, 1e-2]),
                "cap": 20000, "rate": 1e-5, "visc": 1e-5, "dt": 0.05}
    return {"kind": kind, "grids": rng.randint(16, 96)}


# ------------------------------------------------------------------- inputs


def _reflect(u, v):
    u[1:-1, 0] = -u[1:-1, 1]
    u[1:-1, -1] = -u[1:-1, -2]
    u[0, 1:-1] = u[1, 1:-1]
    u[-1, 1:-1] = u[-2, 1:-1]
    v[0, 1:-1] = -v[1, 1:-1]
    v[-1, 1:-1] = -v[-2, 1:-1]
    v[1:-1, 0] = v[1:-1, 1]
    v[1:-1, -1] = v[1:-1, -2]


def _fields(rows, cols, seed):
    """Density, u, v: vortices with cores of 1-4 % of the side, noise in [0, 1]."""
    rng = np.random.default_rng(seed)
    side = math.sqrt(rows * cols)
    count = min(64, max(4, int(round(16 * (side / 1024.0) ** 2))))
    ii = torch.arange(rows, dtype=torch.float32, device=DEV)[:, None]
    jj = torch.arange(cols, dtype=torch.float32, device=DEV)[None, :]
    u = torch.zeros((rows, cols), dtype=torch.float32, device=DEV)
    v = torch.zeros_like(u)
    for _ in range(count):
        cy, cx = rng.uniform(1.0, rows - 2.0), rng.uniform(1.0, cols - 2.0)
        rad = rng.uniform(max(3.0, side / 100.0), max(6.0, side / 25.0))
        gam = rng.uniform(-50.0, 50.0)
        dy, dx = ii - cy, jj - cx
        r2 = (dx * dx + dy * dy).clamp_(min=1e-12)
        f = torch.expm1(r2 * (-1.0 / (rad * rad))).mul_(-gam / (2.0 * math.pi)).div_(r2)
        u.addcmul_(f, dy.expand_as(f), value=-1.0)
        v.addcmul_(f, dx.expand_as(f))
    _reflect(u, v)
    d = torch.zeros_like(u)
    for _ in range(8):
        kx, ky = (int(x) for x in rng.integers(1, 5, size=2))
        ph, a = rng.uniform(0, 2 * math.pi), rng.uniform(0.2, 1.0)
        d += a * torch.sin(2 * math.pi * (kx * jj / cols + ky * ii / rows) + ph)
    d -= d.min()
    d /= d.max()
    return d, u, v


def _sources(rows, cols, seed):
    """Host grids' sources: two density blobs, a faint push on the velocity."""
    rng = np.random.default_rng(seed + 7919)
    ii = torch.arange(rows, dtype=torch.float32, device=DEV)[:, None]
    jj = torch.arange(cols, dtype=torch.float32, device=DEV)[None, :]

    def blob(amp):
        cy, cx = rng.uniform(1.0, rows - 2.0), rng.uniform(1.0, cols - 2.0)
        g = amp * torch.exp(-((ii - cy) ** 2 + (jj - cx) ** 2) / 72.0)
        g[0], g[-1], g[:, 0], g[:, -1] = 0.0, 0.0, 0.0, 0.0
        return g

    return blob(100.0) + blob(100.0), blob(0.02), blob(-0.02)


def _point(case, seed):
    rng = np.random.default_rng(seed + 31)
    i, j = int(rng.integers(2, case["rows"] - 2)), int(rng.integers(2, case["cols"] - 2))
    cells = case["rows"] * case["cols"]
    ang = rng.uniform(0, 2 * math.pi)
    return i, j, 100.0 / cells, 2.0 * math.cos(ang) / cells, 2.0 * math.sin(ang) / cells


def _shapes(case, seed):
    """Uneven (rows, cols) of a batch: half of them square, the sizes spread evenly."""
    rng = np.random.default_rng(seed + 17)
    lo, hi, n = case["smallest"], case["largest"], case["count"]
    out = []
    for k in range(n):
        r = lo + (hi - lo) * k // max(1, n - 1)
        c = r if k % 2 else lo + (hi - lo) * ((5 * k + 2) % n) // max(1, n - 1)
        out.append((r + 2, c + 2))
    order = rng.permutation(n)
    return [out[k] for k in order]


class _View:
    """A field of a handle, as the CUDA array interface; keeps the handle alive."""

    def __init__(self, solver, ptr, view):
        self.solver = solver
        self.__cuda_array_interface__ = {"shape": (view.rows, view.cols), "strides": (view.pitch * 4, 4),
                                         "typestr": "<f4", "data": (int(ptr), False), "version": 2}


class _Held(np.ndarray):
    """A view of page-locked memory that keeps the memory's owner alive."""

    owner = None


def _resident(solver, fields, sources=None):
    """Puts device tensors into a handle's state and returns views of the state."""
    view = solver.device_view()
    ptrs = [view.density, view.u, view.v, view.density_source, view.u_source, view.v_source]
    views = [torch.as_tensor(_View(solver, p, view), device=DEV) for p in ptrs]
    for dst, src in zip(views, list(fields) + list(sources or [])):
        dst.copy_(src)
    torch.cuda.synchronize()
    return views[:3]


def _np(*ts):
    return [np.ascontiguousarray(t.cpu().numpy()) for t in ts]


def _train_inputs(case, seed):
    """Normalised coarse residuals and targets of the network, and its parameters."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    n = case["grids"]
    x = torch.zeros((n * 32, 32, 32), dtype=torch.bfloat16, device=DEV)
    x[:, :, 0] = torch.randn((n * 32, 32), generator=g, device=DEV).to(torch.bfloat16)
    t = 0.5 * torch.randn((n * 32, 32), generator=g, device=DEV)
    return x, t, torch.from_numpy(np.load(PARAMS)).to(DEV)


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind in ("step", "frame", "residual"):
        cfg = {"diffuse_iterations": case["kd"], "device": 0}
        if kind == "residual":
            cfg.update(pressure_tolerance=case["tol"], pressure_max_iterations=case["cap"],
                       warm_start=fluid.FS_WARM_PREVIOUS)
        else:
            cfg["pressure_iterations"] = case["kp"]
        s = fluid.Solver(case["rows"], case["cols"], **cfg)
        st["solver"] = s
        st["out"] = _resident(s, _fields(case["rows"], case["cols"], seed))
        if kind == "frame":
            st["point"] = _point(case, seed)
    elif kind in ("gs", "learned"):
        n = case["n"]
        if kind == "gs":
            s = fluid.FluidSolverGaussSeidel(n, diffuse_iterations=case["kd"], pressure_iterations=case["kp"], device=0)
        else:
            s = fluid.Solver(n, n, diffuse_iterations=case["kd"], pressure_tolerance=case["tol"],
                             pressure_max_iterations=case["cap"], warm_start=fluid.FS_WARM_LEARNED, device=0)
            s.set_network(np.load(PARAMS))
        st["solver"] = s
        st["out"] = _resident(s, _fields(n, n, seed))
    elif kind == "host":
        rows, cols = case["rows"], case["cols"]
        grids = _np(*_fields(rows, cols, seed), *_sources(rows, cols, seed))
        if case["pinned"]:
            pins = [fluid.PinnedArray(rows, cols) for _ in grids]
            for p, a in zip(pins, grids):
                p.array[:] = a
            grids = [p.array.view(_Held) for p in pins]
            for a, p in zip(grids, pins):
                a.owner = p
        st["grids"] = grids
        st["solver"] = fluid.FluidSolverGPU(rows, cols, diffuse_iterations=case["kd"],
                                            pressure_iterations=case["kp"], device=0)
    elif kind == "batch":
        shapes = _shapes(case, seed)
        b = fluid.Batch(shapes, diffuse_iterations=case["kd"], pressure_iterations=case["kp"], device=0)
        for k, (r, c) in enumerate(shapes):
            b.upload(k, *_np(*_fields(r, c, seed + 100 * k)))
        st["batch"] = b
    else:
        from fluid2d_gb300 import learned

        x, t, params = _train_inputs(case, seed)
        st.update(learned=learned, x=x, t=t, net=learned.Net(case["grids"], params))
        st["adam"] = learned.Adam(st["net"], lr=1e-4)
    torch.cuda.synchronize()
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind in ("step", "gs", "learned"):
        st["solver"].step(case["rate"], case["visc"], case["dt"])
        return st["out"]
    if kind == "residual":
        try:
            st["solver"].step(case["rate"], case["visc"], case["dt"])
        except fluid.FluidError as e:
            if e.code != fluid.FS_ERR_NOT_CONVERGED:  # the cap ended the solve, as it should here
                raise
        return st["out"]
    if kind == "frame":
        s = st["solver"]
        i, j, amount, horizontal, vertical = st["point"]
        s.add_density_source(i, j, amount)
        s.add_velocity_source(i, j, horizontal, vertical)
        s.update(case["rate"], case["visc"], case["dt"])
        return st["out"]
    if kind == "host":
        d, u, v, ds, us, vs = st["grids"]
        st["solver"].solve(d, ds, case["rate"], u, v, us, vs, case["visc"], case["dt"])
        return [d, u, v]
    if kind == "batch":
        b = st["batch"]
        b.step(case["rate"], case["visc"], case["dt"], case["steps"], sync=False)
        out = [b.download(k) for k in range(len(b))]
        # one array per field: all grids behind one another
        return [np.concatenate([g[f].ravel() for g in out]) for f in range(3)]
    learned, net = st["learned"], st["net"]
    y = net.forward(st["x"])
    loss, dy = learned.mse_loss(net, st["t"])
    grad = net.backward(st["x"], dy)
    st["adam"].step(grad)
    return [y[:, :, 0], loss, grad, net.params]


# --------------------------------------------------------------------- work


def work(case):
    kind = case["kind"]
    if kind == "train":
        # forward, backward-data and weight gradients of 8 convolutions, 32 -> 32, 3 x 3
        px = case["grids"] * (3 * 1024 + 3 * 256 + 2 * 64)
        params = 8 * (32 * 9 * 32 + 32)
        return {"bytes": case["grids"] * 1024 * (2 * 32 + 4 + 4) + params * 4 * 8, "flops": 3 * px * 2 * 9 * 32 * 32}
    if kind == "batch":
        cells = sum(r * c for r, c in _shapes(case, 0))
        kd, kp, n = case["kd"], case["kp"], case["steps"]
        return {"bytes": 36 * cells, "flops": n * cells * (3 * 6 * kd + 2 * 5 * kp + 100)}
    rows, cols = (case["n"], case["n"]) if "n" in case else (case["rows"], case["cols"])
    cells = rows * cols
    kp = {"residual": case.get("cap"), "learned": 200}.get(kind, case.get("kp"))
    # state and sources in, state out; sweeps, divergence, gradient and advection
    return {"bytes": 36 * cells, "flops": cells * (3 * 6 * case["kd"] + 2 * 5 * kp + 100)}


# -------------------------------------------------------------------- exact


def _fill(x, lr, tb, corners=False):
    x[1:-1, 0] = lr * x[1:-1, 1]
    x[1:-1, -1] = lr * x[1:-1, -2]
    x[0, 1:-1] = tb * x[1, 1:-1]
    x[-1, 1:-1] = tb * x[-2, 1:-1]
    if corners:
        x[0, 0] = 0.5 * (x[0, 1] + x[1, 0])
        x[0, -1] = 0.5 * (x[0, -2] + x[1, -1])
        x[-1, 0] = 0.5 * (x[-1, 1] + x[-2, 0])
        x[-1, -1] = 0.5 * (x[-1, -2] + x[-2, -1])


_SIGNS = {"d": (1.0, 1.0), "u": (-1.0, 1.0), "v": (1.0, -1.0)}


def _nbrs(x):
    return x[1:-1, :-2] + x[1:-1, 2:] + x[:-2, 1:-1] + x[2:, 1:-1]


def _jacobi(x, c, a, den, sweeps, signs):
    x = x.clone()
    for _ in range(sweeps):
        x[1:-1, 1:-1] = (c[1:-1, 1:-1] + a * _nbrs(x)) / den
        _fill(x, *signs)
    return x


def _gauss_seidel(x, c, a, den, sweeps, signs):
    """Lexicographic in-place sweeps, all of them in flight: sweep s updates cell (i, j) at
    time i + j + 2s from values of the time before. A cell next to an edge reads what the
    fill left there: its own value of the sweep before, times the sign."""
    if sweeps == 0:
        return x
    m = x.shape[0] - 2
    lr, tb = signs
    x = x.clone()
    g, cin = x[1:-1, 1:-1], c[1:-1, 1:-1].contiguous()
    init = g.clone()
    i = torch.arange(m, device=x.device)
    shift = i[None, :] + 2 * torch.arange(sweeps, device=x.device)[:, None]
    val = torch.zeros((sweeps, m), dtype=x.dtype, device=x.device)
    old = val
    first, last = i == 0, i == m - 1
    below = torch.roll(i, -1)
    for t in range(2 * m - 1 + 2 * (sweeps - 1)):
        j = t - shift
        jc = j.clamp(0, m - 1)
        up, left = torch.roll(val, 1, 1), val
        before = torch.roll(val, 1, 0)
        j0 = jc[0]
        before[0] = init[i, (j0 + 1).clamp(max=m - 1)]
        right, down = before, torch.roll(before, -1, 1)
        down[0] = init[below, j0]
        own = torch.roll(old, 1, 0)
        lo, hi = lr * own, lr * own
        top, bot = tb * own, tb * own
        lo[0], hi[0], top[0], bot[0] = x[1:-1, 0], x[1:-1, -1], x[0, 1 + j0], x[-1, 1 + j0]
        left, right = torch.where(j == 0, lo, left), torch.where(j == m - 1, hi, right)
        up, down = torch.where(first, top, up), torch.where(last, bot, down)
        val, old = (cin[i, jc] + a * (up + down + left + right)) / den, val
        done = (j[-1] >= 0) & (j[-1] < m)
        g[i[done], j[-1][done]] = val[-1][done]
    _fill(x, *signs, corners=True)
    return x


def _targets(x, y):
    j0, i0 = x.floor(), y.floor()
    return i0.long(), j0.long(), x - j0, y - i0


def _axes(a):
    i = torch.arange(1, a.shape[0] - 1, dtype=a.dtype, device=a.device)[:, None]
    j = torch.arange(1, a.shape[1] - 1, dtype=a.dtype, device=a.device)[None, :]
    return i, j


def _splat(d, u, v, dt0):
    rows, cols = d.shape
    i, j = _axes(d)
    x, y = j + dt0 * u[1:-1, 1:-1], i + dt0 * v[1:-1, 1:-1]
    ok = (x >= 0.5) & (x <= cols - 1.5) & (y >= 0.5) & (y <= rows - 1.5)
    x, y, w = x[ok], y[ok], d[1:-1, 1:-1][ok]
    i0, j0, s0, s2 = _targets(x, y)
    acc = torch.zeros_like(d)
    flat = acc.view(-1)
    at = i0 * cols + j0
    flat.index_add_(0, at, (1 - s0) * (1 - s2) * w)
    flat.index_add_(0, at + cols, (1 - s0) * s2 * w)
    flat.index_add_(0, at + 1, s0 * (1 - s2) * w)
    flat.index_add_(0, at + cols + 1, s0 * s2 * w)
    return acc


def _gather(u, v, dt0):
    rows, cols = u.shape
    i, j = _axes(u)
    x = (j - dt0 * u[1:-1, 1:-1]).clamp(1.5, cols - 1.5)
    y = (i - dt0 * v[1:-1, 1:-1]).clamp(1.5, rows - 1.5)
    i0, j0, s0, s2 = _targets(x, y)
    at = i0 * cols + j0
    out = []
    for f in (u, v):
        g, q = f.clone(), f.reshape(-1)
        g[1:-1, 1:-1] = (1 - s2) * ((1 - s0) * q[at] + s0 * q[at + 1]) + s2 * (
            (1 - s0) * q[at + cols] + s0 * q[at + cols + 1])
        out.append(g)
    return out


def _project(u, v, solve, corners):
    h = 1.0 / math.sqrt(u.numel())
    div, zero = torch.zeros_like(u), torch.zeros_like(u)
    div[1:-1, 1:-1] = -0.5 * h * (u[1:-1, 2:] - u[1:-1, :-2] + v[2:, 1:-1] - v[:-2, 1:-1])
    p = solve(zero, div)
    u, v = u.clone(), v.clone()
    u[1:-1, 1:-1] -= 0.5 * (p[1:-1, 2:] - p[1:-1, :-2]) / h
    v[1:-1, 1:-1] -= 0.5 * (p[2:, 1:-1] - p[:-2, 1:-1]) / h
    _fill(u, *_SIGNS["u"], corners=corners)
    _fill(v, *_SIGNS["v"], corners=corners)
    return u, v


def _step64(case, d, u, v, ds=None, us=None, vs=None):
    """One step in float64: add sources, diffuse, advect and smooth the density, project,
    advect the velocity by itself, project."""
    gs = case["kind"] == "gs"
    kp = case.get("cap") or case["kp"]
    cells, dt = d.numel(), case["dt"]
    dt0 = math.sqrt(cells) * dt
    f = {"d": d.double(), "u": u.double(), "v": v.double()}
    u0, v0 = f["u"].clone(), f["v"].clone()
    sweep = _gauss_seidel if gs else _jacobi
    for k, s, rate in (("d", ds, case["rate"]), ("u", us, case["visc"]), ("v", vs, case["visc"])):
        if s is not None:
            f[k][1:-1, 1:-1] += dt * s.double()[1:-1, 1:-1]
        a = dt * cells * rate
        f[k] = sweep(f[k], f[k], a, 1.0 + 4.0 * a, case["kd"], _SIGNS[k])
    acc = _splat(f["d"], u0, v0, dt0)
    _fill(acc, *_SIGNS["d"], corners=gs)
    if not gs:
        out = acc.clone()
        out[1:-1, 1:-1] = 0.2 * (acc[1:-1, 1:-1] + _nbrs(acc))
        acc = out

    def solve(p, div):
        return sweep(p, div, 1.0, 4.0, kp, _SIGNS["d"])

    u, v = _project(f["u"], f["v"], solve, gs)
    u, v = _gather(u, v, dt0)
    _fill(u, *_SIGNS["u"], corners=gs)
    _fill(v, *_SIGNS["v"], corners=gs)
    u, v = _project(u, v, solve, gs)
    return [acc, u, v]


def _train64(case, seed):
    """The training step with every value in float64 (the network rounds operands to BF16)."""
    x, t, params = _train_inputs(case, seed)
    from fluid2d_gb300 import learned

    n = case["grids"]
    w = params.double().requires_grad_()
    conv = torch.nn.functional.conv2d

    def layer(k, a, skip=None, relu=True):
        q = w[k * 9248:(k + 1) * 9248]
        y = conv(a, q[:9216].view(32, 3, 3, 32).permute(0, 3, 1, 2), q[9216:], padding=1)
        y = y if skip is None else y + skip
        return y.relu() if relu else y

    pool = torch.nn.functional.avg_pool2d
    e1 = layer(0, x.double().view(n, 32, 32, 32).permute(0, 3, 1, 2))
    e3 = layer(2, layer(1, pool(e1, 2)))
    b2 = layer(4, layer(3, pool(e3, 2)))
    d1 = layer(5, b2.repeat_interleave(2, 2).repeat_interleave(2, 3), e3)
    d2 = layer(6, d1.repeat_interleave(2, 2).repeat_interleave(2, 3), e1)
    y = layer(7, d2, relu=False)[:, 0].reshape(n * 32, 32)
    loss = ((y - t.double()) ** 2).mean()
    loss.backward()
    grad = w.grad
    live = torch.from_numpy(learned.frozen_mask() == 0).to(DEV)
    # first Adam step: m / (1 - b1) = grad, v / (1 - b2) = grad^2
    step = 1e-4 * grad / (grad.abs() + 1e-8)
    return [y.detach(), loss.detach(), grad, (w - torch.where(live, step, torch.zeros_like(step))).detach()]


def exact(case, seed):
    kind = case["kind"]
    if kind == "learned":
        return None  # stops where its own residual does
    with torch.enable_grad() if kind == "train" else torch.no_grad():
        if kind == "train":
            return _train64(case, seed)
        if kind == "batch":
            per = []
            for k, (r, c) in enumerate(_shapes(case, seed)):
                q = list(_fields(r, c, seed + 100 * k))
                for _ in range(case["steps"]):
                    q = _step64(case, *q)
                per.append(q)
            return [torch.cat([g[f].reshape(-1) for g in per]) for f in range(3)]
        rows, cols = (case["n"], case["n"]) if "n" in case else (case["rows"], case["cols"])
        fields, src = _fields(rows, cols, seed), [None, None, None]
        if kind == "host":
            src = _sources(rows, cols, seed)
        elif kind == "frame":
            i, j, *amounts = _point(case, seed)
            src = [torch.zeros((rows, cols), dtype=torch.float64, device=DEV) for _ in range(3)]
            for s, a in zip(src, amounts):
                s[i, j] = a * rows * cols
        return _step64(case, *fields, *src)
