"""What users of this framework have it do, as cases that can be timed.

Four kinds of work, each through the Python mirror of the C-ABI:

  solve   a plan that a program keeps: load a device-resident FP32 grid, run
          some steps, read the result back into a device grid
  host    one call: host grid in, steps, host grid out (sweep_host)
  batch   many grids of mixed sizes, stencils and precisions in one run
  serve   a burst of requests to the continuous-batching server

Sizes, step counts, distributions and mixes are those of the benchmark
configurations (bench.py, tcstencil_gb300/workloads.py) and of the sweep
harness, with ragged shapes beside the square ones.
"""
import math

import numpy as np
import torch

import tcstencil_gb300 as tcs
from tcstencil_gb300 import workloads

STENCILS = ("star2d1r", "star2d2r", "box2d1r", "box2d2r")
ENGINE_PRECISIONS = (("auto", "f16"), ("tensor", "f16"), ("auto", "split"), ("cudacore", "f16"), ("cudacore", "f32"))
SIDE = (64, 16386)          # smallest and largest grid side
STEPS = (1, 200)
MAX_CELLS = 16386 * 16386
# Point updates of one pass at most (the 16386 x 16386, 50-step solve's).
MAX_UPDATES = {"f16": 1.3e10, "split": 1.3e10, "f32": 1.0e10}
FLOPS = {"star2d1r": 10, "star2d2r": 18, "box2d1r": 18, "box2d2r": 50}


def listed():
    return [
        # the smallest solves: every step is a few microseconds, so launches
        # and step boundaries are what a user waits for
        _solve("small star2d1r f16 256", "auto", "f16", "star2d1r", 256, 256, 10, "unit"),
        # the first benchmark configuration (1024 x 1024 interior, 10 steps)
        _solve("star2d1r f16 1026", "auto", "f16", "star2d1r", 1026, 1026, 10, "unit"),
        # a ragged grid stepped for longer, radius 2
        _solve("box2d2r f16 333x1517", "auto", "f16", "box2d2r", 333, 1517, 64, "signed"),
        # a large ragged radius-1 sweep
        _solve("box2d1r f16 6000x10001", "auto", "f16", "box2d1r", 6000, 10001, 50, "signed"),
        # the headline configuration (8192 x 8192 interior, 100 steps)
        _solve("box2d2r f16 8196", "tensor", "f16", "box2d2r", 8196, 8196, 100, "signed"),
        # the same configuration's other stencil on the CUDA-core engine
        _solve("cudacore star2d2r f16 8196", "cudacore", "f16", "star2d2r", 8196, 8196, 100, "signed"),
        # results bit for bit as the CPU reference gives them: FP32 storage
        _solve("cudacore box2d1r f32 2051x4099", "cudacore", "f32", "box2d1r", 2051, 4099, 20, "signed"),
        # FP32-level accuracy from the tensor cores, mid-size and ragged
        _solve("split star2d2r 1500x2701", "auto", "split", "star2d2r", 1500, 2701, 30, "smooth"),
        # the split configuration, up to its first drift check (50 steps)
        _solve("split box2d1r 16386", "auto", "split", "box2d1r", 16386, 16386, 50, "smooth"),
        # the one-call form on host memory
        dict(name="host box2d1r f16 3000x5003", kind="host", engine="tensor", precision="f16", stencil="box2d1r",
             ny=3000, nx=5003, steps=20, values="signed"),
        # the batched configuration: 512 mixed grids, half FP16, half split
        dict(name="batch 512 mixed", kind="batch", count=512, side_lo=64, side_hi=2048, steps_lo=1, steps_hi=64, mix=4),
        # the served configuration, as a burst
        dict(name="serve 48 requests", kind="serve", count=48, side_lo=128, side_hi=4096, steps_lo=1, steps_hi=200, mix=5),
    ]


def _solve(name, engine, precision, stencil, ny, nx, steps, values):
    return dict(name=name, kind="solve", engine=engine, precision=precision, stencil=stencil, ny=ny, nx=nx, steps=steps,
                values=values)


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(("solve", "host", "batch", "serve"), (9, 2, 2, 1))[0]
    if kind == "batch":
        return dict(kind="batch", count=_log_int(rng, 4, 512), side_lo=64, side_hi=_log_int(rng, 256, 2048), steps_lo=1,
                    steps_hi=_log_int(rng, 4, 64), mix=rng.randrange(10, 1000))
    if kind == "serve":
        return dict(kind="serve", count=rng.randrange(8, 49), side_lo=128, side_hi=_log_int(rng, 512, 4096), steps_lo=1,
                    steps_hi=_log_int(rng, 8, 200), mix=rng.randrange(10, 1000))
    engine, precision = rng.choice(ENGINE_PRECISIONS)
    ny, nx = _log_int(rng, *SIDE), _log_int(rng, *SIDE)
    if kind == "host":  # the copies take longer than the sweep: sides of the served range
        ny, nx = min(ny, 8196), min(nx, 8196)
    while ny * nx * STEPS[0] > MAX_UPDATES[precision]:
        ny, nx = ny // 2, nx // 2
    steps = _log_int(rng, STEPS[0], max(STEPS[0], min(STEPS[1], int(MAX_UPDATES[precision] / (ny * nx)))))
    return dict(kind=kind, engine=engine if kind == "solve" or engine != "auto" else "tensor", precision=precision,
                stencil=rng.choice(STENCILS), ny=ny, nx=nx, steps=steps, values=rng.choice(("unit", "signed", "smooth")))


# ------------------------------------------------------------------ inputs --
def _grid(case_values, ny, nx, border, seed):
    """A seeded FP32 grid on the GPU: "unit" U[0,1), "signed" U[-1,1), "smooth"
    U[-1,1) + sin(2 pi x) sin(2 pi y), with a zero border."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    g = torch.rand((ny, nx), generator=gen, device="cuda", dtype=torch.float32)
    if case_values != "unit":
        g = g * 2 - 1
    if case_values == "smooth":
        y = torch.linspace(0, 1, ny, device="cuda")
        x = torch.linspace(0, 1, nx, device="cuda")
        g += torch.sin(2 * math.pi * y)[:, None] * torch.sin(2 * math.pi * x)[None, :]
    g[:border] = 0
    g[-border:] = 0
    g[:, :border] = 0
    g[:, -border:] = 0
    return g


def _coeffs(stencil, seed):
    return workloads.normalized_coeffs(np.random.default_rng(seed), stencil)


def _specs(case):
    """The grids of a mixed workload (shapes, stencils, coefficients, steps)."""
    return workloads.mixed_batch(case["count"], (case["side_lo"], case["side_hi"]), (case["steps_lo"], case["steps_hi"]),
                                 case["mix"])


def _mixed_inputs(case, seed):
    """The grids of a mixed workload, FP32: per precision one flat tensor that
    holds its grids one after another (each on a 256-byte boundary, as device
    allocators give them), and all grids as views in spec order."""
    specs = _specs(case)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    flats = {}
    for prec in sorted({s.precision for s in specs}):
        flats[prec] = torch.empty(sum(_room(s) for s in specs if s.precision == prec), device="cuda")
        flats[prec].uniform_(-1, 1, generator=gen)
    views = _views(flats, specs)
    for s, v in zip(specs, views):
        r = workloads.RADIUS[s.stencil]
        v[:r] = 0
        v[-r:] = 0
        v[:, :r] = 0
        v[:, -r:] = 0
    return specs, flats, views


def _pinned(shape):
    return torch.zeros(shape, dtype=torch.float32, pin_memory=True)


def _room(spec):
    return -(-spec.ny * spec.nx // 64) * 64


def _views(flats, specs):
    out, at = [], dict.fromkeys(flats, 0)
    for s in specs:
        a = at[s.precision]
        out.append(flats[s.precision][a:a + s.ny * s.nx].view(s.ny, s.nx))
        at[s.precision] = a + _room(s)
    return out


# ----------------------------------------------------------------- the work --
def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        specs, flats, views = _mixed_inputs(case, seed)
        b = tcs.Batch()
        for s in specs:
            b.add(s.ny, s.nx, s.stencil, s.coeffs, s.steps, s.precision)
        out = {k: torch.zeros_like(f) for k, f in flats.items()}
        state = dict(kind=kind, batch=b, grids=views, out=out, outs=_views(out, specs))
        b.upload(0, views[0])  # allocates the batch's planes
        return state
    if kind == "serve":
        specs, flats, _ = _mixed_inputs(case, seed)
        h_in = {k: _pinned(f.shape) for k, f in flats.items()}
        out = {k: _pinned(f.shape) for k, f in flats.items()}
        for k, f in flats.items():
            h_in[k].copy_(f)
        server = tcs.Server(8 << 30)
        reqs = [(a.numpy(), b.numpy(), s.stencil, s.coeffs, s.steps, s.precision)
                for a, b, s in zip(_views(h_in, specs), _views(out, specs), specs)]
        return dict(kind=kind, server=server, reqs=reqs, out=out, h_in=h_in)
    border = workloads.RADIUS[case["stencil"]]
    grid = _grid(case["values"], case["ny"], case["nx"], border, seed)
    coeffs = _coeffs(case["stencil"], seed)
    if kind == "host":
        h_in, h_out = _pinned(grid.shape), _pinned(grid.shape)
        h_in.copy_(grid)
        return dict(kind=kind, case=case, h_in=h_in.numpy(), h_out=h_out.numpy(), held=(h_in, h_out), coeffs=coeffs)
    plan = tcs.Plan(case["ny"], case["nx"], case["stencil"], coeffs, engine=case["engine"], precision=case["precision"])
    return dict(kind=kind, plan=plan, grid=grid, out=torch.empty_like(grid), steps=case["steps"])


def run(state):
    kind = state["kind"]
    if kind == "solve":
        p = state["plan"]
        p.upload(state["grid"])
        p.run(state["steps"])
        p.download(state["out"])
        return state["out"]
    if kind == "host":
        c = state["case"]
        return tcs.sweep_host(state["h_in"], c["steps"], c["stencil"], state["coeffs"], engine=c["engine"],
                              precision=c["precision"], h_out=state["h_out"])
    if kind == "batch":
        b = state["batch"]
        for i, g in enumerate(state["grids"]):
            b.upload(i, g)
        b.run()
        for i, o in enumerate(state["outs"]):
            b.download(i, o)
        return state["out"]
    server = state["server"]
    tickets = [server.submit(a, b, stencil, coeffs, steps, precision)
               for a, b, stencil, coeffs, steps, precision in state["reqs"]]
    for t in tickets:
        server.wait(t)
    return state["out"]


# ----------------------------------------------------------- what is needed --
def _updates(ny, nx, stencil, steps):
    r = workloads.RADIUS[stencil]
    return (ny - 2 * r) * (nx - 2 * r) * steps


def work(case):
    """Each FP32 grid read once and written once; two operations a tap."""
    if case["kind"] in ("batch", "serve"):
        specs = _specs(case)
    else:
        specs = [workloads.GridSpec(0, case["stencil"], case["precision"], case["ny"], case["nx"], case["steps"], None)]
    return {"bytes": sum(8 * s.ny * s.nx for s in specs),
            "flops": sum(FLOPS[s.stencil] * _updates(s.ny, s.nx, s.stencil, s.steps) for s in specs)}


# -------------------------------------------------------------- in 64 bits --
def _sweep64(grid, stencil, coeffs, steps):
    """`steps` Jacobi steps of an FP32 grid in FP64; the border stays."""
    r = workloads.RADIUS[stencil]
    ny, nx = grid.shape
    star = stencil.startswith("star")
    taps = [(dy, dx, float(coeffs[dy, dx])) for dy in range(2 * r + 1) for dx in range(2 * r + 1)
            if not star or dy == r or dx == r]
    a = grid.double()
    b = a.clone()
    for _ in range(steps):
        acc = b[r:ny - r, r:nx - r]
        acc.zero_()
        for dy, dx, c in taps:
            acc.add_(a[dy:dy + ny - 2 * r, dx:dx + nx - 2 * r], alpha=c)
        a, b = b, a
    return a


def exact(case, seed):
    if case["kind"] in ("batch", "serve"):
        specs, flats, views = _mixed_inputs(case, seed)
        out = {k: torch.zeros(f.shape, dtype=torch.float64, device="cuda") for k, f in flats.items()}
        for s, v, o in zip(specs, views, _views(out, specs)):
            o.copy_(_sweep64(v, s.stencil, s.coeffs, s.steps))
        return out
    grid = _grid(case["values"], case["ny"], case["nx"], workloads.RADIUS[case["stencil"]], seed)
    return _sweep64(grid, case["stencil"], _coeffs(case["stencil"], seed), case["steps"])
