"""Timed cases of the dataflow hot path, through the package's public entry points.

A case is a dict of plain values; `op` says which entry point it takes:

  tile     one heat tile task as its own launch (heat_tile)
  step     one whole Jacobi step (heat_step)
  axpby    y = a*x + b*y over whole vectors (axpby)
  graph    a resolved heat graph on the persistent scheduler (Scheduler.run, or run_periodic
           with a two-step window), one pass = every step of the graph
  chain    chunked axpby passes with moving chunk boundaries, resolved from their segment
           accesses, on the persistent scheduler
  resolve  dependency resolution of a batch of matrix accesses (Resolver.add + graph) on a
           resolver that is reset and reused, as a runtime does between waits
  program  resolve a heat graph, hand its tasks over and run it (Resolver + Scheduler), as a
           program does for a graph it has not run before
  serve    a closed-loop batch of heat requests with host inputs and results (Server.run)
"""
import math

import numpy as np
import torch

import xkaapi_b200 as xk
from xkaapi_b200.heat import ACCESS_REC

COEF = 0.2                       # diffusion coefficient of every heat case (stable: <= 0.25)
AX, BY = 0.75, 0.25              # axpby scalars: repeated passes stay bounded
EDGES_PER_TASK = 64              # room for the successor list of a `resolve` case


# ---- the cases -----------------------------------------------------------------------------
def listed():
    return [
        # the smallest call: a program's own per-task launch of one 128 x 128 tile
        {"name": "tile-f64-128", "op": "tile", "nx": 1024, "ny": 1024, "ld": 1024, "tsx": 128, "tsy": 128, "f32": False},
        # the fused form of one step on the headline grid
        {"name": "step-f64-16384", "op": "step", "nx": 16384, "ny": 16384, "ld": 16384, "f32": False},
        # a step on a ragged FP32 grid, whose odd leading dimension rules out aligned vectors
        {"name": "step-f32-ragged", "op": "step", "nx": 5003, "ny": 4001, "ld": 5003, "f32": True},
        # the axpby body on long vectors of an odd length
        {"name": "axpby-100M", "op": "axpby", "n": 100_000_007, "shift": 0},
        # 10 axpby passes over one vector pair, chunks of 64 KiB to 16 MiB that move between passes
        {"name": "chain-64M", "op": "chain", "n": 1 << 26, "passes": 10, "min_chunk": 65536, "max_chunk": 1 << 24, "layout": 2026},
        # the small heat graph (6400 tile tasks): task latency counts, every grid fits in L2
        {"name": "graph-f64-1024", "op": "graph", "nx": 1024, "ny": 1024, "ld": 1024, "tsx": 128, "tsy": 128, "steps": 100,
         "f32": False, "periodic": False},
        # the headline grid and tile: 16,384 tasks per step streaming 4 GiB of grids
        {"name": "graph-f64-16384", "op": "graph", "nx": 16384, "ny": 16384, "ld": 16384, "tsx": 128, "tsy": 128, "steps": 20,
         "f32": False, "periodic": False},
        # FP32 storage with FP64 arithmetic, as a two-step window repeated
        {"name": "graph-f32-8192", "op": "graph", "nx": 8192, "ny": 8192, "ld": 8192, "tsx": 128, "tsy": 128, "steps": 50,
         "f32": True, "periodic": True},
        # ragged: sides that are no multiple of the tile, rectangular tiles, a partial last window
        {"name": "graph-f32-ragged", "op": "graph", "nx": 2500, "ny": 3100, "ld": 2500, "tsx": 90, "tsy": 150, "steps": 31,
         "f32": True, "periodic": True},
        # the dependency microbench: 65,536 tasks of 1-4 accesses on an 8192^2 matrix
        {"name": "resolve-65536", "op": "resolve", "tasks": 65536},
        # a mid-size graph met for the first time: resolve 10,240 tasks, then run them
        {"name": "program-f64-4096", "op": "program", "nx": 4096, "ny": 4096, "ld": 4096, "tsx": 128, "tsy": 128, "steps": 10,
         "f32": False},
        # a served batch: 24 graphs of mixed sizes, steps and storage types, host input and result
        {"name": "serve-24", "op": "serve", "requests": 24, "min_side": 256, "max_side": 2048, "max_steps": 100, "slots": 8,
         "layout": 7},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid(rng, lo, hi):
    """A grid: half of them multiples of 128, the rest any size, some with a padded column."""
    nx, ny = _log(rng, lo, hi), _log(rng, lo, hi)
    if rng.random() < 0.5:
        nx, ny = max(128, nx // 128 * 128), max(128, ny // 128 * 128)
    return {"nx": nx, "ny": ny, "ld": nx + rng.choice([0, 0, 0, 1, 4, 6])}


def draw(rng):
    op = rng.choice(["tile", "step", "axpby", "chain", "graph", "graph", "graph", "resolve", "program", "serve"])
    if op == "tile":
        return {"op": op, **_grid(rng, 256, 8192), "tsx": _log(rng, 16, 512), "tsy": _log(rng, 16, 512), "f32": rng.random() < 0.5}
    if op == "step":
        return {"op": op, **_grid(rng, 128, 16384), "f32": rng.random() < 0.5}
    if op == "axpby":
        return {"op": op, "n": _log(rng, 1000, 1 << 27), "shift": rng.choice([0, 0, 1])}
    if op == "chain":
        return {"op": op, "n": _log(rng, 1 << 20, 1 << 26), "passes": rng.randint(2, 10), "min_chunk": 65536,
                "max_chunk": 1 << rng.randint(18, 24), "layout": rng.randint(0, 9999)}
    if op == "resolve":
        return {"op": op, "tasks": _log(rng, 500, 65536)}
    if op == "serve":
        return {"op": op, "requests": rng.randint(4, 24), "min_side": 256, "max_side": 256 << rng.randint(0, 3),
                "max_steps": rng.randint(20, 100), "slots": rng.choice([4, 8, 16]), "layout": rng.randint(0, 9999)}
    # graph, program: square tiles of the autotuner's range, or ragged ones; at most about 330,000
    # tasks and the bytes of the largest listed graph
    g = _grid(rng, 256, 8192)
    t = rng.choice([64, 128, 128, 256, 0])
    tsx, tsy = (t, t) if t else (rng.randint(48, 200), rng.randint(48, 200))
    if g["nx"] % tsx == 1:                   # a tile of boundary cells only has no destination access
        g["nx"], g["ld"] = g["nx"] + 1, g["ld"] + 1
    if g["ny"] % tsy == 1:
        g["ny"] += 1
    steps = rng.randint(2, 100) if op == "graph" else rng.randint(2, 20)
    cap = 327680 if op == "graph" else 40960
    steps = max(2, min(steps, cap // (-(-g["nx"] // tsx) * -(-g["ny"] // tsy)), 20 * 16384 ** 2 // (g["nx"] * g["ny"])))
    case = {"op": op, **g, "tsx": tsx, "tsy": tsy, "steps": steps, "f32": rng.random() < 0.5}
    if op == "graph":
        case["periodic"] = rng.random() < 0.3
    return case


# ---- inputs --------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _heat_grid(case, seed):
    """U[0, 1) interior, zero boundary; column-major with leading dimension ld (columns are rows of
    the tensor), as the heat example initialises it."""
    nx, ny, ld = case["nx"], case["ny"], case["ld"]
    dtype = torch.float32 if case["f32"] else torch.float64
    g = torch.rand((ny, ld), dtype=dtype, device="cuda", generator=_gen(seed))
    g[0, :] = 0
    g[ny - 1, :] = 0
    g[:, 0] = 0
    g[:, nx - 1:] = 0
    return g


def _vectors(case, seed):
    gen = _gen(seed)
    x = torch.rand(case["n"], dtype=torch.float64, device="cuda", generator=gen) - 0.5
    y = torch.rand(case["n"] + 1, dtype=torch.float64, device="cuda", generator=gen) - 0.5
    return x, y[case.get("shift", 0):][:case["n"]]


def _chunks(case):
    """(lo, hi) element ranges of every pass: log-uniform chunk sizes, so the boundaries move."""
    rng = np.random.default_rng(case["layout"])
    out = []
    for _ in range(case["passes"]):
        lo = 0
        while lo < case["n"]:
            size = math.exp(rng.uniform(math.log(case["min_chunk"]), math.log(case["max_chunk"])))
            hi = min(case["n"], lo + max(1, int(size) // 8))
            out.append((lo, hi))
            lo = hi
    return np.array(out, dtype=np.int64)


def _chain_records(chunks, x, y):
    """Segment accesses of the chain's tasks: R on the x chunk, RW on the y chunk."""
    recs = np.zeros(2 * len(chunks), dtype=ACCESS_REC)
    recs["task"] = np.repeat(np.arange(len(chunks), dtype=np.uint32), 2)
    recs["type"] = 1
    for part, base, mode in ((recs[0::2], x, 1), (recs[1::2], y, 3)):
        part["mode"] = mode
        part["addr"] = base + 8 * chunks[:, 0]
        part["ld"] = base + 8 * chunks[:, 1]
    return recs


def _mixed_records(case, seed):
    """1-4 accesses per task on an 8192 x 8192 FP64 matrix: rectangles aligned to 64 elements with
    sides 64 * U{1..32}, modes R 60 %, W 20 %, RW 20 %."""
    rng = np.random.default_rng(seed)
    n, align = 8192, 64
    per_task = rng.integers(1, 5, case["tasks"])
    total, units = int(per_task.sum()), n // align
    m, k = rng.integers(1, 33, total), rng.integers(1, 33, total)
    mode = rng.integers(0, 10, total)
    recs = np.zeros(total, dtype=ACCESS_REC)
    recs["task"] = np.repeat(np.arange(case["tasks"], dtype=np.uint32), per_task)
    recs["type"] = 2
    recs["mode"] = np.where(mode < 6, 1, np.where(mode < 8, 2, 3))
    recs["addr"], recs["ld"], recs["sizeof_type"] = 1 << 40, n, 8
    recs["offset_m"] = (rng.random(total) * (units - m + 1)).astype(np.int64) * align
    recs["offset_n"] = (rng.random(total) * (units - k + 1)).astype(np.int64) * align
    recs["m"], recs["n"] = m * align, k * align
    return recs


def _serve_shapes(case):
    """(side, steps, f32) of every request: sides log-uniform, multiples of the 128 tile."""
    rng = np.random.default_rng(case["layout"])
    k = case["requests"]
    side = np.exp(rng.uniform(math.log(case["min_side"]), math.log(case["max_side"] + 1), k))
    side = np.clip(np.round(side / 128).astype(int) * 128, case["min_side"], case["max_side"])
    steps = rng.integers(10, case["max_steps"] + 1, k)
    return [(int(s), int(t), bool(i % 2)) for i, (s, t) in enumerate(zip(side, steps))]


def _heat_graph(case, a, b, steps):
    """A resolver, and the access records of `steps` steps on the grids a, b."""
    size = (case["nx"], case["ny"])
    recs = xk.heat_access_records(*size, case["tsx"], case["tsy"], 0, steps, a.data_ptr(), b.data_ptr(),
                                  esize=a.element_size(), ld=case["ld"])
    return xk.Resolver(), recs


def _heat_descs(case, a, b, steps):
    return xk.heat_task_descs((a.data_ptr(), b.data_ptr()), case["nx"], case["ny"], case["ld"], case["tsx"], case["tsy"], steps,
                              COEF, f32=case["f32"])


def prepare(case, seed):
    op = case["op"]
    state = {"case": case}
    if op in ("tile", "step"):
        a = _heat_grid(case, seed)
        state.update(src=a, dst=a.clone())
    elif op == "axpby":
        state["x"], state["y"] = _vectors(case, seed)
    elif op == "chain":
        x, y = state["x"], state["y"] = _vectors(case, seed)
        chunks = _chunks(case)
        descs = np.zeros(len(chunks), dtype=xk.axpby_desc_dtype())
        descs["kind"], descs["x"], descs["y"] = xk.TASK_AXPBY, x.data_ptr(), y.data_ptr()
        descs["lo"], descs["hi"], descs["a"], descs["b"] = chunks[:, 0], chunks[:, 1], AX, BY
        res, sch = xk.Resolver(), xk.Scheduler()
        res.add(_chain_records(chunks, x.data_ptr(), y.data_ptr()))
        sch.set_tasks(descs)
        state.update(res=res, sch=sch, graph=res.graph())
    elif op == "graph":
        a = _heat_grid(case, seed)
        b = a.clone()
        window = 2 if case["periodic"] else case["steps"]
        res, recs = _heat_graph(case, a, b, 6 if case["periodic"] else case["steps"])
        res.add(recs)
        sch = xk.Scheduler()
        sch.set_tasks(_heat_descs(case, a, b, window))
        per_step = len(recs) // 2 // (6 if case["periodic"] else case["steps"])
        state.update(a=a, b=b, res=res, sch=sch, per_step=per_step,
                     graph=res.periodic(2 * per_step) if case["periodic"] else res.graph())
    elif op == "resolve":
        state.update(res=xk.Resolver(), recs=_mixed_records(case, seed),
                     succ=torch.zeros(EDGES_PER_TASK * case["tasks"], dtype=torch.int32, device="cuda"))
    elif op == "program":
        a = _heat_grid(case, seed)
        b = a.clone()
        res, recs = _heat_graph(case, a, b, case["steps"])
        state.update(a=a, b=b, res=res, recs=recs, sch=xk.Scheduler(), descs=_heat_descs(case, a, b, case["steps"]))
    elif op == "serve":
        shapes = _serve_shapes(case)
        reqs = (xk.Request * len(shapes))()
        grids, results = [], []
        for k, (side, steps, f32) in enumerate(shapes):
            g = _heat_grid({"nx": side, "ny": side, "ld": side, "f32": f32}, seed * 1000 + k)
            grids.append(g.cpu().pin_memory())
            results.append(torch.zeros_like(grids[-1]).pin_memory())
            r = reqs[k]
            r.arrival_s, r.nx, r.ny, r.ts, r.steps, r.f32, r.c = 0.0, side, side, 128, steps, int(f32), COEF
            r.input, r.result = grids[-1].data_ptr(), results[-1].data_ptr()
        state.update(srv=xk.Server(budget_bytes=2 << 30, slots=case["slots"]), reqs=reqs, grids=grids, results=results)
    return state


# ---- one pass ------------------------------------------------------------------------------
class _DeviceArray:
    """A library-owned device array as a tensor, without a copy; keeps its owner alive."""

    def __init__(self, owner, ptr, n):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<i4", "data": (ptr, False), "version": 3}


def _view(owner, ptr, n):
    return torch.as_tensor(_DeviceArray(owner, ptr, n), device="cuda")


def run(state):
    case = state["case"]
    op = case["op"]
    if op == "tile":
        # a tile away from the grid's corner: halo cells on every side
        tx, ty = (case["nx"] // case["tsx"]) // 2, (case["ny"] // case["tsy"]) // 2
        xk.heat_tile(state["src"], state["dst"], case["nx"], case["ny"], case["ld"], tx, ty, case["tsx"], case["tsy"], COEF)
        return state["dst"]
    if op == "step":
        xk.heat_step(state["src"], state["dst"], case["nx"], case["ny"], case["ld"], COEF)
        return state["dst"]
    if op == "axpby":
        xk.axpby(AX, state["x"], BY, state["y"])
        return state["y"]
    if op == "chain":
        state["sch"].run(state["graph"])
        state["sch"].wait()
        return state["y"]
    if op == "graph":
        sch = state["sch"]
        if case["periodic"]:
            sch.run_periodic(state["graph"], (case["steps"] + 1) // 2, state["per_step"] * (1 if case["steps"] % 2 else 2))
        else:
            sch.run(state["graph"])
        sch.wait()
        return state["a"], state["b"]
    if op == "resolve":
        res = state["res"]
        res.reset()
        res.add(state["recs"])
        g = res.graph()
        state["succ"][:g.nedges].copy_(_view(res, g.succ, g.nedges))
        return _view(res, g.succ_ptr, g.ntasks + 1), _view(res, g.npred, g.ntasks), state["succ"]
    if op == "program":
        res, sch = state["res"], state["sch"]
        res.reset()
        res.add(state["recs"])
        sch.set_tasks(state["descs"])
        sch.run(res.graph())
        sch.wait()
        return state["a"], state["b"]
    if op == "serve":
        state["srv"].run(state["reqs"])
        return list(state["results"])
    raise ValueError(op)


# ---- what a pass cannot do without ---------------------------------------------------------
def work(case):
    """Each input read once and each output written once; 8 FP64 operations per cell and step."""
    op = case["op"]
    esz = 4 if case.get("f32") else 8
    if op == "tile":
        cells = min(case["tsx"], case["nx"] - 2) * min(case["tsy"], case["ny"] - 2)
        return {"bytes": 2 * esz * cells, "flops": 8 * cells}
    if op == "step":
        cells = (case["nx"] - 2) * (case["ny"] - 2)
        return {"bytes": 2 * esz * cells, "flops": 8 * cells}
    if op == "axpby":
        return {"bytes": 24 * case["n"], "flops": 3 * case["n"]}
    if op == "chain":
        return {"bytes": 24 * case["n"], "flops": 3 * case["n"] * case["passes"]}
    if op in ("graph", "program"):
        # one grid in, both grids out; a step's intermediate grid need not leave the chip
        cells = (case["nx"] - 2) * (case["ny"] - 2)
        tasks = -(-case["nx"] // case["tsx"]) * -(-case["ny"] // case["tsy"]) * case["steps"]
        return {"bytes": 3 * esz * cells + (192 * tasks if op == "program" else 0), "flops": 8 * cells * case["steps"]}
    if op == "resolve":
        # 2.5 accesses of 64 bytes in, about 20 successors of 4 bytes and two counts out per task
        return {"bytes": case["tasks"] * (160 + 80 + 8), "flops": 0}
    shapes = _serve_shapes(case)
    cells = [(s * s, t, 4 if f32 else 8) for s, t, f32 in shapes]
    return {"bytes": sum(2 * c * e for c, _, e in cells), "flops": sum(8 * c * t for c, t, _ in cells)}


# ---- the same results in 64 bits -----------------------------------------------------------
def _steps64(g, nx, ny, steps):
    """`steps` Jacobi steps of the grid in FP64: (grid after them, grid after one step fewer)."""
    a = g.double()
    b = a.clone()
    for _ in range(steps):
        s = a[1:ny - 1, 1:nx - 1]
        lap = (a[1:ny - 1, 2:nx] - 2.0 * s).add_(a[1:ny - 1, 0:nx - 2])
        lap.add_((a[2:ny, 1:nx - 1] - 2.0 * s).add_(a[0:ny - 2, 1:nx - 1]))
        torch.add(s, lap.mul_(COEF), out=b[1:ny - 1, 1:nx - 1])
        a, b = b, a
    return a, b


def exact(case, seed):
    op = case["op"]
    if op in ("tile", "step"):
        g = _heat_grid(case, seed)
        full, _ = _steps64(g, case["nx"], case["ny"], 1)
        if op == "step":
            return full
        out = g.double()
        x0 = (case["nx"] // case["tsx"]) // 2 * case["tsx"]
        y0 = (case["ny"] // case["tsy"]) // 2 * case["tsy"]
        x1, y1 = min(x0 + case["tsx"], case["nx"]), min(y0 + case["tsy"], case["ny"])
        out[y0:y1, x0:x1] = full[y0:y1, x0:x1]
        return out
    if op in ("axpby", "chain"):
        x, y = _vectors(case, seed)
        for _ in range(case.get("passes", 1)):
            y = AX * x + BY * y
        return y
    if op in ("graph", "program"):
        last, before = _steps64(_heat_grid(case, seed), case["nx"], case["ny"], case["steps"])
        return (last, before) if case["steps"] % 2 == 0 else (before, last)
    if op == "serve":
        out = []
        for k, (side, steps, f32) in enumerate(_serve_shapes(case)):
            g = _heat_grid({"nx": side, "ny": side, "ld": side, "f32": f32}, seed * 1000 + k)
            out.append(_steps64(g, side, side, steps)[0].cpu())
        return out
    return None                  # resolve: whole numbers
