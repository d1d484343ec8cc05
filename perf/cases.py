"""Performance cases: what a user of the framework has it do, timed through its public entry points.

A case is a dict of plain values. `listed()` gives the named ones, `draw(rng)` one more of the same
ranges, `prepare(case, seed)` the inputs, recorded chunks, batches and result buffers that a user's
program holds before the call, `run(state)` one pass (queued on the device's stream wherever the
entry point queues), `work(case)` the bytes and operations of one pass, and `exact(case, seed)` the
same outputs in 64 bits by plain torch.

Sizes and distributions are those of bench.py's workloads and of the tests (n = 1,021 up to 2^28
elements, products up to 8192^3, solves up to order 8192, batches of thousands of uneven items),
with odd and ragged sizes beside the round ones.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from libsci_b200 import chunk as C
from libsci_b200.device import Device, DeviceArray
from libsci_b200.native import SolveReport, check, lib

TORCH = {"float32": torch.float32, "float64": torch.float64, "int8": torch.int8, "int16": torch.int16,
         "int32": torch.int32, "int64": torch.int64, "uint8": torch.uint8}
SIZE = {"float32": 4, "float64": 8, "int8": 1, "int16": 2, "int32": 4, "int64": 8, "uint8": 1}

_held: dict = {}  # the process's device, and the programs whose specialised kernels are ready


def _device() -> Device:
    if "device" not in _held:
        _held["device"] = Device(0)
    return _held["device"]


def listed() -> list[dict]:
    return [
        # a script's small arrays: three calls on about a thousand elements, where each call's latency counts
        {"name": "expression_small", "kind": "expression", "dtype": "float32", "count": 1021},
        # large fused chunks: the streaming workload the backend exists for, 1 GiB per array
        {"name": "fused_large", "kind": "fused", "dtype": "float32", "count": 1 << 28, "holes": 1e-6},
        # the same chunks in double over a ragged mid-size array (simulation state, statistics)
        {"name": "fused_wide_ragged", "kind": "fused", "dtype": "float64", "count": 3000017, "holes": 0.0},
        # differentiation of a fused expression: loss gradients over 2^26 parameters
        {"name": "gradient_large", "kind": "gradient", "dtype": "float32", "count": 1 << 26},
        # integer arrays: counters and indices, stored and reduced
        {"name": "elements_int32_ragged", "kind": "elements", "dtype": "int32", "count": 100000007},
        # numpy-style tables: broadcasting against rows and columns, statistics along either axis
        {"name": "shapes_ragged", "kind": "shapes", "dtype": "float32", "rows": 5001, "columns": 7003},
        # a layer-like product with its adjoints, dimensions that fit no tile, FP32-accurate (the default mode)
        {"name": "product_ragged_training", "kind": "product", "dtype": "float32", "rows": 1000, "columns": 700,
         "depth": 1300, "mode": 3, "backward": True},
        # the large product on bf16 operands
        {"name": "product_large_bf16", "kind": "product", "dtype": "float32", "rows": 8192, "columns": 8192,
         "depth": 8192, "mode": 0, "backward": False},
        # a small linear system inside a differentiable program: solve, then its adjoint
        {"name": "solve_small_training", "kind": "solve", "dtype": "float64", "order": 200, "width": 3,
         "refine": True, "backward": True},
        # the large dense solve, FP32 factors refined to FP64
        {"name": "solve_large_refined", "kind": "solve", "dtype": "float64", "order": 8192, "width": 16,
         "refine": True, "backward": False},
        # many uneven expressions in one replayed launch
        {"name": "batch_uneven", "kind": "batch", "dtype": "float32", "items": 2048, "least": 256, "most": 1 << 20,
         "lengths": 0},
        # thousands of small systems in one replayed launch
        {"name": "solve_batch", "kind": "solve_batch", "systems": 4096, "least": 8, "most": 256, "lengths": 0},
    ]


def _log_int(rng, low: int, high: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _size(rng, low: int, high: int) -> int:
    """A size spread over its logarithm: odd as often as a multiple of 64."""
    n = _log_int(rng, low, high)
    return n | 1 if rng.random() < 0.5 else max(64, n // 64 * 64)


def draw(rng) -> dict:
    kind = rng.choice(["expression", "fused", "gradient", "elements", "shapes", "product", "solve", "batch",
                       "solve_batch"])
    if kind == "expression":
        return {"kind": kind, "dtype": rng.choice(["float32", "float64"]), "count": _size(rng, 256, 1 << 22)}
    if kind == "fused":
        dtype = rng.choice(["float32", "float32", "float64"])
        return {"kind": kind, "dtype": dtype, "count": _size(rng, 1 << 20, 1 << (28 if dtype == "float32" else 25)),
                "holes": 0.0}
    if kind == "gradient":
        dtype = rng.choice(["float32", "float32", "float64"])
        return {"kind": kind, "dtype": dtype, "count": _size(rng, 1 << 14, 1 << (26 if dtype == "float32" else 24))}
    if kind == "elements":
        dtype = rng.choice(["int8", "int16", "int32", "int64", "uint8"])
        return {"kind": kind, "dtype": dtype, "count": _size(rng, 1 << 16, (1 << 29) // SIZE[dtype])}
    if kind == "shapes":
        return {"kind": kind, "dtype": rng.choice(["float32", "float32", "float64"]), "rows": _size(rng, 100, 10000),
                "columns": _size(rng, 100, 10000)}
    if kind == "product":
        dtype = rng.choice(["float32", "float32", "float32", "float64"])
        most = 4096 if dtype == "float32" else 2048
        return {"kind": kind, "dtype": dtype, "rows": _size(rng, 64, most), "columns": _size(rng, 64, most),
                "depth": _size(rng, 64, most), "mode": rng.choice([3, 3, 1, 0]) if dtype == "float32" else 2,
                "backward": rng.random() < 0.5}
    if kind == "solve":
        dtype = rng.choice(["float64", "float64", "float64", "float32"])
        refine = dtype == "float64" and rng.random() < 0.7
        return {"kind": kind, "dtype": dtype, "order": _size(rng, 16, 4096 if refine else 2048),
                "width": rng.choice([1, 1, 3, 16, 64]), "refine": refine, "backward": rng.random() < 0.4}
    if kind == "batch":
        most = rng.choice([4096, 65536, 1 << 20])
        return {"kind": kind, "dtype": rng.choice(["float32", "float32", "float64"]),
                "items": _log_int(rng, 64, 1024 if most == 1 << 20 else 4096), "least": 256, "most": most,
                "lengths": rng.randrange(1 << 20)}
    least = rng.choice([4, 8, 32])
    return {"kind": kind, "systems": _log_int(rng, 64, 4096), "least": least,
            "most": rng.choice([48, 96, 128, 200, 256]), "lengths": rng.randrange(1 << 20)}


# ---- inputs ---------------------------------------------------------------------------------------


def _generator(seed: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _normal(shape, dtype, g):
    return torch.randn(shape, generator=g, device="cuda", dtype=TORCH[dtype])


def _uniform(shape, low, high, dtype, g):
    return torch.rand(shape, generator=g, device="cuda", dtype=TORCH[dtype]) * (high - low) + low


def _uneven(case):
    """The lengths of a batch's items: log-uniform in [least, most], the same for every seed of the inputs."""
    rng = np.random.default_rng(case["lengths"])
    return np.exp(rng.uniform(math.log(case["least"]), math.log(case["most"]), case["items"])).astype(np.int64)


def _orders(case):
    """The orders of a batch's systems: uniform in [least, most], the same for every seed of the inputs."""
    return np.random.default_rng(case["lengths"]).integers(case["least"], case["most"] + 1, case["systems"])


def _inputs(case: dict, seed: int) -> dict:
    """The case's input tensors, from the seed alone."""
    g, kind, dtype = _generator(seed), case["kind"], case.get("dtype", "float64")
    if kind == "expression":
        n = case["count"]
        return {"a": torch.linspace(0, 1, n, device="cuda", dtype=TORCH[dtype]), "b": _uniform(n, -1.0, 1.0, dtype, g),
                "c": torch.ones(n, device="cuda", dtype=TORCH[dtype])}
    if kind == "fused":
        n = case["count"]
        x, y, z = _normal(n, dtype, g), _uniform(n, 0.1, 10.0, dtype, g), _uniform(n, -1.0, 1.0, dtype, g)
        if case["holes"] > 0:
            z[torch.randint(0, n, (max(1, int(n * case["holes"])),), generator=g, device="cuda")] = math.nan
        return {"x": x, "y": y, "z": z}
    if kind == "gradient":
        return {k: _normal(case["count"], dtype, g) for k in "abc"}
    if kind == "elements":
        high = min(torch.iinfo(TORCH[dtype]).max, 1 << 20)
        low = 1 if dtype == "uint8" else -high
        made = {k: torch.randint(low, high, (case["count"],), generator=g, device="cuda", dtype=TORCH[dtype]) for k in "abc"}
        made["b"] = torch.where(made["b"] == 0, torch.ones_like(made["b"]), made["b"])  # a divisor
        return made
    if kind == "shapes":
        r, c = case["rows"], case["columns"]
        return {"x": _normal((r, c), dtype, g), "y": _uniform((r, c), -2.0, 2.0, dtype, g),
                "column": _normal((r, 1), dtype, g).round(), "row": _normal((1, c), dtype, g)}
    if kind == "product":
        m, n, k = case["rows"], case["columns"], case["depth"]
        made = {"left": _uniform((m, k), -1.0, 1.0, dtype, g), "right": _uniform((k, n), -1.0, 1.0, dtype, g)}
        if case["backward"]:
            made["upstream"] = _normal((m, n), dtype, g)
        return made
    if kind == "solve":
        n, w = case["order"], case["width"]
        a = _normal((n, n), dtype, g)
        a.diagonal().add_(float(n))
        made = {"matrix": a, "right": _normal((n, w), dtype, g)}
        if case["backward"]:
            made["upstream"] = _normal((n, w), dtype, g)
        return made
    if kind == "batch":
        counts = _uneven(case)
        offsets = np.concatenate([[0], np.cumsum((counts + 63) // 64 * 64)])  # items as separate allocations lie
        return {"counts": counts, "offsets": offsets, **{k: _normal(int(offsets[-1]), dtype, g) for k in "abc"}}
    orders = _orders(case)
    matrices = _normal(int((orders * orders).sum()), "float64", g)
    starts = np.concatenate([[0], np.cumsum(orders * orders)])
    at = np.concatenate([s + np.arange(n) * (n + 1) for s, n in zip(starts, orders)])
    add = np.repeat(orders.astype(np.float64), orders)
    matrices[torch.from_numpy(at).cuda()] += torch.from_numpy(add).cuda()
    return {"orders": orders, "starts": starts, "matrices": matrices, "rights": _normal(int(orders.sum()), "float64", g)}


def _on_device(tensor) -> DeviceArray:
    """The framework's array over memory that the program holds."""
    name = str(tensor.dtype).replace("torch.", "")
    return DeviceArray(_device(), tensor.data_ptr(), tensor.numel(), np.dtype(name))


def _batch_chunk(precision: int) -> C.Chunk:
    """t = a*b + c stored and tanh(t) reduced in one chunk."""
    chunk = C.Chunk(precision)
    chunk.arguments, chunk.temporaries, chunk.length = 3, 2, 3
    for index, (code, target, sources) in enumerate((
            ("fuse", C.TEMPORARY | 0, (0, 1, 2)),
            ("copy", C.OUTPUT, (C.TEMPORARY | 0, C.NONE, C.NONE)),
            ("tanh", C.TEMPORARY | 1, (C.TEMPORARY | 0, C.NONE, C.NONE)))):
        ins = chunk.instructions[index]
        ins.code, ins.target = C.CODE[code], target
        ins.sources[0], ins.sources[1], ins.sources[2] = sources
    chunk.result = C.TEMPORARY | 1
    return chunk


class _Held:
    """A batch handle that is given back with the state that holds it."""

    def __init__(self, batch):
        self.batch = batch

    def __del__(self):
        self.batch.close()


def prepare(case: dict, seed: int) -> dict:
    device, kind, dtype = _device(), case["kind"], case.get("dtype", "float64")
    state = {"case": case, **_inputs(case, seed)}
    like = lambda shape, dt=None: torch.empty(shape, device="cuda", dtype=TORCH[dt or dtype])  # noqa: E731
    if kind == "expression":
        a, b, c = (_on_device(state[k]).expression() for k in "abc")
        state["t"], state["e"] = like(case["count"]), like(case["count"])
        t = _on_device(state["t"]).expression()
        state["chunks"] = (C.record_output(a * b + c * 2.0), C.record_output(C.unary("exponential", t) * 0.5),
                           C.record_reduce(C.unary("sin", t)))
    elif kind == "fused":
        x, y, z = (_on_device(state[k]).expression() for k in "xyz")
        for name in ("stored", "lower", "upper"):
            state[name] = like(case["count"])
        state["chunks"] = {
            "stored": C.record_output(C.unary("root", C.unary("absolute", x)) * C.unary("logarithm", y) + C.unary("tanh", z)),
            "lower": C.record_output(C.binary("minimum", x, z)), "upper": C.record_output(C.binary("maximum", x, z)),
            "mean": C.record_reduce(C.unary("exponential", -x * x)),
            "peak": C.record_reduce(C.unary("sin", x) * C.unary("cos", z)), "dot": C.record_reduce(x * z)}
    elif kind == "gradient":
        a, b, c = (_on_device(state[k]).expression() for k in "abc")
        state["chunk"] = C.record_reduce(C.unary("exponential", -a * a) * C.unary("sin", b) + C.unary("logarithm", 1 + c * c))
        state["gradients"] = [like(case["count"]) for _ in range(3)]
        state["slots"] = (ctypes.c_void_p * 3)(*[t.data_ptr() for t in state["gradients"]])
    elif kind == "elements":
        a, b, c = (_on_device(state[k]).expression() for k in "abc")
        state["fused"], state["ratio"] = like(case["count"]), like(case["count"])
        state["chunks"] = (C.record_output(a * b + c), C.record_output(C.binary("maximum", a, c) / b),
                           C.record_reduce(a * b))
    elif kind == "shapes":
        r, c = case["rows"], case["columns"]
        state.update(outer=like((r, c)), chosen=like((r, c)), centred=like((r, c)), sums=like(c), means=like((r, 1)))
    elif kind == "product":
        m, n, k = case["rows"], case["columns"], case["depth"]
        state["out"] = like((m, n))
        if case["backward"]:
            state["left_gradient"], state["right_gradient"] = like((m, k)), like((k, n))
    elif kind == "solve":
        n, w = case["order"], case["width"]
        state["solution"], state["report"] = like((n, w)), SolveReport()
        if case["backward"]:
            state.update(again=like((n, w)), matrix_gradient=like((n, n)), right_gradient=like((n, w)))
    elif kind == "batch":
        size, counts = SIZE[dtype], state["counts"]
        starts = state["offsets"][:-1]
        state["t"] = torch.zeros(int(state["offsets"][-1]), device="cuda", dtype=TORCH[dtype])
        state["results"] = torch.zeros(case["items"], device="cuda", dtype=torch.float64)
        pointers = np.stack([state[k].data_ptr() + size * starts for k in "abc"], axis=1).astype(np.uint64)
        outputs = (state["t"].data_ptr() + size * starts).astype(np.uint64)
        torch.cuda.synchronize()  # the batch is tuned on these inputs as it is made
        state["held"] = _Held(device.batch(_batch_chunk(C.WIDE if dtype == "float64" else C.SINGLE), C.SUM, pointers,
                                           counts, outputs, _on_device(state["results"])))
    elif kind == "solve_batch":
        orders = state["orders"]
        state["solutions"] = torch.zeros(int(orders.sum()), device="cuda", dtype=torch.float64)
        state["errors"] = torch.zeros(len(orders), device="cuda", dtype=torch.float64)
        rows = np.concatenate([[0], np.cumsum(orders)])[:-1]
        pointers = [(state[k].data_ptr() + 8 * at).astype(np.uint64)
                    for k, at in (("matrices", state["starts"][:-1]), ("rights", rows), ("solutions", rows))]
        torch.cuda.synchronize()  # the batch is tuned on these inputs as it is made
        state["held"] = _Held(device.solve_batch(orders, *pointers, _on_device(state["errors"])))
    if kind in ("expression", "fused", "gradient") and (kind, dtype) not in _held:
        # a program's chunks run specialised kernels once these are compiled: wait for that once per program
        torch.cuda.synchronize()
        run(state)
        device.jit_wait()
        device.synchronize()
        _held[(kind, dtype)] = True
    return state


# ---- one pass -------------------------------------------------------------------------------------


def _broadcast(device, precision, code, shape, operands, out):
    """out = code(operands...) with numpy broadcasting, through the C ABI into memory the program holds."""
    number = C.EXTRA[code] if code in C.EXTRA else C.CODE[code]
    inputs = (ctypes.c_void_p * len(operands))(*[t.data_ptr() for t in operands])
    extents = (ctypes.c_uint64 * (2 * len(operands)))(*[e for t in operands for e in t.shape])
    check(lib.sci_cuda_broadcast(device.handle, precision, number, 2, (ctypes.c_uint64 * 2)(*shape), len(operands), inputs,
                                 extents, out.data_ptr()), device.handle)


def run(state: dict):
    case, device = state["case"], _device()
    kind = case["kind"]
    precision = C.WIDE if case.get("dtype") == "float64" else C.SINGLE
    if kind == "expression":
        n, (first, second, third) = case["count"], state["chunks"]
        device.execute(first, state["t"].data_ptr(), n)
        device.execute(second, state["e"].data_ptr(), n)
        return {"t": state["t"], "e": state["e"], "s": device.reduce_chunk(third, C.SUM, n)}
    if kind == "fused":
        n, chunks, out = case["count"], state["chunks"], {}
        for name in ("stored", "lower", "upper"):
            device.execute(chunks[name], state[name].data_ptr(), n)
            out[name] = state[name]
        out["mean"] = device.reduce_chunk(chunks["mean"], C.SUM, n) / n
        out["peak"] = device.reduce_chunk(chunks["peak"], C.MAXIMUM, n)
        out["dot"] = device.reduce_chunk(chunks["dot"], C.SUM, n)
        return out
    if kind == "gradient":
        value = ctypes.c_double()
        check(lib.sci_cuda_gradient(device.handle, ctypes.byref(state["chunk"]), case["count"], 1.0, state["slots"],
                                    ctypes.byref(value), 0), device.handle)
        return {"value": value.value, "gradients": state["gradients"]}
    if kind == "elements":
        n, dtype, (fused, ratio, total) = case["count"], case["dtype"], state["chunks"]
        device.execute_elements(dtype, fused, state["fused"].data_ptr(), n)
        device.execute_elements(dtype, ratio, state["ratio"].data_ptr(), n)
        return {"fused": state["fused"], "ratio": state["ratio"], "total": int(device.reduce_elements(dtype, total, C.SUM, n))}
    if kind == "shapes":
        x, y, column, row = (state[k] for k in ("x", "y", "column", "row"))
        full = tuple(x.shape)
        extents = (ctypes.c_uint64 * 2)(*full)
        check(lib.sci_cuda_reduce_axis(device.handle, precision, C.SUM, x.data_ptr(), 2, extents, 0,
                                       state["sums"].data_ptr()), device.handle)
        check(lib.sci_cuda_reduce_axis(device.handle, precision, C.AXIS_MEAN, x.data_ptr(), 2, extents, 1,
                                       state["means"].data_ptr()), device.handle)
        _broadcast(device, precision, "subtract", full, (x, state["means"]), state["centred"])
        _broadcast(device, precision, "add", full, (column, row), state["outer"])
        _broadcast(device, precision, "where", full, (column, x, y), state["chosen"])
        return {k: state[k] for k in ("sums", "means", "centred", "outer", "chosen")}
    if kind == "product":
        m, n, k = case["rows"], case["columns"], case["depth"]
        left, right, out = (_on_device(state[key]) for key in ("left", "right", "out"))
        device.product(left, right, m, n, k, case["mode"], out)
        made = {"out": state["out"]}
        if case["backward"]:
            check(lib.sci_cuda_product_gradient(device.handle, precision, case["mode"], left.pointer, right.pointer,
                                                state["upstream"].data_ptr(), state["left_gradient"].data_ptr(),
                                                state["right_gradient"].data_ptr(), m, n, k), device.handle)
            made.update(left_gradient=state["left_gradient"], right_gradient=state["right_gradient"])
        return made
    if kind == "solve":
        n, w = case["order"], case["width"]
        matrix, right, solution = (_on_device(state[key]) for key in ("matrix", "right", "solution"))
        device.solve(matrix, right, n, w, case["refine"], solution)
        made = {"solution": state["solution"]}
        if case["backward"]:
            check(lib.sci_cuda_solve_gradient(device.handle, precision, 1 if case["refine"] else 0, matrix.pointer,
                                              right.pointer, state["upstream"].data_ptr(), state["again"].data_ptr(),
                                              state["matrix_gradient"].data_ptr(), state["right_gradient"].data_ptr(), n, w,
                                              ctypes.byref(state["report"])), device.handle)
            made.update({k: state[k] for k in ("again", "matrix_gradient", "right_gradient")})
        return made
    state["held"].batch.launch()
    if kind == "batch":
        return {"t": state["t"], "results": state["results"]}
    return {"solutions": state["solutions"]}


# ---- what a pass cannot do without ------------------------------------------------------------------


def work(case: dict) -> dict:
    kind, size = case["kind"], SIZE[case.get("dtype", "float64")]
    if kind == "expression":  # a, b, c -> t; t -> e; t -> s
        return {"bytes": 7 * size * case["count"], "flops": 6 * case["count"]}
    if kind == "fused":  # 4 + 3 + 3 arrays touched by the stored chunks, 1 + 2 + 2 by the reductions
        return {"bytes": 15 * size * case["count"], "flops": 16 * case["count"]}
    if kind == "gradient":
        return {"bytes": 6 * size * case["count"], "flops": 20 * case["count"]}
    if kind == "elements":
        return {"bytes": 10 * size * case["count"], "flops": 6 * case["count"]}
    if kind == "shapes":
        r, c = case["rows"], case["columns"]
        return {"bytes": 8 * size * r * c + size * (4 * r + 2 * c), "flops": 5 * r * c}
    if kind == "product":
        m, n, k = case["rows"], case["columns"], case["depth"]
        passes = 3 if case["backward"] else 1
        return {"bytes": size * passes * (m * k + k * n + m * n), "flops": 2.0 * passes * m * n * k}
    if kind == "solve":
        n, w = case["order"], case["width"]
        one = {"bytes": size * (n * n + 2 * n * w), "flops": 2 / 3 * n ** 3 + 2.0 * n * n * w}
        if not case["backward"]:
            return one
        return {"bytes": 2 * one["bytes"] + size * (n * n + 2 * n * w), "flops": 2 * one["flops"] + 4.0 * n * n * w}
    if kind == "batch":
        mean = (case["most"] - case["least"]) / math.log(case["most"] / case["least"])
        return {"bytes": 4.0 * size * case["items"] * mean, "flops": 3.0 * case["items"] * mean}
    low, high = case["least"], case["most"]
    orders = np.arange(low, high + 1, dtype=np.float64)
    return {"bytes": float(case["systems"] * np.mean(8 * orders ** 2 + 16 * orders)),
            "flops": float(case["systems"] * np.mean(2 / 3 * orders ** 3 + 2 * orders ** 2))}


# ---- the outputs in 64 bits ---------------------------------------------------------------------------


def exact(case: dict, seed: int):
    kind, t = case["kind"], _inputs(case, seed)
    if kind == "elements":
        return None  # whole numbers
    wide = {k: v.double() for k, v in t.items() if isinstance(v, torch.Tensor)}
    if kind == "expression":
        out = wide["a"] * wide["b"] + wide["c"] * 2.0
        return {"t": out, "e": torch.exp(out) * 0.5, "s": float(torch.sin(out).sum())}
    if kind == "fused":
        x, y, z = wide["x"], wide["y"], wide["z"]
        return {"stored": x.abs().sqrt_().mul_(y.log()).add_(z.tanh()),
                # minimum and maximum give the right operand unless the left one is strictly better or NaN
                "lower": torch.where(x < z, x, z), "upper": torch.where(x > z, x, z),
                "mean": float(torch.exp(-x * x).sum()) / case["count"], "peak": float((x.sin() * z.cos()).max()),
                "dot": float((x * z).sum())}
    if kind == "gradient":
        a, b, c = wide["a"], wide["b"], wide["c"]
        e = torch.exp(-a * a)
        return {"value": float((e * b.sin() + torch.log1p(c * c)).sum()),
                "gradients": [-2.0 * a * e * b.sin(), e * b.cos(), 2.0 * c / (1.0 + c * c)]}
    if kind == "shapes":
        x, y, column, row = (wide[k] for k in ("x", "y", "column", "row"))
        means = x.mean(dim=1, keepdim=True)
        return {"sums": x.sum(dim=0), "means": means, "centred": x - means, "outer": column + row,
                "chosen": torch.where(column != 0, x, y)}
    if kind == "product":
        made = {"out": wide["left"] @ wide["right"]}
        if case["backward"]:
            made.update(left_gradient=wide["upstream"] @ wide["right"].T, right_gradient=wide["left"].T @ wide["upstream"])
        return made
    if kind == "solve":
        solution = torch.linalg.solve(wide["matrix"], wide["right"])
        made = {"solution": solution}
        if case["backward"]:
            adjoint = torch.linalg.solve(wide["matrix"].T, wide["upstream"])
            made.update(again=solution, right_gradient=adjoint, matrix_gradient=-adjoint @ solution.T)
        return made
    if kind == "batch":
        out = torch.addcmul(wide["c"], wide["a"], wide["b"])
        folded, spans = out.tanh(), list(zip(t["offsets"][:-1], t["counts"]))
        values = torch.zeros_like(out)
        for start, count in spans:
            values[start:start + count] = out[start:start + count]
        return {"t": values, "results": torch.stack([folded[s:s + n].sum() for s, n in spans])}
    solutions, row = [], 0
    for start, n in zip(t["starts"][:-1], t["orders"]):
        solutions.append(torch.linalg.solve(wide["matrices"][start:start + n * n].view(n, n), wide["rights"][row:row + n]))
        row += n
    return {"solutions": torch.cat(solutions)}
