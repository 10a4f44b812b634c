"""Performance cases of the framework: what a user's program has it do, through its public entry points.

Kinds of case:

* ``map``, ``reduce``, ``matmul``: Sarek kernels in IR text, launched with ``run_vectors`` on vectors that are already on
  the device (left there by an earlier launch), in the default numeric mode;
* ``gemm``: the direct operator ``sb200_gemm_f32`` on the caller's device matrices, with the numeric mode, strides and
  epilogue the caller chooses;
* ``host``: a matmul kernel whose operands are in host memory and whose result is read on the host.

``listed`` gives the fixed cases, ``draw`` one more case of the same ranges, ``prepare`` what the program holds before
the call, ``run`` one pass, ``work`` the bytes and operations a pass cannot do without, ``tolerance`` how far another
correct implementation may be off.
"""
from __future__ import annotations

import sys

import numpy as np
import torch

from spoc_b200 import Backend, Vector, _lib as L, dims1d, dims2d, run_vectors, sarek_ir

MODES = {"3xtf32": L.MODE_3XTF32, "tf32": L.MODE_TF32, "3xmixed": L.MODE_3XMIXED, "3xf16": L.MODE_3XF16, "f16": L.MODE_F16}
MAX_MACS = 65536 * 4096 * 4096      # the largest product of the listed cases
EPILOGUE = dict(alpha=1.5, beta=0.5, c="c", bias="bias", relu=True)


def listed() -> list[dict]:
    return [
        # STREAM triad at the size the benchmark driver takes by default: one short launch, most of it latency
        {"name": "triad_1e6", "kind": "map", "op": "triad", "n": 1000000},
        # the fused two-kernel chain over vectors far larger than L2: HBM bandwidth
        {"name": "chain_2p28", "kind": "map", "op": "chain", "n": 1 << 28},
        # a user's own element-wise kernel (three inputs, two outputs, division, square root, a branch), odd length
        {"name": "generic_map_1e7", "kind": "map", "op": "generic", "n": 10000019},
        # dot product of two long vectors, one partial sum per block of 256, ragged last block
        {"name": "dot_5e7", "kind": "reduce", "op": "dot", "n": 50000017},
        # the smallest product: 64 x 64 x 64, the 4096-element size the tiled benchmark is run at
        {"name": "matmul_64", "kind": "matmul", "form": "tiled", "m": 64, "n": 64, "k": 64, "epilogue": False},
        # the ordinary product of the benchmarks
        {"name": "matmul_1024", "kind": "matmul", "form": "tiled", "m": 1024, "n": 1024, "k": 1024, "epilogue": False},
        # a ragged product: no dimension a multiple of 4, so that no row starts on a 16-byte boundary
        {"name": "matmul_ragged", "kind": "matmul", "form": "naive", "m": 1531, "n": 2047, "k": 1021, "epilogue": False},
        # a large product with the fused epilogue (scaling, accumulated matrix, bias, clamp)
        {"name": "matmul_8192_epilogue", "kind": "matmul", "form": "tiled", "m": 8192, "n": 8192, "k": 8192, "epilogue": True},
        # a few rows against a large matrix (a small batch through one layer), TF32, bias and clamp: B is read once
        {"name": "gemm_64_rows_tf32", "kind": "gemm", "mode": "tf32", "m": 64, "n": 4096, "k": 4096, "pad": 0, "data": "uniform",
         "epilogue": True},
        # a mid-size product in the half-precision three-term split
        {"name": "gemm_2048_3xf16", "kind": "gemm", "mode": "3xf16", "m": 2048, "n": 2048, "k": 2048, "pad": 0, "data": "uniform",
         "epilogue": True},
        # many rows against a square matrix, normally distributed operands, the mixed mode
        {"name": "gemm_skinny_mixed", "kind": "gemm", "mode": "3xmixed", "m": 65536, "n": 4096, "k": 4096, "pad": 0, "data": "normal",
         "epilogue": False},
        # host to host: new operands in host memory, launch, result read on the host
        {"name": "host_matmul_2048", "kind": "host", "m": 2048, "n": 2048, "k": 2048},
    ]


def _log(rng, low: float, high: float) -> int:
    return int(round(low * (high / low) ** rng.random()))


def _dims(rng, low: int, high: int, limit: int) -> tuple[int, int, int]:
    """Three dimensions, half of the time multiples of 32, else as they fall; their product at most `limit`."""
    while True:
        m, n, k = (_log(rng, low, high) for _ in range(3))
        if rng.random() < 0.5:
            m, n, k = ((d + 31) // 32 * 32 for d in (m, n, k))
        if m * n * k <= limit:
            return m, n, k


def draw(rng) -> dict:
    kind = rng.choice(("map", "map", "reduce", "matmul", "matmul", "gemm", "gemm", "gemm", "host"))
    if kind == "map":
        return {"kind": "map", "op": rng.choice(("vector_add", "triad", "chain", "generic")), "n": _log(rng, 1000, 1 << 28)}
    if kind == "reduce":
        return {"kind": "reduce", "op": rng.choice(("sum", "dot")), "n": _log(rng, 1000, 1 << 28)}
    if kind == "matmul":
        m, n, k = _dims(rng, 16, 8192, MAX_MACS)
        return {"kind": "matmul", "form": rng.choice(("naive", "tiled")), "m": m, "n": n, "k": k, "epilogue": rng.random() < 0.5}
    if kind == "gemm":
        m, n, k = _dims(rng, 16, 16384, MAX_MACS)
        return {"kind": "gemm", "mode": rng.choice(tuple(MODES)), "m": m, "n": n, "k": k, "pad": rng.choice((0, 0, 8, 3)),
                "data": rng.choice(("uniform", "normal")), "epilogue": rng.random() < 0.5}
    m, n, k = _dims(rng, 64, 4096, 4096 ** 3)
    return {"kind": "host", "m": m, "n": n, "k": k}


# ------------------------------------------------------------------ state
_backend: Backend | None = None


def _ready() -> tuple[Backend, object]:
    global _backend
    if _backend is None:
        _backend = Backend()
        _backend.Device.init()
    dev = _backend.Device.get(0)
    _backend.Device.set_current(dev)
    return _backend, dev


class _Resident:
    """A vector whose valid copy is on the device, as after a launch that wrote it, and a torch view of that copy."""

    def __init__(self, n: int):
        backend, dev = _ready()
        self.vector = Vector(backend, np.empty(n, dtype=np.float32))
        self.vector.buffer = backend.Memory.alloc(dev, n, np.float32)
        self.vector.location = Vector.STALE_CPU
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f4", "data": (self.vector.buffer.ptr, False), "version": 2}

    def __del__(self):
        if not sys.is_finalizing():
            self.vector.free()


def _resident(n: int) -> tuple[Vector, torch.Tensor]:
    holder = _Resident(n)
    view = torch.as_tensor(holder, device="cuda")    # keeps the holder, and with it the buffer
    return holder.vector, view.zero_()


def _generator(seed: int) -> torch.Generator:
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _vectors(g: torch.Generator, counts, random) -> tuple[list[Vector], list[torch.Tensor]]:
    vecs, views = [], []
    for n, filled in zip(counts, random):
        v, t = _resident(n)
        if filled:
            t.uniform_(-1.0, 1.0, generator=g)
        vecs.append(v)
        views.append(t)
    return vecs, views


def _launch(case: dict, ir: str, vecs, views, scalars, block, grid, outputs) -> dict:
    backend, dev = _ready()
    torch.cuda.synchronize()        # the vectors' contents are there for whichever stream uses them
    return {"kind": case["kind"], "backend": backend, "device": dev, "ir": ir, "args": list(vecs) + scalars, "views": views,
            "block": block, "grid": grid, "out": [views[i] for i in outputs]}


def _matmul_launch(form: str, m: int, n: int):
    if form == "tiled":
        return dims2d(16, 16), dims2d((n + 15) // 16, (m + 15) // 16)
    return dims1d(256), dims1d((m * n + 255) // 256)


def prepare(case: dict, seed: int) -> dict:
    kind, g = case["kind"], _generator(seed)
    if kind == "map":
        n, op = case["n"], case["op"]
        block, grid = dims1d(256), dims1d((n + 255) // 256)
        if op == "vector_add":
            vecs, views = _vectors(g, [n] * 3, (True, True, False))
            return _launch(case, sarek_ir.vector_add_ir(), vecs, views, [("int32", n)], block, grid, [2])
        if op == "triad":
            vecs, views = _vectors(g, [n] * 3, (False, True, True))
            return _launch(case, sarek_ir.stream_triad_ir(), vecs, views, [("float32", 3.0), ("int32", n)], block, grid, [0])
        if op == "chain":       # the fused chain has no guard: the vectors are padded to whole blocks
            padded = grid.x * block.x
            vecs, views = _vectors(g, [padded] * 3, (False, True, True))
            return _launch(case, sarek_ir.chain_fused_ir(3.0), vecs, views, [], block, grid, [0])
        vecs, views = _vectors(g, [n] * 5, (False, False, True, True, True))
        return _launch(case, sarek_ir.generic_example_ir(), vecs, views, [("float32", 1.25), ("int32", n)], block, grid, [0, 1])
    if kind == "reduce":
        n, inputs = case["n"], 2 if case["op"] == "dot" else 1
        blocks = (n + 255) // 256
        vecs, views = _vectors(g, [n] * inputs + [blocks], [True] * inputs + [False])
        return _launch(case, sarek_ir.block_reduce_ir(case["op"], 256), vecs, views, [("int32", n)], dims1d(256), dims1d(blocks),
                       [inputs])
    m, n, k = case["m"], case["n"], case["k"]
    if kind == "matmul":
        epilogue = EPILOGUE if case["epilogue"] else None
        ir = (sarek_ir.matmul_tiled_ir if case["form"] == "tiled" else sarek_ir.matmul_naive_ir)(epilogue=epilogue)
        counts = [m * k, k * n, m * n] + ([n, m * n] if epilogue else [])
        vecs, views = _vectors(g, counts, (True, True, True, True, False) if epilogue else (True, True, False))
        block, grid = _matmul_launch(case["form"], m, n)
        return _launch(case, ir, vecs, views, [("int32", m), ("int32", n), ("int32", k)], block, grid, [len(counts) - 1])
    if kind == "gemm":
        _ready()
        pad = case["pad"]

        def matrix(rows, cols, scale=1.0):
            t = torch.empty(rows, cols + pad, device="cuda")
            if case["data"] == "normal":
                return t.normal_(0.0, scale, generator=g)
            return t.uniform_(-1.0, 1.0, generator=g)

        a, b = matrix(m, k), matrix(k, n, k ** -0.5)
        c, bias = (matrix(m, n), matrix(1, n)) if case["epilogue"] else (None, None)
        d = torch.zeros(m, n + pad, device="cuda")
        torch.cuda.synchronize()
        return {"kind": kind, "lib": L.load(), "mode": MODES[case["mode"]], "m": m, "n": n, "k": k, "a": a, "b": b, "c": c, "bias": bias,
                "d": d}
    backend, dev = _ready()
    host = [torch.empty(count, device="cuda").uniform_(-1.0, 1.0, generator=g).cpu().numpy() for count in (m * k, k * n)]
    vecs = [Vector(backend, host[0]), Vector(backend, host[1]), Vector.create(backend, m * n)]
    block, grid = _matmul_launch("tiled", m, n)
    return {"kind": kind, "backend": backend, "device": dev, "ir": sarek_ir.matmul_tiled_ir(), "block": block, "grid": grid,
            "vectors": _HostVectors(vecs), "args": vecs + [("int32", m), ("int32", n), ("int32", k)]}


class _HostVectors:
    """Gives the vectors' device buffers back when the program is done with them."""

    def __init__(self, vecs):
        self.vecs = vecs

    def __del__(self):
        if not sys.is_finalizing():
            for v in self.vecs:
                v.free()


def run(state: dict):
    if state["kind"] == "gemm":
        a, b, c, bias, d = state["a"], state["b"], state["c"], state["bias"], state["d"]
        rc = state["lib"].sb200_gemm_f32(0, 0, state["mode"], state["m"], state["n"], state["k"], a.data_ptr(), a.stride(0),
                                         b.data_ptr(), b.stride(0), d.data_ptr(), d.stride(0), 1.5 if c is not None else 1.0,
                                         c.data_ptr() if c is not None else 0, c.stride(0) if c is not None else 0,
                                         0.5 if c is not None else 0.0, bias.data_ptr() if bias is not None else 0,
                                         L.ACT_RELU if c is not None else L.ACT_NONE)
        if rc != 0:
            raise RuntimeError(state["lib"].sb200_last_error_string().decode())
        return d
    if state["kind"] == "host":
        a, b, d = state["args"][:3]
        a.location = b.location = Vector.CPU        # the program has put new operands into the host arrays
        run_vectors(state["backend"], device=state["device"], ir=state["ir"], args=state["args"], block=state["block"],
                    grid=state["grid"])
        return d.to_array()
    run_vectors(state["backend"], device=state["device"], ir=state["ir"], args=state["args"], block=state["block"],
                grid=state["grid"])
    return state["out"]


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "map":
        vectors, flops = {"vector_add": (3, 1), "triad": (3, 2), "chain": (3, 4), "generic": (5, 9)}[case["op"]]
        return {"bytes": 4.0 * vectors * case["n"], "flops": float(flops * case["n"])}
    if kind == "reduce":
        inputs = 2 if case["op"] == "dot" else 1
        return {"bytes": 4.0 * (inputs * case["n"] + (case["n"] + 255) // 256), "flops": float(inputs * case["n"])}
    m, n, k = case["m"], case["n"], case["k"]
    extra = m * n + n if case.get("epilogue") else 0
    return {"bytes": 4.0 * (m * k + k * n + m * n + extra), "flops": 2.0 * m * n * k}


def tolerance(case: dict) -> dict:
    kind = case["kind"]
    if kind in ("map", "reduce"):       # at most one rounding of a float32 apart
        return {"rel": 1e-6, "max": 1e-6}
    if case.get("mode") in ("tf32", "f16"):     # operands rounded to 11 significant bits
        return {"rel": 5e-4, "max": 5e-3}
    # float32 sums in the tensor core's accumulator, which truncates: the loss grows with the number of terms and is 7e-9 of
    # the result per term against a float64 product, for terms of random sign
    rel = 1e-5 + 1e-8 * case["k"]
    return {"rel": rel, "max": 8 * rel}
