"""The calls that stand for this library's use, for timing and comparison.

Every case is one call of a public entry point (opensycl_b200.capi, or the
C-ABI plan that a program with fixed segments keeps) on device data, with the
value distributions of the repository's benchmark and tests: uniform
integers, N(0,1) and |N(0,1)| floats of which one in eight is scaled by 1e-6,
truncated Zipf(1.2) bytes, log-uniform segment lengths.

  listed()            the fixed cases
  draw(rng)           another case of the same ranges
  prepare(case, seed) what a program holds before the call
  run(state)          one pass; returns the call's outputs
  work(case)          the bytes the call cannot do without
  exact(case, seed)   the outputs in 64 bits, from plain torch
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from opensycl_b200 import capi as C

DEV = "cuda"
TORCH = {"i32": torch.int32, "i64": torch.int64, "u32": torch.uint32, "f32": torch.float32,
         "f64": torch.float64, "bf16": torch.bfloat16, "u8": torch.uint8}
SIZE = {"i32": 4, "i64": 8, "u32": 4, "f32": 4, "f64": 8, "bf16": 2, "u8": 1}
ACC = {**SIZE, "bf16": 4}  # bf16 inputs accumulate in, and write, fp32
CHUNK = 1 << 25


def listed():
    return [
        # a reduction inside a host loop (a convergence check, a counter): launch and host latency
        {"name": "reduce_i32_1k", "op": "reduce", "dtype": "i32", "n": 1021},
        # the headline step's first half: the dot product of two 1 GiB vectors
        {"name": "dot_f32_2p28", "op": "dot", "dtype": "f32", "n": 1 << 28},
        # offsets from counts (CSR row pointers, compaction slots) of a few hundred thousand items
        {"name": "exscan_u32_300k", "op": "scan", "dtype": "u32", "n": 300007, "inclusive": False},
        # the headline step's second half: prefix sums of a 1 GiB vector
        {"name": "scan_f32_2p28", "op": "scan", "dtype": "f32", "n": 1 << 28, "inclusive": True},
        # prefix sums of bf16 data (probabilities, weights) into fp32, an odd size
        {"name": "scan_bf16_50m", "op": "scan", "dtype": "bf16", "n": 50000003, "inclusive": True},
        # stream compaction of the benchmark's shape, three of eight elements kept
        {"name": "copy_if_u32_2p28", "op": "copy_if", "dtype": "u32", "n": 1 << 28, "keep8": 3},
        # byte histogram with a few hot bins
        {"name": "histogram_zipf_2p28", "op": "histogram", "dtype": "u8", "n": 1 << 28},
        # per-group sums whose offsets change from call to call: the direct segmented call
        {"name": "segreduce_f32_10k", "op": "segreduce", "dtype": "f32", "n": (1 << 28) - 1234, "nseg": 10000,
         "plan": False},
        # per-group prefix sums over fixed offsets: the captured plan
        {"name": "segscan_i64_plan", "op": "segscan", "dtype": "i64", "n": (1 << 27) - 77, "nseg": 10000,
         "plan": True},
        # the largest sort of the benchmark
        {"name": "sort_i32_2p28", "op": "sort", "dtype": "i32", "n": 1 << 28, "desc": False},
        # an ordinary sort of wide keys (scores, timestamps), largest first
        {"name": "sort_f64_1m", "op": "sort", "dtype": "f64", "n": 1000003, "desc": True},
        # merging a large sorted run with a smaller one (an update of a sorted table)
        {"name": "merge_f32_130m", "op": "merge", "dtype": "f32", "na": 100000007, "nb": 33333331, "desc": False},
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["reduce", "dot", "scan", "scan", "copy_if", "histogram", "segreduce", "segscan", "sort", "merge"])
    if op == "reduce":
        dt = rng.choice(["i32", "i64", "f32", "bf16", "f64"])
        return {"op": op, "dtype": dt, "n": _size(rng, 1000, (1 << 31) // max(4, SIZE[dt]))}
    if op == "dot":
        dt = rng.choice(["f32", "bf16"])
        return {"op": op, "dtype": dt, "n": _size(rng, 1000, 1 << 28)}
    if op == "scan":
        dt = rng.choice(["i32", "u32", "i64", "f32", "bf16"])
        return {"op": op, "dtype": dt, "n": _size(rng, 1000, (1 << 30) // max(4, SIZE[dt])),
                "inclusive": rng.random() < 0.5}
    if op == "copy_if":
        dt = rng.choice(["u32", "u32", "i64"])
        return {"op": op, "dtype": dt, "n": _size(rng, 1000, (1 << 30) // SIZE[dt]), "keep8": rng.randint(1, 7)}
    if op == "histogram":
        return {"op": op, "dtype": "u8", "n": _size(rng, 1000, 1 << 28)}
    if op in ("segreduce", "segscan"):
        dt = rng.choice(["f32", "i64", "i32"])
        n = _size(rng, 1 << 16, (1 << 30) // SIZE[dt])
        return {"op": op, "dtype": dt, "n": n, "nseg": _size(rng, 16, min(20000, n // 64)),
                "plan": rng.random() < 0.5}
    if op == "sort":
        dt = rng.choice(["i32", "u32", "f32", "i64", "f64"])
        return {"op": op, "dtype": dt, "n": _size(rng, 1000, (1 << 28) // (1 if SIZE[dt] == 4 else 4)),
                "desc": rng.random() < 0.5}
    dt = rng.choice(["i32", "f32", "i64"])
    top = (1 << 28) // (SIZE[dt] // 4) // 2
    return {"op": "merge", "dtype": dt, "na": _size(rng, 1000, top), "nb": _size(rng, 1000, top),
            "desc": rng.random() < 0.5}


# ------------------------------------------------------------------ inputs

def _gen(seed, k=0):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 8 + k)


def _ints(g, n, dt):
    if dt == "i64":
        return torch.randint(-(1 << 20), (1 << 20) + 1, (n,), generator=g, device=DEV, dtype=torch.int64)
    if dt == "u32":
        x = torch.randint(-(1 << 31), 1 << 31, (n,), generator=g, device=DEV, dtype=torch.int32)
        return x.view(torch.uint32)
    return torch.randint(-1000, 1001, (n,), generator=g, device=DEV, dtype=torch.int32)


def _floats(g, n, dt, positive):
    """N(0,1) (or |N(0,1)|), one in eight scaled by 1e-6."""
    x = torch.randn(n, generator=g, device=DEV, dtype=torch.float64 if dt == "f64" else torch.float32)
    for i in range(0, n, CHUNK):
        v = x[i:i + CHUNK]
        v *= torch.where(torch.rand(v.numel(), generator=g, device=DEV) < 0.125, 1e-6, 1.0)
        if positive:
            v.abs_()
    return x.to(TORCH[dt])


def _values(g, n, dt, positive=False):
    return _ints(g, n, dt) if dt in ("i32", "i64", "u32") else _floats(g, n, dt, positive)


def _keys(g, n, dt):
    """Sort keys over the whole range of the type."""
    if dt in ("f32", "f64"):
        return torch.randn(n, generator=g, device=DEV, dtype=TORCH[dt])
    if dt == "i64":
        return torch.randint(-(1 << 62), 1 << 62, (n,), generator=g, device=DEV, dtype=torch.int64)
    x = torch.randint(-(1 << 31), 1 << 31, (n,), generator=g, device=DEV, dtype=torch.int32)
    return x.view(torch.uint32) if dt == "u32" else x


def _zipf(g, n):
    p = 1.0 / torch.arange(1, 257, device=DEV, dtype=torch.float64) ** 1.2
    cdf = (torch.cumsum(p, 0) / p.sum()).float()[:-1].contiguous()
    out = torch.empty(n, dtype=torch.uint8, device=DEV)
    for i in range(0, n, CHUNK):
        m = min(CHUNK, n - i)
        out[i:i + m] = torch.bucketize(torch.rand(m, generator=g, device=DEV), cdf, out_int32=True)
    return out


def _offsets(seed, nseg, n):
    """CSR offsets: lengths log-uniform in [1, 2^20], scaled to n elements in all."""
    u = np.random.default_rng(int(seed)).random(nseg)
    ends = np.cumsum(np.floor(2.0 ** (20.0 * u)) + 1.0)
    offs = np.concatenate([[0], np.floor(ends * (n / ends[-1]))]).astype(np.int64)
    offs[-1] = n
    return torch.from_numpy(offs).to(DEV)


class _Plan:
    """A segmented plan (b2p_plan_segmented) over fixed buffers."""

    def __init__(self, prim, x, offsets, out):
        self.x, self.offsets, self.out = x, offsets, out
        self.handle = ctypes.c_void_p()
        stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        C.check(C.lib().b2p_plan_segmented(ctypes.byref(self.handle), prim, C.dtype_code(x), C.SUM, x.data_ptr(),
                                           out.data_ptr(), offsets.data_ptr(), offsets.numel() - 1, x.numel(),
                                           C.AUTO, stream), "b2p_plan_segmented")

    def launch(self):
        stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        C.check(C.lib().b2p_plan_launch(self.handle, stream), "b2p_plan_launch")
        return self.out

    def __del__(self):
        if self.handle:
            torch.cuda.synchronize()
            C.lib().b2p_plan_destroy(self.handle)


def prepare(case, seed):
    op, dt = case["op"], case["dtype"]
    g = _gen(seed)
    st = {"op": op}
    if op == "reduce":
        st["x"] = _values(g, case["n"], dt)
    elif op == "dot":
        st["x"], st["y"] = _values(g, case["n"], dt), _values(_gen(seed, 1), case["n"], dt)
    elif op == "scan":
        st["x"], st["inclusive"] = _values(g, case["n"], dt, positive=True), case["inclusive"]
    elif op == "copy_if":
        st["x"] = _keys(g, case["n"], dt)
        st["keep8"] = case["keep8"]
        st["out"] = torch.zeros(case["n"] * SIZE[dt] // 4, dtype=torch.int32, device=DEV).view(TORCH[dt])
        st["count"] = C.zeros(1, torch.uint64, DEV)
    elif op == "histogram":
        st["x"] = _zipf(g, case["n"])
    elif op in ("segreduce", "segscan"):
        st["x"], st["offsets"] = _values(g, case["n"], dt), _offsets(seed, case["nseg"], case["n"])
        if case["plan"]:
            prim = C.PRIM_SEG_REDUCE if op == "segreduce" else C.PRIM_SEG_SCAN
            out = torch.zeros(case["nseg"] if op == "segreduce" else case["n"], dtype=TORCH[dt], device=DEV)
            st["plan"] = _Plan(prim, st["x"], st["offsets"], out)
    elif op == "sort":
        st["x"], st["desc"] = _keys(g, case["n"], dt), case["desc"]
    else:
        st["desc"] = case["desc"]
        for name, k in (("a", 0), ("b", 1)):
            st[name] = torch.sort(_keys(_gen(seed, k), case["n" + name], dt), descending=case["desc"])[0]
    return st


def _signed(x):
    """The same bits as a type that torch computes with (uint32 and uint64 tensors only hold data)."""
    signed = {torch.uint32: torch.int32, torch.uint64: torch.int64}.get(x.dtype)
    return x if signed is None else x.view(signed)


def run(st):
    op = st["op"]
    if op == "reduce":
        return C.reduce(st["x"])
    if op == "dot":
        return C.dot(st["x"], st["y"])
    if op == "scan":
        return _signed(C.inclusive_scan(st["x"]) if st["inclusive"] else C.exclusive_scan(st["x"], 0))
    if op == "copy_if":  # (x & 7) < keep8, into buffers that the program keeps
        out, count = C.copy_if(st["x"], 7, C.CMP_LT, st["keep8"], out=st["out"], count=st["count"])
        return _signed(out), _signed(count)
    if op == "histogram":
        return C.histogram_u8(st["x"])
    if op in ("segreduce", "segscan"):
        if "plan" in st:
            return st["plan"].launch()
        return (C.segmented_reduce if op == "segreduce" else C.segmented_scan)(st["x"], st["offsets"])
    if op == "sort":  # the sort is in place: the program keeps its input
        return _signed(C.sort_(st["x"].clone(), descending=st["desc"]))
    return C.merge(st["a"], st["b"], descending=st["desc"])


def work(case):
    op, dt = case["op"], case["dtype"]
    es, eo = SIZE[dt], ACC[dt]
    if op == "merge":
        return {"bytes": 2 * es * (case["na"] + case["nb"]), "flops": 0}
    n = case["n"]
    if op == "reduce":
        return {"bytes": es * n + eo, "flops": n}
    if op == "dot":
        return {"bytes": 2 * es * n + eo, "flops": 2 * n}
    if op == "scan":
        return {"bytes": (es + eo) * n, "flops": n}
    if op == "copy_if":
        return {"bytes": es * n + es * n * case["keep8"] / 8 + 8, "flops": 0}
    if op == "histogram":
        return {"bytes": n + 1024, "flops": 0}
    if op == "segreduce":
        return {"bytes": es * n + (8 + eo) * case["nseg"] + 8, "flops": n}
    if op == "segscan":
        return {"bytes": (es + eo) * n + 8 * case["nseg"] + 8, "flops": n}
    return {"bytes": 2 * es * n, "flops": 0}


# --------------------------------------------------------------- 64 bits

def _wide(x):
    return x.to(torch.float64)


def exact(case, seed):
    """Floating outputs only: whole numbers and bytes are the same or wrong."""
    op, dt = case["op"], case["dtype"]
    if dt not in ("f32", "bf16", "f64") or op in ("copy_if", "histogram"):
        return None
    st = prepare({**case, "plan": False}, seed)
    if op == "reduce":
        return sum(_wide(st["x"][i:i + CHUNK]).sum() for i in range(0, case["n"], CHUNK)).reshape(1)
    if op == "dot":
        return sum((_wide(st["x"][i:i + CHUNK]) * _wide(st["y"][i:i + CHUNK])).sum()
                   for i in range(0, case["n"], CHUNK)).reshape(1)
    if op == "scan":
        y = torch.cumsum(_wide(st["x"]), 0)
        return y if case["inclusive"] else torch.cat([y.new_zeros(1), y[:-1]])
    if op in ("segreduce", "segscan"):
        offs = st["offsets"].tolist()
        x = _wide(st["x"])
        if op == "segreduce":
            return torch.stack([x[a:b].sum() for a, b in zip(offs, offs[1:])])
        return torch.cat([torch.cumsum(x[a:b], 0) for a, b in zip(offs, offs[1:])])
    if op == "sort":
        return torch.sort(_wide(st["x"]), descending=case["desc"])[0]
    return torch.sort(torch.cat([_wide(st["a"]), _wide(st["b"])]), descending=case["desc"])[0]
