"""GPU parity of b2p_merge / b2p_sort (the hipsycl::algorithms::merge /
sort path) against the oracle's stable merge and sort, through the C-ABI.

Bar: bit-exact (keys are moved, never computed), including the order of
keys that compare equal but differ in their bits (-0.0 / +0.0: the stable
order).  Cases: the known answers of the reference's tests/pstl/merge.cpp
and sort.cpp (tests/golden/merge_sort_cases.npz), every key type in both
directions at sizes around the merge and radix tiles (b2p_sort runs the
radix sort from 2^15 keys on), ragged and empty inputs, extreme keys,
duplicates-heavy keys, and at 2^28 keys size-independent properties
(sorted, the same multiset as the input: the sum of the keys and the
histogram of their top byte).
"""
import ctypes
import os

import numpy as np
import pytest
import torch

from opensycl_b200 import capi as C
from oracle import oracle as O

pytestmark = pytest.mark.gpu

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "merge_sort_cases.npz")
DT = [C.I32, C.I64, C.U32, C.U64, C.F32, C.F64]
NP = {C.I32: np.int32, C.I64: np.int64, C.U32: np.uint32, C.U64: np.uint64, C.F32: np.float32,
      C.F64: np.float64}
# around the merge sort's 4096-key tiles, the radix sort's start (2^15 keys)
# and its 8192-key tiles
SIZES = [1, 2, 7, 255, 2047, 2048, 2049, 4096, 3 * 2048 + 17, 32767, 32768, 5 * 8192, 5 * 8192 + 1, 100003,
         (1 << 20) + 5]


def keys(rng, code, n, dup=False):
    if dup:  # few distinct values: long runs of equal keys
        v = rng.integers(0, 17, n)
        if code in (C.F32, C.F64):  # equal keys with different bits: -0.0 and +0.0
            v = np.where(v == 0, np.where(rng.random(n) < 0.5, -0.0, 0.0), v - 8.0)
        return v.astype(NP[code])
    if code in (C.F32, C.F64):
        return rng.standard_normal(n).astype(NP[code])
    info = np.iinfo(NP[code])
    return rng.integers(info.min, info.max, n, dtype=NP[code], endpoint=True)


def same_bits(got, ref):
    return got.dtype == ref.dtype and np.array_equal(got.view(np.uint8), ref.view(np.uint8))


def test_golden_merge_and_sort(dev):
    g = np.load(GOLDEN)
    names = sorted({k.rsplit("/", 1)[0] for k in g.files})
    for nm in names:
        if nm.startswith("merge/"):
            out = C.merge(dev_t(g[nm + "/a"]), dev_t(g[nm + "/b"]))
            assert np.array_equal(out.cpu().numpy(), g[nm + "/out"]), nm
        else:
            t = dev_t(g[nm + "/in"])
            C.sort_(t)
            assert np.array_equal(t.cpu().numpy(), g[nm + "/out"]), nm
    torch.cuda.synchronize()


def dev_t(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("code", DT)
@pytest.mark.parametrize("desc", [False, True])
def test_sort_parity(dev, code, desc):
    rng = np.random.default_rng(100 + code + 10 * desc)
    for n in SIZES:
        for dup in (False, True):
            x = keys(rng, code, n, dup)
            t = dev_t(x)
            C.sort_(t, descending=desc)
            assert same_bits(t.cpu().numpy(), O.sort(x, desc)), (n, dup)


@pytest.mark.parametrize("code", DT)
@pytest.mark.parametrize("desc", [False, True])
def test_merge_parity(dev, code, desc):
    rng = np.random.default_rng(200 + code + 10 * desc)
    for na, nb in [(0, 0), (0, 5), (5, 0), (1, 1), (2047, 1), (2048, 2048), (3000, 100003), (100003, 3000),
                   ((1 << 20) + 1, (1 << 19) + 7)]:
        for dup in (False, True):
            a = O.sort(keys(rng, code, na, dup), desc)
            b = O.sort(keys(rng, code, nb, dup), desc)
            out = C.merge(dev_t(a), dev_t(b), descending=desc)
            assert same_bits(out.cpu().numpy(), O.merge(a, b, desc)), (na, nb, dup)


def test_merge_disjoint_and_interleaved(dev):
    """All of a before all of b, the reverse, and a perfect interleave: the
    merge path runs along the matrix edges and the diagonal."""
    n = 1 << 20
    lo, hi = np.arange(n, dtype=np.int64), np.arange(n, 2 * n, dtype=np.int64)
    ev, od = np.arange(0, 2 * n, 2, dtype=np.int64), np.arange(1, 2 * n, 2, dtype=np.int64)
    for a, b in [(lo, hi), (hi, lo), (ev, od), (od, ev)]:
        out = C.merge(dev_t(a), dev_t(b)).cpu().numpy()
        assert np.array_equal(out, O.merge(a, b))


def test_sort_full_size_properties(dev):
    """2^28 uint32 keys (1 GiB): sorted, and the same multiset (the sum of the
    keys is unchanged and the counts of the top byte match)."""
    n = 1 << 28
    g = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randint(0, 1 << 31, (n,), generator=g, device="cuda", dtype=torch.int64).to(torch.int32)
    x = x.view(torch.uint32)
    xi = x.view(torch.int32).to(torch.int64)
    s0 = int(xi.sum())
    h0 = torch.bincount((x.view(torch.int32).to(torch.int64) >> 24) & 0xFF, minlength=256)
    C.sort_(x)
    xi = x.view(torch.int32).to(torch.int64)
    u = xi & 0xFFFFFFFF
    assert bool((u[1:] >= u[:-1]).all())
    assert int(xi.sum()) == s0
    assert torch.equal(torch.bincount((xi >> 24) & 0xFF, minlength=256), h0)
    del xi, u


def test_sort_descending_int64_full_size_properties(dev):
    n = 1 << 26
    g = torch.Generator(device="cuda").manual_seed(6)
    x = torch.randint(-(1 << 62), 1 << 62, (n,), generator=g, device="cuda", dtype=torch.int64)
    s0 = int(x.sum())
    C.sort_(x, descending=True)
    assert bool((x[1:] <= x[:-1]).all())
    assert int(x.sum()) == s0


def test_bf16_and_bad_args_are_rejected(dev):
    t = torch.zeros(16, dtype=torch.bfloat16, device="cuda")
    with pytest.raises(C.B2PError):
        C.sort_(t)
    L = C.lib()
    a = dev_t(np.arange(8, dtype=np.int32))
    assert L.b2p_sort(C.I32, a.data_ptr(), 1 << 16, 0, None, 0, None) == C.ERR_SCRATCH
    o = torch.empty(16, dtype=torch.int32, device="cuda")
    assert L.b2p_merge(99, a.data_ptr(), 8, a.data_ptr(), 8, o.data_ptr(), 0, None, 0, None) == C.ERR_INVALID_ARG
    assert L.b2p_merge(C.I32, a.data_ptr(), 8, a.data_ptr(), 8, o.data_ptr(), 0, None, 0, None) == C.ERR_SCRATCH
    host = np.zeros(8, dtype=np.int32)
    assert L.b2p_sort(C.I32, host.ctypes.data, 8, 0, None, 0, None) == C.ERR_INVALID_PTR


@pytest.mark.parametrize("code", DT)
def test_sort_extreme_and_uniform_keys(dev, code):
    """Every key the same (one digit value in every radix pass), and the
    extremes of the type (minimum, maximum, infinities, both zeros) mixed
    into random keys, in both directions."""
    rng = np.random.default_rng(300 + code)
    n = 100003
    same = np.full(n, 5, dtype=NP[code])
    t = dev_t(same)
    C.sort_(t)
    assert same_bits(t.cpu().numpy(), same)
    x = keys(rng, code, n)
    if code in (C.F32, C.F64):
        ext = np.array([np.inf, -np.inf, 0.0, -0.0, np.finfo(NP[code]).max, np.finfo(NP[code]).min,
                        np.finfo(NP[code]).tiny, -np.finfo(NP[code]).tiny], dtype=NP[code])
    else:
        info = np.iinfo(NP[code])
        ext = np.array([info.min, info.max, 0, 1, info.max - 1, info.min + 1], dtype=NP[code])
    idx = rng.integers(0, n, 4000)
    x[idx] = ext[rng.integers(0, ext.size, idx.size)]
    for desc in (False, True):
        t = dev_t(x)
        C.sort_(t, descending=desc)
        assert same_bits(t.cpu().numpy(), O.sort(x, desc)), desc


def test_sort_largest_radix_input(dev):
    """2^31 - 5 int32 keys (8 GiB), just below the radix sort's 2^31 limit of
    32-bit output slots: sorted, and the same multiset (sum of the keys and
    counts of the top byte)."""
    n = (1 << 31) - 5
    g = torch.Generator(device="cuda").manual_seed(9)
    x = torch.randint(-(1 << 31), (1 << 31) - 1, (n,), generator=g, device="cuda", dtype=torch.int32)
    s0 = int(torch.sum(x, dtype=torch.int64))
    h0 = torch.bincount(((x >> 24) & 0xFF).to(torch.int32), minlength=256)
    C.sort_(x)
    assert bool((x[1:] >= x[:-1]).all())
    assert int(torch.sum(x, dtype=torch.int64)) == s0
    assert torch.equal(torch.bincount(((x >> 24) & 0xFF).to(torch.int32), minlength=256), h0)
    del x
    torch.cuda.empty_cache()


@pytest.mark.parametrize("code", [C.I32, C.F32, C.I64, C.F64])
@pytest.mark.parametrize("offset", [0, 1])
def test_radix_tile_edges(dev, code, offset):
    """Around the radix sort's 32 KiB tiles (8192 4-byte or 4096 8-byte keys)
    and around one tile per resident block, where a block starts to walk
    several tiles; keys that start 16-byte aligned (staged by cp.async) or one
    element later; random digits, few distinct keys, and keys already in
    order (a whole tile in one digit of the upper passes)."""
    rng = np.random.default_rng(400 + code)
    tile = 8192 if code in (C.I32, C.F32) else 4096
    blocks = 3 * torch.cuda.get_device_properties(0).multi_processor_count
    for n in (8 * tile - 1, 8 * tile, 8 * tile + 1, blocks * tile, blocks * tile + 1, 2 * blocks * tile - 1):
        for kind in ("random", "dup", "sorted"):
            x = keys(rng, code, n, kind == "dup")
            if kind == "sorted":
                x.sort()
            desc = bool(n & 1)
            t = torch.empty(n + offset, dtype=dev_t(x[:1]).dtype, device="cuda")[offset:]
            t.copy_(dev_t(x))
            C.sort_(t, descending=desc)
            assert same_bits(t.cpu().numpy(), O.sort(x, desc)), (n, kind)


@pytest.mark.parametrize("code", [C.F32, C.I64])
def test_merge_many_tiles(dev, code):
    """More than 4096 tiles, where a partition warp takes 32 of them: the sum of
    the keys kept and the result sorted, for sides of very different length
    and an odd number of tiles."""
    n = 4100 * (4960 if code == C.F32 else 2400) + 77
    for na in (1000, n // 3):
        g = torch.Generator(device="cuda").manual_seed(na)
        x = torch.randint(-(1 << 23), 1 << 23, (n,), generator=g, device="cuda")
        x = x.to(torch.float32 if code == C.F32 else torch.int64)
        a, b = torch.sort(x[:na])[0], torch.sort(x[na:])[0]
        assert torch.equal(C.merge(a, b), torch.sort(x)[0])


@pytest.mark.parametrize("code", DT)
@pytest.mark.parametrize("desc", [False, True])
def test_merge_tile_edges(dev, code, desc):
    """Around the merge's tiles (4960 4-byte or 2400 8-byte keys) with one side
    empty, short or equal, unaligned output, sides that do not interleave at
    all, the type's extreme keys$
    sides' sentinel) and infinities among the keys, and both zeros (the
    serial tiles)."""
    rng = np.random.default_rng(500 + code + 10 * desc)
    tile = 4960 if NP[code]().itemsize == 4 else 2400
    flt = code in (C.F32, C.F64)
    last = [np.inf, -np.inf] if flt else [np.iinfo(NP[code]).max, np.iinfo(NP[code]).min]
    for total in (tile - 1, tile, tile + 1, 8 * tile, 8 * tile + 1, 16 * tile - 1):
        for na in (0, 1, 31, total // 2, total - 16, total):
            for kind in ("random", "dup", "last", "apart"):
                x = keys(rng, code, total, kind == "dup")
                if kind == "last":
                    x[rng.random(total) < 0.3] = last[0]
                    x[rng.random(total) < 0.3] = last[1]
                if kind == "apart":
                    x.sort()
                    if (total + na) % 2:
                        x = x[::-1]
                a, b = O.sort(x[:na].copy(), desc), O.sort(x[na:].copy(), desc)
                off = total % 2
                out = torch.empty(total + off, dtype=dev_t(x[:1].copy()).dtype, device="cuda")[off:]
                C.merge(dev_t(a), dev_t(b), out=out, descending=desc)
                assert same_bits(out.cpu().numpy(), O.merge(a, b, desc)), (total, na, kind)


@pytest.mark.parametrize("code", [C.F32, C.F64])
@pytest.mark.parametrize("desc", [False, True])
def test_merge_with_nans_writes_only_keys(dev, code, desc):
    """NaNs compare as unordered, at the end of a side or anywhere in it, so
    the order of the result is not specified; every key that it holds is one
    of the inputs' keys.  Less than a tile, several tiles, and numbers of
    tiles on both sides of the limit where a partition warp takes 32 of them."""
    dt, bits = (torch.float32, torch.int32) if code == C.F32 else (torch.float64, torch.int64)
    tile = 4960 if code == C.F32 else 2400
    g = torch.Generator(device="cuda").manual_seed(600 + code + 10 * desc)
    for total in (tile - 1, tile, 7 * tile + 5, 3000 * tile, 3000 * tile + 1):
        for na in (total // 2, total // 9):
            for where in ("end", "anywhere"):
                sides = []
                for n in (na, total - na):
                    x = torch.sort(torch.randn(n, generator=g, device="cuda", dtype=dt), descending=desc)[0]
                    if where == "end":
                        x[n - n // 7:] = float("nan")
                    else:
                        x[torch.rand(n, generator=g, device="cuda") < 0.1] = float("nan")
                    sides.append(x)
                out = C.merge(*sides, descending=desc)
                assert torch.isin(out.view(bits), torch.cat(sides).view(bits)).all(), (total, na, where)


@pytest.mark.parametrize("op", ["merge", "sort"])
def test_a_failed_launch_is_reported_once(dev, op):
    """A merge or sort on a stream whose capture has become invalid returns
    ERR_CUDA, and leaves no error behind for the next caller of the CUDA
    runtime to find."""
    cudart = ctypes.CDLL("libcudart.so.12")
    x = torch.sort(torch.randn(100000, device="cuda"))[0]
    out = torch.empty(200000, device="cuda")
    n = x.numel()
    nbytes = C.lib().b2p_scratch_bytes(C.PRIM_SORT, C.F32, 2 * n, 0, C.AUTO)
    tmp = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    handle = ctypes.c_void_p(st.cuda_stream)
    assert cudart.cudaStreamBeginCapture(handle, 2) == 0  # relaxed: other streams' calls go on
    assert cudart.cudaStreamSynchronize(handle) != 0  # not allowed: the capture is invalid from here on
    cudart.cudaGetLastError()
    if op == "merge":
        status = C.lib().b2p_merge(C.F32, x.data_ptr(), n, x.data_ptr(), n, out.data_ptr(), 0, tmp.data_ptr(), nbytes,
                                   handle)
    else:
        status = C.lib().b2p_sort(C.F32, x.data_ptr(), n, 0, tmp.data_ptr(), nbytes, handle)
    left = cudart.cudaGetLastError()
    graph = ctypes.c_void_p()
    assert cudart.cudaStreamEndCapture(handle, ctypes.byref(graph)) != 0 and not graph
    cudart.cudaGetLastError()
    assert status == C.ERR_CUDA and left == 0


@pytest.mark.parametrize("code", [C.F32, C.F64])
@pytest.mark.parametrize("n", [5000, 20000, 32767])
def test_sort_with_nans_writes_only_keys(dev, code, n):
    """Sorts of several tiles below the radix sort's size, with NaNs anywhere:
    the merge passes' runs are then in no order, and the order of the result
    is not specified; every key that it holds is one of the input's."""
    dt, bits = (torch.float32, torch.int32) if code == C.F32 else (torch.float64, torch.int64)
    g = torch.Generator(device="cuda").manual_seed(700 + code)
    for share in (0.001, 0.1, 0.9):
        for desc in (False, True):
            x = torch.randn(n, generator=g, device="cuda", dtype=dt)
            x[torch.rand(n, generator=g, device="cuda") < share] = float("nan")
            y = C.sort_(x.clone(), descending=desc)
            assert torch.isin(y.view(bits), x.view(bits)).all(), (share, desc)


@pytest.mark.parametrize("code", [C.I32, C.F64])
def test_merge_at_the_route_rules(dev, code):
    """Totals on both sides of every rule of the merge's route (2^18 and 7 x 2^18
    keys, the lopsided 8-byte merges up to 2^24 keys, 4,096 and 16,384 tiles),
    sides of equal and of very different length, both orders: the bits of the
    sorted whole."""
    dt = torch.int32 if code == C.I32 else torch.float64
    tile = 4960 if code == C.I32 else 2400
    g = torch.Generator(device="cuda").manual_seed(code)
    for total in (1 << 18, 7 << 18, 1 << 24, 4096 * tile, 16384 * tile):
        for n in (total - 1, total, total + 1):
            x = torch.randint(-(1 << 31), 1 << 31, (n,), generator=g, device="cuda").to(dt)
            for na, desc in ((n // 2, False), (n // 65, True), (n - 3, False)):
                a, b = torch.sort(x[:na], descending=desc)[0], torch.sort(x[na:], descending=desc)[0]
                ref = torch.sort(x, descending=desc)[0]
                assert torch.equal(C.merge(a, b, descending=desc), ref), (n, na, desc)


@pytest.mark.parametrize("n", [100003, 1000003])
def test_sort_and_merge_in_a_captured_graph(dev, n):
    """Sorts and merges whose kernels start early, captured into a graph: right
    behind a copy, behind another call's last kernel, as the first work of a
    forked stream and as the first after two streams join.  Replays on new
    inputs sort and merge those."""
    g = torch.Generator(device="cuda").manual_seed(n)

    def new(k):
        return torch.randint(-(1 << 31), 1 << 31, (k,), generator=g, device="cuda", dtype=torch.int32)

    x, a, b = new(n), torch.sort(new(n))[0], torch.sort(new(n // 2))[0]
    y, z = torch.empty_like(x), torch.empty_like(x)
    ab, aab = torch.empty(n + n // 2, dtype=torch.int32, device="cuda"), torch.empty(2 * n + n // 2, dtype=torch.int32,
                                                                                    device="cuda")
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        main = torch.cuda.current_stream()
        side.wait_stream(main)
        with torch.cuda.stream(side):
            C.merge(a, b, out=ab, stream=side)
            C.merge(a, ab, out=aab, stream=side)
        y.copy_(x)
        C.sort_(y, stream=main)
        z.copy_(y)
        main.wait_stream(side)
        C.sort_(z, descending=True, stream=main)
    for _ in range(3):
        x.copy_(new(n))
        a.copy_(torch.sort(new(n))[0])
        b.copy_(torch.sort(new(n // 2))[0])
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, torch.sort(x)[0]) and torch.equal(z, torch.sort(x, descending=True)[0])
        assert torch.equal(ab, torch.sort(torch.cat([a, b]))[0])
        assert torch.equal(aab, torch.sort(torch.cat([a, a, b]))[0])
