"""GPU parity: every primitive of libb2p against the CPU oracle (oracle/),
through the C-ABI, on seeded inputs.

Bars:
  * integer / index / byte results: bit-exact against the oracle;
  * fp32 / bf16 SUM (reduce, dot, scan): |got - ref| <= 1e-6 |ref| + 1e-12 S
    where ref is the FP64 oracle and S the sum of magnitudes (the second
    term only matters when the exact result cancels to ~0);
  * float MIN / MAX: bit-exact against numpy;
  * float PROD: relative 4 n 2^-24 against FP64 (plain arithmetic).
"""
import numpy as np
import pytest
import torch

from opensycl_b200 import capi as C
from oracle import oracle as O

pytestmark = pytest.mark.gpu

INT_DT = [C.I32, C.I64, C.U32, C.U64]
FLOAT_DT = [C.F32, C.BF16, C.F64]
NP = {C.I32: np.int32, C.I64: np.int64, C.U32: np.uint32, C.U64: np.uint64,
      C.F32: np.float32, C.BF16: np.uint16, C.F64: np.float64}
TD = {C.I32: torch.int32, C.I64: torch.int64, C.U32: torch.uint32, C.U64: torch.uint64,
      C.F32: torch.float32, C.BF16: torch.bfloat16, C.F64: torch.float64}
SIZES = [1, 2, 5, 127, 128, 1000, 4099, 65537, (1 << 20) + 3]
REDUCE_CONFIGS = [0, 9, 22, 47, C.AUTO]
SCAN_CONFIGS = [0, 6, 19, 22, 23, 26, 41, C.AUTO]
FLOAT_TOL = 1e-6


def valid(prim, code, cfgs):
    """Configs of `cfgs` the library accepts for this primitive and dtype."""
    L = C.lib()
    return [c for c in cfgs if c == C.AUTO or L.b2p_config_valid(prim, code, c)]


def to_dev(a, code, offset=0):
    """numpy -> device tensor; `offset` elements of padding in front make the
    returned view start off a 16-byte boundary."""
    if offset:
        a = np.concatenate([np.zeros(offset, dtype=a.dtype), a])
    if code == C.BF16:
        t = torch.from_numpy(a.view(np.int16)).cuda().view(torch.bfloat16)
    else:
        t = torch.from_numpy(np.ascontiguousarray(a)).cuda()
    return t[offset:]


def to_np(t):
    if t.dtype == torch.bfloat16:
        return t.view(torch.int16).cpu().numpy().view(np.uint16)
    return t.cpu().numpy()


def rand_ints(rng, code, n, op):
    if op == C.PROD:  # keep products meaningful: mostly ones, some twos/threes
        v = rng.choice(np.array([1, 1, 1, 1, 2, 3, -1] if code in (C.I32, C.I64) else [1, 1, 1, 2, 3]), n)
        return v.astype(NP[code])
    info = np.iinfo(NP[code])
    return rng.integers(info.min, info.max, n, dtype=NP[code], endpoint=True)


def rand_floats(rng, code, n, positive=False):
    x = rng.standard_normal(n)
    x[rng.random(n) < 0.125] *= 1e-6
    if positive:
        x = np.abs(x)
    if code == C.BF16:
        return O.bf16_round(x.astype(np.float32))
    return x.astype(NP[code])


def as_f64(a, code):
    return O.bf16_to_f32(a).astype(np.float64) if code == C.BF16 else a.astype(np.float64)


def float_ok(got, ref, sabs):
    return abs(float(got) - ref) <= FLOAT_TOL * abs(ref) + 1e-12 * sabs


# ------------------------------------------------------------------ reduce

@pytest.mark.parametrize("code", INT_DT)
@pytest.mark.parametrize("op", [C.SUM, C.PROD, C.MIN, C.MAX, C.AND, C.OR, C.XOR])
def test_reduce_int_bit_exact(dev, code, op):
    rng = np.random.default_rng(100 + 7 * code + op)
    for n in SIZES:
        x = rand_ints(rng, code, n, op)
        init = rand_ints(rng, code, 1, op)[0]
        ref = O.reduce(code, op, x, init)
        for off in (0, 1):
            xd = to_dev(x, code, off)
            for cfg in REDUCE_CONFIGS:
                got = C.reduce(xd, op, init=init, config=cfg)
                assert to_np(got)[0] == ref, (n, off, cfg)


@pytest.mark.parametrize("code", FLOAT_DT)
def test_reduce_float_sum_vs_fp64(dev, code):
    rng = np.random.default_rng(200 + code)
    for n in SIZES:
        x = rand_floats(rng, code, n)
        ref, sabs = O.fp64_sum(code, x, init=0.5)
        for off in (0, 3):
            xd = to_dev(x, code, off)
            for cfg in REDUCE_CONFIGS:
                got = to_np(C.reduce(xd, "sum", init=0.5, config=cfg))[0]
                assert float_ok(got, ref, sabs), (n, off, cfg, got, ref)


@pytest.mark.parametrize("code", FLOAT_DT)
@pytest.mark.parametrize("op", [C.MIN, C.MAX, C.PROD])
def test_reduce_float_other_ops(dev, code, op):
    rng = np.random.default_rng(300 + code * 3 + op)
    for n in SIZES:
        if op == C.PROD:
            x64 = 1.0 + (rng.random(n) - 0.5) * 1e-3
            x = O.bf16_round(x64.astype(np.float32)) if code == C.BF16 else x64.astype(NP[code])
        else:
            x = rand_floats(rng, code, n)
        xd = to_dev(x, code)
        xf = as_f64(x, code)
        for cfg in (0, 22, C.AUTO):
            got = to_np(C.reduce(xd, op, init=1.0 if op == C.PROD else (np.inf if op == C.MIN else -np.inf),
                                 config=cfg))[0]
            if op == C.MIN:
                assert got == xf.min()
            elif op == C.MAX:
                assert got == xf.max()
            else:
                ref = np.prod(xf)
                eps = 2.0 ** -24 if code != C.F64 else 2.0 ** -53
                assert abs(got - ref) <= 4 * n * eps * abs(ref)


def test_reduce_float_config_independent(dev):
    """fp32 SUM is bit-identical for all 48 launch configurations."""
    rng = np.random.default_rng(7)
    for n in (1000, 65537, (1 << 22) + 5):
        x = rand_floats(rng, C.F32, n)
        xd = to_dev(x, C.F32, 1)
        vals = {to_np(C.reduce(xd, "sum", init=0.0, config=c))[0].tobytes() for c in range(48)}
        assert len(vals) == 1, n
        bd = to_dev(rand_floats(rng, C.F32, n), C.F32)
        dots = {to_np(C.dot(xd, bd, config=c))[0].tobytes() for c in range(48)}
        assert len(dots) == 1, n


def test_reduce_no_init_combines_with_out(dev):
    x = to_dev(np.arange(1000, dtype=np.int32), C.I32)
    out = torch.tensor([7], dtype=torch.int32, device="cuda")
    C.reduce(x, "sum", init=None, out=out)
    C.reduce(x, "sum", init=None, out=out)
    assert out.item() == 7 + 2 * 499500  # incremental sycl::reduction (reduction.cpp:326-350)


def test_reduce_empty_leaves_out_untouched(dev):
    x = torch.zeros(0, dtype=torch.float32, device="cuda")
    out = torch.tensor([42.0], device="cuda")
    C.reduce(x, "sum", init=1.0, out=out)
    assert out.item() == 42.0


# ------------------------------------------------------------------ dot

@pytest.mark.parametrize("code", FLOAT_DT)
def test_dot_vs_fp64(dev, code):
    rng = np.random.default_rng(400 + code)
    for n in SIZES:
        a = rand_floats(rng, code, n)
        b = rand_floats(rng, code, n)
        ref, sabs = O.fp64_sum(code, a, b, init=0.25)
        for oa, ob in ((0, 0), (1, 1), (0, 1)):  # (0, 1): differently aligned -> scalar path
            ad, bd = to_dev(a, code, oa), to_dev(b, code, ob)
            for cfg in (0, 22, C.AUTO):
                got = to_np(C.dot(ad, bd, init=0.25, config=cfg))[0]
                assert float_ok(got, ref, sabs), (n, oa, ob, cfg, got, ref)


# ------------------------------------------------------------------ scan

@pytest.mark.parametrize("code", INT_DT)
@pytest.mark.parametrize("op", [C.SUM, C.PROD, C.MIN, C.MAX, C.AND, C.OR, C.XOR])
def test_scan_int_bit_exact(dev, code, op):
    rng = np.random.default_rng(500 + 7 * code + op)
    sizes = [1, 31, 512, 513, 4096, 8191, 8192, 8193, 100003]
    for n in sizes:
        x = rand_ints(rng, code, n, op)
        init = rand_ints(rng, code, 1, op)[0]
        r_inc = O.scan(code, op, True, x)
        r_inc_i = O.scan(code, op, True, x, init)
        r_exc = O.scan(code, op, False, x, init)
        for off in (0, 1):
            xd = to_dev(x, code, off)
            for cfg in valid(C.PRIM_SCAN, code, SCAN_CONFIGS):
                assert np.array_equal(to_np(C.scan(xd, True, op, None, config=cfg)), r_inc), (n, off, cfg)
                assert np.array_equal(to_np(C.scan(xd, True, op, init, config=cfg)), r_inc_i), (n, off, cfg)
                assert np.array_equal(to_np(C.scan(xd, False, op, init, config=cfg)), r_exc), (n, off, cfg)


@pytest.mark.parametrize("code", FLOAT_DT)
def test_scan_float_sum_vs_fp64(dev, code):
    rng = np.random.default_rng(600 + code)
    for n in [1, 31, 4097, 100003, (1 << 20) + 7]:
        x = rand_floats(rng, code, n, positive=True)
        ref_i = O.fp64_scan(code, True, x, 0.0)
        ref_e = O.fp64_scan(code, False, x, 1.5)
        xd = to_dev(x, code)
        for cfg in valid(C.PRIM_SCAN, code, SCAN_CONFIGS):
            gi = to_np(C.scan(xd, True, "sum", None, config=cfg)).astype(np.float64)
            ge = to_np(C.scan(xd, False, "sum", 1.5, config=cfg)).astype(np.float64)
            pos = ref_i > 0
            assert np.max(np.abs(gi - ref_i)[pos] / ref_i[pos]) <= FLOAT_TOL, (n, cfg)
            assert np.max(np.abs(ge - ref_e) / ref_e) <= FLOAT_TOL, (n, cfg)


# Pipelined (TMA) scan configurations: 128 x 32, 256 x 16, 256 x 32 (512 x 16,
# configuration 26, has no pipelined kernel and runs the two-phase kernel).
TMA_SCAN_CONFIGS = [19, 22, 23]


@pytest.mark.parametrize("code", [C.I32, C.I64, C.U32])
def test_scan_pipelined_row_tails(dev, code):
    """Sizes around tile and 128-byte-row boundaries: the last tile may be
    partly or wholly past the complete rows that the bulk tensor copies
    cover, and the elements after them go through plain loads and stores."""
    rng = np.random.default_rng(550 + code)
    es = np.dtype(NP[code]).itemsize
    epr = 128 // es
    for cfg in TMA_SCAN_CONFIGS:
        blk, items = C.config_describe(cfg)[:2]
        tile = blk * items
        for n in [tile, tile + 1, 3 * tile - 1, 3 * tile + epr - 1, 5 * tile + 256 * epr,
                  5 * tile + 256 * epr + 3, 7 * tile + tile // 2 + 5]:
            x = rand_ints(rng, code, n, C.SUM)
            init = rand_ints(rng, code, 1, C.SUM)[0]
            xd = to_dev(x, code)
            assert np.array_equal(to_np(C.scan(xd, True, C.SUM, None, config=cfg)),
                                  O.scan(code, C.SUM, True, x)), (cfg, n)
            assert np.array_equal(to_np(C.scan(xd, False, C.SUM, init, config=cfg)),
                                  O.scan(code, C.SUM, False, x, init)), (cfg, n)


def test_scan_pipelined_bf16_in_fp32_out(dev):
    """bf16 input, fp32 output through the pipelined kernel (the output tile
    sits beside the input tile in each stage): SUM against FP64, MAX exact,
    around 64-element input rows and 32-element output rows."""
    rng = np.random.default_rng(570)
    for cfg in TMA_SCAN_CONFIGS:
        blk, items = C.config_describe(cfg)[:2]
        tile = blk * items
        for n in [tile, 2 * tile + 63, 3 * tile + 32 * 5 + 7, 5 * tile + tile // 2 + 1]:
            x = rand_floats(rng, C.BF16, n, positive=True)
            xd = to_dev(x, C.BF16)
            ref_i = O.fp64_scan(C.BF16, True, x, 0.0)
            ref_e = O.fp64_scan(C.BF16, False, x, 1.5)
            gi = to_np(C.scan(xd, True, "sum", None, config=cfg)).astype(np.float64)
            ge = to_np(C.scan(xd, False, "sum", 1.5, config=cfg)).astype(np.float64)
            pos = ref_i > 0
            assert np.max(np.abs(gi - ref_i)[pos] / ref_i[pos]) <= FLOAT_TOL, (cfg, n)
            assert np.max(np.abs(ge - ref_e) / ref_e) <= FLOAT_TOL, (cfg, n)
            xs = O.bf16_to_f32(rand_floats(rng, C.BF16, n))
            xsd = to_dev(O.bf16_round(xs), C.BF16)
            gm = to_np(C.scan(xsd, True, C.MAX, None, config=cfg))
            assert np.array_equal(gm, np.maximum.accumulate(xs).astype(np.float32)), (cfg, n)


def test_scan_pipelined_fp32_long_exclusive(dev):
    """fp32 SUM longer than 2^24 (FP64 tile carries) through the pipelined
    kernel, inclusive and exclusive with init."""
    rng = np.random.default_rng(560)
    n = (1 << 24) + 12345
    x = rand_floats(rng, C.F32, n, positive=True)
    ref_i = O.fp64_scan(C.F32, True, x, 0.0)
    ref_e = O.fp64_scan(C.F32, False, x, 1.5)
    xd = to_dev(x, C.F32)
    for cfg in (22, 23):
        gi = to_np(C.scan(xd, True, "sum", None, config=cfg)).astype(np.float64)
        ge = to_np(C.scan(xd, False, "sum", 1.5, config=cfg)).astype(np.float64)
        assert np.max(np.abs(gi - ref_i) / ref_i) <= FLOAT_TOL, cfg
        assert np.max(np.abs(ge - ref_e) / ref_e) <= FLOAT_TOL, cfg


@pytest.mark.parametrize("code", [C.F32, C.F64])
@pytest.mark.parametrize("op", [C.MIN, C.MAX])
def test_scan_float_minmax_exact(dev, code, op):
    rng = np.random.default_rng(700 + code + op)
    x = rand_floats(rng, code, 100003)
    ref = (np.minimum if op == C.MIN else np.maximum).accumulate(x)
    got = to_np(C.scan(to_dev(x, code), True, op, None, config=C.AUTO))
    assert np.array_equal(got, ref.astype(got.dtype))


def test_scan_in_place(dev):
    rng = np.random.default_rng(8)
    x = rng.integers(-1000, 1000, 50001).astype(np.int32)
    xd = to_dev(x, C.I32)
    C.scan(xd, True, "sum", None, out=xd)
    assert np.array_equal(to_np(xd), O.scan(C.I32, C.SUM, True, x))
    xd = to_dev(x, C.I32)
    C.scan(xd, False, "sum", 3, out=xd)
    assert np.array_equal(to_np(xd), O.scan(C.I32, C.SUM, False, x, 3))


def test_scan_repeated_calls_share_scratch(dev):
    """Epoch-tagged tile status: back-to-back calls on one scratch buffer
    never read a previous call's status words."""
    rng = np.random.default_rng(9)
    for n in (70001, 9000, 300000, 9000):
        x = rng.integers(-5, 5, n).astype(np.int64)
        xd = to_dev(x, C.I64)
        for _ in range(3):
            assert np.array_equal(to_np(C.scan(xd, True, "sum", None, config=0)),
                                  O.scan(C.I64, C.SUM, True, x))


# ------------------------------------------------------------------ copy_if

@pytest.mark.parametrize("code", [C.U32, C.I32, C.F32, C.I64, C.U64])
def test_copy_if_bit_exact(dev, code):
    rng = np.random.default_rng(800 + code)
    for n in [1, 2, 100, 4095, 4096, 4097, 100003, (1 << 20) + 1]:
        bits = rng.integers(0, 1 << 32, n, dtype=np.uint64)
        if np.dtype(NP[code]).itemsize == 8:
            u = bits | (rng.integers(0, 1 << 32, n, dtype=np.uint64) << np.uint64(32))
        else:
            u = bits.astype(np.uint32)
        x = u.view(NP[code])
        for mask, cmp, rhs in ((7, C.CMP_LT, 3), (1, C.CMP_EQ, 0), (0, C.CMP_EQ, 0), (0xFF, C.CMP_GT, 255)):
            keep = {C.CMP_LT: (u & mask) < rhs, C.CMP_EQ: (u & mask) == rhs,
                    C.CMP_GT: (u & mask) > rhs}[cmp]
            ref = x[keep]
            for off in (0, 1):
                xd = to_dev(x, code, off)
                for cfg in valid(C.PRIM_COPY_IF, code, (0, 6, 19, 22, 23, 26, C.AUTO)):
                    out, cnt = C.copy_if(xd, mask, cmp, rhs, config=cfg)
                    k = int(cnt.item())
                    assert k == ref.size, (n, mask, cmp, off, cfg)
                    assert np.array_equal(to_np(out[:k]).view(u.dtype), ref.view(u.dtype))


@pytest.mark.parametrize("code", [C.U32, C.U64])
def test_copy_if_pipelined_unaligned_output(dev, code):
    """Pipelined copy_if writes the 16-byte-aligned middle of each tile's
    output with one bulk copy and the ends with plain stores: outputs that
    start at every 16-byte phase, sizes around tile and row boundaries."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(810 + code)
    es = np.dtype(NP[code]).itemsize
    for cfg in TMA_SCAN_CONFIGS:
        blk, items = C.config_describe(cfg)[:2]
        tile = blk * items
        for n in [tile, 3 * tile + 5, 6 * tile + 128 // es * 7 + 1]:
            u = rng.integers(0, 1 << 32, n, dtype=np.uint64).astype(NP[code])
            keep = (u & 7) < 3
            ref = u[keep]
            xd = to_dev(u, code)
            for shift in range(16 // es):
                big = torch.empty(n + 4, dtype=TD[code], device="cuda")
                out = big[shift:shift + n]
                _, cnt = C.copy_if(xd, 7, C.CMP_LT, 3, out=out, config=cfg)
                k = int(cnt.item())
                assert k == ref.size, (cfg, n, shift)
                assert np.array_equal(to_np(out[:k]), ref), (cfg, n, shift)


@pytest.mark.parametrize("code", [C.U32, C.U64])
def test_copy_if_pipelined_regular_patterns(dev, code):
    """Regular keep patterns through the pipelined copy_if kernels: all kept
    (the output is the input), none kept, every other element, one element
    per tile; sizes with a partial last tile."""
    rng = np.random.default_rng(870 + code)
    for cfg in TMA_SCAN_CONFIGS:
        blk, items = C.config_describe(cfg)[:2]
        tile = blk * items
        n = 5 * tile + 77
        u = rng.integers(0, 1 << 32, n, dtype=np.uint64).astype(NP[code])
        u = (u & ~np.array(7, dtype=NP[code])) | (np.arange(n) % 8).astype(NP[code])  # low 3 bits = index mod 8
        xd = to_dev(u, code)
        for cmp, rhs in [(C.CMP_LT, 8), (C.CMP_GT, 7), (C.CMP_EQ, 0), (C.CMP_LT, 4)]:
            keep = (u & 7) < 8 if (cmp, rhs) == (C.CMP_LT, 8) else \
                (u & 7) > 7 if cmp == C.CMP_GT else (u & 7) == 0 if cmp == C.CMP_EQ else (u & 7) < 4
            ref = u[keep]
            out, cnt = C.copy_if(xd, 7, cmp, rhs, config=cfg)
            k = int(cnt.item())
            assert k == ref.size, (cfg, cmp, rhs)
            assert np.array_equal(to_np(out[:k]), ref), (cfg, cmp, rhs)
        # one kept element per tile
        v = np.zeros(n, dtype=NP[code])
        v[::tile] = 1
        out, cnt = C.copy_if(to_dev(v, code), 1, C.CMP_EQ, 1, config=cfg)
        assert int(cnt.item()) == v[::tile].size and np.all(to_np(out[:int(cnt.item())]) == 1)


def test_copy_if_oracle_u32(dev):
    rng = np.random.default_rng(11)
    x = rng.integers(0, 1 << 32, 1 << 20, dtype=np.uint64).astype(np.uint32)
    ref, cnt = O.copy_if_u32(x, 7, C.CMP_LT, 3)
    out, c = C.copy_if(to_dev(x, C.U32), 7, C.CMP_LT, 3)
    assert int(c.item()) == cnt and np.array_equal(to_np(out[:cnt]), ref)


# ------------------------------------------------------------------ histogram

def test_histogram_bit_exact(dev):
    rng = np.random.default_rng(12)
    for n in [1, 15, 16, 17, 1000, 100003, (1 << 22) + 9]:
        for dist in ("uniform", "zipf", "single"):
            if dist == "uniform":
                k = rng.integers(0, 256, n).astype(np.uint8)
            elif dist == "zipf":
                k = C.synth_fill(4, int(rng.integers(1 << 30)), n, 1.2)
            else:
                k = np.full(n, 7, dtype=np.uint8)
            for nbins in (256, 100):
                base = rng.integers(0, 1000, nbins).astype(np.int32)
                ref = O.histogram_u8(k, nbins, bins=base.astype(np.uint32)).astype(np.int64)
                for off in (0, 5):
                    for cfg in (0, 30, C.AUTO):
                        bins = torch.from_numpy(base.copy()).cuda()
                        kd = torch.from_numpy(np.concatenate([np.zeros(off, np.uint8), k])).cuda()[off:]
                        C.histogram_u8(kd, bins=bins, nbins=nbins, config=cfg)
                        assert np.array_equal(bins.cpu().numpy().astype(np.int64), ref), (n, dist, nbins, off, cfg)


def test_histogram_streamed_chunks(dev):
    """Grid mode 1 streams keys through a ring of shared stages with bulk
    copies: many chunks per block (the ring wraps), a partial last chunk,
    unaligned heads and ragged tails; the scratch-less error word stays clear."""
    rng = np.random.default_rng(13)
    for n in [(40 << 20) + 3, (9 << 20) + 4095]:
        k = C.synth_fill(4, int(rng.integers(1 << 30)), n, 1.2)
        ref = O.histogram_u8(k, 256).astype(np.int64)
        for off in (0, 1, 15):
            for cfg in (23, 30, 31):
                assert C.config_describe(cfg)[2] == 1
                bins = torch.zeros(256, dtype=torch.int32, device="cuda")
                kd = torch.from_numpy(np.concatenate([np.zeros(off, np.uint8), k])).cuda()[off:]
                C.histogram_u8(kd, bins=bins, config=cfg)
                assert np.array_equal(bins.cpu().numpy().astype(np.int64), ref), (n, off, cfg)
    assert C.device_error(scratchless=True) == C.OK


# ------------------------------------------------------------------ errors

def test_errors_are_status_codes(dev):
    L = C.lib()
    import ctypes
    host = np.zeros(1024, dtype=np.float32)
    out = torch.zeros(1, device="cuda")
    sp, sb = C.scratch_for(C.PRIM_REDUCE, C.F32, 1024)
    rc = L.b2p_reduce(C.F32, C.SUM, host.ctypes.data_as(ctypes.c_void_p), 1024, out.data_ptr(),
                      None, sp, sb, 0, None)
    assert rc in (C.ERR_INVALID_PTR, C.OK)  # OK only where pageable memory is device-accessible
    x = torch.zeros(1024, device="cuda")
    assert L.b2p_reduce(C.F32, C.AND, x.data_ptr(), 1024, out.data_ptr(), None, sp, sb, 0, None) == C.ERR_INVALID_ARG
    assert L.b2p_reduce(C.F32, C.SUM, x.data_ptr(), 1024, out.data_ptr(), None, sp, sb, 48, None) == C.ERR_INVALID_ARG
    assert L.b2p_reduce(C.F32, C.SUM, x.data_ptr(), 1024, out.data_ptr(), None, sp, 8, 0, None) == C.ERR_SCRATCH
    assert L.b2p_scan(C.F32, C.SUM, 0, x.data_ptr(), x.data_ptr(), 1024, None, sp, sb, 0, None) == C.ERR_INVALID_ARG
    # misaligned element pointer
    assert L.b2p_reduce(C.F32, C.SUM, x.data_ptr() + 2, 10, out.data_ptr(), None, sp, sb, 0, None) == C.ERR_INVALID_PTR
    torch.cuda.synchronize()
    assert C.device_error() == C.OK


def test_kernels_are_sm100a(dev):
    """The kernels the CUDA runtime loads from libb2p are sm_100a machine code
    (cudaFuncGetAttributes binaryVersion 100), with no PTX to JIT."""
    import ctypes
    b, p = ctypes.c_int(0), ctypes.c_int(-1)
    C.check(C.lib().b2p_kernel_arch(ctypes.byref(b), ctypes.byref(p)), "b2p_kernel_arch")
    assert b.value == 100, b.value


@pytest.mark.parametrize("code", [C.I32, C.I64, C.F32, C.BF16, C.F64])
def test_reduce_one_block_limit(dev, code):
    """Sizes on both sides of the one-block reduce's limit (32 runs of 8 KiB),
    of a run, of a vector, and starts up to seven elements off a 16-byte
    boundary: integers exact, floats within 1e-6 of the FP64 sum, the same bits
    in every launch configuration; combining with *out; the dot product."""
    es = {C.I32: 4, C.I64: 8, C.F32: 4, C.BF16: 2, C.F64: 8}[code]
    run = 8192 // es
    g = torch.Generator(device="cuda").manual_seed(code)
    for n in (1, 2, 16 // es, run - 1, run, run + 1, 32 * run - 1, 32 * run, 32 * run + 1, 33 * run + 5):
        for off in (0, 1, 3):
            if code in (C.I32, C.I64):
                base = torch.randint(-1000, 1000, (n + off,), generator=g, device="cuda")
                x = base.to(torch.int32 if code == C.I32 else torch.int64)[off:]
            else:
                base = torch.randn(n + off, generator=g, device="cuda", dtype=torch.float64)
                x = base.to({C.F32: torch.float32, C.BF16: torch.bfloat16, C.F64: torch.float64}[code])[off:]
            ref = x.to(torch.float64).sum().item()
            scale = x.to(torch.float64).abs().sum().item()
            bits = set()
            for cfg in (C.AUTO, 0, 15, 17, 47):
                got = C.reduce(x, "sum", init=0, config=cfg)
                bits.add(got.view(torch.uint8).cpu().numpy().tobytes())
                assert abs(got.item() - ref) <= 1e-6 * abs(ref) + 1e-12 * scale, (n, off, cfg)
            assert len(bits) == 1, (n, off)
            if code in (C.I32, C.I64):
                assert C.reduce(x, "min", init=5).item() == min(5, int(x.min()))
                keep = torch.full((1,), 7, dtype=x.dtype, device="cuda")
                assert C.reduce(x, "sum", init=None, out=keep).item() == 7 + int(x.sum())
            else:
                d = C.dot(x, x, init=1.0).item()
                rd = 1.0 + (x.to(torch.float64) ** 2).sum().item()
                assert abs(d - rd) <= 1e-6 * rd, (n, off)


@pytest.mark.parametrize("code", [C.I32, C.I64, C.F32, C.BF16])
def test_scan_and_copy_if_at_the_tile_rules(dev, code):
    """Sizes on both sides of every size rule of the automatic configuration
    (one look-back tile per block with its own index as tile id, then the
    pipelined kernel): the scan against torch's cumulative sum, copy_if
    against a mask, integers exact, floats within 1e-6."""
    g = torch.Generator(device="cuda").manual_seed(code)
    for n in (1, 2048, 2049, 1 << 18, (1 << 18) + 1, 1 << 19, (1 << 19) + 1, 1 << 20, (1 << 20) + 1, 1 << 21,
              (1 << 21) + 1, 13 << 18, (13 << 18) + 1, 1 << 22, (1 << 22) + 1):
        if code in (C.I32, C.I64):
            x = torch.randint(0, 1 << 20, (n,), generator=g, device="cuda")
            x = x.to(torch.int32 if code == C.I32 else torch.int64)
            ref = torch.cumsum(x, 0).to(x.dtype)
            assert torch.equal(C.inclusive_scan(x), ref), n
            ex = C.exclusive_scan(x, 5)
            assert ex[0].item() == 5 and torch.equal(ex[1:], ref[:-1] + 5), n
            out, cnt = C.copy_if(x, 7, C.CMP_LT, 3)
            keep = x[(x & 7) < 3]
            assert int(cnt.item()) == keep.numel() and torch.equal(out[:keep.numel()], keep), n
        else:
            x = torch.rand(n, generator=g, device="cuda").to(torch.float32 if code == C.F32 else torch.bfloat16)
            ref = torch.cumsum(x.to(torch.float64), 0)
            got = C.inclusive_scan(x).to(torch.float64)
            assert ((got - ref).abs() <= 1e-6 * ref.abs() + 1e-30).all(), n


@pytest.mark.parametrize("code", [C.U32, C.I64, C.F32, C.BF16])
def test_pipelined_look_back_units(dev, code):
    """Tile counts around the rule for two tiles per look-back unit (three per
    SM), with a last unit of one tile and ragged last tiles: integer scans and
    copy_if (few, some and all kept) exact, float scans within 1e-6 of FP64."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    g = torch.Generator(device="cuda").manual_seed(code)
    for items in (16, 32):
        if code == C.I64 and items == 32:
            continue
        cfg = 16 + 4 + (2 if items == 16 else 3)
        tile = 256 * items
        for n in [t * tile + d for t in (3 * sms - 1, 3 * sms, 3 * sms + 1) for d in (-1, 0, 1, 5)]:
            if code in (C.U32, C.I64):
                x = torch.randint(0, 1 << 20, (n,), generator=g, device="cuda")
                ref = torch.cumsum(x, 0)
                y = x if code == C.I64 else x.to(torch.uint32)
                got = C.inclusive_scan(y, config=cfg).to(torch.int64)
                assert torch.equal(got, ref if code == C.I64 else ref & 0xFFFFFFFF), (items, n)
                for rhs in (0, 1, 3, 8):
                    out, cnt = C.copy_if(y, 7, C.CMP_LT, rhs, config=cfg)
                    keep = x[(x & 7) < rhs]
                    k = int(cnt.item())
                    assert k == keep.numel() and torch.equal(out[:k].to(torch.int64), keep), (items, n, rhs)
            else:
                x = torch.rand(n, generator=g, device="cuda").to(torch.float32 if code == C.F32 else torch.bfloat16)
                ref = torch.cumsum(x.to(torch.float64), 0)
                got = C.inclusive_scan(x, config=cfg).to(torch.float64)
                assert ((got - ref).abs() <= 1e-6 * ref).all(), (items, n)


@pytest.mark.parametrize("code", [C.F32, C.BF16])
def test_pipelined_scan_special_values(dev, code):
    """Denormals and signed zeros scan like other values; from an infinity or a
    NaN on, and only there, the outputs are not finite."""
    n = 6 << 20
    dt = torch.float32 if code == C.F32 else torch.bfloat16
    g = torch.Generator(device="cuda").manual_seed(code)
    bits = torch.randint(0, 1 << (23 if code == C.F32 else 7), (n,), generator=g, device="cuda")
    tiny = bits.to(torch.int32 if code == C.F32 else torch.int16).view(dt)
    ref = torch.cumsum(tiny.to(torch.float64), 0)
    got = C.inclusive_scan(tiny).to(torch.float64)
    # one fp32 rounding: relative, or half a denormal step of 2^-149
    assert ((got - ref).abs() <= 1e-6 * ref + 2.0**-149).all()
    assert (C.inclusive_scan(torch.full((n,), -0.0, device="cuda", dtype=dt)) == 0).all()
    x = torch.rand(n, generator=g, device="cuda").to(dt)
    for at, value in ((n // 2 + 3, float("inf")), (n // 3, float("-inf")), (n - 2, float("nan"))):
        y = x.clone()
        y[at] = value
        ref = torch.cumsum(y.to(torch.float64), 0)
        for got, start in ((C.inclusive_scan(y), at), (C.exclusive_scan(y, 0.0), at + 1)):
            # (the double-float carry of an infinity is (inf, NaN): NaN in later tiles)
            assert not torch.isfinite(got[start:]).any()
            assert got[start].item() == value or value != value
            assert torch.isfinite(got[:start]).all()
        inc = C.inclusive_scan(y)[:at].to(torch.float64)
        assert ((inc - ref[:at]).abs() <= 1e-6 * ref[:at]).all()


@pytest.mark.parametrize("busy", ["elementwise", "sort", "scans"])
def test_small_look_back_calls_beside_another_stream(dev, busy):
    """Scans and copy_if whose blocks all fit on an empty GPU, while another
    stream's work holds most of it (elementwise kernels, a sort's persistent
    blocks, or look-back calls of its own), so that their blocks start late
    and not together: exact results, and no wait has run out."""
    ours, other = torch.cuda.Stream(), torch.cuda.Stream()
    g = torch.Generator(device="cuda").manual_seed(3)
    big = torch.randint(0, 1 << 30, (1 << 26,), generator=g, device="cuda", dtype=torch.int32)
    x = torch.randint(0, 1 << 20, ((1 << 20) + 3,), generator=g, device="cuda", dtype=torch.int32)
    ref = torch.cumsum(x, 0).to(torch.int32)
    keep = x[(x & 7) < 3]
    torch.cuda.synchronize()
    for n in (5000, 300007, (1 << 20) + 3):
        kept = int(((x[:n] & 7) < 3).sum())
        torch.cuda.synchronize()
        if busy == "elementwise":
            with torch.cuda.stream(other):
                y = big.float()
                for _ in range(6):
                    y = torch.sin(y)
        elif busy == "sort":
            with torch.cuda.stream(other):
                y = big.clone()
            C.sort_(y, stream=other)
        got = []
        for _ in range(40):
            with torch.cuda.stream(ours):
                got.append((C.inclusive_scan(x[:n], stream=ours), C.copy_if(x[:n], 7, C.CMP_LT, 3, stream=ours)))
            if busy == "scans":
                with torch.cuda.stream(other):
                    y = C.inclusive_scan(x, stream=other)
        torch.cuda.synchronize()
        for s, (out, cnt) in got:
            assert torch.equal(s, ref[:n]), n
            assert int(cnt.item()) == kept and torch.equal(out[:kept], keep[:kept]), n
        assert C.device_error(ours) == C.OK and C.device_error(other) == C.OK


@pytest.mark.parametrize("code", [C.U32, C.I64, C.F32, C.BF16, C.F64])
def test_scan_and_copy_if_at_the_wave_rules(dev, code):
    """Sizes on both sides of the rules that count the look-back blocks an SM
    holds (7 x 2^18, 37 x 2^15, 37 x 2^16, 110 x 2^14 and 55 x 2^16 elements): scans
    against torch's cumulative sum, copy_if against a mask, integers exact,
    floats within 1e-6."""
    g = torch.Generator(device="cuda").manual_seed(code)
    for edge in (1 << 20, 37 << 15, 110 << 14, 7 << 18, 1 << 21, 37 << 16, 55 << 16):
        for n in (edge, edge + 1):
            if code in (C.U32, C.I64):
                x = torch.randint(0, 1 << 20, (n,), generator=g, device="cuda")
                ref = torch.cumsum(x, 0)
                y = x if code == C.I64 else x.to(torch.uint32)
                got = C.inclusive_scan(y).to(torch.int64)
                assert torch.equal(got, ref if code == C.I64 else ref & 0xFFFFFFFF), n
                out, cnt = C.copy_if(y, 7, C.CMP_LT, 5)
                keep, k = x[(x & 7) < 5], int(cnt.item())
                assert k == keep.numel() and torch.equal(out[:k].to(torch.int64), keep), n
            else:
                dt = {C.F32: torch.float32, C.BF16: torch.bfloat16, C.F64: torch.float64}[code]
                x = torch.rand(n, generator=g, device="cuda").to(dt)
                ref = torch.cumsum(x.to(torch.float64), 0)
                got = C.inclusive_scan(x).to(torch.float64)
                assert ((got - ref).abs() <= 1e-6 * ref.abs() + 1e-30).all(), n


def canonical_sum(x, init, chains, lift, off_bytes):
    """The canonical sum of a 1-D array as numpy restates it: runs of 32 lanes x
    16 vectors of 16 bytes, `chains` accumulators per lane, a lane butterfly, the
    512-wide halving tree over the runs, then head, body and tail.  fp32 and
    bf16 (chains 2 and 4) accumulate in double-float, fp64 plainly."""
    df = chains > 1
    ft = np.float32 if df else np.float64

    def two_sum(a, b):
        s = a + b
        bp = s - a
        return s, (a - (s - bp)) + (b - bp)

    def add(acc, v):
        if not df:
            return (acc[0] + v,)
        s, e = two_sum(acc[0], v)
        return s, acc[1] + e

    def comb(a, b):
        if not df:
            return (a[0] + b[0],)
        s, e = two_sum(a[0], b[0])
        e = e + (a[1] + b[1])
        h = s + e
        return h, e - (h - s)

    def norm(a):
        if not df:
            return a
        h = a[0] + a[1]
        return h, a[1] - (h - a[0])

    def zero(shape=()):
        return tuple(np.zeros(shape, ft) for _ in range(2 if df else 1))

    def ends(part):
        acc = zero()
        for v in lift(part):
            acc = add(acc, v)
        return norm(acc)

    es = x.itemsize
    vec = 16 // es
    head = min((16 - off_bytes % 16) % 16 // es, x.size)
    nvec = (x.size - head) // vec
    body = lift(x[head:head + nvec * vec]).reshape(nvec, vec)
    runs = -(-nvec // 512)
    padded = np.zeros((runs * 512, vec), ft)
    padded[:nvec] = body
    real = (np.arange(runs * 512) < nvec).reshape(runs, 16, 32)
    padded = padded.reshape(runs, 16, 32, vec)
    accs = [zero((runs, 32)) for _ in range(chains)]
    for j in range(16):
        for e in range(vec):
            new = add(accs[e % chains], padded[:, j, :, e])
            accs[e % chains] = tuple(np.where(real[:, j], n, o) for n, o in zip(new, accs[e % chains]))
    if chains == 4:
        accs = [comb(accs[0], accs[1]), comb(accs[2], accs[3])]
    lane = norm(comb(accs[0], accs[1]) if df else accs[0])
    for m in (16, 8, 4, 2, 1):
        lane = comb(lane, tuple(a[:, np.arange(32) ^ m] for a in lane))
    slots = zero(512)
    for s, a in zip(slots, lane):
        s[:runs] = a[:, 0]
    slots = comb(zero(512), slots)
    w = 256
    while w:
        slots = comb(tuple(s[:w] for s in slots), tuple(s[w:2 * w] for s in slots))
        w //= 2
    total = comb(comb(ends(x[:head]), tuple(s[0] for s in slots)), ends(x[head + nvec * vec:]))
    total = comb((ft(init), ft(0)) if df else (ft(init),), total)
    return ft(total[0] + total[1]) if df else ft(total[0])


@pytest.mark.parametrize("code", [C.F32, C.BF16, C.F64])
def test_reduce_bits_follow_the_canonical_tree(dev, code):
    """Sums of up to 32 runs (the one-block kernel) and of 33 to 70 (the kernel of
    the long reduces), at starts on and off a 16-byte boundary: the bits of the
    canonical tree restated in numpy."""
    es = {C.F32: 4, C.BF16: 2, C.F64: 8}[code]
    run = 8192 // es
    rng = np.random.default_rng(code)
    for n in (1, 16 // es, run - 1, run, 5 * run + 3, 31 * run + 7, 32 * run, 32 * run + 16 // es, 33 * run + 5, 70 * run):
        for off in (0, 1):
            x = rng.standard_normal(n) * np.exp(rng.standard_normal(n) * 4)
            if code == C.BF16:
                t = torch.from_numpy(x).to(torch.bfloat16)
                bits = t.view(torch.int16).numpy().view(np.uint16)
                ref = canonical_sum(bits, 0.5, 4, lambda b: (b.astype(np.uint32) << 16).view(np.float32), off * es)
            else:
                ft = np.float32 if code == C.F32 else np.float64
                x = x.astype(ft)
                t = torch.from_numpy(x)
                ref = canonical_sum(x, 0.5, 2 if code == C.F32 else 1, lambda b: b, off * es)
            base = torch.zeros(n + off, dtype=t.dtype, device="cuda")
            base[off:] = t.cuda()
            for cfg in (C.AUTO, 0, 47):
                got = C.reduce(base[off:], "sum", init=0.5, config=cfg).cpu().numpy()[0]
                assert got.tobytes() == ref.tobytes(), (n, off, cfg, got, ref)
