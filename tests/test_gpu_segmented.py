"""Segmented reduce / scan (one persistent launch for all segments) and the
CUDA-graph plans, against per-segment oracle calls."""
import ctypes

import numpy as np
import pytest
import torch

from opensycl_b200 import capi as C
from oracle import oracle as O

pytestmark = pytest.mark.gpu

NP = {C.I32: np.int32, C.I64: np.int64, C.F32: np.float32, C.F64: np.float64}
SEG_CONFIGS = [0, 6, 22, 41, C.AUTO]


def make_offsets(rng, nseg, kind):
    if kind == "small":
        lens = rng.integers(0, 40, nseg)
    elif kind == "mixed":
        lens = np.floor(2.0 ** (rng.random(nseg) * 17)).astype(np.int64)
        lens[rng.random(nseg) < 0.1] = 0
    else:  # long: many pieces per segment
        lens = rng.integers(20000, 90000, nseg)
    return np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)


def values(rng, code, n):
    if code in (C.F32, C.F64):
        return rng.standard_normal(n).astype(NP[code])
    return rng.integers(-(1 << 20), 1 << 20, n).astype(NP[code])


def valid(code, cfgs):
    L = C.lib()
    return [c for c in cfgs if c == C.AUTO or L.b2p_config_valid(C.PRIM_SEG_REDUCE, code, c)]


@pytest.mark.parametrize("kind", ["small", "mixed", "long"])
@pytest.mark.parametrize("code", [C.I32, C.I64, C.F32])
def test_segmented_reduce(dev, kind, code):
    rng = np.random.default_rng(hash((kind, code)) % 2**32)
    nseg = {"small": 3000, "mixed": 700, "long": 40}[kind]
    offs = make_offsets(rng, nseg, kind)
    x = values(rng, code, int(offs[-1]))
    xd = torch.from_numpy(x).cuda()
    od = torch.from_numpy(offs).cuda()
    if code == C.F32:
        ref = O.fp64_segmented_sum(code, x, offs)
        sabs = np.array([np.abs(x[offs[s]:offs[s + 1]]).astype(np.float64).sum() for s in range(nseg)])
    else:
        ref = O.segmented_reduce(code, C.SUM, x, offs)
    for cfg in valid(code, SEG_CONFIGS):
        got = C.segmented_reduce(xd, od, "sum", config=cfg).cpu().numpy()
        if code == C.F32:
            err = np.abs(got.astype(np.float64) - ref)
            assert np.all(err <= 1e-6 * np.abs(ref) + 1e-12 * sabs + 1e-30), (kind, cfg)
        else:
            assert np.array_equal(got, ref), (kind, cfg)
    if code != C.F32:
        for op in (C.MIN, C.MAX):
            got = C.segmented_reduce(xd, od, op, config=C.AUTO).cpu().numpy()
            info = np.iinfo(NP[code])
            ident = info.max if op == C.MIN else info.min
            exp = np.array([(x[offs[s]:offs[s + 1]].min() if op == C.MIN else x[offs[s]:offs[s + 1]].max())
                            if offs[s + 1] > offs[s] else ident for s in range(nseg)], dtype=NP[code])
            assert np.array_equal(got, exp)


@pytest.mark.parametrize("kind", ["small", "mixed", "long"])
@pytest.mark.parametrize("code", [C.I64, C.F32])
def test_segmented_scan(dev, kind, code):
    rng = np.random.default_rng(7 + hash((kind, code)) % 2**31)
    nseg = {"small": 2000, "mixed": 500, "long": 30}[kind]
    offs = make_offsets(rng, nseg, kind)
    x = values(rng, code, int(offs[-1]))
    if code == C.F32:
        x = np.abs(x)
    xd = torch.from_numpy(x).cuda()
    od = torch.from_numpy(offs).cuda()
    for cfg in valid(code, SEG_CONFIGS):
        for inclusive, init in ((True, None), (True, 3), (False, 5)):
            got = C.segmented_scan(xd, od, inclusive, "sum", init, config=cfg).cpu().numpy()
            if code == C.F32:
                ref = np.concatenate([O.fp64_scan(O.F32, inclusive, x[offs[s]:offs[s + 1]],
                                                  float(init or 0)) for s in range(nseg)
                                      if offs[s + 1] > offs[s]])
                ok = np.abs(got.astype(np.float64) - ref) <= 1e-6 * np.abs(ref) + 1e-30
                assert ok.all(), (kind, cfg, inclusive)
            else:
                ref = O.segmented_scan(code, C.SUM, inclusive, x, offs, init)
                assert np.array_equal(got, ref), (kind, cfg, inclusive, init)


def test_segmented_plan_graph(dev):
    rng = np.random.default_rng(3)
    offs = make_offsets(rng, 1000, "mixed")
    x = values(rng, C.I64, int(offs[-1]))
    xd = torch.from_numpy(x).cuda()
    od = torch.from_numpy(offs).cuda()
    out = torch.zeros(1000, dtype=torch.int64, device="cuda")
    L = C.lib()
    plan = ctypes.c_void_p()
    s = torch.cuda.current_stream()
    C.check(L.b2p_plan_segmented(ctypes.byref(plan), C.PRIM_SEG_REDUCE, C.I64, C.SUM, xd.data_ptr(),
                                 out.data_ptr(), od.data_ptr(), 1000, int(offs[-1]), C.AUTO,
                                 ctypes.c_void_p(s.cuda_stream)), "plan")
    ref = O.segmented_reduce(C.I64, C.SUM, x, offs)
    for _ in range(3):
        out.zero_()
        C.check(L.b2p_plan_launch(plan, ctypes.c_void_p(s.cuda_stream)), "launch")
        assert np.array_equal(out.cpu().numpy(), ref)
    assert 0 <= L.b2p_plan_config(plan) < 48
    L.b2p_plan_destroy(plan)


@pytest.mark.parametrize("flat", [18, 22, 23])
def test_segmented_kernels_share_scratch_at_every_epoch(dev, flat):
    """The pipelined kernel's boundary records (a tile without a boundary
    inside holds tile + 1 = 0x801, 0x1001 or 0x2001) and the piece kernel's
    pieces stay in the scratch body; a look-back of the other kernel over the
    same bytes must not take one for a status word of its launch, whatever
    the launch's epoch (those values once read as "aggregate of epoch 8, 16
    or 32")."""
    rng = np.random.default_rng(flat)
    lens = rng.integers(20000, 40000, 60)
    offs = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    x = values(rng, C.I32, int(offs[-1]))
    xd, od = torch.from_numpy(x).cuda(), torch.from_numpy(offs).cuda()
    ref = O.segmented_reduce(C.I32, C.SUM, x, offs)
    C.Scratch.release()
    C.Scratch.get(C.lib().b2p_scratch_bytes(C.PRIM_SEG_REDUCE, C.I32, x.size, 60, C.AUTO) + 256)
    assert np.array_equal(C.segmented_reduce(xd, od, "sum", config=0).cpu().numpy(), ref)  # epoch 0
    for epoch in range(1, 35, 2):
        assert np.array_equal(C.segmented_reduce(xd, od, "sum", config=flat).cpu().numpy(), ref), epoch
        assert np.array_equal(C.segmented_reduce(xd, od, "sum", config=0).cpu().numpy(), ref), epoch + 1


@pytest.mark.parametrize("nseg", [1024, 1025, 16 * 1024 + 1, 40000])
def test_segmented_offsets_checked_on_device(dev, nseg):
    """Offset arrays on both sides of the limits of the device-side check (one
    block up to 16,384 segments) and of a tile's boundary record (62): many
    empty segments at one place and at the end, hundreds of boundaries in one
    tile, and one long segment over many tiles.  A decreasing pair anywhere,
    or a negative first offset, is refused and leaves the output alone."""
    rng = np.random.default_rng(nseg)
    lens = rng.integers(0, 30, nseg)
    lens[nseg // 3:nseg // 3 + 200] = 0
    lens[nseg // 2] = 300000
    lens[-5:] = 0
    offs = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    x = values(rng, C.I64, int(offs[-1]))
    xd, od = torch.from_numpy(x).cuda(), torch.from_numpy(offs).cuda()
    got = C.segmented_reduce(xd, od, "sum").cpu().numpy()
    assert np.array_equal(got, O.segmented_reduce(C.I64, C.SUM, x, offs))
    got = C.segmented_scan(xd, od, False, "sum", 5).cpu().numpy()
    assert np.array_equal(got, O.segmented_scan(C.I64, C.SUM, False, x, offs, 5))
    for at in (1, nseg // 2 + 1, nseg - 1):
        bad = offs.copy()
        bad[at] = bad[at + 1] + 1
        out = torch.full((nseg,), 7, dtype=torch.int64, device="cuda")
        with pytest.raises(C.B2PError) as e:
            C.segmented_reduce(xd, torch.from_numpy(bad).cuda(), "sum", out=out)
        assert e.value.status == C.ERR_INVALID_ARG and bool((out == 7).all())
    bad = offs.copy()
    bad[0] = -1
    with pytest.raises(C.B2PError):
        C.segmented_reduce(xd, torch.from_numpy(bad).cuda(), "sum")


@pytest.mark.parametrize("code", [C.F32, C.BF16])
@pytest.mark.parametrize("inclusive", [True, False])
def test_segmented_scan_special_values(dev, code, inclusive):
    """Long and short segments with denormals, and an infinity or a NaN in some
    of them: those segments are not finite from that element on, every other
    output is within 1e-6 of FP64 sums."""
    n, dt = 3 * 8192 * 40 + 777, torch.float32 if code == C.F32 else torch.bfloat16
    rng = np.random.default_rng(int(code) + inclusive)
    cuts = np.unique(np.concatenate([rng.integers(0, n, 60), rng.integers(n // 2, n // 2 + 4000, 200), [0, n]]))
    x = torch.from_numpy(rng.random(n).astype(np.float32)).to(dt)
    x[1000:9000] = torch.finfo(dt).tiny / 4
    seg = np.searchsorted(cuts, np.arange(n), side="right") - 1
    bad_at = {int(seg[i]): int(i) for i in (n // 3, n // 2 + 1500, n - 5)}
    for (s, i), v in zip(sorted(bad_at.items()), (float("inf"), float("-inf"), float("nan"))):
        x[i] = v
    xd = x.to(dev)
    offsets = torch.from_numpy(cuts.astype(np.int64)).to(dev)
    got = C.segmented_scan(xd, offsets, inclusive=inclusive, init=None if inclusive else 0.0).double().cpu().numpy()
    xs = x.double().numpy()
    for s in range(len(cuts) - 1):
        a, b = cuts[s], cuts[s + 1]
        fin = bad_at[s] + (0 if inclusive else 1) if s in bad_at else b
        ref = np.cumsum(xs[a:b]) if inclusive else np.concatenate([[0.0], np.cumsum(xs[a:b])[:-1]])
        k = fin - a
        assert (np.abs(got[a:fin] - ref[:k]) <= 1e-6 * np.abs(ref[:k]) + 2.0**-149).all(), s
        assert not np.isfinite(got[fin:b]).any(), s


def test_segmented_reduce_sixteen_stage_tiles(dev):
    """bf16 at 256 x 16 (8 KiB tiles, the shape with the most input stages):
    many tiles per reducer group, sums within 1e-6 of FP64."""
    n, nseg, cfg = (1 << 24) + 321, 900, 16 + 4 + 2
    g = torch.Generator(device="cuda").manual_seed(5)
    x = torch.rand(n, generator=g, device="cuda").to(torch.bfloat16)
    cuts = torch.sort(torch.randint(0, n, (nseg - 1,), generator=g, device="cuda")).values
    offsets = torch.cat([cuts.new_zeros(1), cuts, cuts.new_full((1,), n)])
    total = torch.cat([cuts.new_zeros(1, dtype=torch.float64), torch.cumsum(x.double(), 0)])
    ref = total[offsets[1:]] - total[offsets[:-1]]
    got = C.segmented_reduce(x, offsets, config=cfg).double()
    assert ((got - ref).abs() <= 1e-6 * ref + 1e-6).all()


@pytest.mark.parametrize("prim", [C.PRIM_SEG_REDUCE, C.PRIM_SEG_SCAN])
@pytest.mark.parametrize("shape", ["long", "many", "min"])
def test_plan_with_offsets_in_host_memory(dev, prim, shape):
    """A plan takes offsets in pageable host memory: long segments (boundary
    records), hundreds of boundaries in a tile (offsets read by the launch),
    and an operator of the piece kernel.  The offsets may change afterwards."""
    rng = np.random.default_rng(11)
    lens = rng.integers(20000, 40000, 40) if shape != "many" else rng.integers(0, 30, 20000)
    offs = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    op = C.MIN if shape == "min" else C.SUM
    x = values(rng, C.I64, int(offs[-1]))
    ref = O.segmented_reduce(C.I64, op, x, offs) if prim == C.PRIM_SEG_REDUCE else \
        O.segmented_scan(C.I64, op, True, x, offs)
    xd = torch.from_numpy(x).cuda()
    out = torch.zeros(ref.size, dtype=torch.int64, device="cuda")
    plan, st = ctypes.c_void_p(), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    host = offs.copy()
    C.check(C.lib().b2p_plan_segmented(ctypes.byref(plan), prim, C.I64, op, xd.data_ptr(), out.data_ptr(),
                                       host.ctypes.data, lens.size, x.size, C.AUTO, st))
    host[:] = -1
    for _ in range(2):
        out.zero_()
        C.check(C.lib().b2p_plan_launch(plan, st))
        assert np.array_equal(out.cpu().numpy(), ref)
    torch.cuda.synchronize()
    C.lib().b2p_plan_destroy(plan)
