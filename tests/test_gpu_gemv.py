"""GemvQuant parity: CUDA (through the C ABI) against the oracle's dequantise-then-dot.

Tolerance: 1e-3 relative / 1e-4 absolute against the oracle's double-precision accumulation of the
same bit-exact weights, the absolute term in units of the output vector's RMS (the synthetic block
scales give outputs of order 1e2..1e3, where 1e-4 in absolute terms is below what any f32 summation
order can resolve).  The oracle's f32 result (sequential summation, as nalgebra does) carries its own
rounding error of up to about K * 2^-24 * sum|w x|, so against it the absolute term is widened by
that bound."""
import numpy as np
import pytest
import torch

import oracle
from conftest import ATOL, RTOL, assert_close
from wgml_b200 import ops, synth

pytestmark = pytest.mark.gpu
ALL = [ops.F32, ops.F16, ops.Q4_0, ops.Q4_1, ops.Q5_0, ops.Q5_1, ops.Q8_0, ops.Q4_K, ops.Q5_K, ops.Q6_K, ops.Q8_K]


def make(qtype, nrows, ncols, seed):
    qt, arr = synth.matrix(qtype, nrows, ncols, seed, f"m{qtype}")
    x = np.random.default_rng(seed + 1).standard_normal(ncols).astype(np.float32)
    return np.ascontiguousarray(arr).view(np.uint8), x


def check(qtype, raw, nrows, ncols, x, out):
    o32, o64 = oracle.gemv_quant(qtype, raw, nrows, ncols, x, want_f64=True)
    atol = ATOL * max(1.0, float(np.sqrt(np.mean(o64 ** 2))))
    assert_close(out, o64, RTOL, atol, f"qtype {qtype} {nrows}x{ncols} vs f64 oracle")
    w = oracle.dequantize(qtype, raw).reshape(nrows, ncols)
    bound = ncols * 2.0 ** -24 * (np.abs(w.astype(np.float64)) @ np.abs(x.astype(np.float64)))
    err = np.abs(out.astype(np.float64) - o32)
    assert (err <= atol + RTOL * np.abs(o32) + bound).all(), f"qtype {qtype}: vs f32 oracle, worst {err.max()}"


@pytest.mark.parametrize("qtype", ALL)
@pytest.mark.parametrize("shape", [(4, 256), (37, 512), (1757, 768), (1024, 2816)])
def test_gemv_small(qtype, shape):
    nrows, ncols = shape
    raw, x = make(qtype, nrows, ncols, 7)
    m = ops.GpuQuantMatrix(qtype, raw, nrows, ncols)
    out = torch.full((nrows,), float("nan"), device="cuda")
    ops.GemvQuant.from_device().dispatch(out, m, torch.from_numpy(x).cuda())
    check(qtype, raw, nrows, ncols, x, out.cpu().numpy())


@pytest.mark.parametrize("qtype", [ops.Q4_K, ops.Q8_0, ops.Q6_K, ops.Q5_0, ops.F32])
def test_gemv_raw_blocks_on_device(qtype):
    nrows, ncols = 130, 1024
    raw, x = make(qtype, nrows, ncols, 11)
    out = torch.zeros(nrows, device="cuda")
    ops.GemvQuant.from_device().dispatch_raw(out, qtype, torch.from_numpy(raw).cuda(), nrows, ncols, torch.from_numpy(x).cuda())
    check(qtype, raw, nrows, ncols, x, out.cpu().numpy())


@pytest.mark.parametrize("qtype", [ops.Q8_0, ops.Q4_K, ops.Q6_K])
@pytest.mark.parametrize("shape", [(4096, 4096), (11008, 4096), (4096, 11008), (32000, 4096)])
def test_gemv_microbench_shapes_vs_oracle(qtype, shape):
    """The GEMV microbench configurations at full size."""
    nrows, ncols = shape
    raw, x = make(qtype, nrows, ncols, 13)
    m = ops.GpuQuantMatrix(qtype, raw, nrows, ncols)
    out = torch.zeros(nrows, device="cuda")
    g = ops.GemvQuant.from_device()
    xd = torch.from_numpy(x).cuda()
    g.dispatch(out, m, xd)
    o = out.cpu().numpy()
    check(qtype, raw, nrows, ncols, x, o)
    # linearity: W(2x - 3y) = 2Wx - 3Wy (size-independent property)
    y = torch.randn(ncols, device="cuda", generator=torch.Generator("cuda").manual_seed(3))
    out_y, out_c = torch.zeros_like(out), torch.zeros_like(out)
    g.dispatch(out_y, m, y)
    g.dispatch(out_c, m, (2 * xd - 3 * y).contiguous())
    lin = (2 * out - 3 * out_y).cpu().numpy()
    scale = float(np.abs(lin).max())
    assert np.abs(out_c.cpu().numpy() - lin).max() <= 1e-5 * scale


def test_gemv_70b_and_gpt2_shapes():
    for qtype, (nrows, ncols) in [(ops.Q4_K, (1024, 8192)), (ops.Q4_K, (8192, 28672)), (ops.Q8_0, (2304, 768)),
                                  (ops.Q8_0, (50257, 768)), (ops.Q8_0, (768, 3072))]:
        raw, x = make(qtype, nrows, ncols, 17)
        m = ops.GpuQuantMatrix(qtype, raw, nrows, ncols)
        out = torch.zeros(nrows, device="cuda")
        ops.GemvQuant.from_device().dispatch(out, m, torch.from_numpy(x).cuda())
        check(qtype, raw, nrows, ncols, x, out.cpu().numpy())


def test_gemv_dimension_mismatch_is_an_error():
    raw, x = make(ops.Q4_K, 8, 256, 1)
    m = ops.GpuQuantMatrix(ops.Q4_K, raw, 8, 256)
    g = ops.GemvQuant.from_device()
    with pytest.raises(ops.WgbError):
        g.dispatch(torch.zeros(8, device="cuda"), m, torch.zeros(255, device="cuda"))
    with pytest.raises(ops.WgbError):
        ops.GpuQuantMatrix(ops.Q4_K, raw, 8, 250)
    with pytest.raises(ops.WgbError):
        ops.GpuQuantMatrix(9, raw, 8, 256)  # Q8_1: unsupported by the reference as well


@pytest.mark.parametrize("qtype", [ops.Q4_K, ops.Q6_K, ops.Q8_0])
def test_gemv_outlier_inputs(qtype):
    """The fast kernels read the input in block fixed point (one exponent per 32 columns, 23 bits).  Inputs that
    stress it: twelve decades inside one 32-column group, groups of zeros, one huge element, denormal-sized
    values -- against the f64 oracle, same tolerance as everywhere."""
    nrows, ncols = 512, 4096
    raw, _ = make(qtype, nrows, ncols, 23)
    rng = np.random.default_rng(5)
    cases = {}
    x = rng.standard_normal(ncols).astype(np.float32)
    x[:32] *= np.float32(10.0) ** rng.uniform(-6, 6, 32).astype(np.float32)      # 12 decades in the first group
    x[32:64] = 0.0                                                                # an all-zero group
    x[64:96] = np.where(np.arange(32) == 7, np.float32(1e4), np.float32(1e-8))    # one outlier among tiny values
    cases["decades"] = x
    x = np.zeros(ncols, np.float32)
    x[1000] = 3.0e30
    x[1001] = -2.5
    cases["one huge element"] = x
    cases["tiny"] = (rng.standard_normal(ncols) * 1e-30).astype(np.float32)
    cases["zeros"] = np.zeros(ncols, np.float32)
    m = ops.GpuQuantMatrix(qtype, raw, nrows, ncols)
    g = ops.GemvQuant.from_device()
    for name, xv in cases.items():
        out = torch.full((nrows,), float("nan"), device="cuda")
        g.dispatch(out, m, torch.from_numpy(xv).cuda())
        o = out.cpu().numpy()
        assert np.isfinite(o).all(), name
        _, o64 = oracle.gemv_quant(qtype, raw, nrows, ncols, xv, want_f64=True)
        atol = ATOL * float(np.sqrt(np.mean(o64 ** 2))) if name != "zeros" else 0.0
        assert_close(o, o64, RTOL, atol, f"qtype {qtype}, {name}")


@pytest.mark.parametrize("qtype,cols", [(ops.Q4_K, (256, 2048, 2304, 4352, 51200)), (ops.Q6_K, (256, 2048, 2304, 4352, 48640)),
                                        (ops.Q8_0, (32, 96, 1024, 1056, 2080, 46080)), (ops.F32, (4, 60, 512, 516, 1088, 25600))])
@pytest.mark.parametrize("nrows", [1, 7, 9, 16, 1184, 1185, 2376])
def test_gemv_tile_edges(qtype, cols, nrows):
    """Rows around a tile of eight, of sixteen and the line between the two (148 tiles of eight); columns around a unit, a stage of
    eight units and two of them, down to one block and up to the longest row the fused kernel has ever taken.
    The input is held as 23-bit fixed point against the largest of 32 columns (2^-23 of it at most), the sums of a row are f32 in
    fewer than K / 32 + 64 steps, each within 2^-24 of the sum of magnitudes."""
    for ncols in cols:
        if ncols > 20000 and nrows > 16:
            continue
        raw, x = make(qtype, nrows, ncols, 29)
        out = torch.full((nrows,), float("nan"), device="cuda")
        ops.GemvQuant.from_device().dispatch(out, ops.GpuQuantMatrix(qtype, raw, nrows, ncols), torch.from_numpy(x).cuda())
        w = np.abs(oracle.dequantize(qtype, raw).reshape(nrows, ncols).astype(np.float64))
        pad = -ncols % 32
        top = np.repeat(np.abs(np.pad(x, (0, pad))).reshape(-1, 32).max(axis=1), 32)[:ncols].astype(np.float64)
        mags = w @ np.abs(x.astype(np.float64))
        if qtype in (ops.Q4_K, ops.Q6_K):   # codes and mins of a group are summed apart: magnitudes before the two cancel
            mags = mags + 2.0 * np.abs(w).reshape(nrows, -1, 32).max(axis=2) @ np.abs(x.astype(np.float64)).reshape(-1, 32).sum(axis=1)
        bound = 2.0 ** -23 * (w @ top) + (ncols / 32 + 64) * 2.0 ** -24 * mags
        _, o64 = oracle.gemv_quant(qtype, raw, nrows, ncols, x, want_f64=True)
        err = np.abs(out.cpu().numpy().astype(np.float64) - o64)
        assert (err <= bound).all(), f"qtype {qtype} {nrows}x{ncols}: {(err / np.maximum(bound, 1e-300)).max()}"


@pytest.mark.parametrize("qtype,cols", [(ops.F32, (48960, 48964, 53056, 53060)), (ops.Q4_K, (64768, 67584)), (ops.Q6_K, (57344, 61440)), (ops.Q8_0, (67488, 70304))])
def test_gemv_rows_around_the_longest(qtype, cols):
    """More rows than eight-row tiles for every block, rows around the two lines of the fused kernel: the longest that leaves room for a
    stage of sixteen rows, then stages of eight, then the general kernel.  Bound: 23-bit inputs and f32 sums in fewer than K / 32 + 64
    steps (general kernel: a chain of K / 32 per lane), as in test_gemv_tile_edges."""
    nrows = 1185
    for ncols in cols:
        raw, x = make(qtype, nrows, ncols, 31)
        out, xd = torch.full((nrows,), float("nan"), device="cuda"), torch.from_numpy(x).cuda()
        ops.GemvQuant.from_device().dispatch(out, ops.GpuQuantMatrix(qtype, raw, nrows, ncols), xd)
        w = torch.from_numpy(oracle.dequantize(qtype, raw).reshape(nrows, ncols)).cuda().double()
        exp = w @ xd.double()
        w.abs_()
        pad = torch.nn.functional.pad(xd.abs(), (0, -ncols % 32)).view(-1, 32)
        mags = w @ xd.abs().double()
        if qtype in (ops.Q4_K, ops.Q6_K):
            mags += 2.0 * w.view(nrows, -1, 32).amax(2) @ pad.sum(1).double()
        bound = 2.0 ** -23 * (w @ pad.amax(1).repeat_interleave(32)[:ncols].double()) + (ncols / 32 + 64) * 2.0 ** -24 * mags
        err = (out.double() - exp).abs()
        assert (err <= bound).all(), f"qtype {qtype} {nrows}x{ncols}: {(err / bound).max()}"


@pytest.mark.parametrize("qtype,ncols,stage", [(ops.F32, 11008, 512), (ops.F32, 22016, 512), (ops.Q8_0, 28672, 1024), (ops.Q8_0, 46080, 1024)])
def test_gemv_long_rows_are_not_one_chain(qtype, ncols, stage):
    """All weights 1, 2^24 in the first stage of columns and a 1 in each later one: an addition to the large sum loses the 1 (a tie, to
    even).  Stages go to four sums in turn, so a quarter of the additions are to the large one, and a few at the end (three between
    the sums, one between halves of a row): each within half an ulp, 1."""
    n = 24
    w = np.ones((n, ncols), np.float32)
    if qtype == ops.F32:
        raw = w.view(np.uint8)
    else:
        raw = np.concatenate([np.full((n * ncols // 32, 1), 1.0, np.float16).view(np.uint8).reshape(-1, 2), np.ones((n * ncols // 32, 32), np.uint8)], axis=1)
    assert np.array_equal(oracle.dequantize(qtype, raw.reshape(-1)).reshape(n, ncols), w)
    x = np.zeros(ncols, np.float32)
    x[0], x[stage + 64::stage] = 2.0 ** 24, 1.0
    stages = -(-ncols // stage)
    out = torch.zeros(n, device="cuda")
    ops.GemvQuant.from_device().dispatch(out, ops.GpuQuantMatrix(qtype, raw.reshape(-1), n, ncols), torch.from_numpy(x).cuda())
    err = np.abs(out.cpu().numpy().astype(np.float64) - x.astype(np.float64).sum()).max()
    assert err <= stages / 4 + 4, (err, stages)


@pytest.mark.parametrize("qtype,nrows,ncols", [
    (ops.F32, 32000, 288),      # one stage a tile: the consumer groups take tiles in turn, three epilogue warps
    (ops.F32, 60000, 32),       # the same with one unit at work
    (ops.Q8_0, 50257, 768),     # six units of a stage at work
    (ops.Q4_K, 26000, 4096),    # two stages a tile: a group always has the same columns
    (ops.Q4_K, 26000, 6144),    # three: they alternate
    (ops.Q6_K, 32000, 4096),    # a ring of six slots, an odd number would fit
    (ops.Q4_K, 9000, 28672),    # fourteen stages a tile, a ring of six: one epilogue warp
])
def test_ring_slots_used_many_times(qtype, nrows, ncols):
    """Matrices whose blocks go around the ring several times, in the ways consumer and epilogue warps can meet a slot's uses;
    called again and again, every output has the same bits."""
    raw, x = make(qtype, nrows, ncols, 17)
    m, xd, op = ops.GpuQuantMatrix(qtype, raw, nrows, ncols), torch.from_numpy(x).cuda(), ops.GemvQuant.from_device()
    outs = [torch.full((nrows,), float("nan"), device="cuda") for _ in range(16)]
    for o in outs:
        op.dispatch(o, m, xd)
    ops.device_status()
    for o in outs[1:]:
        assert torch.equal(o, outs[0])
    _, o64 = oracle.gemv_quant(qtype, raw, nrows, ncols, x, want_f64=True)
    assert_close(outs[0].cpu().numpy(), o64, RTOL, ATOL * max(1.0, float(np.sqrt(np.mean(o64 ** 2)))), f"qtype {qtype} {nrows}x{ncols}")
