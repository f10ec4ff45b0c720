"""The kernels that multiply raw quants on the warp-level tensor-core instructions - csrc/gemv_hm.cu (16-bit activations, 1..8 rows), csrc/gemv_mb.cu
(Q5_K, Q4_0, Q6_K with any activations, 1..8 rows) and csrc/gemm_mm.cu (Q5_K, Q4_0, from nine tokens) - against the oracle's 64-bit sums.
gemv_hm multiplies the activations as they are; the other two hold them in fixed point (30 bits, 62 for one FP32 row) or as FP16 terms (22 bits of
each value) and leave rows that these do not hold to a plain FP32 loop, so in all of them a result is a sum of a few hundred FP32 terms with
errors of at most 2^-22 each (sqrt(K / 32 + 16) * 2^-24 and less than 2^-21 for the terms: below 2e-6 over a row for K <= 14336), which is the bound.
Sizes: one row, ragged tiles of 16, fewer rows than SMs, several row tiles per CTA, several passes over a CTA's rows, K of one block, of
an odd number of blocks (Q6_K rows that start on any even byte) and of more blocks than a CTA has warps."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

import oracle
from brotensor_b200 import _capi, synth

PLAIN, DP, HM, MB, MM = 1, 3, 6, 7, 8  # what the option "last_kernel" calls them
FMTS = [synth.Q4_K, synth.Q5_K, synth.Q6_K, synth.Q8_0, synth.Q4_0]
SHAPES = [(1, 256), (15, 512), (37, 768), (300, 6912), (2373, 1024), (40, 14336), (20000, 256)]
DT = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}


@pytest.fixture
def ops_raw():
    from brotensor_b200 import ops
    yield ops
    for key in ("gemv_hm", "gemv_mb", "gemm_mm"):
        ops.set_option(key, 1)
    ops.set_option("pdl", 0)
    assert ops.device_status() == 0


def _last_kernel():
    v = ctypes.c_int(0)
    _capi.check(_capi.lib().b200q_get_option(b"last_kernel", ctypes.byref(v)))
    return v.value


def _operands(fmt, N, K, M, dtype):
    Wh = synth.make_blocks(fmt, N, K, seed=N + K)
    x = torch.from_numpy(synth.make_activations(M, K, seed=M + K)).to(DT[dtype])
    b = torch.from_numpy(synth.make_activations(1, N, seed=5).reshape(-1)).to(DT[dtype])
    want = oracle.cpu().matmul(fmt, Wh, x.float().numpy(), bias=b.float().numpy(), threads=8, want_f64=True)[1]
    return torch.from_numpy(Wh).cuda(), x.cuda(), b.cuda(), want


@pytest.mark.gpu
@pytest.mark.parametrize("N,K", SHAPES + [(40000, 768)])  # the last: several row sets per CTA, activations resident in gemv_hm
@pytest.mark.parametrize("fmt", FMTS)
def test_decode_rows(fmt, N, K, ops_raw):
    ops = ops_raw
    for M, dtype in ((1, "f16"), (2, "bf16"), (3, "f32"), (5, "bf16"), (7, "f32"), (8, "bf16"), (8, "f16")):
        W, x, b, want = _operands(fmt, N, K, M, dtype)
        for kernel in ("gemv_hm", "gemv_mb"):
            if kernel == "gemv_hm" and dtype == "f32":
                continue
            ops.set_option("gemv_hm", 2 if kernel == "gemv_hm" else 0)
            ops.set_option("gemv_mb", 2)
            if kernel == "gemv_mb" and fmt in (synth.Q4_K, synth.Q8_0):
                continue
            y = ops.gemv(fmt, W, x, N, bias=b, out_dtype=torch.float32)
            assert _last_kernel() == (HM if kernel == "gemv_hm" else MB), (kernel, M, dtype)
            assert oracle.rel_l2(y.cpu().numpy(), want) < 2e-6, (kernel, M, dtype)
            assert torch.equal(y, ops.gemv(fmt, W, x, N, bias=b, out_dtype=torch.float32))  # fixed order of additions
            for early in (-1, 1):
                ops.set_option("pdl", early)
                assert torch.equal(y, ops.gemv(fmt, W, x, N, bias=b, out_dtype=torch.float32))
            ops.set_option("pdl", 0)
            half = ops.gemv(fmt, W, x, N, bias=b, out_dtype=torch.float16)
            assert torch.equal(half, y.half())  # one rounding of the same sums


@pytest.mark.gpu
@pytest.mark.parametrize("N,K", SHAPES)
@pytest.mark.parametrize("fmt", [synth.Q5_K, synth.Q4_0])
def test_a_few_dozen_tokens(fmt, N, K, ops_raw):
    ops = ops_raw
    for M, dtype in ((9, "f16"), (17, "f32"), (33, "bf16"), (64, "f16"), (65, "f32"), (131, "f16")):
        if N * K * M > 4e8:
            continue
        W, x, b, want = _operands(fmt, N, K, M, dtype)
        ops.set_option("gemv_hm", 0)  # (up to sixteen rows of 16-bit activations are its)
        y = ops.linear(fmt, W, x, N, bias=b, out_dtype=torch.float32)
        assert _last_kernel() == MM, (M, dtype)
        assert oracle.rel_l2(y.cpu().numpy(), want) < 2e-6, (M, dtype)
        assert torch.equal(y, ops.linear(fmt, W, x, N, bias=b, out_dtype=torch.float32))


@pytest.mark.gpu
@pytest.mark.parametrize("fmt,N,K", [(synth.Q8_0, 640, 14336), (synth.Q8_0, 640, 4096), (synth.Q6_K, 1024, 12288), (synth.Q5_K, 300, 8192), (synth.Q4_K, 40, 4096)])
def test_matrices_of_few_rows_and_many_activations(fmt, N, K, ops_raw):
    """Blocks of long rows beside eight activation rows: as many per stage as fit, on the same kernel."""
    ops = ops_raw
    for M in (6, 7, 8, 9, 16):
        W, x, b, want = _operands(fmt, N, K, M, "f16")
        ops.set_option("gemv_i8", 0)  # (K = 4096 of Q8_0 / Q4_K has another kernel for eight rows)
        ops.set_option("gemv_hm", 2)
        y = ops.linear(fmt, W, x, N, bias=b, out_dtype=torch.float32)
        ops.set_option("gemv_i8", 1)
        assert _last_kernel() == HM, M
        assert oracle.rel_l2(y.cpu().numpy(), want) < 2e-6, M


@pytest.mark.gpu
@pytest.mark.parametrize("fmt,N,K,M,kernel", [(synth.Q6_K, 2048, 4096, 2, HM), (synth.Q6_K, 2048, 8192, 2, DP), (synth.Q6_K, 1024, 14336, 2, DP),
                                              (synth.Q6_K, 2048, 14336, 3, HM), (synth.Q4_K, 2048, 4096, 2, HM), (synth.Q4_K, 3072, 4096, 2, DP),
                                              (synth.Q4_K, 6912, 2560, 2, HM), (synth.Q4_0, 20000, 512, 1, HM), (synth.Q5_K, 9000, 512, 1, MB)])
def test_where_the_lines_lie(fmt, N, K, M, kernel, ops_raw):
    W, x, b, want = _operands(fmt, N, K, M, "f16")
    y = ops_raw.gemv(fmt, W, x, N, bias=b, out_dtype=torch.float32)
    assert _last_kernel() == kernel
    assert oracle.rel_l2(y.cpu().numpy(), want) < (2e-3 if kernel == DP else 2e-6)  # (15-bit fixed point in the integer-dot kernel)


@pytest.mark.gpu
def test_weights_on_two_byte_boundaries(ops_raw):
    """Q6_K rows may start anywhere; the other formats' unaligned weights keep going to the plain kernel."""
    ops = ops_raw
    for fmt, shift in ((synth.Q6_K, 2), (synth.Q6_K, 14), (synth.Q8_0, 2), (synth.Q4_0, 6), (synth.Q5_K, 4)):
        N, K = 77, 1280
        for M, dtype in ((1, "f16"), (4, "f32"), (20, "f16")):
            W, x, b, want = _operands(fmt, N, K, M, dtype)
            buf = torch.zeros(W.numel() + 64, dtype=torch.uint8, device="cuda")
            moved = buf[shift:shift + W.numel()]
            moved.copy_(W.reshape(-1))
            y = ops.linear(fmt, moved, x, N, bias=b, out_dtype=torch.float32)
            assert _last_kernel() == (PLAIN if fmt != synth.Q6_K else MB if dtype == "f32" else HM), (fmt, shift, M)
            assert oracle.rel_l2(y.cpu().numpy(), want) < 2e-6, (fmt, shift, M)


@pytest.mark.gpu
@pytest.mark.parametrize("fmt", FMTS)
def test_activations_that_are_not_finite(fmt, ops_raw):
    """Infinities and NaN give what FP32 arithmetic on the decoded weights gives."""
    ops = ops_raw
    N, K = 200, 1024
    W = torch.from_numpy(synth.make_blocks(fmt, N, K, seed=3)).cuda()
    plain = fmt in (synth.Q5_K, synth.Q4_0)  # formats whose every form sums in FP32
    for M, dtype in ((3, "f16"), (3, "f32"), (20, "f16"), (20, "f32")):
        if not plain and (M > 8 or (dtype == "f32" and fmt != synth.Q6_K)):
            continue
        for value in (float("inf"), float("-inf"), float("nan")):
            x = torch.from_numpy(synth.make_activations(M, K, seed=4)).to(DT[dtype]).cuda()
            x[1, 77] = value
            y = ops.linear(fmt, W, x, N, out_dtype=torch.float32)
            ops.set_option("gemv_path", 1)
            want = torch.cat([ops.gemv(fmt, W, x[i:i + 1], N, out_dtype=torch.float32) for i in range(M)])
            ops.set_option("gemv_path", 0)
            assert torch.equal(torch.isnan(y), torch.isnan(want)) and torch.equal(torch.isinf(y), torch.isinf(want))
            ok = torch.isfinite(want)
            assert torch.allclose(y[ok], want[ok], rtol=1e-4, atol=1e-4)


@pytest.mark.gpu
@pytest.mark.parametrize("fmt", FMTS)
def test_scales_that_are_not_finite(fmt, ops_raw):
    """A block whose FP16 scale is infinite gives what FP32 arithmetic on the decoded weights gives, also where its quants sum up to nothing."""
    ops = ops_raw
    N, K = 200, 1280
    at = 208 if fmt == synth.Q6_K else 0
    blocks = synth.make_blocks(fmt, N, K, seed=3).reshape(-1, synth.BLOCK_BYTES[fmt])
    per_row = blocks.shape[0] // N
    for row, bits in ((3, 0x7C00), (77, 0xFC00), (130, 0x7E00)):
        blocks[row * per_row + 1, at:at + 2] = (bits & 255, bits >> 8)
    W = torch.from_numpy(blocks.reshape(-1).copy()).cuda()
    for M, dtype in ((1, "f32"), (1, "f16"), (3, "f16"), (3, "f32"), (7, "f32"), (20, "f16"), (20, "f32")):
        if fmt not in (synth.Q5_K, synth.Q4_0) and (M > 8 or (dtype == "f32" and fmt != synth.Q6_K)):
            continue  # (formats and types with other kernels)
        x = torch.from_numpy(synth.make_activations(M, K, seed=4)).to(DT[dtype]).cuda()
        x[0] = 0
        for hm in (1, 2, 0):
            if fmt in (synth.Q4_K, synth.Q8_0) and hm != 2:
                continue
            ops.set_option("gemv_hm", hm)
            y = ops.linear(fmt, W, x, N, out_dtype=torch.float32)
            assert _last_kernel() in (HM, MB, MM)
            ops.set_option("gemv_path", 1)
            want = torch.cat([ops.gemv(fmt, W, x[i:i + 1], N, out_dtype=torch.float32) for i in range(M)])
            ops.set_option("gemv_path", 0)
            assert not torch.isfinite(want).all()
            assert torch.equal(torch.isnan(y), torch.isnan(want)) and torch.equal(y[torch.isinf(y)], want[torch.isinf(want)])
            ok = torch.isfinite(want)
            assert torch.allclose(y[ok], want[ok], rtol=1e-4, atol=1e-4)


def _wide_operands(fmt, N, K, M, dtype, base=10.0):
    """Weights that are zero in one channel of every 256 and activations that are base^m times the others there (row m): the channel adds nothing to a
    result, but it sets the scale of whatever represents the 256 together."""
    blocks = synth.make_blocks(fmt, N, K, seed=N).reshape(-1, synth.BLOCK_BYTES[fmt])
    if fmt == synth.Q4_0:  # element 5 of every eighth block: nibble 8
        z = blocks.reshape(N, -1, 18)[:, ::8]
        z[..., 2 + 5] = (z[..., 2 + 5] & 0xF0) | 8
    elif fmt == synth.Q6_K:  # 6-bit value 32
        blocks[:, 5] &= 0xF0
        blocks[:, 128 + 5] = (blocks[:, 128 + 5] & 0xFC) | 2
    else:  # Q5_K: q = 0 and no min in the first sub-block
        blocks[:, 8] &= 0xC0
        blocks[:, 16 + 5] &= 0xFE
        blocks[:, 48 + 5] &= 0xF0
    x = synth.make_activations(M, K, seed=K)
    x[:, 5::256] *= (base ** np.arange(M, dtype=np.float64)[:, None]).astype(np.float32)
    x = torch.from_numpy(x).to(DT[dtype])
    assert torch.isfinite(x).all()
    want = oracle.cpu().matmul(fmt, blocks.reshape(-1), x.float().numpy(), threads=8, want_f64=True)[1]
    return torch.from_numpy(blocks.reshape(-1).copy()).cuda(), x.cuda(), want


@pytest.mark.gpu
@pytest.mark.parametrize("fmt", [synth.Q5_K, synth.Q6_K, synth.Q4_0])
def test_a_channel_far_above_the_others(fmt, ops_raw):
    """What a channel without weight costs the rest of its block: nothing, in FP32 as in the 16-bit types."""
    ops = ops_raw
    N, K = 90, 2304
    for M, dtype, base in ((8, "f32", 10), (8, "bf16", 10), (6, "f16", 6), (4, "f32", 100), (2, "f32", 1000), (2, "f32", 1e5)):
        W, x, want = _wide_operands(fmt, N, K, M, dtype, base)
        ops.set_option("gemv_hm", 0)
        ops.set_option("gemv_mb", 2)
        rows = ops.gemv(fmt, W, x, N, out_dtype=torch.float32)
        assert _last_kernel() == MB
        each = torch.cat([ops.gemv(fmt, W, x[m:m + 1], N, out_dtype=torch.float32) for m in range(M)])
        for m in range(M):
            for y in (rows, each):
                assert oracle.rel_l2(y[m].cpu().numpy(), want[m]) < 2e-6, (M, dtype, m)


@pytest.mark.gpu
@pytest.mark.parametrize("fmt", [synth.Q5_K, synth.Q4_0])
def test_a_channel_far_above_the_others_in_a_prompt(fmt, ops_raw):
    ops = ops_raw
    N, K = 90, 2304
    for M, dtype, base in ((20, "f32", 10), (20, "bf16", 30), (17, "f32", 30), (12, "f16", 2.2)):
        W, x, want = _wide_operands(fmt, N, K, M, dtype, base)
        ops.set_option("gemv_hm", 0)  # (up to sixteen rows of 16-bit activations are its)
        y = ops.linear(fmt, W, x, N, out_dtype=torch.float32).cpu().numpy()
        assert _last_kernel() == MM
        for m in range(M):
            assert oracle.rel_l2(y[m], want[m]) < 2e-6, (M, dtype, m)
    # the other end: a token whose largest value is near FP16's, and one far below FP32's normal scale
    Wh = synth.make_blocks(fmt, N, K, seed=2)
    for dtype, scale in (("f16", 12000.0), ("f32", 1e-35)):
        x = (torch.from_numpy(synth.make_activations(24, K, seed=9)) * scale).to(DT[dtype])
        want = oracle.cpu().matmul(fmt, Wh, x.float().numpy(), threads=8, want_f64=True)[1]
        y = ops.linear(fmt, torch.from_numpy(Wh).cuda(), x.cuda(), N, out_dtype=torch.float32).cpu().numpy()
        assert oracle.rel_l2(y / np.float32(scale), want / scale) < 2e-6


@pytest.mark.gpu
def test_magnitudes_that_fp16_cannot_hold(ops_raw):
    """FP32 and BF16 activations far outside FP16's range are scaled, not rounded away."""
    ops = ops_raw
    fmt, N, K = synth.Q5_K, 96, 2048
    Wh = synth.make_blocks(fmt, N, K, seed=8)
    W = torch.from_numpy(Wh).cuda()
    for M in (1, 2, 6, 24):
        for dtype in ("f32", "bf16"):
            for scale in (1e-30, 1e-25, 1e-6, 1e6, 1e25, 1e30):
                x = (torch.from_numpy(synth.make_activations(M, K, seed=9)) * scale).to(DT[dtype])
                want = oracle.cpu().matmul(fmt, Wh, x.float().numpy(), threads=8, want_f64=True)[1]
                y = ops.linear(fmt, W, x.cuda(), N, out_dtype=torch.float32).cpu().numpy()
                assert oracle.rel_l2(y / np.float32(scale), want / scale) < 2e-6
