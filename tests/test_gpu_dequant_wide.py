"""The wide decode kernels (32 values per thread, 16-bit outputs) and the generic one behind FP32, bit for bit against the oracle: rows of one
block and of an odd number of blocks, sizes below and above one thread block, the regrouped Q6_K layout, and weights that are not aligned for whole-header
loads (those take the generic kernel)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import oracle
from brotensor_b200 import synth

DT = {torch.float32: None, torch.float16: 1, torch.bfloat16: 4}


def _want(fmt, Wh, rows, K, dt):
    cpu = oracle.cpu()
    return cpu.dequant_f32(fmt, Wh, rows, K).view(np.uint32) if DT[dt] is None else cpu.dequant_16(fmt, Wh, rows, K, DT[dt])


def _bits(t, dt):
    return t.view(torch.int32 if dt == torch.float32 else torch.int16).cpu().numpy().view(np.uint32 if dt == torch.float32 else np.uint16)


@pytest.mark.gpu
@pytest.mark.parametrize("rows,K", [(1, 256), (3, 768), (37, 2048), (515, 6912), (4096, 1024)])
@pytest.mark.parametrize("fmt", [synth.Q4_K, synth.Q5_K, synth.Q6_K, synth.Q8_0, synth.Q4_0])
def test_decode_is_exact(fmt, rows, K):
    from brotensor_b200 import ops
    Wh = synth.make_blocks(fmt, rows, K, seed=rows + K)
    W = torch.from_numpy(Wh).cuda()
    buf = torch.zeros(W.numel() + 16, dtype=torch.uint8, device="cuda")
    shifted = buf[4:4 + W.numel()]  # on a 4-byte boundary only
    shifted.copy_(W.reshape(-1))
    for dt in DT:
        want = _want(fmt, Wh, rows, K, dt)
        assert np.array_equal(_bits(ops.dequant(fmt, W, rows, K, dt), dt), want.reshape(rows, K))
        assert np.array_equal(_bits(ops.dequant(fmt, shifted, rows, K, dt), dt), want.reshape(rows, K))
        if fmt == synth.Q6_K and K % 2048 == 0:
            R = ops.repack(fmt, W, rows, K)
            assert np.array_equal(_bits(ops.dequant(ops.repacked_fmt(fmt, K), R, rows, K, dt), dt), want.reshape(rows, K))


@pytest.mark.gpu
@pytest.mark.parametrize("rows,K", [(1, 32), (7, 96), (5, 64), (33, 320), (9, 384)])
@pytest.mark.parametrize("fmt", [synth.Q8_0, synth.Q4_0])
def test_rows_of_a_few_blocks(fmt, rows, K):
    """Rows that are not whole groups of four (Q8_0) or two (Q4_0) blocks take the generic kernel."""
    from brotensor_b200 import ops
    Wh = synth.make_blocks(fmt, rows, K, seed=rows + K)
    W = torch.from_numpy(Wh).cuda()
    for dt in DT:
        assert np.array_equal(_bits(ops.dequant(fmt, W, rows, K, dt), dt), _want(fmt, Wh, rows, K, dt).reshape(rows, K))
