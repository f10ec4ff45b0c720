"""How a long prompt is cut into token passes and K splits inside one launch of the prefill GEMM: token counts around the
passes' edges (one token into a second pass, a last pass of a few tokens, several passes with and without a split K) against the
oracle on a sample of the columns (prefill bound, rel-L2 <= 2e-3), and against the one-CTA kernel, which takes 512 tokens after another."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import oracle
from brotensor_b200 import _capi, synth


@pytest.mark.gpu
@pytest.mark.parametrize("fmt,N,K,M", [(synth.Q4_K, 300, 1024, 513), (synth.Q4_K, 14336, 512, 1000), (synth.Q8_0, 4096, 2048, 1025), (synth.Q6_K, 1000, 2560, 777),
                                       (synth.Q4_K, 2560, 2560, 2000), (synth.Q6_K, 257, 4096, 1537)])
def test_long_prompts(fmt, N, K, M):
    from brotensor_b200 import ops
    Wh, xh = synth.make_blocks(fmt, N, K, seed=N + M), synth.make_activations(M, K, seed=M)
    bh = synth.make_activations(1, N, seed=5).reshape(-1)
    W, X, b = torch.from_numpy(Wh).cuda(), torch.from_numpy(xh).cuda(), torch.from_numpy(bh).cuda()
    y = ops.gemm(fmt, W, X, N, bias=b)
    assert torch.equal(y, ops.gemm(fmt, W, X, N, bias=b))
    half = ops.gemm(fmt, W, X.half(), N, bias=b.half(), out_dtype=torch.float16)
    rows = np.arange(0, N, max(1, N // 100))
    want = oracle.cpu().matmul(fmt, Wh.reshape(N, -1)[rows].reshape(-1), xh, threads=16) + bh[None, rows]
    cols = torch.from_numpy(rows).cuda()
    assert oracle.rel_l2(y[:, cols].cpu().numpy(), want) < 2e-3
    assert oracle.rel_l2(half[:, cols].float().cpu().numpy(), want) < 2e-3
    try:
        ops.set_option("gemm_pair", 0)
        one = ops.gemm(fmt, W, X, N, bias=b)
    finally:
        ops.set_option("gemm_pair", 1)
    assert oracle.rel_l2(y.cpu().numpy(), one.cpu().numpy()) < 1e-5  # the order of the FP32 additions of a split K alone
    assert ops.device_status() == 0


def _workspace(fmt, M, N, K, dtype=_capi.F16):
    return _capi.lib().b200q_gemm_workspace_bytes(fmt, dtype, M, N, K)


@pytest.mark.parametrize("fmt", [synth.Q4_K, synth.Q6_K, synth.Q8_0, synth.Q5_K, synth.Q4_0])
@pytest.mark.parametrize("N,K", [(4096, 4096), (1024, 4096), (14336, 4096), (4096, 14336), (640, 2560), (10240, 10240), (300, 1024), (257, 2048)])
def test_a_workspace_covers_every_shorter_prompt(fmt, N, K):
    sizes = [_workspace(fmt, M, N, K) for M in list(range(1, 1200)) + list(range(1200, 9000, 97))]
    assert all(a <= b for a, b in zip(sizes, sizes[1:]))


@pytest.mark.gpu
@pytest.mark.parametrize("N,K", [(4096, 4096), (1024, 4096)])
def test_results_do_not_depend_on_a_larger_workspace(N, K):
    from brotensor_b200 import ops
    W = torch.from_numpy(synth.make_blocks(synth.Q4_K, N, K, seed=1)).cuda()
    X = torch.from_numpy(synth.make_activations(2000, K, seed=2)).half().cuda()
    ws = torch.empty(_workspace(synth.Q4_K, 2000, N, K), dtype=torch.uint8, device="cuda")
    for M in (17, 45, 300, 512, 513, 1100, 2000):
        own = torch.empty(_workspace(synth.Q4_K, M, N, K), dtype=torch.uint8, device="cuda")
        a, b = (ops.gemm(synth.Q4_K, W, X[:M], N, out_dtype=torch.float32, ws=w) for w in (own, ws))
        assert torch.equal(a, b), M


@pytest.mark.gpu
@pytest.mark.parametrize("fmt,N,K", [(synth.Q4_K, 2560, 2560), (synth.Q6_K, 1024, 4096), (synth.Q8_0, 640, 2560)])
def test_nine_to_sixteen_rows_need_their_workspace(fmt, N, K):
    """Also where the GEMM hands the call to two passes of the decode GEMV, which read none."""
    from brotensor_b200 import ops
    W = torch.from_numpy(synth.make_blocks(fmt, N, K, seed=1)).cuda()
    room = torch.empty(_workspace(fmt, 16, N, K) + 256, dtype=torch.uint8, device="cuda")
    for M in (9, 16):
        X = torch.from_numpy(synth.make_activations(M, K, seed=2)).half().cuda()
        y = torch.zeros(M, N, dtype=torch.float32, device="cuda")
        for ws, n in ((None, 0), (room.data_ptr(), 1024), (room.data_ptr() + 16, room.numel() - 256)):
            rc = _capi.lib().b200q_gemm(fmt, W.data_ptr(), X.data_ptr(), _capi.F16, None, y.data_ptr(), _capi.F32, M, N, K, ws, n, None)
            assert rc == _capi.ERR_WORKSPACE
        torch.cuda.synchronize()
        assert not y.any()
        assert ops.gemm(fmt, W, X, N, ws=room).any()


@pytest.mark.gpu
def test_more_passes_than_a_grid_holds():
    """One token into pass 65536 (activations and their image: 34 GB)."""
    from brotensor_b200 import ops
    fmt, M, N, K = synth.Q8_0, 65535 * 512 + 1, 4, 256
    if torch.cuda.mem_get_info()[0] < 60e9:
        pytest.skip("not enough free device memory")
    W = torch.from_numpy(synth.make_blocks(fmt, N, K, seed=1)).cuda()
    X = torch.zeros(M, K, dtype=torch.float16, device="cuda")
    at = torch.tensor([0, 511, 512, M // 2, M - 514, M - 2, M - 1], device="cuda")
    X[at] = torch.from_numpy(synth.make_activations(len(at), K, seed=2)).half().cuda()
    y = ops.gemm(fmt, W, X, N, out_dtype=torch.float32)
    want = ops.gemv(fmt, W, X[at].contiguous(), N, out_dtype=torch.float32)
    assert oracle.rel_l2(y[at].cpu().numpy(), want.cpu().numpy()) < 2e-3
    assert torch.count_nonzero(y) == len(at) * N
    del X, y
    torch.cuda.empty_cache()
