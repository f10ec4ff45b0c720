"""The kernels that start before their predecessor has finished (the default launch form) read nothing too early: weights and
activations that the launch before them in the stream has just written, in eager order and in a captured graph with a forked
branch, give the bits of plain launches."""
import pytest

torch = pytest.importorskip("torch")

from brotensor_b200 import synth


@pytest.fixture
def ops_pdl():
    from brotensor_b200 import ops
    yield ops
    ops.set_option("pdl", 0)


@pytest.mark.gpu
@pytest.mark.parametrize("fmt,N,K,M", [(synth.Q4_K, 14336, 4096, 1), (synth.Q4_K, 4096, 4096, 1), (synth.Q4_K, 1024, 2560, 2), (synth.Q4_K, 4096, 4096, 6),
                                       (synth.Q6_K, 4096, 14336, 1), (synth.Q6_K, 4096, 4096, 6), (synth.Q8_0, 4096, 4096, 3), (synth.Q5_K, 3000, 2560, 1),
                                       (synth.Q4_0, 700, 1024, 20), (synth.Q4_K, 1024, 4096, 40), (synth.Q6_K, 300, 8192, 17), (synth.Q8_0, 600, 2048, 600)])
def test_predecessor_writes_the_operands(fmt, N, K, M, ops_pdl):
    ops = ops_pdl
    Ws = [torch.from_numpy(synth.make_blocks(fmt, N, K, seed=s)).cuda() for s in (1, 2)]
    xs = [torch.from_numpy(synth.make_activations(M, K, seed=s)).cuda() for s in (3, 4)]
    ops.set_option("pdl", -1)
    gemv = ops.gemv if M <= 8 else ops.gemm
    want = [gemv(fmt, W, x, N) for W, x in zip(Ws, xs)]
    ops.set_option("pdl", 0)
    W, x = torch.empty_like(Ws[0]), torch.empty_like(xs[0])

    def load(i):  # elementwise kernels, not copies: a copy would be waited for in any case
        torch.bitwise_or(Ws[i & 1], 0, out=W)
        torch.mul(xs[i & 1], 1.0, out=x)

    outs = []
    for i in range(12):
        load(i)
        outs.append(gemv(fmt, W, x, N))
    side, graph, captured = torch.cuda.Stream(), torch.cuda.CUDAGraph(), []
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        main = torch.cuda.current_stream()
        for i in range(4):
            load(i)
            side.wait_stream(main)
            with torch.cuda.stream(side):
                a = gemv(fmt, W, x, N)
            b = gemv(fmt, W, x, N)
            main.wait_stream(side)
            captured.append((i, a, b, gemv(fmt, W, x, N)))
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(y, want[i & 1]) for i, y in enumerate(outs))
    assert all(torch.equal(y, want[c[0] & 1]) for c in captured for y in c[1:])
    assert ops.device_status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("fmt,N,K,M,dtype", [(synth.Q5_K, 3000, 2560, 1, torch.float32), (synth.Q6_K, 700, 2304, 2, torch.float16), (synth.Q4_K, 1024, 4096, 6, torch.float16),
                                             (synth.Q8_0, 700, 1024, 4, torch.bfloat16), (synth.Q4_0, 700, 1024, 20, torch.float32)])
def test_predecessor_writes_operands_that_are_not_finite(fmt, N, K, M, dtype, ops_pdl):
    """The FP32 loop that takes over for such activations reads the weights again, and no earlier."""
    ops = ops_pdl
    Ws = [torch.from_numpy(synth.make_blocks(fmt, N, K, seed=s)).cuda() for s in (1, 2)]
    x = torch.from_numpy(synth.make_activations(M, K, seed=3)).to(dtype).cuda()
    x[M // 2, 300] = float("inf")
    ops.set_option("pdl", -1)
    want = [ops.linear(fmt, W, x, N, out_dtype=torch.float32).view(torch.int32) for W in Ws]
    ops.set_option("pdl", 0)
    assert not torch.equal(*want)
    W = torch.empty_like(Ws[0])
    for i in range(40):
        torch.bitwise_or(Ws[i & 1], 0, out=W)
        assert torch.equal(ops.linear(fmt, W, x, N, out_dtype=torch.float32).view(torch.int32), want[i & 1])
    assert ops.device_status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("M", [1, 2, 3, 4])
@pytest.mark.parametrize("pdl", [-1, 0, 1])
def test_predecessor_writes_the_activations(pdl, M, ops_pdl):
    """The integer-dot kernel in each launch form: plain launches read the activations on the read-only path, overlapped ones behind the wait."""
    ops, fmt, N, K = ops_pdl, synth.Q4_K, 1024, 8192
    W = torch.from_numpy(synth.make_blocks(fmt, N, K, seed=1)).cuda()
    for dtype in (torch.float32, torch.float16):
        xs = [torch.from_numpy(synth.make_activations(M, K, seed=s)).to(dtype).cuda() for s in (3, 4)]
        ops.set_option("pdl", -1)
        want = [ops.gemv(fmt, W, x, N) for x in xs]
        ops.set_option("pdl", pdl)
        x = torch.empty_like(xs[0])
        for i in range(20):
            torch.mul(xs[i & 1], 1.0, out=x)
            assert torch.equal(ops.gemv(fmt, W, x, N), want[i & 1])
    assert ops.device_status() == 0
