"""Decode calls on both sides of each line between the warp-MMA and the tcgen05 kernel (token counts 16/17, 32/33, 48/49 and matrix sizes),
plain, with a norm and with a gate: the output of the separate quantiser and forward GEMM, bit for bit, and the same through the
static-array call."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def ops(pkg):
    return pkg.int2_tc_ops


@pytest.mark.parametrize("M", [16, 17, 31, 32, 33, 48, 49, 63, 64])
@pytest.mark.parametrize("K,N", [(192, 100), (1088, 8192), (2048, 3000), (4096, 8000), (12352, 264)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_every_route_gives_the_forward_pass(ops, M, K, N, dtype):
    g = torch.Generator(device=DEV).manual_seed(M + K + N)
    x = torch.randn(M, K, generator=g, device=DEV).to(dtype)
    up = torch.randn(M, K, generator=g, device=DEV).to(dtype)
    W = torch.randint(0, 256, (N, K // 4), generator=g, device=DEV, dtype=torch.uint8)
    nw = torch.rand(K, generator=g, device=DEV) + 0.5
    for u, w in ((None, None), (None, nw), (up, nw), (up, None)):
        y = x if u is None and w is None else ops.prelinear_rows(x, u, w)
        q, a = ops.quantize_rows(y)
        want = ops.matmul_rows(q, W, a, 0.02, dtype, 1)
        for _ in range(2):
            assert torch.equal(ops.linear_decode(x, W, 0.02, dtype, None, u, w), want)
    q, a = ops.quantize_rows(x)
    assert torch.equal(ops.linear_decode_static(x, W, 0.02, torch.empty(M, N, dtype=dtype, device=DEV)), ops.matmul_rows(q, W, a, 0.02, dtype, 1))
    ops.check_device_status(torch.device(DEV))


# both sides of the lines in matrix size: 2048 outputs or inputs (49 tokens up), 9 million weights, 8192 outputs and 7168 inputs (33 to 48),
# 16384 outputs, 32 million weights and 2368 outputs (17 to 32)
@pytest.mark.parametrize("M,K,N", [(49, 2048, 2048), (64, 2048, 2064), (64, 2112, 100), (40, 2944, 3056), (48, 2944, 3060), (33, 256, 8200), (40, 7168, 72),
                                   (40, 7104, 72), (17, 64, 16384), (32, 64, 16380), (24, 13568, 2368), (24, 13568, 2376), (32, 13504, 2364)])
def test_lines_in_matrix_size(ops, M, K, N):
    g = torch.Generator(device=DEV).manual_seed(M + K + N)
    x = torch.randn(M, K, generator=g, device=DEV).bfloat16()
    W = torch.randint(0, 256, (N, K // 4), generator=g, device=DEV, dtype=torch.uint8)
    nw = torch.rand(K, generator=g, device=DEV) + 0.5
    for w in (None, nw):
        q, a = ops.quantize_rows(x if w is None else ops.prelinear_rows(x, None, w))
        assert torch.equal(ops.linear_decode(x, W, 0.02, None, None, None, w), ops.matmul_rows(q, W, a, 0.02, torch.bfloat16, 1))
    ops.check_device_status(torch.device(DEV))


def test_calls_in_a_chain_and_under_capture(ops):
    """Each call is a programmatic dependent launch behind its quantiser: a chain of layers that feed one another, eager and replayed."""
    g = torch.Generator(device=DEV).manual_seed(3)
    Ws = [torch.randint(0, 256, (2048, 512), generator=g, device=DEV, dtype=torch.uint8) for _ in range(6)]
    x = torch.randn(64, 2048, generator=g, device=DEV).bfloat16()

    def chain(f):
        y = x
        for w in Ws:
            y = f(y, w)
        return y

    def separate(y, w):
        q, a = ops.quantize_rows(y)
        return ops.matmul_rows(q, w, a, 0.02, y.dtype, 1)

    want = chain(separate)
    one = lambda y, w: ops.linear_decode(y, w, 0.02)
    assert torch.equal(chain(one), want)
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        chain(one)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            out = chain(one)
    for _ in range(5):
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)
    ops.check_device_status(torch.device(DEV))
