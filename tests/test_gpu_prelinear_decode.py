"""The decode call that forms and quantises its input itself (norm, gate or both) equals the two separate calls bit for bit: token
counts around every kernel choice, widths around the one-group-per-thread limit, non-finite tokens, strided gate and up."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def ops(pkg):
    return pkg.int2_tc_ops


@pytest.mark.parametrize("M", [1, 2, 8, 9, 17, 33, 64])
@pytest.mark.parametrize("K,N", [(64, 40), (1536, 100), (4160, 512), (12288, 48), (16384, 130)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
def test_prelinear_decode_equals_the_separate_calls(ops, pkg, M, K, N, dtype):
    g = torch.Generator(device=DEV).manual_seed(M * 7 + K + N)
    gu = (torch.randn(M, 2 * K, generator=g, device=DEV) * 2.0).to(dtype)
    x, up = gu[:, :K], gu[:, K:]
    if M > 2:
        gu[1] = 0.0
        gu[2, 5] = float("nan")
        gu[M - 1, K - 1] = float("inf")
    w = 1.0 + 0.3 * torch.randn(K, generator=g, device=DEV)
    W = torch.randint(0, 256, (N, K // 4), generator=g, device=DEV, dtype=torch.uint8)
    for u, nw in ((None, w), (up, None), (up, w)):
        want = ops.linear_decode(ops.prelinear_rows(x, u, nw, 1e-6), W, 0.03)
        got = ops.linear_decode(x, W, 0.03, None, None, u, nw, 1e-6)
        assert got.dtype == dtype and torch.equal(got, want)
    ops.check_device_status(torch.device(DEV))
    with pytest.raises(RuntimeError, match="norm_weight must be a contiguous float32"):
        ops.linear_decode(x, W, 0.03, None, None, None, w[:-1])


def test_prelinear_decode_refuses_what_it_cannot_run(ops, pkg):
    x = torch.zeros(2, 16448, dtype=torch.bfloat16, device=DEV)
    with pytest.raises(pkg.ElleciError) as e:
        ops.linear_decode(x, torch.zeros(16, 4112, dtype=torch.uint8, device=DEV), 1.0, norm_weight=torch.ones(16448, device=DEV))
    assert e.value.status == pkg._lib.EL_ERR_UNSUPPORTED_SHAPE


@pytest.mark.parametrize("M,K,N", [(32, 6208, 100), (17, 8192, 5000), (33, 11008, 2400), (64, 16384, 2384), (16, 16384, 40), (9, 12800, 16)])
def test_decode_of_tokens_that_exceed_shared_memory(ops, M, K, N):
    """Rows too long for shared memory are multiplied a chunk of the reduction at a time: chunk ends inside and at a round of the
    sixteen warps, one and several row groups per CTA, a remainder of tokens; the output is the prefill kernels' bit for bit."""
    g = torch.Generator(device=DEV).manual_seed(M + K + N)
    x = torch.randn(M, K, generator=g, device=DEV).bfloat16()
    W = torch.randint(0, 256, (N, K // 4), generator=g, device=DEV, dtype=torch.uint8)
    Xq, a = ops.quantize_rows(x)
    want = ops.matmul_rows(Xq, W, a, 0.02)
    assert torch.equal(ops.linear_decode(x, W, 0.02), want)
    ops.check_device_status(torch.device(DEV))
