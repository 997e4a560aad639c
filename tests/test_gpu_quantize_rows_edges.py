"""The per-token quantiser where its row cache changes size or ends (4096, 12288, 16384 elements) and where its rounding changes form: rows
with an infinity or a NaN, rows below the floor, and a floor so small that the scale overflows."""
import numpy as np
import pytest
import torch

from oracle import int2_oracle as O

from helpers import t2n

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("K", [8, 4096, 4104, 12288, 12296, 16384, 16392, 20000])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("eps", [1e-5, 1e-30])
def test_against_the_oracle(pkg, K, dtype, eps):
    g = torch.Generator().manual_seed(K)
    x = torch.randn(9, K, generator=g)
    x[1, K // 2], x[2, K - 1], x[3, 0] = float("inf"), float("nan"), float("-inf")
    x[4] *= 1e-7
    x[5] = 0.0
    x = x.to(dtype)
    x[6] = 127.0 * torch.rand(K, generator=g).round().to(dtype)       # many exact ties at +-0.5 of a step
    x[6, 0] = 254.0
    q, a = pkg.int2_tc_ops.quantize_rows(x.to(DEV), eps)
    qo, ao = O.quantize_rows(t2n(x), eps)
    assert np.array_equal(a.cpu().numpy(), ao) and np.array_equal(q.cpu().numpy(), qo)


def test_a_scale_that_overflows(pkg):
    """Zeros times an infinite scale are NaN and become 0; the largest value saturates."""
    x = torch.zeros(3, 64)
    x[1, 5], x[2, 7] = 1e-40, -1e-41
    q, a = pkg.int2_tc_ops.quantize_rows(x.to(DEV), 1e-42)
    want = torch.zeros(3, 64, dtype=torch.int8)
    want[1, 5], want[2, 7] = 127, -128
    assert torch.equal(q.cpu(), want)
