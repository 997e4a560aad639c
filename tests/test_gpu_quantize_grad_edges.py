"""The gradient quantiser at row lengths around the two vectors a thread takes per turn (2048 and 4096 elements), with values beyond the
given maximum (clamped), exact ties, infinities, NaN, and maxima and row scales that are zero, infinite or NaN."""
import numpy as np
import pytest
import torch

from helpers import t2n

pytestmark = pytest.mark.gpu
DEV = "cuda"


def expected(dy, xa, g):
    """int8 of (dY * x_absmax/127) * 127/g in float32, half to even, clamped to +-127; what is not a number, or not finite in dY, is 0."""
    with np.errstate(all="ignore"):
        inv = np.float32(127.0) / np.float32(g) if g >= 1e-30 else np.float32(0)
        sx = (xa / np.float32(127.0)).astype(np.float32)
        y = np.where(np.isfinite(dy), dy, np.float32(np.nan)) * sx[:, None]
        r = np.clip(np.rint(y * inv), -127, 127)
        return np.where(np.isnan(r), 0, r).astype(np.int8)


@pytest.mark.parametrize("N", [8, 2040, 2048, 2056, 4096, 4104, 6152, 11008])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("g", [4.0, 1.0, 127.0, 0.0, 1e-31, float("inf"), float("nan")])
def test_against_the_definition(pkg, N, dtype, g):
    gen = torch.Generator().manual_seed(N)
    dy = torch.randn(8, N, generator=gen)
    dy[1, N // 2], dy[2, N - 1], dy[3, 0] = float("inf"), float("nan"), float("-inf")
    dy[4] = torch.randint(-255, 256, (N,), generator=gen) * 0.5          # with g = 127 and a row scale of 1: exact ties
    dy = dy.to(dtype)
    xa = torch.tensor([3.0, 2.0, 1.0, 0.5, 127.0, float("inf"), float("nan"), 0.0])
    q = pkg.int2_tc_ops.quantize_grad(dy.to(DEV), xa.to(DEV), torch.tensor([g], device=DEV))
    assert np.array_equal(q.cpu().numpy(), expected(t2n(dy).astype(np.float32), xa.numpy(), g))
