"""Layers of 16, 32 or 48 inputs: the streaming forward and dX kernels against the oracle's integers and scaled outputs."""
import numpy as np
import pytest
import torch

from oracle import int2_oracle as O

from helpers import t2n

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def ops(pkg):
    return pkg.int2_tc_ops


# token counts around the 16-row tile and beyond one wave of CTAs; output widths around the 64-column warp block, the
# 512-column CTA block and the shared-memory chunk of dX (8192 reduction rows at 16 inputs, 2688 at 48); widths that no
# 16-byte store takes (20, 36) fall to the general kernel
@pytest.mark.parametrize("M,K,N", [(1, 16, 8), (15, 16, 64), (17, 16, 520), (33, 32, 1000), (130, 48, 2752), (5, 48, 48),
                                   (16, 16, 8192), (40, 16, 8256), (31, 32, 20), (7, 16, 36), (2600, 16, 96)])
def test_narrow_layers_match_oracle(ops, M, K, N):
    rng = np.random.default_rng(M * 31 + K * 7 + N)
    Xq = rng.integers(-128, 128, (M, K)).astype(np.int8)
    Gq = rng.integers(-128, 128, (M, N)).astype(np.int8)
    Wp = rng.integers(0, 256, (N, K // 4)).astype(np.uint8)          # every code, also the reserved one
    W = O.unpack_ternary(Wp, K).astype(np.int64)
    ax = (rng.random(M) + 0.5).astype(np.float32)
    X, G, Wd, A = (torch.from_numpy(np.ascontiguousarray(a)).to(DEV) for a in (Xq, Gq, Wp, ax))
    y = Xq.astype(np.int64) @ W.T
    dx = Gq.astype(np.int64) @ W
    assert np.array_equal(ops.matmul_rows(X, Wd, A, 0.02, torch.int32).cpu().numpy(), y)
    assert np.array_equal(ops.backward_input_rows(G, Wd, A, 0.02, K, torch.int32).cpu().numpy(), dx)
    sc = (ax / np.float32(127.0)) * np.float32(0.02)
    for dt in (torch.bfloat16, torch.float16, torch.float32):
        for got, acc in ((ops.matmul_rows(X, Wd, A, 0.02, dt), y), (ops.backward_input_rows(G, Wd, A, 0.02, K, dt), dx)):
            want = torch.from_numpy(acc.astype(np.float32) * sc[:, None]).to(dt)
            assert np.array_equal(t2n(got), t2n(want))
    # one scale for the whole tensor, and both against the general kernel
    one = A[:1].contiguous()
    assert torch.equal(ops.matmul_int8(X, Wd, one, 0.02), ops.matmul_int8(X, Wd, one, 0.02, path=1))
    assert torch.equal(ops.backward_input_int8(G, Wd, one, 0.02, K), ops.backward_input_int8(G, Wd, one, 0.02, K, path=1))
