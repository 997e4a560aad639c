"""Problems with few output tiles run on 128-column tiles of the single-CTA kernel: forward, dX and the fused weight gradient at
tile edges, against the general CUDA-core kernel's integers and the separate weight-gradient and update kernels."""
import numpy as np
import pytest
import torch

from helpers import random_packed

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def ops(pkg):
    return pkg.int2_tc_ops


# rows around the 128-row tile, columns around the 128-column tile (also a last tile of 64 and of 8 columns), reductions that
# end inside a 128-deep block, and the sizes on both sides of the rule on the B200's 148 SMs (74 tiles of 128 x 256)
@pytest.mark.parametrize("M,N,K", [(129, 64, 64), (255, 136, 192), (256, 192, 320), (300, 1032, 128), (1024, 1536, 1536), (1184, 2048, 256),
                                   (1300, 2048, 256), (2048, 192, 2048)])
def test_narrow_tiles_match_general_kernel(ops, M, N, K):
    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    Xq = torch.randint(-127, 128, (M, K), generator=g, device=DEV, dtype=torch.int8)
    Gq = torch.randint(-127, 128, (M, N), generator=g, device=DEV, dtype=torch.int8)
    W = torch.from_numpy(np.ascontiguousarray(random_packed(N, K, seed=K)[0])).to(DEV)
    a = torch.rand(M, generator=g, device=DEV) + 0.5
    for dt in (torch.int32, torch.bfloat16, torch.float32):
        assert torch.equal(ops.matmul_rows(Xq, W, a, 0.02, dt), ops.matmul_rows(Xq, W, a, 0.02, dt, path=1))
        if N % 16 == 0 and K % 64 == 0:
            assert torch.equal(ops.backward_input_rows(Gq, W, a, 0.02, K, dt), ops.backward_input_rows(Gq, W, a, 0.02, K, dt, path=1))
    if ops.dw_hysteresis_supported(N, K):
        gmax = torch.full((1,), 3e-6, device=DEV)
        H = torch.randint(0, 256, (N, K // 2), generator=g, device=DEV, dtype=torch.uint8)
        W1, H1, W2, H2 = W.clone(), H.clone(), W.clone(), H.clone()
        ops.dw_hysteresis(Gq, Xq, gmax, W1, H1, 0.02, 5.0, 3, 0.001, 7)
        ops.hysteresis_step_v2(ops.weight_grad(Gq, Xq, gmax, path=1), W2, H2, 0.02, 5.0, 3, 0.001, 7)
        assert torch.equal(W1, W2) and torch.equal(H1, H2) and not torch.equal(W1, W)
    ops.check_device_status(torch.device(DEV))
