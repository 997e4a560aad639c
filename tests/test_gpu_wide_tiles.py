"""The 256-column tiles of the single-CTA kernel beyond the rule for 128-column ones (more than 74 tiles of 128 x 256 on 148 SMs), with
a last column tile that is only partly inside: forward, dX, the weight gradient and its fused update."""
import numpy as np
import pytest
import torch

from oracle import int2_oracle as O
from oracle import native

from helpers import random_packed

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def ops(pkg):
    return pkg.int2_tc_ops


# 33 row tiles of weights: two bands of 16 and a band of one; a last column tile of 64 and of 96 columns, whose second
# 128-column operand box is wholly outside; idx_base aligned to 32 (one hash fold per chunk) and not
@pytest.mark.parametrize("M,N,K", [(300, 4176, 1088), (300, 4176, 1376), (130, 2064, 2496)])
@pytest.mark.parametrize("idx_base", [0, 1000])
def test_fused_update_on_ragged_wide_tiles(ops, M, N, K, idx_base):
    rng = np.random.default_rng(M + N + K)
    Gq = rng.integers(-127, 128, (M, N)).astype(np.int8)
    Xq = rng.integers(-128, 128, (M, K)).astype(np.int8)
    Wp, _ = random_packed(N, K, 5)
    Hp = O.pack_counters(rng.integers(-3, 4, (N, K)).astype(np.int8))
    g = np.float32(2e-3)
    G, X, W, H = (torch.from_numpy(np.ascontiguousarray(a)).to(DEV) for a in (Gq, Xq, Wp, Hp))
    gmax = torch.tensor([g], device=DEV)
    dW = O.dw_from_acc(O.gemm_dw_acc(Gq, Xq), g)
    assert np.array_equal(ops.weight_grad(G, X, gmax).cpu().numpy(), dW)
    ops.dw_hysteresis(G, X, gmax, W, H, 1e-2, 5.0, 3, 0.01, 3, idx_base=idx_base)
    ops.check_device_status(torch.device(DEV))
    Wo, Ho = native.c_hysteresis_step(dW, Wp, Hp, 1e-2, 5.0, 3, 0.01, 3, K, idx_base=idx_base)
    assert np.array_equal(W.cpu().numpy(), Wo) and np.array_equal(H.cpu().numpy(), Ho)
    assert (O.unpack_ternary(Wo, K) != O.unpack_ternary(Wp, K)).mean() > 0.01


# 11 row tiles x 9 column tiles, the last one of 64 or 192 columns
@pytest.mark.parametrize("M,N,K", [(1300, 2112, 2240), (1300, 2240, 2112)])
def test_forward_and_dx_on_ragged_wide_tiles(ops, pkg, M, N, K):
    rng = np.random.default_rng(M + N + K)
    Xq = rng.integers(-128, 128, (M, K)).astype(np.int8)
    dYq = rng.integers(-128, 128, (M, N)).astype(np.int8)
    Wp, _ = random_packed(N, K, 6)
    X, G, W = (torch.from_numpy(np.ascontiguousarray(a)).to(DEV) for a in (Xq, dYq, Wp))
    a = torch.rand(M, device=DEV) + 0.5
    single = pkg._lib.EL_PATH_TC_SINGLE
    assert np.array_equal(ops.matmul_rows(X, W, a, 1.0, torch.int32, path=single).cpu().numpy(), O.gemm_fwd_acc(Xq, Wp, K))
    assert torch.equal(ops.matmul_rows(X, W, a, 0.02, path=single), ops.matmul_rows(X, W, a, 0.02, path=1))
    assert torch.equal(ops.backward_input_rows(G, W, a, 1.0, K, torch.int32, path=single), ops.backward_input_rows(G, W, a, 1.0, K, torch.int32, path=1))
    assert torch.equal(ops.backward_input_rows(G, W, a, 0.02, K, path=single), ops.backward_input_rows(G, W, a, 0.02, K, path=1))
    ops.check_device_status(torch.device(DEV))
