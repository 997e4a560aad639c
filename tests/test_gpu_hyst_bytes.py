"""The hysteresis update that works on four weights as the bytes of one word: every threshold, counters over the whole int4 range (-8 too),
all four codes, no, some and certain decay, and gradients from nothing to infinite, through the stand-alone kernel and the fused one."""
import numpy as np
import pytest
import torch

from oracle import int2_oracle as O
from oracle import native

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def ops(pkg):
    return pkg.int2_tc_ops


def _state(N, K, seed):
    rng = np.random.default_rng(seed)
    return rng, rng.integers(0, 256, (N, K // 4)).astype(np.uint8), rng.integers(0, 256, (N, K // 2)).astype(np.uint8)


@pytest.mark.parametrize("thr", [1, 2, 3, 4, 5, 6, 7])
@pytest.mark.parametrize("decay", [0.0, 0.3, 1.0])
@pytest.mark.parametrize("ftz", [True, False])
def test_stand_alone(ops, thr, decay, ftz):
    N, K = 64, 96
    rng, Wp, Hp = _state(N, K, thr)
    dW = (rng.standard_normal((N, K)) * 10.0 ** rng.integers(-7, 4, (N, K))).astype(np.float32)
    dW.reshape(-1)[:9] = [np.nan, np.inf, -np.inf, 0.0, -0.0, 1e-45, -1e-42, 3.4e38, 1.2e-38]
    for idx_base in (0, 33):
        W, H = torch.from_numpy(Wp).to(DEV), torch.from_numpy(Hp).to(DEV)
        ops.hysteresis_step_v2(torch.from_numpy(dW).to(DEV), W, H, 1e-2, 5.0, thr, decay, 9, idx_base=idx_base, ftz=ftz)
        Wo, Ho = native.c_hysteresis_step(dW, Wp, Hp, 1e-2, 5.0, thr, decay, 9, K, idx_base=idx_base, ftz=ftz)
        assert np.array_equal(W.cpu().numpy(), Wo) and np.array_equal(H.cpu().numpy(), Ho)


@pytest.mark.parametrize("N,K", [(48, 96), (4128, 1120)])       # narrow tiles, and pairs with ragged last tiles
@pytest.mark.parametrize("thr,decay,g", [(1, 0.0, 1e-3), (3, 0.3, 0.1), (7, 1.0, 30.0)])
def test_fused(ops, N, K, thr, decay, g):
    rng, Wp, Hp = _state(N, K, N)
    Gq, Xq = rng.integers(-127, 128, (40, N)).astype(np.int8), rng.integers(-128, 128, (40, K)).astype(np.int8)
    G, X, W, H = (torch.from_numpy(a).to(DEV) for a in (Gq, Xq, Wp, Hp))
    ops.dw_hysteresis(G, X, torch.tensor([g], device=DEV), W, H, 1e-2, 5.0, thr, decay, 3)
    Wo, Ho = native.c_hysteresis_step(O.dw_from_acc(O.gemm_dw_acc(Gq, Xq), np.float32(g)), Wp, Hp, 1e-2, 5.0, thr, decay, 3, K)
    assert np.array_equal(W.cpu().numpy(), Wo) and np.array_equal(H.cpu().numpy(), Ho)
    ops.check_device_status(torch.device(DEV))
