"""The pair GEMM hands expanded weights from one CTA to an MMA that the other one issues.  Many launches of one problem, with other
work between them so that the CTAs meet in other ways, give the general kernel's integers every time."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def ops(pkg):
    return pkg.int2_tc_ops


# 2 x 16 and 8 x 7 pair tiles for 74 pairs, and 8 x 32: several tiles per pair, both accumulators in turn
@pytest.mark.parametrize("M,N,K", [(512, 4096, 1024), (2048, 1792, 2048), (2048, 8192, 1024)])
@pytest.mark.parametrize("lean", [False, True])
def test_repeated_launches_give_the_same_integers(ops, pkg, M, N, K, lean):
    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    Xq = torch.randint(-128, 128, (M, K), generator=g, device=DEV, dtype=torch.int8)
    Gq = torch.randint(-128, 128, (M, N), generator=g, device=DEV, dtype=torch.int8)
    W = torch.randint(0, 256, (N, K // 4), generator=g, device=DEV, dtype=torch.uint8)
    a = torch.ones(M, device=DEV)
    path = pkg._lib.EL_PATH_TC | (pkg._lib.EL_FLAG_LEAN if lean else 0)
    y = ops.matmul_rows(Xq, W, a, 1.0, torch.int32, path=1)
    dx = ops.backward_input_rows(Gq, W, a, 1.0, K, torch.int32, path=1)
    other = torch.empty(32 << 20, dtype=torch.uint8, device=DEV)
    wrong = torch.zeros((), dtype=torch.int64, device=DEV)
    for i in range(40):
        other[:(i % 4) << 23].fill_(i)
        wrong += (ops.matmul_rows(Xq, W, a, 1.0, torch.int32, path=path) != y).sum()
        wrong += (ops.backward_input_rows(Gq, W, a, 1.0, K, torch.int32, path=path) != dx).sum()
    ops.check_device_status(torch.device(DEV))
    assert int(wrong) == 0
