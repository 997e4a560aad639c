"""Forward and dX with the weights in tensor memory, at the edges of every token tile (32, 64, 128, 256), of the 256-feature tile and of
the reduction step (128 or 256 deep): the exact int32 sums and the scaled outputs against the CUDA-core kernel, whose sums other
tests compare with the oracle."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def ops(pkg):
    return pkg.int2_tc_ops


def _check(ops, pkg, M, N, K, dx):
    g = torch.Generator(device=DEV).manual_seed(M + 7 * N + 13 * K)
    W = torch.randint(0, 256, (N, K // 4), generator=g, device=DEV, dtype=torch.uint8)       # all four codes
    a = torch.rand(M, generator=g, device=DEV) + 0.5
    q = torch.randint(-128, 128, (M, N if dx else K), generator=g, device=DEV, dtype=torch.int8)

    def call(dtype, path):
        return ops.backward_input_rows(q, W, a, 0.02, K, dtype, path) if dx else ops.matmul_rows(q, W, a, 0.02, dtype, path)

    for dtype in (torch.int32, torch.bfloat16, torch.float16, torch.float32):
        want = call(dtype, pkg._lib.EL_PATH_SIMPLE)
        for path in (pkg._lib.EL_PATH_TC, pkg._lib.EL_PATH_TC | pkg._lib.EL_FLAG_LEAN):
            assert torch.equal(call(dtype, path), want), (dtype, path)
    ops.check_device_status(torch.device(DEV))


# one token more and less than each tile; features around the 64 of a warp pair, the 128 of a CTA and the 256 of a pair; reductions
# of an odd number of 128-blocks and of a part of one; features that leave an output pitch no TMA store takes (70, 100, 321)
@pytest.mark.parametrize("M", [1, 31, 33, 63, 65, 127, 129, 255, 257])
@pytest.mark.parametrize("N,K", [(70, 64), (128, 192), (200, 320), (321, 384), (1000, 1088)])
def test_forward_edges(ops, pkg, M, N, K):
    _check(ops, pkg, M, N, K, False)


@pytest.mark.parametrize("M", [1, 32, 33, 65, 128, 129, 256, 300])
@pytest.mark.parametrize("N,K", [(16, 64), (48, 128), (144, 192), (272, 320), (1104, 576)])
def test_dx_edges(ops, pkg, M, N, K):
    _check(ops, pkg, M, N, K, True)


# more tiles than pairs at each token tile: both accumulators in turn, stages and slots many times round
@pytest.mark.parametrize("M,N,K", [(20, 40000, 512), (60, 40064, 384), (128, 40000, 640), (2500, 4096, 1536), (5000, 8200, 256)])
def test_several_tiles_per_pair(ops, pkg, M, N, K):
    _check(ops, pkg, M, N, K, False)


@pytest.mark.parametrize("M,N,K", [(20, 512, 40000), (60, 400, 40064), (128, 640, 40000), (2500, 1536, 4096), (5000, 256, 8256)])
def test_several_tiles_per_pair_dx(ops, pkg, M, N, K):
    _check(ops, pkg, M, N, K, True)
