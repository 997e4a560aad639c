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


# Scaled outputs of sums up to the edge of 2^22 and beyond: tokens of -128 against weights of one sign, reductions of up to 32767 (the sums are
# converted by an addition) and from 32768 on (by the conversion unit); some rows of ordinary tokens between them.
@pytest.mark.parametrize("D", [32704, 32752, 32768, 65536])
@pytest.mark.parametrize("dx", [False, True])
@pytest.mark.parametrize("M", [40, 300])
@pytest.mark.parametrize("byte", [0x00, 0xAA])       # all weights -1, all +1
def test_large_sums(ops, pkg, D, dx, M, byte):
    if not dx and D % 64:
        pytest.skip("the forward reduction is a multiple of 64")
    g = torch.Generator(device=DEV).manual_seed(D + M)
    C = 192
    W = torch.full((D, C // 4) if dx else (C, D // 4), byte, device=DEV, dtype=torch.uint8)
    a = torch.rand(M, generator=g, device=DEV) + 0.5
    q = torch.full((M, D), -128, device=DEV, dtype=torch.int8)
    q[::3] = torch.randint(-128, 128, q[::3].shape, generator=g, device=DEV, dtype=torch.int8)

    def call(dtype, path):
        return ops.backward_input_rows(q, W, a, 0.02, C, dtype, path) if dx else ops.matmul_rows(q, W, a, 0.02, dtype, path)

    assert int(call(torch.int32, pkg._lib.EL_PATH_SIMPLE).abs().max()) == 128 * D
    for dtype in (torch.bfloat16, torch.float32):
        want = call(dtype, pkg._lib.EL_PATH_SIMPLE)
        for path in (pkg._lib.EL_PATH_TC, pkg._lib.EL_PATH_TC | pkg._lib.EL_FLAG_LEAN):
            assert torch.equal(call(dtype, path), want), (dtype, path)
    ops.check_device_status(torch.device(DEV))
