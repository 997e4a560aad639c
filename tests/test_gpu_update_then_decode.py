"""A weight update followed at once by a decode call, many times without a synchronisation: the decode kernels request packed weights
while the quantiser in front of them still runs, so each output has to be that of the weights the update has left."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
M, K, N, STEPS = 2048, 4096, 2048, 12


@pytest.fixture(scope="module")
def ops(pkg):
    return pkg.int2_tc_ops


# 5 tokens: one launch that quantises them itself; 24: quantiser and warp MMA; 64: quantiser and tcgen05
@pytest.mark.parametrize("tokens", [1, 5, 24, 64])
@pytest.mark.parametrize("norm", [False, True])
@pytest.mark.parametrize("captured", [False, True])
def test_decode_reads_the_updated_weights(ops, tokens, norm, captured):
    g = torch.Generator(device=DEV).manual_seed(tokens)
    dY = torch.randn(M, N, generator=g, device=DEV).mul_(1e-3).bfloat16()
    dYs = (dY, -dY)             # back and forth, so that every step moves weights
    Xq = torch.randint(-127, 128, (M, K), generator=g, device=DEV, dtype=torch.int8)
    ax = torch.rand(M, generator=g, device=DEV) + 0.5
    W = torch.randint(0, 256, (N, K // 4), generator=g, device=DEV, dtype=torch.uint8)
    H = torch.randint(0, 256, (N, K // 2), generator=g, device=DEV, dtype=torch.uint8)
    x = torch.randn(tokens, K, generator=g, device=DEV).bfloat16()
    nw = torch.rand(K, generator=g, device=DEV) + 0.5 if norm else None

    def steps():
        outs = []
        for step in range(STEPS):
            ops.weight_update(dYs[step % 2], ax, Xq, W, H, False, 0.5, 5.0, 3, 0.01, step)
            y = ops.linear_decode(x, W, 0.02, torch.bfloat16, None, None, nw)
            outs.append((y, W.clone()))
        return outs

    if captured:
        s = torch.cuda.Stream()
        s.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(s):
            steps()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=s):
                outs = steps()
            graph.replay()
        torch.cuda.synchronize()
    else:
        outs = steps()
    q, a = ops.quantize_rows(x if nw is None else ops.prelinear_rows(x, None, nw))
    before = None
    for y, w in outs:
        assert before is None or not torch.equal(w, before)
        assert torch.equal(y, ops.matmul_rows(q, w, a, 0.02, torch.bfloat16, 1))
        before = w
    ops.check_device_status(torch.device(DEV))
