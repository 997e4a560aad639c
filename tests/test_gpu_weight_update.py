"""The one-call weight update of a layer against the operator calls it stands for, bit for bit: every gradient type and layout, one
scale per token and per tensor, widths with and without the fused kernel, and shapes that have to be refused."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def ops(pkg):
    return pkg.int2_tc_ops


def _dy(kind, M, N, g):
    dy = torch.randn(M, N, generator=g, device=DEV) * 1e-3
    return {"bf16": dy.bfloat16(), "fp16": dy.half(), "fp32": dy, "fp64": dy.double(), "transposed": dy.bfloat16().t().contiguous().t(),
            "column window": torch.cat([dy, dy], 1).bfloat16()[:, :N], "three dimensions": dy.bfloat16().view(3, M // 3, N),
            "expanded": dy[:1].bfloat16().expand(M, N)}[kind]


@pytest.mark.parametrize("kind", ["bf16", "fp16", "fp32", "fp64", "transposed", "column window", "three dimensions", "expanded"])
@pytest.mark.parametrize("N,K", [(96, 64), (40, 48)])               # the second: no fused kernel
@pytest.mark.parametrize("per_tensor", [False, True])
def test_equals_the_separate_calls(ops, kind, N, K, per_tensor):
    M = 33
    g = torch.Generator(device=DEV).manual_seed(N + K)
    dY = _dy(kind, M, N, g)
    Xq = torch.randint(-127, 128, (M, K), generator=g, device=DEV, dtype=torch.int8)
    ax = torch.rand(1 if per_tensor else M, generator=g, device=DEV) + 0.5
    W = torch.randint(0, 256, (N, (K + 3) // 4), generator=g, device=DEV, dtype=torch.uint8)
    H = torch.randint(0, 256, (N, (K + 1) // 2), generator=g, device=DEV, dtype=torch.uint8)
    W1, H1, W2, H2 = W.clone(), H.clone(), W.clone(), H.clone()
    rows = ax.expand(M).contiguous()
    d = dY.reshape(-1, N)
    d = d if d.dtype in (torch.float16, torch.bfloat16, torch.float32) else d.float()
    d = (d.half() if per_tensor else d).contiguous()
    q, a, gmax = ops.quantize_rows(d, 1e-30, fold_absmax=rows)
    Gq = ops.quantize_grad(d, rows, gmax)
    if ops.dw_hysteresis_supported(N, K):
        ops.dw_hysteresis(Gq, Xq, gmax, W1, H1, 0.5, 5.0, 3, 0.01, 7, 128)
    else:
        ops.hysteresis_step_v2(ops.weight_grad(Gq, Xq, gmax), W1, H1, 0.5, 5.0, 3, 0.01, 7, 128)
    assert not torch.equal(W1, W)
    q2, a2 = ops.weight_update(dY, ax, Xq, W2, H2, per_tensor, 0.5, 5.0, 3, 0.01, 7, 128)
    assert q2.shape == dY.shape and torch.equal(q2.reshape(-1, N), q) and torch.equal(a2, a)
    assert torch.equal(W1, W2) and torch.equal(H1, H2)


def test_refusals(ops):
    t = lambda *s, dtype=torch.uint8: torch.zeros(*s, dtype=dtype, device=DEV)
    dY, ax, Xq, W, H = t(4, 32, dtype=torch.bfloat16), t(4, dtype=torch.float32), t(4, 64, dtype=torch.int8), t(32, 16), t(32, 32)
    upd = (False, 0.1, 5.0, 3, 0.0, 1)
    for args, msg in [((dY.cpu(), ax, Xq, W, H), "dY must be a CUDA tensor"), ((dY, ax[:3], Xq, W, H), "fold_absmax must be float32"),
                      ((dY, ax.double(), Xq, W, H), "fold_absmax must be float32"), ((dY, ax, Xq.short(), W, H), "must be int8"),
                      ((dY[:3], ax, Xq, W, H), "same number of tokens"), ((dY, ax, Xq, W[:, :8], H), "shape mismatch"),
                      ((dY, ax, Xq, W, H[:, :8]), "shape mismatch"), ((dY, ax, Xq, t(32, 32)[:, ::2], H), "must be contiguous"),
                      ((dY, ax, Xq, W.char(), H), "must be uint8"), ((dY, ax, Xq, W.cpu(), H), "must be uint8")]:
        with pytest.raises(RuntimeError, match=msg):
            ops.weight_update(*args, *upd)


@pytest.mark.parametrize("shape", ["flat", "rows joined", "rows cut in two"])
@pytest.mark.parametrize("N,K", [(96, 64), (40, 48)])
def test_gradient_of_another_shape(ops, pkg, shape, N, K):
    """M*N gradient elements whose last dimension is not N: one scale per tensor takes them as [M, N], one per token refuses them before
    anything changes."""
    B, T = 3, 10
    M = B * T
    g = torch.Generator(device=DEV).manual_seed(N)
    rows = torch.randn(M, N, generator=g, device=DEV).mul_(1e-3).half()
    dY = {"flat": rows.flatten(), "rows joined": rows.view(B, T * N), "rows cut in two": rows.view(2 * M, N // 2)}[shape]
    Xq = torch.randint(-127, 128, (M, K), generator=g, device=DEV, dtype=torch.int8)
    ax = torch.rand(1, generator=g, device=DEV) + 0.5
    W = torch.randint(0, 256, (N, (K + 3) // 4), generator=g, device=DEV, dtype=torch.uint8)
    H = torch.randint(0, 256, (N, (K + 1) // 2), generator=g, device=DEV, dtype=torch.uint8)
    W1, H1, W2, H2 = W.clone(), H.clone(), W.clone(), H.clone()
    q1, a1 = ops.weight_update(rows, ax, Xq, W1, H1, True, 0.5, 5.0, 3, 0.01, 7)
    q2, a2 = ops.weight_update(dY, ax, Xq, W2, H2, True, 0.5, 5.0, 3, 0.01, 7)
    assert q2.shape == (M, N) and torch.equal(q1, q2) and torch.equal(a1, a2)
    assert not torch.equal(W1, W) and torch.equal(W1, W2) and torch.equal(H1, H2)
    W0, H0 = W.clone(), H.clone()
    with pytest.raises(RuntimeError, match="last dimension"):
        ops.weight_update(dY, ax.expand(M).contiguous(), Xq, W, H, False, 0.5, 5.0, 3, 0.01, 7)
    assert torch.equal(W, W0) and torch.equal(H, H0)
    for mode in ("per_token", "per_tensor"):                 # the same through a layer
        layer = pkg.Int2LinearTC(K, N, threshold=3, quant_mode=mode).to(DEV)
        layer.init_from_float(torch.randn(N, K, generator=g, device=DEV))
        before, counters = layer.W_packed.clone(), layer.H_packed.clone()
        layer(torch.randn(B, T, K, generator=g, device=DEV).half())
        if mode == "per_tensor":
            layer.hysteresis_update(dY, 0.5)
            assert not torch.equal(layer.H_packed, counters)
        else:
            with pytest.raises(RuntimeError, match="last dimension"):
                layer.hysteresis_update(dY, 0.5)
            assert torch.equal(layer.W_packed, before) and torch.equal(layer.H_packed, counters)
