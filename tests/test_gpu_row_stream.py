"""The streaming norm and gate kernels at the edges of their ranges, bit for bit against the oracle: many tokens per CTA (the
ring of rows wraps), columns that fill no warp's vectors, the widths where one form hands over to the next, tokens with
non-finite values between ordinary ones."""
import numpy as np
import pytest
import torch

from oracle import int2_oracle as O

from helpers import t2n

pytestmark = pytest.mark.gpu
DEV = "cuda"
_IO = {torch.bfloat16: "bf16", torch.float16: "f16", torch.float32: "f32"}


@pytest.fixture(scope="module")
def ops(pkg):
    return pkg.int2_tc_ops


# 256: 32 CTAs per SM walk over several tokens each; 1032: a last warp with one vector; 6152 / 8200 / 12296: float32 and 16-bit
# backward forms change there; 16384 / 16392: the last streaming width and the first beyond it
@pytest.mark.parametrize("M,K", [(5000, 256), (601, 1032), (7, 6152), (6, 8200), (6, 12288), (5, 12296), (4, 16384), (3, 16392)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
def test_norm_kernels_at_their_edges(ops, M, K, dtype):
    g = torch.Generator().manual_seed(M + K)
    x = (torch.randn(M, K, generator=g) * 1.5).to(dtype)
    gy = (torch.randn(M, K, generator=g) * 1e-2).to(dtype)
    w = (1.0 + 0.3 * torch.randn(K, generator=g)).float()
    rstd = torch.from_numpy(O.rmsnorm_rstd(t2n(x), 1e-6))
    dx, dw = ops.rmsnorm_backward(gy.to(DEV), x.to(DEV), w.to(DEV), rstd.to(DEV))
    dxo, dwo = O.rmsnorm_backward(t2n(gy), t2n(x), w.numpy(), rstd.numpy(), _IO[dtype])
    assert np.array_equal(t2n(dx), dxo) and np.array_equal(dw.cpu().numpy(), dwo)
    x[M // 2, K // 2] = float("inf")
    x[M - 1, K - 1] = float("nan")
    q, a, r = ops.rmsnorm_quantize_rows(x.to(DEV), w.to(DEV), 1e-6, 1e-5)
    with np.errstate(all="ignore"):
        qo, ao, ro = O.rmsnorm_quantize_rows(t2n(x), w.numpy(), 1e-6, 1e-5, _IO[dtype])
    assert np.array_equal(r.cpu().numpy(), ro, equal_nan=True)
    assert np.array_equal(a.cpu().numpy(), ao) and np.array_equal(q.cpu().numpy(), qo)


@pytest.mark.parametrize("M,H", [(3000, 256), (401, 1032), (6, 5640), (6, 6152), (5, 11272), (5, 12288), (4, 12296), (3, 16384), (3, 16392)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
def test_gate_kernels_at_their_edges(ops, M, H, dtype):
    g = torch.Generator().manual_seed(M * 3 + H)
    gu = (torch.randn(M, 2 * H, generator=g) * 2.0).to(dtype)
    gy = (torch.randn(M, H, generator=g) * 1e-2).to(dtype)
    w = (1.0 + 0.3 * torch.randn(H, generator=g)).float()
    gate, up = t2n(gu[:, :H]), t2n(gu[:, H:])
    h, _, _ = O.swiglu_hidden(gate, up, _IO[dtype])
    rstd = O.rmsnorm_rstd(h, 1e-6)
    d = gu.to(DEV)
    dg, du, dw = ops.swiglu_backward(gy.to(DEV), d[:, :H], d[:, H:], w.to(DEV), torch.from_numpy(rstd).to(DEV))
    dgo, duo, dwo = O.swiglu_backward(t2n(gy), gate, up, w.numpy(), rstd, _IO[dtype])
    assert np.array_equal(t2n(dg), dgo) and np.array_equal(t2n(du), duo) and np.array_equal(dw.cpu().numpy(), dwo)
    gu[M // 2, 0] = float("nan")
    gu[M - 1, H + 1] = float("inf")
    d = gu.to(DEV)
    for norm in (True, False):
        q, a, r = ops.swiglu_quantize_rows(d[:, :H], d[:, H:], w.to(DEV) if norm else None, 1e-6, 1e-5)
        with np.errstate(all="ignore"):
            qo, ao, ro = O.swiglu_quantize_rows(t2n(gu[:, :H]), t2n(gu[:, H:]), w.numpy() if norm else None, 1e-6, 1e-5, _IO[dtype])
        assert np.array_equal(a.cpu().numpy(), ao) and np.array_equal(q.cpu().numpy(), qo)
        if norm:
            assert np.array_equal(r.cpu().numpy(), ro, equal_nan=True)
