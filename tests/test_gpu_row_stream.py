"""The streaming norm and gate kernels, bit for bit against the oracle: at the edges of their ranges (columns that fill no warp's
vectors, the widths where one form hands over to the next, tokens with non-finite values between ordinary ones), with so many
tokens that every CTA refills its slots several times, and with products below the normal range of the type."""
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


# 256: CTAs of one warp; 1032: a last warp with one vector; 6152 / 8200 / 12296: float32 and 16-bit
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


def _some_rows(M, first, n=48):
    """Row 0, the last row and n between them, half of them from `first` on."""
    rng = np.random.default_rng(M)
    rows = np.concatenate([[0, M - 1], rng.choice(np.arange(1, first), n // 2, False), rng.choice(np.arange(first, M - 1), n // 2, False)])
    return np.unique(rows)


# Five tokens or more per CTA, on several warps, by the grid of each launch on 148 SMs: 16-bit norm forward 8 CTAs per SM at 4096
# columns and 2 at 11008 (float32: 4 and 1), gate forward 6 and 2, norm and gate backward 3 at 4096 (float32: 2).  The slots
# hold two rows (norm backward: three), so that rows from the third (fourth) on are read from refilled slots, and from
# the third on reuse the first row's reduction buffers.  `at`: a row that no CTA takes before its third.
@pytest.mark.parametrize("M,K,at", [(6000, 4096, 3000), (1500, 11008, 700)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
def test_norm_forward_over_refilled_slots(ops, M, K, at, dtype):
    g = torch.Generator().manual_seed(M + K)
    x = (torch.randn(M, K, generator=g) * 1.5).to(dtype)
    w = (1.0 + 0.3 * torch.randn(K, generator=g)).float()
    x[at, K // 2] = float("inf")
    x[at + 1, 3] = float("nan")
    x[M - 2, K - 1] = float("-inf")
    rows = np.union1d(_some_rows(M, at), [at - 1, at, at + 1, at + 2, M - 2])
    q, a, r = ops.rmsnorm_quantize_rows(x.to(DEV), w.to(DEV), 1e-6, 1e-5)
    with np.errstate(all="ignore"):
        qo, ao, ro = O.rmsnorm_quantize_rows(t2n(x[rows]), w.numpy(), 1e-6, 1e-5, _IO[dtype])
    assert np.array_equal(r.cpu().numpy()[rows], ro, equal_nan=True)
    assert np.array_equal(a.cpu().numpy()[rows], ao) and np.array_equal(q.cpu().numpy()[rows], qo)


@pytest.mark.parametrize("M,H,at", [(4500, 4096, 2000), (1500, 11008, 700)])
@pytest.mark.parametrize("norm", [True, False])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_gate_forward_over_refilled_slots(ops, M, H, at, norm, dtype):
    g = torch.Generator().manual_seed(M * 3 + H)
    gu = (torch.randn(M, 2 * H, generator=g) * 2.0).to(dtype)
    w = (1.0 + 0.3 * torch.randn(H, generator=g)).float() if norm else None
    gu[at, H - 1] = float("nan")
    gu[at + 1, H + 7] = float("inf")
    gu[M - 2, 2 * H - 1] = float("-inf")
    rows = np.union1d(_some_rows(M, at), [at - 1, at, at + 1, at + 2, M - 2])
    d = gu.to(DEV)
    q, a, r = ops.swiglu_quantize_rows(d[:, :H], d[:, H:], w.to(DEV) if norm else None, 1e-6, 1e-5)
    h = t2n(gu[rows])
    with np.errstate(all="ignore"):
        qo, ao, ro = O.swiglu_quantize_rows(h[:, :H], h[:, H:], w.numpy() if norm else None, 1e-6, 1e-5, _IO[dtype])
    assert np.array_equal(a.cpu().numpy()[rows], ao) and np.array_equal(q.cpu().numpy()[rows], qo)
    if norm:
        assert np.array_equal(r.cpu().numpy()[rows], ro, equal_nan=True)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
def test_backward_over_refilled_slots(ops, dtype):
    M, K = 2500, 4096
    g = torch.Generator().manual_seed(9)
    gu, gy = (torch.randn(M, 2 * K, generator=g) * 2.0).to(dtype), (torch.randn(M, K, generator=g) * 1e-2).to(dtype)
    w = (1.0 + 0.3 * torch.randn(K, generator=g)).float()
    d = gu.to(DEV)
    x, up = t2n(gu[:, :K]), t2n(gu[:, K:])
    rstd = O.rmsnorm_rstd(x, 1e-6)
    dx, dw = ops.rmsnorm_backward(gy.to(DEV), d[:, :K].contiguous(), w.to(DEV), torch.from_numpy(rstd).to(DEV))
    dxo, dwo = O.rmsnorm_backward(t2n(gy), x, w.numpy(), rstd, _IO[dtype])
    assert np.array_equal(t2n(dx), dxo) and np.array_equal(dw.cpu().numpy(), dwo)
    h, _, _ = O.swiglu_hidden(x, up, _IO[dtype])
    rstd = O.rmsnorm_rstd(h, 1e-6)
    dg, du, dw = ops.swiglu_backward(gy.to(DEV), d[:, :K], d[:, K:], w.to(DEV), torch.from_numpy(rstd).to(DEV))
    dgo, duo, dwo = O.swiglu_backward(t2n(gy), x, up, w.numpy(), rstd, _IO[dtype])
    assert np.array_equal(t2n(dg), dgo) and np.array_equal(t2n(du), duo) and np.array_equal(dw.cpu().numpy(), dwo)


# gradients whose packed 16-bit products lie around and below the smallest normal number of the type, down to half its
# smallest subnormal one: one rounding there has to give what float32 and then the type give (row_stream.cuh, mul_raw)
@pytest.mark.parametrize("dtype,scale", [(torch.bfloat16, 1e-38), (torch.bfloat16, 1e-40), (torch.float16, 1e-5), (torch.float16, 2e-7)])
def test_backward_below_the_normal_range(ops, dtype, scale):
    M, K = 40, 1032
    g = torch.Generator().manual_seed(5)
    gu, gy = torch.randn(M, 2 * K, generator=g).to(dtype), (torch.randn(M, K, generator=g).double() * scale).to(dtype)
    w = (1.0 + 0.3 * torch.randn(K, generator=g)).float()
    d = gu.to(DEV)
    x, up = t2n(gu[:, :K]), t2n(gu[:, K:])
    rstd = O.rmsnorm_rstd(x, 1e-6)
    dx, dw = ops.rmsnorm_backward(gy.to(DEV), d[:, :K].contiguous(), w.to(DEV), torch.from_numpy(rstd).to(DEV))
    dxo, dwo = O.rmsnorm_backward(t2n(gy), x, w.numpy(), rstd, _IO[dtype])
    assert np.count_nonzero(dxo) > M * K // 4
    assert np.array_equal(t2n(dx), dxo) and np.array_equal(dw.cpu().numpy(), dwo)
    h, _, _ = O.swiglu_hidden(x, up, _IO[dtype])
    rstd = O.rmsnorm_rstd(h, 1e-6)
    dg, du, dw = ops.swiglu_backward(gy.to(DEV), d[:, :K], d[:, K:], w.to(DEV), torch.from_numpy(rstd).to(DEV))
    dgo, duo, dwo = O.swiglu_backward(t2n(gy), x, up, w.numpy(), rstd, _IO[dtype])
    assert np.array_equal(t2n(dg), dgo) and np.array_equal(t2n(du), duo) and np.array_equal(dw.cpu().numpy(), dwo)
