"""Several training steps of one layer whose output gradient arrives in the same buffer every time, with new values: dX, output and packed
state of each step against the oracle, in both update orders, and what a pass leaves behind when it ends early."""
import numpy as np
import pytest
import torch

from oracle import int2_oracle as O
from oracle import native

from helpers import make_layer_inputs, t2n

pytestmark = pytest.mark.gpu
DEV = "cuda"
M, K, N, LR = 64, 128, 96, 0.5


def _layer(pkg, d, order="reference", hook=True, **kw):
    cls = pkg.Int2LinearTCWithGradHook if hook else pkg.Int2LinearTC
    layer = cls(K, N, threshold=2, lr_scale=5.0, decay_rate=0.001, hysteresis_order=order, **kw).to(DEV)
    layer.init_from_float(d["W"].to(DEV), scale=d["gamma"])
    if hook:
        layer.set_lr(LR)
    return layer.train()


def _gradient(step):
    return (torch.randn(M, N, generator=torch.Generator().manual_seed(100 + step)) * 1e-2).bfloat16()


def _oracle_step(d, dY, Wp, Hp, step, order, dY_for_dx=None):
    _, Xq, ax = O.bitlinear_forward(t2n(d["x"]), Wp, d["gamma"], K, out="bf16")
    dW, _, _ = O.bitlinear_dw(t2n(dY), Xq, ax)
    Wn, Hn = native.c_hysteresis_step(dW, Wp, Hp, LR, 5.0, 2, 0.001, step, K)
    w = Wp if order == "after_dx" else Wn
    return O.bitlinear_backward_dx(t2n(dY if dY_for_dx is None else dY_for_dx), w, d["gamma"], K, out="bf16"), Wn, Hn


def _check(layer, x, want, Wn, Hn):
    assert np.array_equal(t2n(x.grad), want)
    assert np.array_equal(layer.W_packed.cpu().numpy(), Wn) and np.array_equal(layer.H_packed.cpu().numpy(), Hn)


@pytest.mark.parametrize("order", ["reference", "after_dx"])
@pytest.mark.parametrize("refill", ["copy_", "data.copy_", "no hook"])
def test_one_gradient_buffer_refilled_each_step(pkg, order, refill):
    """"no hook": the update is the caller's own call after the backward pass."""
    d = make_layer_inputs(M, K, N, seed=1)
    hook = refill != "no hook"
    if not hook and order == "reference":
        order = "after_dx"
    layer, Wp, Hp = _layer(pkg, d, order, hook), d["Wp"], d["Hp"]
    buf = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
    x = d["x"].to(DEV).requires_grad_(True)
    for step in range(1, 5):
        dY = _gradient(step)
        (buf.data if refill == "data.copy_" else buf).copy_(dY)
        x.grad = None
        layer(x).backward(buf)
        if not hook:
            layer.hysteresis_update(buf, LR)
        want, Wp, Hp = _oracle_step(d, dY, Wp, Hp, step, order)
        _check(layer, x, want, Wp, Hp)


@pytest.mark.parametrize("order", ["reference", "after_dx"])
def test_gradient_changed_by_a_later_hook(pkg, order):
    """A hook of the caller's that runs after the layer's own and doubles the gradient where it lies: dX is that of the doubled one; the
    update before dX has seen the first, the update after dX the doubled."""
    d = make_layer_inputs(M, K, N, seed=2)
    layer, Wp, Hp = _layer(pkg, d, order), d["Wp"], d["Hp"]
    x = d["x"].to(DEV).requires_grad_(True)
    for step in (1, 2):
        dY = _gradient(step)
        x.grad = None
        y = layer(x)
        y.register_hook(lambda g: g.mul_(2))
        y.backward(dY.to(DEV))
        want, Wp, Hp = _oracle_step(d, dY if order == "reference" else dY * 2, Wp, Hp, step, order, dY * 2)
        _check(layer, x, want, Wp, Hp)


@pytest.mark.parametrize("order", ["reference", "after_dx"])
@pytest.mark.parametrize("first", ["stops at the output", "needs no dX", "accumulation"])
def test_pass_that_forms_no_dx(pkg, order, first):
    """What the hook of such a pass left is not taken for the gradient of the next one, which comes in the same buffer."""
    d = make_layer_inputs(M, K, N, seed=3)
    layer, Wp, Hp = _layer(pkg, d, order, bias=True), d["Wp"], d["Hp"]
    buf, x = _gradient(0).to(DEV), d["x"].to(DEV).requires_grad_(True)
    updated = False
    if first == "stops at the output":
        y = layer(x)
        torch.autograd.grad(y, [y], buf)
        updated = order == "reference"
    elif first == "needs no dX":
        layer(x.detach()).backward(buf)
        updated = True
    else:
        pkg.disable_hysteresis()
        try:
            layer(x).backward(buf)
        finally:
            pkg.enable_hysteresis()
    steps = 1
    if updated:
        _, Wp, Hp = _oracle_step(d, _gradient(0), Wp, Hp, 1, order)
        steps = 2
    dY = _gradient(1)
    buf.data.copy_(dY)
    x.grad = None
    layer(x).backward(buf)
    want, Wp, Hp = _oracle_step(d, dY, Wp, Hp, steps, order)
    _check(layer, x, want, Wp, Hp)


@pytest.mark.parametrize("order", ["reference", "after_dx"])
def test_a_step_quantises_the_gradient_once_and_keeps_nothing(pkg, order, monkeypatch):
    d = make_layer_inputs(M, K, N, seed=4)
    layer = _layer(pkg, d, order)
    x = d["x"].to(DEV).requires_grad_(True)
    calls = []
    ops = pkg.int2_tc_ops
    quantise, update = ops.quantize_rows, ops.weight_update
    monkeypatch.setattr(ops, "quantize_rows", lambda *a, **k: (calls.append("rows"), quantise(*a, **k))[1])
    monkeypatch.setattr(ops, "weight_update", lambda *a, **k: (calls.append("update"), update(*a, **k))[1])
    y = layer(x)
    calls.clear()
    y.backward(_gradient(1).to(DEV))
    assert calls == (["update"] if order == "reference" else ["rows", "update"])

    def tensors(v):
        return isinstance(v, torch.Tensor) or (isinstance(v, tuple) and any(map(tensors, v)))

    assert [name for name, v in vars(layer).items() if tensors(v)] == []
