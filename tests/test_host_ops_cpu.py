"""The native operator calls (csrc/host_ops.cpp): the module loads, names every operator that int2_tc_ops forwards to, and refuses
what the Python checks refused, with the same exception type and message.  No call here reaches a GPU."""
import importlib.util
import os
import re

import pytest
import torch

from conftest import ROOT, load_package


@pytest.fixture(scope="module")
def pkg():
    return load_package()


def test_every_forwarded_operator_exists(pkg):
    src = open(os.path.join(ROOT, "elleci-training-vast_b200", "int2_tc_ops.py")).read()
    names = set(re.findall(r"host_ops\(\)\.(\w+)\(", src))
    assert len(names) >= 10
    host = pkg._lib.host_ops()
    for name in names:
        assert callable(getattr(host, name)), name


@pytest.mark.parametrize("call,message", [
    (lambda o, t: o.quantize_rows(t), "x must be a CUDA tensor"),
    (lambda o, t: o.quantize_rows(None), "x must be a CUDA tensor"),
    (lambda o, t: o.quantize_grad(t, t, t), "dY must be a CUDA tensor"),
    (lambda o, t: o.quantize_activation(t), "Input must be a CUDA tensor"),
    (lambda o, t: o.rmsnorm_quantize_rows(t, t), "x must be a CUDA tensor"),
    (lambda o, t: o.rmsnorm_backward(t, t, t, t), "g must be a CUDA tensor"),
    (lambda o, t: o.swiglu_quantize_rows(t, t), "gate must be a CUDA tensor"),
    (lambda o, t: o.swiglu_backward(t, t, t), "gy must be a CUDA tensor"),
    (lambda o, t: o.prelinear_rows(t), "x must be a CUDA tensor"),
    (lambda o, t: o.matmul_rows(t, t, t, 1.0), "X_int8 must be a CUDA tensor"),
    (lambda o, t: o.backward_input_rows(t, t, t, 1.0, 8), "dY_int8 must be a CUDA tensor"),
    (lambda o, t: o.dw_hysteresis(t, t, t, t, t, 0.1, 5.0, 3, 0.0, 1), "Gq must be a CUDA tensor"),
    (lambda o, t: o.linear_decode(t, t, 1.0), "x must be a CUDA tensor"),
])
def test_arguments_that_are_no_cuda_tensors_are_refused(pkg, call, message):
    with pytest.raises(RuntimeError, match=message):
        call(pkg.int2_tc_ops, torch.zeros(2, 8))


def test_a_wrong_number_of_arguments_is_a_type_error(pkg):
    with pytest.raises(TypeError):
        pkg._lib.host_ops().quantize_rows(torch.zeros(2, 8))


def _refused_calls(o, t):
    """Every native operator on arguments that pass its checks; `t(shape, dtype)` makes them."""
    f, i8, u8 = torch.float32, torch.int8, torch.uint8
    x, row, one, w = t((4, 64), torch.bfloat16), t((4,), f), t((1,), f), t((64,), f)
    xq, gq, W, H = t((4, 64), i8), t((4, 32), i8), t((32, 16), u8), t((32, 32), u8)
    return {
        "quantize_rows": lambda: o.quantize_rows(x),
        "quantize_rows_fold": lambda: o.quantize_rows(x, fold_absmax=row),
        "quantize_grad": lambda: o.quantize_grad(x, row, one),
        "quantize_tensor": lambda: o.quantize_activation_async(x, one),
        "rmsnorm_quantize_rows": lambda: o.rmsnorm_quantize_rows(x, w),
        "rmsnorm_backward": lambda: o.rmsnorm_backward(x, x, w, row),
        "swiglu_quantize_rows": lambda: o.swiglu_quantize_rows(x, x, w),
        "swiglu_backward": lambda: o.swiglu_backward(x, x, x, w, row),
        "prelinear_rows": lambda: o.prelinear_rows(x, x, w),
        "gemm_fwd": lambda: o.matmul_rows(xq, W, row, 1.0),
        "gemm_dx": lambda: o.backward_input_rows(gq, W, row, 1.0, 64),
        "dw_hysteresis": lambda: o.dw_hysteresis(gq, xq, one, W, H, 0.1, 5.0, 3, 0.0, 1),
        "linear_decode": lambda: o.linear_decode(x, W, 1.0),
        "linear_decode_norm": lambda: o.linear_decode(x, W, 1.0, norm_weight=w),
    }


NATIVE_CALLS = sorted(_refused_calls(None, lambda s, d: torch.zeros(s, dtype=d)))


@pytest.mark.parametrize("name", NATIVE_CALLS)
def test_a_tensor_without_storage_is_refused_before_anything_is_cached(pkg, name):
    """Under vmap a tensor passes every check but has no data pointer.  Reading it raises, as it did in the Python functions: with the GIL
    held, before an output is allocated or a status word or decode workspace is created.  (The CUDA tensors are fake ones.)"""
    from torch._subclasses.fake_tensor import FakeTensorMode
    o = pkg.int2_tc_ops
    status, decode = dict(o._status_bufs), dict(o._decode_ws)

    def call(batched):
        def make(shape, dtype):
            return (batched + torch.zeros(shape, device="cuda:0")).to(dtype)
        return _refused_calls(o, make)[name]()

    with FakeTensorMode(), pytest.raises(RuntimeError, match="Cannot access data pointer of Tensor that doesn't have storage"):
        torch.func.vmap(call)(torch.zeros(3, 1, device="cuda:0"))
    assert o._status_bufs == status and o._decode_ws == decode


def test_threads_that_meet_in_the_first_call_share_one_status_word(pkg, monkeypatch):
    """The native calls keep the address of a device's status word, so a second thread's first call must not replace it: here the
    other thread's whole call runs while this one is still creating its tensor."""
    o, dev = pkg.int2_tc_ops, torch.device("cpu", 0)
    zeros, other = torch.zeros, []

    def zeros_with_another_thread(*args, **kw):
        if not other:
            other.append(None)
            other[0] = o.device_status(dev)
        return zeros(*args, **kw)

    monkeypatch.setattr(o, "_status_bufs", {})
    monkeypatch.setattr(torch, "zeros", zeros_with_another_thread)
    assert o.device_status(dev) is other[0] and o.device_status(dev) is other[0]


def test_a_module_built_for_another_torch_is_not_loaded(pkg, monkeypatch):
    """The extension module is compiled against one torch: under another one it counts as not built, to the loader and to the build."""
    spec = importlib.util.spec_from_file_location("_elleci_build", os.path.join(ROOT, "elleci-training-vast_b200", "build.py"))
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    built = build.host_path()
    assert os.path.exists(built)
    monkeypatch.setattr(torch, "__version__", "0.0.0+other")
    assert build.host_path() != built and build._stale()
    monkeypatch.setattr(pkg._lib, "_host", None)
    with pytest.raises(pkg.ElleciError, match="is missing: build it with"):
        pkg._lib.host_ops()


def _refusals(o, t):
    """(call, exception, message) for the checks of every native operator behind the first one; `t(shape, dtype)` makes the tensors.
    x [4,64], two weight matrices of 32 rows, and what a caller may get wrong about each argument."""
    f, i8, u8, b16 = torch.float32, torch.int8, torch.uint8, torch.bfloat16
    x, row, one, w = t((4, 64), b16), t((4,), f), t((1,), f), t((64,), f)
    xq, gq, W, H = t((4, 64), i8), t((4, 32), i8), t((32, 16), u8), t((32, 32), u8)
    row5, w2, h64 = t((5,), f), t((64, 2), f)[:, 0], t((4, 64), torch.float16)
    cpu = torch.zeros(1)
    R, K, V, T = RuntimeError, KeyError, ValueError, TypeError
    floats = "must be float16, bfloat16 or float32"
    upd = (0.1, 5.0, 3, 0.0, 1)
    return {
        "quantize_rows": [
            (lambda: o.quantize_rows(xq), R, "x " + floats),
            (lambda: o.quantize_rows(x, "eps"), T, "real number"),
            (lambda: o.quantize_rows(x, fold_absmax=row5), R, r"fold_absmax must be float32 \[M\]"),
            (lambda: o.quantize_rows(x, fold_absmax=row.to(b16)), R, r"fold_absmax must be float32 \[M\]"),
            (lambda: o.quantize_rows(x, fold_absmax=3), T, "fold_absmax must be a tensor"),
            (lambda: o.quantize_rows(x, raw_absmax=row5), R, r"raw_absmax must be a contiguous float32 \[M\]"),
            (lambda: o.quantize_rows(x, raw_absmax=t((4, 2), f)[:, 0]), R, r"raw_absmax must be a contiguous float32 \[M\]"),
            (lambda: o.quantize_rows(x, out=x), R, r"out must be a contiguous int8 CUDA tensor of M\*K elements"),
            (lambda: o.quantize_rows(x, out=gq), R, r"out must be a contiguous int8 CUDA tensor of M\*K elements"),
            (lambda: o.quantize_rows(x, out=t((4, 128), i8)[:, ::2]), R, r"out must be a contiguous int8 CUDA tensor of M\*K elements")],
        "quantize_grad": [
            (lambda: o.quantize_grad(x, row5, one), R, r"x_absmax must be float32 \[M\]"),
            (lambda: o.quantize_grad(x, row, row), R, r"g_absmax must be float32 \[1\]"),
            (lambda: o.quantize_grad(xq, row, one), K, "torch")],
        "quantize_tensor": [
            (lambda: o.quantize_activation_async(x, cpu), R, "d_global_max must be a CUDA tensor"),
            (lambda: o.quantize_activation_async(xq, one), R, "Input must be float16")],
        "rmsnorm_quantize_rows": [
            (lambda: o.rmsnorm_quantize_rows(x, None), R, "weight must be a CUDA tensor"),
            (lambda: o.rmsnorm_quantize_rows(xq, w), R, "x " + floats),
            (lambda: o.rmsnorm_quantize_rows(x, row), R, r"weight must be a contiguous float32 \[K\]"),
            (lambda: o.rmsnorm_quantize_rows(x, w.to(b16)), R, r"weight must be a contiguous float32 \[K\]"),
            (lambda: o.rmsnorm_quantize_rows(x, w2), R, r"weight must be a contiguous float32 \[K\]")],
        "rmsnorm_backward": [
            (lambda: o.rmsnorm_backward(x, h64, w, row), R, "g and x must have the same shape and dtype"),
            (lambda: o.rmsnorm_backward(x[:2], x, w, row), R, "g and x must have the same shape and dtype"),
            (lambda: o.rmsnorm_backward(x, x, row, row), R, r"weight must be float32 \[K\]"),
            (lambda: o.rmsnorm_backward(x, x, w, row5), R, r"rstd must be float32 \[M\]")],
        "swiglu_quantize_rows": [
            (lambda: o.swiglu_quantize_rows(x, h64), R, "gate and up must have the same shape and dtype"),
            (lambda: o.swiglu_quantize_rows(xq, xq), R, "gate and up " + floats),
            (lambda: o.swiglu_quantize_rows(x, x, w2), R, r"norm_weight must be a contiguous float32 \[H\]")],
        "swiglu_backward": [
            (lambda: o.swiglu_backward(x, x, x[:2]), R, "gate and up must have the same shape and dtype"),
            (lambda: o.swiglu_backward(h64, x, x), R, "gy must have the shape and dtype of gate"),
            (lambda: o.swiglu_backward(x, x, x, out=x), R, r"out must be a contiguous \[M, 2H\] tensor"),
            (lambda: o.swiglu_backward(x, x, x, row, row), R, r"norm_weight must be float32 \[H\]"),
            (lambda: o.swiglu_backward(x, x, x, w), R, r"rstd must be float32 \[M\]"),
            (lambda: o.swiglu_backward(x, x, x, w, row5), R, r"rstd must be float32 \[M\]")],
        "prelinear_rows": [
            (lambda: o.prelinear_rows(xq), R, "x " + floats),
            (lambda: o.prelinear_rows(x, cpu), R, "up must be a CUDA tensor"),
            (lambda: o.prelinear_rows(x, h64), R, "gate and up must have the same shape and dtype"),
            (lambda: o.prelinear_rows(x, None, w2), R, r"norm_weight must be a contiguous float32 \[K\]")],
        "gemm_fwd": [
            (lambda: o.matmul_rows(x, W, row, 1.0), R, "X_int8 must be int8"),
            (lambda: o.matmul_rows(xq, xq, row, 1.0), R, "W_packed must be uint8"),
            (lambda: o.matmul_rows(xq, W, row.to(b16), 1.0), R, "d_scale_x must be float32"),
            (lambda: o.matmul_rows(xq, W[0], row, 1.0), R, "W_packed must be 2-D"),
            (lambda: o.matmul_rows(gq, W, row, 1.0), R, "Dimension mismatch: X has 32 features but W_packed has packed_K=16"),
            (lambda: o.matmul_rows(xq, W, row5, 1.0), R, "one absmax per token expected"),
            (lambda: o.matmul_rows(xq, W, row, 1.0, torch.int64), K, "torch"),
            (lambda: o.matmul_rows(xq, W, row, 1.0, "bf16"), T, "torch.dtype"),
            (lambda: o.matmul_rows(xq, W, row, None), T, "real number")],
        "gemm_dx": [
            (lambda: o.backward_input_rows(x, W, row, 1.0, 64), R, "dY_int8 must be int8"),
            (lambda: o.backward_input_rows(gq, gq, row, 1.0, 64), R, "W_packed must be uint8"),
            (lambda: o.backward_input_rows(gq, W, row.to(b16), 1.0, 64), R, "d_scale_dy must be float32"),
            (lambda: o.backward_input_rows(gq, W[0], row, 1.0, 64), V, "W_packed must be 2-D"),
            (lambda: o.backward_input_rows(xq, W, row, 1.0, 64), R, "dY has 64 features but W_packed has 32 rows"),
            (lambda: o.backward_input_rows(gq, W, row, 1.0, 60), R, "K=60 does not match W_packed's packed_K=16"),
            (lambda: o.backward_input_rows(gq, W, row5, 1.0, 64), R, "one absmax per token expected")],
        "dw_hysteresis": [
            (lambda: o.dw_hysteresis(x, xq, one, W, H, *upd), R, "Gq and Xq must be int8"),
            (lambda: o.dw_hysteresis(gq[:2], xq, one, W, H, *upd), R, "Gq and Xq must have the same number of tokens"),
            (lambda: o.dw_hysteresis(gq, xq, one, W, W, *upd), R, "W_packed / H_packed shape mismatch"),
            (lambda: o.dw_hysteresis(gq, xq, one, t((32, 32), u8)[:, ::2], H, *upd), R, "W_packed/H_packed must be contiguous")],
        "linear_decode": [
            (lambda: o.linear_decode(xq, W, 1.0), R, "x " + floats),
            (lambda: o.linear_decode(x, W[0], 1.0), R, "W_packed must be uint8"),
            (lambda: o.linear_decode(x[:, :32], W, 1.0), R, "x has 32 features but W_packed has packed_K=16"),
            (lambda: o.linear_decode(t((65, 64), b16), W, 1.0), R, "linear_decode takes 1..64 tokens"),
            (lambda: o.linear_decode(t((0, 64), b16), W, 1.0), R, "linear_decode takes 1..64 tokens"),
            (lambda: o.linear_decode(x, W, 1.0, torch.int64), K, "torch"),
            (lambda: o.linear_decode(x, W, 1.0, up=h64), R, "gate and up must have the same shape and dtype"),
            (lambda: o.linear_decode(x, W, 1.0, norm_weight=w2), R, r"norm_weight must be a contiguous float32 \[K\]")],
    }


@pytest.mark.parametrize("name", sorted(_refusals(None, lambda s, d: torch.zeros(s, dtype=d))))
def test_arguments_with_the_wrong_type_or_shape_are_refused(pkg, name):
    """Each check of the native operators, on fake CUDA tensors: the exception type and the message that the caller sees."""
    from torch._subclasses.fake_tensor import FakeTensorMode
    with FakeTensorMode():
        cases = _refusals(pkg.int2_tc_ops, lambda shape, dtype: torch.zeros(shape, device="cuda:0").to(dtype))[name]
        for i, (call, error, message) in enumerate(cases):
            with pytest.raises(error, match=message):
                call()
                pytest.fail(f"{name}: case {i} was accepted")
