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
