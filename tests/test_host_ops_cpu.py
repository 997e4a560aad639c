"""The native operator calls (csrc/host_ops.cpp): the module loads, names every operator that int2_tc_ops forwards to, and refuses
what the Python checks refused, with the same exception type and message.  No call here reaches a GPU."""
import re

import os

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
