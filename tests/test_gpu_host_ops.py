"""The native operator calls on the GPU: what torch refuses a data pointer is refused there too, and calls of several threads."""
import os
import subprocess
import sys
import threading

import pytest
import torch

from conftest import ROOT

pytestmark = pytest.mark.gpu


def test_vmap_over_a_layer_raises_and_leaves_the_process_alive():
    """vmap hands the layer tensors without storage: the call raises in Python, and the process goes on to a normal call."""
    code = """
import sys
sys.path.insert(0, {tests!r}); sys.path.insert(0, {root!r})
import torch
from conftest import load_package
pkg = load_package()
layer = pkg.BitLinearInt2(64, 128, use_extra_rmsnorm=False).to("cuda").eval()
x = torch.randn(3, 4, 64, device="cuda", dtype=torch.bfloat16)
with torch.no_grad():
    layer(x)                    # the first call draws the weights
    try:
        torch.func.vmap(layer)(x)
    except RuntimeError as e:
        assert "Cannot access data pointer of Tensor" in str(e), e
    else:
        raise SystemExit("vmap was accepted")
    assert layer(x).shape == (3, 4, 128)
torch.cuda.synchronize()
print("alive")
""".format(tests=os.path.join(ROOT, "tests"), root=ROOT)
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "alive", (r.returncode, r.stdout, r.stderr)


def test_a_call_that_the_library_refuses_raises_and_leaves_the_next_one_alone(pkg):
    """A status other than 0 comes back as ElleciError with the call's name, from each kind of entry point."""
    o, dev = pkg.int2_tc_ops, "cuda"
    x, w, W = torch.randn(4, 64, device=dev), torch.ones(64, device=dev), torch.zeros(32, 16, dtype=torch.uint8, device=dev)
    odd, wide = torch.randn(4, 60, device=dev), torch.randn(4, 60, device=dev, dtype=torch.bfloat16)
    refused = [
        ("el_rmsnorm_quantize_rows", lambda: o.rmsnorm_quantize_rows(wide, torch.ones(60, device=dev))),
        ("el_rmsnorm_backward", lambda: o.rmsnorm_backward(wide, wide, torch.ones(60, device=dev), w[:4])),
        ("el_swiglu_quantize_rows", lambda: o.swiglu_quantize_rows(wide, wide)),
        ("el_linear_decode", lambda: o.linear_decode(odd, W[:, :15], 1.0)),
        ("el_prelinear_decode", lambda: o.linear_decode(odd, W[:, :15], 1.0, norm_weight=torch.ones(60, device=dev))),
        ("el_gemm_fwd_ws", lambda: o.matmul_rows(torch.zeros(4, 60, dtype=torch.int8, device=dev), W[:, :15], w[:4], 1.0, path=pkg._lib.EL_PATH_TC)),
    ]
    good = o.linear_decode(x, W, 1.0, norm_weight=w)
    for name, call in refused:
        with pytest.raises(pkg.ElleciError, match=name):
            call()
        assert torch.equal(o.linear_decode(x, W, 1.0, norm_weight=w), good)
    o.check_device_status(torch.device(dev, torch.cuda.current_device()))


# 64 x 16384: the stream-K kernel, whose partial sums meet in the cached workspace; 5 and 64 x 1024: kernels without one
@pytest.mark.parametrize("M,K,norm", [(64, 16384, False), (64, 16384, True), (64, 1024, True), (5, 1024, False)])
def test_decode_from_several_threads_on_their_own_streams(pkg, M, K, norm):
    """Threads that decode at the same time, each on its own stream and weights, each from its first call on (the call that creates the
    stream's workspace): every output is that of the call alone."""
    o, N, threads, calls = pkg.int2_tc_ops, 2048, 4, 25
    g = torch.Generator(device="cuda").manual_seed(M + K)
    W = [torch.randint(0, 256, (N, K // 4), generator=g, device="cuda", dtype=torch.uint8) for _ in range(threads)]
    x = [torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16) for _ in range(threads)]
    w = torch.rand(K, generator=g, device="cuda") + 0.5 if norm else None
    want = []
    for i in range(threads):
        q, a = o.quantize_rows(x[i]) if w is None else o.rmsnorm_quantize_rows(x[i], w)[:2]
        want.append(o.matmul_rows(q, W[i], a, 0.01))
    torch.cuda.synchronize()
    wrong, errors, start = [0] * threads, [], threading.Barrier(threads)

    def decode(i):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                start.wait(timeout=60)
                outs = [o.linear_decode(x[i], W[i], 0.01, norm_weight=w) for _ in range(calls)]
                wrong[i] = sum(int((y != want[i]).sum()) for y in outs)
        except BaseException as e:          # reported by the main thread
            errors.append(e)

    pool = [threading.Thread(target=decode, args=(i,)) for i in range(threads)]
    for t in pool:
        t.start()
    for t in pool:
        t.join(timeout=120)
    assert not errors and wrong == [0] * threads, (errors, wrong)
    o.check_device_status(torch.device("cuda", torch.cuda.current_device()))


@pytest.mark.parametrize("M,norm", [(1, False), (5, True), (24, False), (64, False), (64, True)])
def test_decode_keeps_no_memory_and_needs_no_workspace(pkg, M, norm):
    """A stream's first decode call holds nothing once its output is gone; a workspace that is given is still checked for its size."""
    o, N, K = pkg.int2_tc_ops, 4096, 256
    x, W = torch.randn(M, K, device="cuda"), torch.randint(0, 256, (N, K // 4), device="cuda", dtype=torch.uint8)
    w = torch.ones(K, device="cuda") if norm else None
    need = pkg._lib.lib().el_decode_workspace_bytes(N)
    want = o.linear_decode(x, W, 0.01, workspace=torch.zeros(need, device="cuda", dtype=torch.uint8), norm_weight=w)
    with pytest.raises(RuntimeError, match="workspace too small"):
        o.linear_decode(x, W, 0.01, workspace=torch.zeros(need - 1, device="cuda", dtype=torch.uint8), norm_weight=w)
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    with torch.cuda.stream(torch.cuda.Stream()):
        y = o.linear_decode(x, W, 0.01, norm_weight=w)
        torch.cuda.synchronize()
        assert torch.equal(y, want)
        del y
    assert torch.cuda.memory_allocated() == before
