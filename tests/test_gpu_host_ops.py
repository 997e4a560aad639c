"""The native operator calls on the GPU: what torch refuses a data pointer is refused there too, and calls of several threads."""
import os
import subprocess
import sys

import pytest

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
