"""The calls whose speed counts: INT2 layers and feed-forward blocks trained and served through the module API.

A case is a dict of plain values.  `kind` says which program is measured:

  train      one optimisation step of a layer: forward, backward (gradient of the input and of the norm weight) and the
             hysteresis update of the packed weights, fired from the output's gradient hook as a trainer has it
  infer      the layer without gradient recording: prefill with many tokens, decode with 1 to 64
  ffn_train  the same step of the SwiGLU feed-forward block (three layers, gate fused with norm and quantiser)
  ffn_infer  the block without gradient recording

Weights are drawn from N(0, 0.02), activations from N(0, 1), output gradients from N(0, 1e-3), counters uniformly from
[-3, 3]; about a sixth of the counters then sit at a threshold of 3, so a step moves a realistic share of the weights.
"""
import importlib.util
import math
import os
import sys

import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if not os.path.isdir(os.path.join(_ROOT, "elleci-training-vast_b200")):
    _ROOT = os.getcwd()


def _package():
    """The package; its directory name has a hyphen, so it is loaded by path (from the working folder's tree)."""
    name = "elleci_training_vast_b200"
    if name not in sys.modules:
        root = os.getcwd() if os.path.isdir(os.path.join(os.getcwd(), "elleci-training-vast_b200")) else _ROOT
        folder = os.path.join(root, "elleci-training-vast_b200")
        spec = importlib.util.spec_from_file_location(name, os.path.join(folder, "__init__.py"), submodule_search_locations=[folder])
        module = importlib.util.module_from_spec(spec)
        sys.modules[name] = module
        spec.loader.exec_module(module)
    return sys.modules[name]


_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
_BYTES = {"bf16": 2, "fp16": 2, "fp32": 4}
LR, LR_SCALE, DECAY = 1e-2, 5.0, 0.001


def _layer(kind, tokens, fin, fout, dtype="bf16", norm=True, mode="per_token", order="reference"):
    return {"kind": kind, "tokens": tokens, "in": fin, "out": fout, "dtype": dtype, "norm": norm, "mode": mode, "order": order}


def _ffn(kind, tokens, width, dtype="bf16"):
    return {"kind": kind, "tokens": tokens, "width": width, "dtype": dtype}


def listed():
    return [
        # a layer of the small model: batch 2 x 512 tokens
        dict(_layer("train", 1024, 1536, 1536, norm=False), name="train_small"),
        # the up and the down projection of the 7B feed-forward block: batch 4 x 1024 tokens
        dict(_layer("train", 4096, 4096, 11008, norm=False, order="after_dx"), name="train_up_7b"),
        dict(_layer("train", 4096, 11008, 4096), name="train_down_7b"),
        # the largest: a large-batch step of the 7B Mamba input projection
        dict(_layer("train", 65536, 4096, 16384, norm=False, order="after_dx"), name="train_long"),
        # the reference's own mode (one scale per tensor, fp16) with a token count that fills no tile
        dict(_layer("train", 1999, 2048, 1536, dtype="fp16", norm=False, mode="per_tensor"), name="train_per_tensor_ragged"),
        # the Mamba step-size projection, whose sixteen inputs fit no tensor-core tile
        dict(_layer("train", 2048, 16, 8192), name="train_dt_proj"),
        # prefill through the MLA latent down projection: few output tiles
        dict(_layer("infer", 4096, 4096, 512), name="prefill_latent"),
        # decode: one sequence, a few, a full batch
        dict(_layer("infer", 1, 4096, 11008), name="decode_1"),
        dict(_layer("infer", 8, 11008, 4096), name="decode_8"),
        dict(_layer("infer", 64, 4096, 11008), name="decode_64"),
        # the whole 7B feed-forward block: a training step, and the generation of a few sequences
        dict(_ffn("ffn_train", 4096, 4096), name="ffn_train_7b"),
        dict(_ffn("ffn_infer", 4, 4096), name="ffn_decode_4"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


_MOST_MACS = 65536 * 4096 * 16384


def draw(rng):
    """Another case of the same ranges: 1 to 65536 tokens (any number), layers from 256 x 256 to 16384 wide in steps of 64
    (the model's widths), now and then one of its narrow projections, all three data types, both quantisation modes."""
    dtype = rng.choice(["bf16"] * 6 + ["fp16"] * 2 + ["fp32"])
    kind = rng.choice(["train"] * 4 + ["infer"] * 2 + ["decode"] * 3 + ["ffn_train", "ffn_infer"])
    if kind in ("ffn_train", "ffn_infer"):
        width = 64 * _log_int(rng, 8, 72)
        tokens = _log_int(rng, 64, 16384) if kind == "ffn_train" else _log_int(rng, 1, 64)
        return _ffn(kind, tokens, width, dtype)
    fin, fout = 64 * _log_int(rng, 4, 256), 64 * _log_int(rng, 4, 256)
    norm = rng.random() < 0.7
    if kind == "decode":
        return _layer("infer", _log_int(rng, 1, 64), fin, fout, dtype, norm)
    tokens = _log_int(rng, 65, 65536)
    if kind == "train" and rng.random() < 0.15:       # the narrow projections: x_proj, dt_proj, the diff gate
        fin, fout = rng.choice([(fin, 48), (fin, 16), (16, fout)])
        tokens = min(tokens, 8192)
    while tokens * fin * fout > _MOST_MACS // 2 or tokens * (fin + fout) > 65536 * 20480 // 2:
        tokens = tokens // 2 + 1
    mode = "per_tensor" if kind == "train" and dtype == "fp16" and rng.random() < 0.6 else "per_token"
    order = rng.choice(["reference", "after_dx"])
    return _layer(kind, tokens, fin, fout, dtype, norm and mode == "per_token", mode, order)


def _fill_layer(layer, gen, dev):
    """Ternarised N(0, 0.02) weights, counters uniform in [-3, 3], a norm weight around one."""
    inner = layer.int2_layer
    n, k = layer.out_features, layer.in_features
    inner.init_from_float(torch.randn(n, k, generator=gen, device=dev) * 0.02)
    h = torch.randint(-3, 4, (n, 2 * inner.H_packed.shape[1]), generator=gen, device=dev, dtype=torch.int8)
    h = (h & 0xF).to(torch.uint8).view(n, -1, 2)
    inner.H_packed.copy_(h[:, :, 0] | (h[:, :, 1] << 4))
    if layer.use_extra_rmsnorm:
        with torch.no_grad():
            layer.extra_rmsnorm.weight.copy_(1.0 + 0.1 * torch.randn(k, generator=gen, device=dev))


def _rows(rows, cols, dtype, gen, dev, scale=1.0):
    x = torch.randn(rows, cols, generator=gen, device=dev, dtype=dtype)
    return x if scale == 1.0 else x.mul_(scale)


def prepare(case, seed):
    """The module with its weights on the GPU, and one batch: tokens and, for training, the gradient of the output."""
    pkg = _package()
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev).manual_seed(int(seed))
    dtype, tokens = _DTYPES[case["dtype"]], case["tokens"]
    training = case["kind"] in ("train", "ffn_train")
    if case["kind"].startswith("ffn"):
        module = pkg.SwiGLUFFNInt2(case["width"], threshold=3, lr_scale=LR_SCALE, decay_rate=DECAY).to(dev)
        layers = [module.w1, module.w2, module.w3]
        fin = fout = case["width"]
    else:
        fin, fout = case["in"], case["out"]
        module = pkg.BitLinearInt2(fin, fout, threshold=3, lr_scale=LR_SCALE, decay_rate=DECAY, use_extra_rmsnorm=case["norm"],
                                   quant_mode=case["mode"], hysteresis_order=case["order"]).to(dev)
        layers = [module]
    for layer in layers:
        _fill_layer(layer, gen, dev)
    module.train(training)
    pkg.set_all_int2_lr(module, LR)
    x = _rows(tokens, fin, dtype, gen, dev)
    state = {"module": module, "layers": layers, "x": x}
    if training:
        x.requires_grad_(True)
        state["dy"] = _rows(tokens, fout, dtype, gen, dev, 1e-3)
        state["norms"] = [layer.extra_rmsnorm.weight for layer in layers if layer.use_extra_rmsnorm]
    return state


def run(state):
    """One pass: a training step returns the output, the gradients and the updated packed state; inference the output."""
    module, x = state["module"], state["x"]
    if "dy" not in state:
        with torch.no_grad():
            return module(x)
    x.grad = None
    for w in state["norms"]:
        w.grad = None
    y = module(x)
    y.backward(state["dy"])
    return {"y": y.detach(), "dx": x.grad, "d_norm": [w.grad for w in state["norms"]],
            "weights": [layer.int2_layer.W_packed for layer in state["layers"]],
            "counters": [layer.int2_layer.H_packed for layer in state["layers"]]}


def _layer_work(tokens, fin, fout, esz, training, norm):
    """Bytes and operations of one layer: tokens in and out, packed weights (2 bits), and for training the two gradients
    and the packed weights and counters (4 bits) written back; three integer products of 2*tokens*in*out operations."""
    weights = fin * fout / 4
    if not training:
        return tokens * (fin + fout) * esz + weights + (4 * fin if norm else 0), 2 * tokens * fin * fout
    return 2 * tokens * (fin + fout) * esz + 2 * weights + fin * fout + (8 * fin if norm else 0), 6 * tokens * fin * fout


def work(case):
    esz, tokens = _BYTES[case["dtype"]], case["tokens"]
    training = case["kind"] in ("train", "ffn_train")
    if case["kind"].startswith("ffn"):
        width = case["width"]
        hidden = 256 * ((int(width * 8 / 3) + 255) // 256)
        # the block's own input and output, and every layer's weights and counters; what lies between may stay on the chip
        state = 3 * width * hidden * (1.5 if training else 0.25)
        ends = tokens * 2 * width * esz * (2 if training else 1)
        return {"bytes": state + ends + (2 if training else 1) * 4 * (2 * width + hidden), "flops": (18 if training else 6) * tokens * width * hidden}
    b, f = _layer_work(tokens, case["in"], case["out"], esz, training, case["norm"])
    return {"bytes": b, "flops": f}


def tolerance(case):
    """About four times what the path differs by from itself in 64 bits (norms, gates, quantisers, products; two passes on
    one state).  The products are exact integer sums; what differs is which way a value halfway between two int8 steps
    goes (bf16 tokens hit such ties on about one value in a thousand), the rounding of outputs to the I/O type and the
    few weights whose stochastic rounding sits on the edge.  In the block these pass through three quantisers, and the
    packed weights of the second step carry the first step's differences."""
    if case["dtype"] == "fp32":
        return {"rel": 2e-4, "max": 0.05, "differ": 5e-5}
    if case["kind"].startswith("ffn"):
        return {"rel": 0.03, "max": 0.9, "differ": 2e-3}
    return {"rel": 5e-3, "max": 0.4, "differ": 5e-5}
