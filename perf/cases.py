"""Workloads that stand for what a user of this library has it do, through its public entry points.

`listed()` holds the named ones; `draw(rng)` gives more of the same ranges. `prepare` makes weights and inputs on the GPU from
a seed, `run` is one pass, `work` the bytes and operations a pass cannot do without, `tolerance` how far a correct
implementation of the same precision may be off.

Kinds of case:
  vit        a DINOv2 model as models.dinov2.dinov2() builds it: features of a batch of images, eager or from a CUDA graph
  blocks     the transformer blocks of a timm-style ViT patched by install_vit_blocks(), eager or under graphs.graphed()
  attention  one attention() call, on the unbound packed qkv buffer or on tensors of their own
  linear     one linear() call with one of its epilogues
  layernorm  one layer_norm() call
"""
import torch
import torch.nn as nn

import fastbb_b200 as fastbb
from fastbb_b200.attention import attention
from fastbb_b200.gemm import linear
from fastbb_b200.graphs import graphed
from fastbb_b200.layernorm import layer_norm
from fastbb_b200.models.dinov2 import ARCH, DinoV2Params, dinov2, swiglu_hidden

PATCH = 14
# blocks whose features dense-prediction heads read (four per model, spread over its depth)
TAPS = {"vits14": (2, 5, 8, 11), "vitb14": (2, 5, 8, 11), "vitl14": (4, 11, 17, 23), "vitg14": (9, 19, 29, 39)}


def listed():
    return [
        # An interactive program that embeds one 224 x 224 image at a time with the smallest model: launches and host time.
        {"name": "vits14_224_b1_eager", "kind": "vit", "arch": "vits14", "registers": 0, "height": 224, "width": 224, "batch": 1,
         "spec": "fh-g0", "graph": False, "call": "features", "image": "fp32"},
        # The same model and size in a service that replays a CUDA graph.
        {"name": "vits14_224_b1_graph", "kind": "vit", "arch": "vits14", "registers": 0, "height": 224, "width": 224, "batch": 1,
         "spec": "fh-g0", "graph": True, "call": "last", "image": "fp32"},
        # Dense prediction on a landscape photo: register tokens, feature maps of four layers as [B, C, h, w], ragged token count (1041).
        {"name": "vitb14reg_392x518_b1_maps", "kind": "vit", "arch": "vitb14", "registers": 4, "height": 392, "width": 518, "batch": 1,
         "spec": "sdpa-g0", "graph": False, "call": "maps", "image": "fp32"},
        # Embedding a data set: a batch of 224 x 224 crops through a large model.
        {"name": "vitl14_224_b32_eager", "kind": "vit", "arch": "vitl14", "registers": 0, "height": 224, "width": 224, "batch": 32,
         "spec": "fh-g2", "graph": False, "call": "features", "image": "fp32"},
        # The headline workload: one 896 x 1344 frame, four layers' tokens (6145 tokens), replayed.
        {"name": "vitl14_896x1344_b1_graph", "kind": "vit", "arch": "vitl14", "registers": 0, "height": 896, "width": 1344, "batch": 1,
         "spec": "fh-g0", "graph": True, "call": "tokens", "image": "fp16"},
        # The largest model at its native resolution, one GPU's share of a batch of 32 (4 x 1370 tokens), fp16 accumulation.
        {"name": "vitg14_518_b4_graph", "kind": "vit", "arch": "vitg14", "registers": 0, "height": 518, "width": 518, "batch": 4,
         "spec": "hh-g1", "graph": True, "call": "last", "image": "fp16"},
        # A timm ViT-B/16 at 1024 x 1024 (4097 tokens) with its blocks patched in place.
        {"name": "vitb16_blocks_4097_b1", "kind": "blocks", "dim": 768, "depth": 12, "tokens": 4097, "batch": 1, "spec": "fh-g1",
         "graph": False, "dtype": "fp16"},
        # The operators on their own, as a program that vendors them calls them: the smallest attention of the ViT range ...
        {"name": "attention_257_h16", "kind": "attention", "tokens": 257, "heads": 16, "batch": 1, "variant": "fh", "packed": True},
        # ... and the longest sequence of the kernel sweep.
        {"name": "attention_16385_h16", "kind": "attention", "tokens": 16385, "heads": 16, "batch": 1, "variant": "hh", "packed": True},
        # An ordinary MLP input layer: tokens of one 518 x 518 image, GELU epilogue.
        {"name": "linear_1370_fc1_gelu", "kind": "linear", "rows": 1370, "k": 1024, "n": 4096, "epilogue": "gelu", "bias": True, "variant": "f32"},
        # The largest layer of the kernel sweep: MLP output with LayerScale and residual, fp16 accumulation.
        {"name": "linear_32768_fc2_residual", "kind": "linear", "rows": 32768, "k": 4096, "n": 1024, "epilogue": "residual", "bias": True, "variant": "h"},
        # LayerNorm of the headline's tokens, fp32 input cast to fp16 on the way out.
        {"name": "layernorm_6145x1024_fp32", "kind": "layernorm", "rows": 6145, "dim": 1024, "dtype": "fp32"},
    ]


# ---------------------------------------------------------------------------------------------------------- more cases
def _spread(rng, lo, hi):
    """A whole number of lo .. hi, even over its logarithm."""
    return min(hi, max(lo, int(round(lo * (hi / lo) ** rng.random()))))


def _draw_vit(rng):
    arch = rng.choice(["vits14", "vitb14", "vitl14", "vitg14"])
    return {"kind": "vit", "arch": arch, "registers": rng.choice([0, 0, 4]), "height": PATCH * _spread(rng, 8, 96), "width": PATCH * _spread(rng, 8, 96),
            "batch": _spread(rng, 1, 32), "spec": rng.choice(["fh", "hh", "sdpa", "ff"]) + "-" + rng.choice(["g0", "g1", "g2", "g3"]),
            "graph": rng.random() < 0.5, "call": rng.choice(["features", "last", "tokens", "maps"]), "image": rng.choice(["fp32", "fp16"])}


def _draw_blocks(rng):
    return {"kind": "blocks", "dim": rng.choice([384, 768, 1024]), "depth": 12, "tokens": _spread(rng, 50, 4097), "batch": _spread(rng, 1, 16),
            "spec": rng.choice(["fh", "hh", "sdpa"]) + "-" + rng.choice(["g0", "g1"]), "graph": rng.random() < 0.3, "dtype": rng.choice(["fp16", "fp32"])}


def _draw_attention(rng):
    return {"kind": "attention", "tokens": _spread(rng, 64, 16385), "heads": rng.choice([6, 12, 16, 24]), "batch": _spread(rng, 1, 32),
            "variant": rng.choice(["fh", "hh", "ff"]), "packed": rng.random() < 0.7}


def _draw_linear(rng):
    c = rng.choice([384, 768, 1024, 1536])
    epilogue = rng.choice(["none", "gelu", "residual", "residual", "swiglu"])
    k, n = {"none": (c, 3 * c), "gelu": (c, 4 * c), "residual": rng.choice([(c, c), (4 * c, c)]), "swiglu": (c, 2 * swiglu_hidden(c))}[epilogue]
    return {"kind": "linear", "rows": _spread(rng, 17, 32768), "k": k, "n": n, "epilogue": epilogue, "bias": rng.random() < 0.8,
            "variant": rng.choice(["f32", "c2", "h"])}


def _draw_layernorm(rng):
    return {"kind": "layernorm", "rows": _spread(rng, 17, 65536), "dim": rng.choice([384, 768, 1024, 1280, 1536, 2048]),
            "dtype": rng.choice(["fp16", "fp32", "bf16"])}


def draw(rng):
    most = 0.7 * max(work(c)["flops"] for c in listed())
    make = rng.choice([_draw_vit] * 4 + [_draw_blocks] + [_draw_attention] * 2 + [_draw_linear] * 2 + [_draw_layernorm])
    while True:
        case = make(rng)
        if work(case)["flops"] <= most:
            return case


# ------------------------------------------------------------------------------------------------- weights and inputs
_DTYPE = {"fp16": torch.float16, "fp32": torch.float32, "bf16": torch.bfloat16}


def _gen(seed):
    return torch.Generator("cuda").manual_seed(seed)


def _normal(g, *shape, std=1.0, dtype=torch.float16):
    return torch.randn(*shape, device="cuda", generator=g, dtype=torch.float32).mul_(std).to(dtype)


def _fill(name, t, g):
    """A parameter as a freshly initialised ViT has it (trunc-normal, std 0.02), with biases, norms and LayerScale of a trained
    one's size, so that every term of the path takes part in the result."""
    if name.endswith("gamma"):
        return t.uniform_(0.05, 0.2, generator=g)
    if t.dim() == 1 and "norm" in name:
        return t.normal_(1.0 if name.endswith("weight") else 0.0, 0.1, generator=g)
    t.normal_(0.0, 0.02, generator=g)
    return t.clamp_(-0.04, 0.04)


def _prepare_vit(case, g):
    with torch.device("meta"):
        shapes = {k: v.shape for k, v in DinoV2Params(case["arch"], num_register_tokens=case["registers"]).state_dict().items()}
    weights = {k: _fill(k, torch.empty(s, device="cuda", dtype=torch.float32 if k == "pos_embed" else torch.float16), g) for k, s in shapes.items()}
    model = dinov2(case["arch"], weights, spec=case["spec"] + ("-graph" if case["graph"] else ""))
    x = _normal(g, case["batch"], 3, case["height"], case["width"], dtype=_DTYPE[case["image"]])
    taps = TAPS[case["arch"]]
    calls = {
        "features": lambda im: model.forward_features(im),
        "last": lambda im: model.get_intermediate_layers(im, n=1, return_class_token=True),
        "tokens": lambda im: model.get_intermediate_layers(im, n=taps, return_class_token=True),
        "maps": lambda im: model.get_intermediate_layers(im, n=taps, reshape=True, return_class_token=True),
    }
    fn = calls[case["call"]]
    if case["graph"]:  # a service captures its graph when it starts
        with torch.inference_mode(False), torch.no_grad():
            fn(torch.zeros_like(x))
    return {"fn": fn, "x": x}


class _Attention(nn.Module):
    def __init__(self, dim):
        super().__init__()
        self.num_heads, self.scale = dim // 64, 64 ** -0.5
        self.qkv, self.proj = nn.Linear(dim, 3 * dim), nn.Linear(dim, dim)


class _Mlp(nn.Module):
    def __init__(self, dim):
        super().__init__()
        self.fc1, self.act, self.fc2 = nn.Linear(dim, 4 * dim), nn.GELU(), nn.Linear(4 * dim, dim)


class _Block(nn.Module):
    """A transformer block with timm's attribute names; its forward is what install_vit_blocks() replaces."""

    def __init__(self, dim):
        super().__init__()
        self.norm1, self.norm2 = nn.LayerNorm(dim, eps=1e-6), nn.LayerNorm(dim, eps=1e-6)
        self.attn, self.mlp, self.ls1, self.ls2 = _Attention(dim), _Mlp(dim), nn.Identity(), nn.Identity()

    def forward(self, x):
        raise RuntimeError("the block was not patched")


def _prepare_blocks(case, g):
    with torch.device("meta"):
        stack = nn.Sequential(*[_Block(case["dim"]) for _ in range(case["depth"])])
    stack = stack.to_empty(device="cuda").requires_grad_(False).eval()
    for name, p in stack.named_parameters():
        _fill(name, p, g)
    if fastbb.install_vit_blocks(stack, case["spec"]) != case["depth"]:
        raise RuntimeError("some block was not patched")
    x = _normal(g, case["batch"], case["tokens"], case["dim"], dtype=_DTYPE[case["dtype"]])
    fn = graphed(stack) if case["graph"] else stack
    if case["graph"]:
        fn(torch.zeros_like(x))
    return {"fn": fn, "x": x}


def _prepare_attention(case, g):
    b, n, h = case["batch"], case["tokens"], case["heads"]
    if case["packed"]:
        q, k, v = _normal(g, b, n, 3, h, 64).unbind(2)
    else:
        q, k, v = (_normal(g, b, n, h, 64) for _ in range(3))
    return {"q": q, "k": k, "v": v, "variant": case["variant"]}


def _prepare_linear(case, g):
    m, n, k = case["rows"], case["n"], case["k"]
    residual = case["epilogue"] == "residual"
    return {"x": _normal(g, m, k), "w": _normal(g, n, k, std=0.02), "b": _normal(g, n, std=0.1) if case["bias"] else None,
            "act": None if residual or case["epilogue"] == "none" else case["epilogue"], "variant": case["variant"],
            "res": _normal(g, m, n) if residual else None, "gamma": _fill("gamma", torch.empty(n, device="cuda", dtype=torch.float16), g) if residual else None}


def _prepare_layernorm(case, g):
    c = case["dim"]
    return {"x": _normal(g, case["rows"], c, dtype=_DTYPE[case["dtype"]]), "w": (1 + _normal(g, c, std=0.1)), "b": _normal(g, c, std=0.1)}


def prepare(case, seed):
    make = {"vit": _prepare_vit, "blocks": _prepare_blocks, "attention": _prepare_attention, "linear": _prepare_linear, "layernorm": _prepare_layernorm}
    with torch.no_grad():
        return {"kind": case["kind"], **make[case["kind"]](case, _gen(seed))}


def run(state):
    kind = state["kind"]
    if kind in ("vit", "blocks"):
        with torch.no_grad():
            return state["fn"](state["x"])
    if kind == "attention":
        return attention(state["q"], state["k"], state["v"], variant=state["variant"])
    if kind == "linear":
        return linear(state["x"], state["w"], state["b"], act=state["act"], res=state["res"], gamma=state["gamma"], variant=state["variant"])
    return layer_norm(state["x"], state["w"], state["b"], 1e-6)


# ------------------------------------------------------------------------------------------------ work and tolerances
def _stack_work(c, depth, hidden, gated, batch, tokens):
    """(flops, weight bytes) of a run of transformer blocks."""
    per_token = 2 * c * (3 * c + c + (3 if gated else 2) * hidden)
    flops = depth * batch * (tokens * per_token + 4 * tokens * tokens * c)
    return flops, 2 * depth * c * (4 * c + (3 if gated else 2) * hidden)


def work(case):
    kind = case["kind"]
    if kind == "vit":
        c, depth, _, ffn = ARCH[case["arch"]]
        b, hw = case["batch"], (case["height"] // PATCH) * (case["width"] // PATCH)
        n = 1 + case["registers"] + hw
        flops, weights = _stack_work(c, depth, 4 * c if ffn == "mlp" else swiglu_hidden(c), ffn != "mlp", b, n)
        patch = 3 * PATCH * PATCH
        flops += 2 * b * hw * c * patch
        weights += 2 * c * (patch + n)
        image = b * 3 * case["height"] * case["width"] * (4 if case["image"] == "fp32" else 2)
        outputs = {"features": 2, "last": 1, "tokens": 4, "maps": 4}[case["call"]] * b * n * c * 2
        return {"flops": flops, "bytes": weights + image + outputs}
    if kind == "blocks":
        c, b, n = case["dim"], case["batch"], case["tokens"]
        flops, weights = _stack_work(c, case["depth"], 4 * c, False, b, n)
        return {"flops": flops, "bytes": weights + 2 * b * n * c * (4 if case["dtype"] == "fp32" else 2)}
    if kind == "attention":
        b, n, h = case["batch"], case["tokens"], case["heads"]
        return {"flops": 4 * b * h * n * n * 64, "bytes": 4 * b * n * h * 64 * 2}
    if kind == "linear":
        m, n, k = case["rows"], case["n"], case["k"]
        out = n // 2 if case["epilogue"] == "swiglu" else n
        return {"flops": 2 * m * n * k, "bytes": 2 * (m * k + n * k + m * out + (m * n if case["epilogue"] == "residual" else 0))}
    m, c = case["rows"], case["dim"]
    return {"flops": 8 * m * c, "bytes": m * c * (2 + (4 if case["dtype"] == "fp32" else 2)) + 4 * c}


def tolerance(case):
    kind = case["kind"]
    if kind in ("vit", "blocks"):
        # fp16 activations are rounded seven times per block (2^-12 relative each), differently by every order of summation: two
        # correct stacks drift apart like the square root of the depth, cls rows of random weights by some times more
        return {"rel": 1e-2}
    if kind == "attention":
        return {"rel": 2e-3}  # fp16 probabilities and outputs
    if kind == "linear":
        # fp16 outputs of an fp32 sum; an fp16 accumulator rounds each partial sum of K / 16 as well
        return {"rel": 1e-2 if case["variant"] == "h" else 1e-3}
    return {"rel": 1e-3}  # fp16 outputs of fp32 statistics
