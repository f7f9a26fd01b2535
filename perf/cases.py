"""The performance cases of the library: what a host engine asks of it, by model shape and token count.

A case is one call of a public entry point (`MoeLayer.forward` / `forward_dev`, `Stack.forward_dev`)
on a layer or a layer stack of one of the shapes in `pelica_b200.synth`:

  olmoe    one layer of C1 (Q4_K; softmax top-8 of 64). The smallest calls of all: one FFN operator of an
           engine that keeps the rest of the model to itself. `io` says where that engine's activations
           live: "device", or "host" (page-locked arrays in and out, the call returns when y is there).
  qwen3    a stack of C2 layers (Q4_K gate/up, Q6_K down; top-8 of 128, renormalised): token-by-token
           decode, decode of a few sequences together, prefill. Fewer layers: the share of a model that
           an engine keeps on this GPU.
  gptoss   a stack of C3 layers (MXFP4, f32 activations, biases, clamped GLU; top-4 of 32).
  dsv3     one layer of C4 (d 7168, 256 experts in 8 groups, sigmoid scores with a selection bias, a shared
           expert): 6.4 GB a layer, so a GPU holds a few layers or a shard.
  zipf     one layer of C5 with skewed routing: a few experts serve most tokens, some none.
  q4x      one layer of the second int8 path (32-value activation blocks; Q8_0, IQ4_NL or IQ4_XS weights,
           softmax over the selected logits; top-8 of 32).

Token counts go from 1 (decode) over a few (several sequences, speculative tokens) to prompts of thousands.
Weights, router, biases and activations are made from the seed: N(0, 0.02) weights quantised to the
shape's types, N(0, 1) activations, RMS-normalised where the engine normalises them before the call.
"""
import numpy as np
import torch

import pelica_b200 as pb
from pelica_b200 import synth

CONFIGS = {"olmoe": synth.C1_OLMOE, "qwen3": synth.C2_QWEN3, "gptoss": synth.C3_GPTOSS, "dsv3": synth.C4_DSV3,
           "zipf": synth.C5_ZIPF}
Q4X = {"q8_0": synth.C6_Q8_0, "iq4_nl": synth.C7_IQ4NL, "iq4_xs": synth.C8_IQ4XS}
STACKS = ("qwen3", "gptoss")
IQ4_LEVELS = [-127, -104, -83, -65, -49, -35, -22, -10, 1, 13, 25, 38, 53, 69, 89, 113]


def listed():
    return [
        # the smallest call: one token through one operator, activations on the GPU
        dict(name="olmoe_decode_1", family="olmoe", tokens=1, io="device"),
        # a short prompt from an engine whose activations are in host memory
        dict(name="olmoe_prefill_64_host", family="olmoe", tokens=64, io="host"),
        # a token through the whole model's experts
        dict(name="qwen3_decode_1", family="qwen3", layers=48, tokens=1),
        # eight sequences decoded together
        dict(name="qwen3_decode_8", family="qwen3", layers=48, tokens=8),
        # a prompt chunk through the whole model's experts
        dict(name="qwen3_prefill_512", family="qwen3", layers=48, tokens=512),
        dict(name="gptoss_decode_1", family="gptoss", layers=24, tokens=1),
        dict(name="gptoss_prefill_2048", family="gptoss", layers=24, tokens=2048),
        # experts much larger than the caches
        dict(name="dsv3_decode_1", family="dsv3", tokens=1),
        # a full decode batch: nearly every expert is read for about two tokens
        dict(name="dsv3_decode_64", family="dsv3", tokens=64),
        dict(name="dsv3_prefill_4096", family="dsv3", tokens=4096),
        # a ragged prompt, its tokens piled on a few experts
        dict(name="zipf_prefill_3001", family="zipf", tokens=3001),
        # a few dozen tokens on 4-bit codebook weights
        dict(name="q4x_iq4xs_33", family="q4x", weights="iq4_xs", tokens=33),
    ]


def _tokens(rng, most):
    """1 .. most, even over the logarithm."""
    return max(1, min(most, int(round(most ** rng.random()))))


def draw(rng):
    family = rng.choice(["olmoe", "qwen3", "gptoss", "dsv3", "zipf", "q4x"])
    case = dict(family=family)
    if family == "olmoe":
        case.update(tokens=_tokens(rng, 512), io=rng.choice(["device", "host"]))
    elif family == "qwen3":
        layers = rng.randint(4, 48)
        case.update(layers=layers, tokens=_tokens(rng, min(2048, 48 * 512 // layers)))
    elif family == "gptoss":
        case.update(layers=rng.randint(2, 24), tokens=_tokens(rng, 2048))
    elif family == "dsv3":
        case.update(tokens=_tokens(rng, 4096))
    elif family == "zipf":
        case.update(tokens=_tokens(rng, 8192))
    else:
        case.update(weights=rng.choice(sorted(Q4X)), tokens=_tokens(rng, 1024))
    return case


def _config(case):
    return Q4X[case["weights"]] if case["family"] == "q4x" else CONFIGS[case["family"]]


# --------------------------------------------------------------------------
# states
# --------------------------------------------------------------------------
_context = None


def _ctx():
    """The process's one context (a GPU, its stream and workspace), as an engine has it."""
    global _context
    if _context is None:
        _context = pb.Context(torch.cuda.current_device())
    return _context


class _Dev:
    """A torch tensor as a device buffer of the library's calls."""

    def __init__(self, t):
        self.t, self.ptr = t, t.data_ptr()


class State:
    """Layers, the stack over them where the case runs one, and the call's buffers."""

    def __init__(self, case):
        self.case = case
        self.layers, self.stack = [], None
        self.x = self.y = None

    def __del__(self):
        if self.stack is not None:
            self.stack.close()
        for layer in self.layers:
            layer.close()


def _quantise_32(ty, w):
    """[rows][cols] f32 on the GPU -> the type's block bytes (blocks of 32 values; 256 for IQ4_XS)."""
    b = w.reshape(-1, 32)
    if ty == synth.Q8_0:
        d = (b.abs().amax(-1) / 127.0).half()
        q = torch.round(b / d.float()[:, None]).clamp(-127, 127).to(torch.int8)
        return torch.cat([d.view(torch.uint8).reshape(-1, 2), q.view(torch.uint8)], 1).reshape(-1)
    levels = torch.tensor(IQ4_LEVELS, dtype=torch.float32, device=w.device)
    edges = (levels[1:] + levels[:-1]) / 2
    if ty == synth.IQ4_NL:
        big = b.gather(1, b.abs().argmax(-1, keepdim=True))[:, 0]
        d = (big / -127.0).half()
        idx = torch.bucketize(b / d.float()[:, None], edges).to(torch.uint8)
        return torch.cat([d.view(torch.uint8).reshape(-1, 2), idx[:, :16] | (idx[:, 16:] << 4)], 1).reshape(-1)
    assert ty == synth.IQ4_XS
    amax = b.abs().amax(-1).reshape(-1, 8)
    d = (amax.amax(-1) / 127.0 / 31.0).half()
    sub = torch.round(amax / 127.0 / d.float()[:, None]).clamp(1, 31)
    scale = (d.float()[:, None] * sub).reshape(-1, 1)
    idx = torch.bucketize(b / scale, edges).to(torch.uint8)
    ls = sub.to(torch.int32) + 32
    high = torch.zeros(ls.shape[0], dtype=torch.int32, device=w.device)
    low = torch.zeros(ls.shape[0], 4, dtype=torch.int32, device=w.device)
    for i in range(8):
        high |= ((ls[:, i] >> 4) & 3) << (2 * i)
        low[:, i // 2] |= (ls[:, i] & 15) << (4 * (i % 2))
    head = torch.cat([torch.stack([high & 255, high >> 8], 1), low], 1).to(torch.uint8)
    quants = (idx[:, :16] | (idx[:, 16:] << 4)).reshape(-1, 128)
    return torch.cat([d.view(torch.uint8).reshape(-1, 2), head, quants], 1).reshape(-1)


def _q4x_weights(cfg, gen):
    dev = gen.device
    shapes = dict(gate=(cfg.type_gate, cfg.ff, cfg.d), up=(cfg.type_up, cfg.ff, cfg.d), down=(cfg.type_down, cfg.d, cfg.ff))
    w = {"router": (torch.randn(cfg.n_exp, cfg.d, device=dev, generator=gen) * cfg.sigma).cpu().numpy()}
    for key, (ty, rows, cols) in shapes.items():
        m = torch.randn(cfg.n_exp * rows, cols, device=dev, generator=gen) * cfg.sigma
        w[key] = _quantise_32(ty, m).reshape(cfg.n_exp, -1).cpu().numpy()
    return w


def prepare(case, seed):
    cfg, family, tokens = _config(case), case["family"], case["tokens"]
    ctx = _ctx()
    gen = torch.Generator(device="cuda").manual_seed(1000003 * seed + 17)
    s = State(case)
    for i in range(case.get("layers", 1)):
        layer = pb.MoeLayer(ctx, cfg)
        s.layers.append(layer)
        if family == "q4x":
            layer.load(_q4x_weights(cfg, gen))
            continue
        layer.fill_synthetic(7919 * i + 104729 * seed + 1, cfg.sigma, cfg.sigma if cfg.logit_bias else 0.0,
                             cfg.select_bias_sigma)
        if family == "zipf":
            w = (torch.randn(cfg.n_exp, cfg.d, device="cuda", generator=gen) * cfg.sigma).cpu().numpy()
            bias = synth.zipf_router_bias(cfg.n_exp, seed, s=1.2, dead=8, strength=0.6)
            pb._check(layer.lib.pm_layer_set_router(layer.h, w.ctypes.data, synth.F32, bias.ctypes.data, None))
    x = torch.randn(tokens, cfg.d, device="cuda", generator=gen)
    if family in STACKS:
        s.stack = pb.Stack(ctx, s.layers)
    else:  # the engine has normalised what it hands to the operator
        x = x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-6)
    if case.get("io") == "host":
        s.x = torch.empty(x.shape, pin_memory=True).copy_(x).numpy()
        s.y = torch.zeros(x.shape, pin_memory=True).numpy()
    else:
        s.x, s.y = _Dev(x), _Dev(torch.zeros_like(x))
    return s


def run(s):
    tokens = s.case["tokens"]
    if s.case.get("io") == "host":
        return s.layers[0].forward(s.x, s.y)
    if s.stack is not None:
        s.stack.forward_dev(s.x, tokens, s.y)
    else:
        s.layers[0].forward_dev(s.x, tokens, s.y)
    return s.y.t


# --------------------------------------------------------------------------
# what a pass cannot do without
# --------------------------------------------------------------------------
def work(case):
    cfg, tokens, layers = _config(case), case["tokens"], case.get("layers", 1)
    # experts that `tokens` tokens touch: of live experts chosen evenly (a skewed router touches fewer)
    live = cfg.n_exp - 8 if case["family"] == "zipf" else cfg.n_exp
    if case["family"] == "zipf":
        p = np.arange(1, live + 1, dtype=np.float64) ** -1.2
        p = np.minimum(1.0, p * cfg.top_k / p.sum())
    else:
        p = np.full(live, cfg.top_k / live)
    touched = float((1.0 - (1.0 - p) ** tokens).sum())
    shared = cfg.scaled(ff=cfg.shared_ff, has_expert_bias=0).expert_bytes() if cfg.shared else 0
    per_layer = touched * cfg.expert_bytes() + shared + 4 * cfg.n_exp * cfg.d
    per_token = 2 * cfg.n_exp * cfg.d + 6 * cfg.d * (cfg.top_k * cfg.ff + (cfg.shared_ff if cfg.shared else 0))
    return {"bytes": layers * per_layer + 2 * 4 * tokens * cfg.d, "flops": float(layers * tokens * per_token)}


def tolerance(case):
    if case["family"] == "q4x":
        # 32-bit sums, then the hidden vector is quantised again: a sum that rounds otherwise moves a few
        # of its int8 values by one
        return {"rel": 1e-4, "max": 1e-2}
    if case["family"] == "gptoss":
        if case["tokens"] < 32:
            return {"rel": 1e-4}  # f32 sums of any order through up to 24 layers
        # Prompts run on the tensor cores with the activations as two bf16 parts (2^-17 a value). Through a
        # stack such a difference now and then turns a near tie of a token's fourth and fifth expert, and that
        # token goes on with another expert of the same weight: a few of 2048 tokens over 24 layers.
        return {"rel": 1e-2, "max": 0.9} if case["layers"] > 1 else {"rel": 1e-4}
    # int8 blocks: integer sums, and float terms in a fixed order; quantising again and routing take every bit
    # of them, so the results are defined to the bit
    return "exact"
