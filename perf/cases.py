"""The mixture-of-experts layer's timed cases: what a program that serves a model with this library has it do.

A model server keeps one ``MoeLayer`` per layer with its weights resident, and calls it once per step: with the few
tokens of a decode step, with a mixed batch of decode tokens and a prompt's next chunk, or with whole prompts.  The
layer is called on device buffers by itself (``forward_dev``), as the whole block with the norm before and the residual
after (``block_forward_dev``), with a shared expert beside the routed ones, on host buffers (``forward``, what the C++
node bindings call) and as the dense FFN (``dense_forward_dev``).

Every tensor of a case comes from one generator seeded with the case's seed.  Device-buffer calls of all states go to
one stream, as the layers of one model do.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from coalsack_b200 import MoeLayer

# gpt-oss-120b, gpt-oss-20b and Qwen3-30B-A3B shaped layers (MXFP4 experts), and a Llama-4 style layer: experts held as
# fp16 matrices (the form Q4_K / Q6_K slices are decoded to), one per token, sigmoid gate applied before the expert,
# a shared dense expert beside them.
GPTOSS_120B = dict(experts=128, top_k=4, hidden=2880, ffn=2880, bias=True, swiglu="modified", router_bias="normal")
GPTOSS_20B = dict(experts=32, top_k=4, hidden=2880, ffn=2880, bias=True, swiglu="modified", router_bias="normal")
QWEN3_30B = dict(experts=128, top_k=8, hidden=2048, ffn=768, bias=False, swiglu="standard", router_bias="none")
SHARED_16 = dict(experts=16, top_k=1, hidden=2048, ffn=2048, bias=False, swiglu="standard", router_bias="none")
DENSE_2880 = dict(experts=1, top_k=1, hidden=2880, ffn=2880, bias=True, swiglu="standard", router_bias="none")


def _case(entry, shape, tokens, **more):
    return dict(entry=entry, tokens=tokens, **{**shape, **more})


def listed():
    return [
        # one user's next token through a 128-expert layer: four experts' weights, and the latency of every launch
        dict(name="decode_1", **_case("layer", GPTOSS_120B, 1)),
        # a small decode batch through the whole block: norm, layer, residual
        dict(name="block_decode_8", **_case("block", GPTOSS_120B, 8)),
        # a full decode batch: most experts are hit, by two rows each
        dict(name="decode_64", **_case("layer", GPTOSS_120B, 64)),
        # decode tokens and a piece of a prompt in one batch, through the whole block
        dict(name="block_mixed_333", **_case("block", GPTOSS_120B, 333)),
        # whole prompts: the benchmark's default workload
        dict(name="prefill_8192", **_case("layer", GPTOSS_120B, 8192)),
        # whole prompts through 32 experts with a Zipf-like load: the first experts get many times the last ones' rows
        dict(name="prefill_4096_zipf", **_case("layer", GPTOSS_20B, 4096, router_bias="zipf")),
        # a decode batch through fine-grained experts: eight of 128 small ones per token, no biases
        dict(name="fine_decode_16", **_case("layer", QWEN3_30B, 16)),
        # whole prompts through fine-grained experts
        dict(name="fine_prefill_2048", **_case("layer", QWEN3_30B, 2048)),
        # a decode batch through the host-buffer call of the node bindings, whose tensors are ordinary (pageable) memory
        dict(name="host_decode_32", **_case("host", GPTOSS_20B, 32, pinned=False)),
        # whole prompts in page-locked host buffers, results back in host memory
        dict(name="host_prefill_8192", **_case("host", GPTOSS_120B, 8192, pinned=True)),
        # the shared expert's dense FFN over whole prompts, fp16 weights
        dict(name="dense_8192", **_case("dense", DENSE_2880, 8192)),
        # a small decode batch through the block with a shared expert; fp16 experts, gate weight applied before them
        dict(name="shared_decode_5", **_case("shared", SHARED_16, 5)),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """Another call of the same kinds: any batch from 1 to 8192 tokens (log-uniform, so odd sizes at every scale),
    through one of the layers above or one of other sizes (hidden and ffn any multiple of 32)."""
    entry = rng.choice(["layer", "layer", "layer", "block", "host", "dense", "shared"])
    tokens = _log_int(rng, 1, 8192)
    if entry in ("dense", "shared"):
        shape = dict(DENSE_2880 if entry == "dense" else SHARED_16)
        if rng.random() < 0.5:
            shape.update(hidden=32 * rng.randint(16, 90), ffn=32 * rng.randint(16, 90), bias=rng.random() < 0.5)
        return _case(entry, shape, tokens)
    pick = rng.randrange(4)
    if pick < 3:
        shape = dict((GPTOSS_120B, GPTOSS_20B, QWEN3_30B)[pick])
        if shape["router_bias"] == "normal" and rng.random() < 0.3:
            shape["router_bias"] = "zipf"
    else:
        shape = dict(experts=rng.choice([8, 16, 32, 64, 128]), top_k=rng.choice([1, 2, 4, 8]),
                     hidden=32 * rng.randint(16, 90), ffn=32 * rng.randint(16, 90), bias=rng.random() < 0.5,
                     swiglu=rng.choice(["modified", "standard"]), router_bias=rng.choice(["normal", "zipf", "none"]))
        shape["top_k"] = min(shape["top_k"], shape["experts"] // 2)
        tokens = min(tokens, 32768 // shape["top_k"])
    return _case(entry, shape, tokens, **({"pinned": rng.random() < 0.5} if entry == "host" else {}))


# ---- inputs ---------------------------------------------------------------------------------------------------------
_stream = None


def _model_stream():
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream


def _normal(g, *shape, scale=1.0):
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float32).mul_(scale)


def _host(t):
    """A CUDA tensor's copy in host memory, as numpy (through torch's pool of page-locked blocks, which makes it quick)."""
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h.numpy()


def _mxfp4(g, count, rows, cols):
    """[count, rows*cols/32*17] MXFP4 blocks: codes uniform, scale exponents uniform in [118, 124]."""
    b = torch.randint(0, 256, (count, rows * cols // 32, 17), generator=g, device="cuda", dtype=torch.uint8)
    b[:, :, 0] = torch.randint(118, 125, b.shape[:2], generator=g, device="cuda", dtype=torch.uint8)
    return _host(b.view(count, -1))


def _biases(g, c, count):
    if not c["bias"]:
        return None, None, None
    return tuple(_host(_normal(g, count, n, scale=0.01)) for n in (c["ffn"], c["ffn"], c["hidden"]))


def _load_mxfp4(g, lay, c):
    E, H, F = c["experts"], c["hidden"], c["ffn"]
    for e in range(0, E, 16):  # sixteen experts' tensors at a time
        n = min(16, E - e)
        lay.load_experts_bulk(e, _mxfp4(g, n, F, H), _mxfp4(g, n, F, H), _mxfp4(g, n, H, F), *_biases(g, c, n))


def _load_f16(g, lay, c, count):
    H, F = c["hidden"], c["ffn"]
    for e in range(count):
        w = [_host(_normal(g, r, k, scale=k ** -0.5).half()) for r, k in ((F, H), (F, H), (H, F))]
        lay.load_expert_f16(e, *w, *(None if b is None else b[0] for b in _biases(g, c, 1)))


def _set_router(g, lay, c):
    E, H = c["experts"], c["hidden"]
    bias = {"none": lambda: None,
            "normal": lambda: _host(_normal(g, E, scale=0.01)),
            "zipf": lambda: (0.5 * np.log(1.0 / (np.arange(E) + 1.0))).astype(np.float32)}[c["router_bias"]]()
    lay.set_router(_host(_normal(g, E, H, scale=0.02)), bias)


def prepare(case, seed):
    c, T, H = case, case["tokens"], case["hidden"]
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    act = 0 if c["swiglu"] == "modified" else 1
    entry = c["entry"]
    f16 = entry in ("dense", "shared")
    lay = MoeLayer(c["experts"], c["top_k"], H, c["ffn"], activation=act, has_bias=c["bias"], max_tokens=T,
                   weights_f16=f16, sigmoid_gating=entry == "shared", weight_before_ffn=entry == "shared")
    if f16:
        _load_f16(g, lay, c, c["experts"])
    else:
        _load_mxfp4(g, lay, c)
    if entry != "dense":
        _set_router(g, lay, c)
    s = dict(entry=entry, layer=lay, T=T, shared=None, stream=_model_stream().cuda_stream)
    if entry in ("block", "shared"):
        lay.set_ffn_norm(_host(1.0 + _normal(g, H, scale=0.1)))
    if entry == "shared":
        s["shared"] = MoeLayer(1, 1, H, c["ffn"], activation=1, has_bias=c["bias"], max_tokens=T, weights_f16=True)
        _load_f16(g, s["shared"], c, 1)
    hidden = _normal(g, T, H)
    if entry != "host":
        s["hidden"] = hidden
        s["out"] = torch.empty(T, H, device="cuda")
        s["router"] = torch.empty(T, c["top_k"], 2, device="cuda")
    elif c["pinned"]:
        s["hidden"] = torch.empty(T, H, pin_memory=True).copy_(hidden)
        s["out"] = torch.empty(T, H, pin_memory=True)
        s["router"] = torch.empty(T, c["top_k"], 2, pin_memory=True)
    else:
        s["hidden"] = hidden.cpu().numpy()
        s["out"] = np.empty((T, H), np.float32)
        s["router"] = np.empty((T, c["top_k"], 2), np.float32)
    torch.cuda.synchronize()
    return s


# ---- one pass -------------------------------------------------------------------------------------------------------
def run(s):
    lay, entry = s["layer"], s["entry"]
    if entry == "layer":
        lay.forward_dev(s["hidden"], s["T"], s["out"], d_router_out=s["router"], stream=s["stream"])
    elif entry in ("block", "shared"):
        lay.block_forward_dev(s["hidden"], s["T"], s["router"], s["out"], stream=s["stream"], shared=s["shared"])
    elif entry == "dense":
        lay.dense_forward_dev(s["hidden"], s["T"], s["out"], stream=s["stream"])
        return s["out"]
    else:
        lay.forward(s["hidden"], out=s["out"], router_out_buf=s["router"])
    return s["out"], s["router"]


def work(case):
    """Bytes: the weights of the experts that T tokens hit when they choose evenly, each once, the gate matrix, and the
    activations in and out.  Flops: three matrices per (token, expert) pair, and the gate."""
    T, E, k, H, F = (case[n] for n in ("tokens", "experts", "top_k", "hidden", "ffn"))
    f16 = case["entry"] in ("dense", "shared")
    per_expert = 3 * H * F * (2 if f16 else 17 / 32) + (4 * (2 * F + H) if case["bias"] else 0)
    hit = E * (1.0 - (1.0 - k / E) ** T)
    pairs = T * k
    if case["entry"] == "shared":
        hit, pairs = hit + 1, pairs + T
    moved = hit * per_expert + 2 * 4 * T * H
    flops = 6 * pairs * H * F
    if case["entry"] != "dense":
        moved += 4 * E * H + 8 * T * k
        flops += 2 * T * E * H
    return {"bytes": moved, "flops": flops}


def tolerance(case):
    """The contractions take fp16 activations (rounded before each of the two) and add in fp32: two implementations
    differ by a rounding of 2^-11 per operand where they round at different points.  The bound on the largest
    difference is the one the tests hold the library to."""
    return {"rel": 1e-3, "max": 2e-2}
