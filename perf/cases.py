"""The work that a program has this package do, as cases that can be timed and checked.

A program that serves a model builds it once (``CausalLM`` from a configuration), keeps its weights, a paged cache and the
state slots of its requests on the device, and then runs steps: prompt portions, decoded tokens, or both in one batch.  A
case is one such step of a whole model, of one layer, or of one sublayer, at sizes of this package's benchmarks:

* ``model``: a decode step of a whole Llama model, from token ids to logits;
* ``layer``: one Llama layer (norm, attention over the paged cache, norm, feed-forward) for a prompt portion, for decoded
  tokens, or for a mixed batch, in bfloat16 or in true 32-bit;
* ``mixer``: a recurrent mixer of another decoder (gated linear attention, delta rule, matrix memory, state space,
  forget-and-write), whose state lives in the requests' slots;
* ``experts``: a routed feed-forward.

Steps of single tokens run as a captured CUDA graph, which is how the engine runs them; everything else is launched as the
engine launches it.  ``exact`` restates every case in plain torch operations in 64 bits.
"""
from __future__ import annotations

import json
import math
import random

import torch

from photon_infer_b200.config.registry import architecture_name, get_architecture
from photon_infer_b200.csrc.build import ensure_built
from photon_infer_b200.kernels import ops
from photon_infer_b200.models.model import CausalLM
from photon_infer_b200.parts.base import GroupView, LayerCache, StepContext
from photon_infer_b200.weights.random_init import random_tensors_on_device

PAGE = 16
DTYPES = {"bf16": torch.bfloat16, "f32": torch.float32}

#: Layer shapes of the Llama models that the benchmarks run: hidden, query heads, key/value heads, head size, feed-forward, the
#: factor of the frequency scaling, layers.
SHAPES = {"llama-3.2-1b": (2048, 32, 8, 64, 8192, 32.0, 16),
          "llama-3.2-3b": (3072, 24, 8, 128, 8192, 32.0, 28),
          "llama-3.1-8b": (4096, 32, 8, 128, 14336, 8.0, 32)}
VOCAB = 128256

MIXERS = ("gla", "delta", "mlstm", "mamba2", "hgrn2")


# ----------------------------------------------------------------------------- the cases

def listed():
    return [
        # eight users of a small model, each waiting for the next token: the engine's headline workload
        {"name": "model_decode_8", "kind": "model", "shape": "llama-3.2-1b", "layers": 16, "requests": 8, "new": 1,
         "context": 640, "ragged": True, "dtype": "bf16"},
        # a layer of a decode step under continuous batching: an odd number of requests of very different lengths
        {"name": "layer_decode_56", "kind": "layer", "shape": "llama-3.2-3b", "requests": 56, "new": 1, "context": 2304,
         "ragged": True, "dtype": "bf16"},
        # a layer over one whole prompt
        {"name": "layer_prompt_2048", "kind": "layer", "shape": "llama-3.2-1b", "requests": 1, "new": 2048, "context": 0,
         "ragged": False, "dtype": "bf16"},
        # a layer over the eighth portion of a long prompt: attention over what the cache holds dominates
        {"name": "layer_prompt_long", "kind": "layer", "shape": "llama-3.1-8b", "requests": 1, "new": 2048, "context": 14336,
         "ragged": False, "dtype": "bf16"},
        # a layer of a mixed step: one request's prompt portion (an odd number of tokens) beside others' decoded tokens
        {"name": "layer_mixed", "kind": "layer", "shape": "llama-3.2-3b", "requests": 41, "new": 1, "context": 1500,
         "ragged": True, "portion": 1093, "dtype": "bf16"},
        # the true 32-bit run: two prompts of odd lengths in one step
        {"name": "layer_prompt_f32", "kind": "layer", "shape": "llama-3.2-1b", "requests": 2, "new": 431, "context": 0,
         "ragged": True, "dtype": "f32"},
        # recurrent mixers over prompts: two whole prompts of one request, two prompts of different lengths in one step, and a
        # short odd portion of a request whose state is not empty
        {"name": "gla_prompt_2048", "kind": "mixer", "mixer": "gla", "width": 2048, "requests": 1, "new": 2048, "context": 0,
         "ragged": False, "dtype": "bf16"},
        {"name": "delta_prompt_2048", "kind": "mixer", "mixer": "delta", "width": 2048, "requests": 1, "new": 2048, "context": 0,
         "ragged": False, "dtype": "bf16"},
        {"name": "mlstm_prompts", "kind": "mixer", "mixer": "mlstm", "width": 2048, "requests": 2, "new": 1531, "context": 0,
         "ragged": True, "dtype": "bf16"},
        {"name": "hgrn2_portion", "kind": "mixer", "mixer": "hgrn2", "width": 2048, "requests": 1, "new": 777, "context": 512,
         "ragged": False, "dtype": "bf16"},
        # routed experts: a prompt portion, and a decode step in which every token reads two experts
        {"name": "experts_prompt_2048", "kind": "experts", "width": 2048, "requests": 1, "new": 2048, "context": 0,
         "ragged": False, "dtype": "bf16"},
        {"name": "experts_decode_8", "kind": "experts", "width": 2048, "requests": 8, "new": 1, "context": 0, "ragged": False,
         "dtype": "bf16"},
    ]


def _spread(rng, low, high):
    """A whole number between the two, spread over the logarithm."""
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    what = rng.choice(("model", "layer_decode", "layer_prompt", "layer_mixed", "layer_f32", "mixer_prompt", "mixer_prompt",
                       "mixer_decode", "experts_prompt", "experts_decode"))
    if what == "model":
        return {"kind": "model", "shape": "llama-3.2-1b", "layers": 16, "requests": _spread(rng, 1, 64), "new": 1,
                "context": _spread(rng, 32, 1024), "ragged": rng.random() < 0.5, "dtype": "bf16"}
    if what == "layer_decode":
        return {"kind": "layer", "shape": rng.choice(sorted(SHAPES)), "requests": _spread(rng, 1, 96), "new": 1,
                "context": _spread(rng, 64, 4096), "ragged": rng.random() < 0.7, "dtype": "bf16"}
    if what == "layer_prompt":
        return {"kind": "layer", "shape": rng.choice(sorted(SHAPES)), "requests": rng.choice((1, 1, 2, 3)),
                "new": _spread(rng, 64, 680), "context": rng.choice((0, 0, rng.randrange(1, 4096))), "ragged": True, "dtype": "bf16"}
    if what == "layer_mixed":
        return {"kind": "layer", "shape": rng.choice(sorted(SHAPES)), "requests": _spread(rng, 2, 64), "new": 1,
                "context": _spread(rng, 64, 2048), "ragged": True, "portion": _spread(rng, 40, 2000), "dtype": "bf16"}
    if what == "layer_f32":
        return {"kind": "layer", "shape": "llama-3.2-1b", "requests": rng.choice((1, 2)), "new": _spread(rng, 1, 256),
                "context": rng.choice((0, rng.randrange(1, 512))), "ragged": rng.random() < 0.5, "dtype": "f32"}
    if what == "mixer_prompt":
        return {"kind": "mixer", "mixer": rng.choice(MIXERS), "width": rng.choice((2048, 2048, 4096)),
                "requests": rng.choice((1, 1, 2, 3)), "new": _spread(rng, 64, 2048), "context": rng.choice((0, 512)), "ragged": True,
                "dtype": "bf16"}
    if what == "mixer_decode":
        return {"kind": "mixer", "mixer": rng.choice(MIXERS), "width": rng.choice((2048, 4096)), "requests": _spread(rng, 1, 48),
                "new": 1, "context": 512, "ragged": False, "dtype": "bf16"}
    if what == "experts_prompt":
        return {"kind": "experts", "width": rng.choice((2048, 2048, 4096)), "requests": 1, "new": _spread(rng, 130, 3000),
                "context": 0, "ragged": False, "dtype": "bf16"}
    return {"kind": "experts", "width": rng.choice((2048, 4096)), "requests": _spread(rng, 1, 64), "new": 1, "context": 0,
            "ragged": False, "dtype": "bf16"}


def _lengths(case):
    """(tokens of each request in the step, tokens of each request in the cache before it): from the case alone."""
    rng = random.Random(json.dumps({k: v for k, v in case.items() if k != "name"}, sort_keys=True))
    n, new, context = case["requests"], case["new"], case["context"]
    some = lambda most: rng.randint(max(1, most // 16), most) if case["ragged"] and most > 1 else most
    news, held = [some(new) for _ in range(n)], [some(context) if context else 0 for _ in range(n)]
    if case.get("portion"):
        news[0] = case["portion"]
    if case["ragged"] and n > 1 and not case.get("portion"):
        news[-1], held[-1] = new, context               # the longest is as long as the case says
    return news, held


def _captured(case):
    return case["new"] == 1 and not case.get("portion")


# ----------------------------------------------------------------------------- configurations and weights

def _config(case):
    if case["kind"] in ("model", "layer"):
        hidden, heads, kv, d, ff, factor, _ = SHAPES[case["shape"]]
        return dict(architectures=["LlamaForCausalLM"], hidden_size=hidden, intermediate_size=ff,
                    num_hidden_layers=case.get("layers", 1), num_attention_heads=heads, num_key_value_heads=kv, head_dim=d,
                    vocab_size=VOCAB if case["kind"] == "model" else 256, max_position_embeddings=131072, rms_norm_eps=1e-5,
                    rope_theta=500000.0, tie_word_embeddings=True,
                    rope_scaling=dict(rope_type="llama3", factor=factor, low_freq_factor=1.0, high_freq_factor=4.0,
                                      original_max_position_embeddings=8192))
    w = case["width"]
    heads = w // 128
    if case["kind"] == "experts":
        mixer = dict(type="gla", mixer=dict(heads=heads, dim=128, vdim=128, tau=16.0),
                     mlp=dict(kind="moe", router=dict(experts=16, top=2), expert=dict(ff=w), shared=dict(ff=2 * w)))
        return dict(architecture="Finelix", vocab=256, width=w, embedding=dict(scale=1.0), norm=dict(eps=1e-5), layers=[mixer], loop=None)
    kind = case["mixer"]
    if kind == "gla":
        layer = dict(type="gla", mixer=dict(heads=heads, dim=128, vdim=128, tau=16.0), mlp=None)
        return dict(architecture="Finelix", vocab=256, width=w, embedding=dict(scale=1.0), norm=dict(eps=1e-5), layers=[layer], loop=None)
    if kind == "delta":
        layer = dict(type="delta", mixer=dict(heads=heads, kv_heads=heads // 2, dim=128, vdim=128, conv=4), mlp=None)
        return dict(architecture="Lerosun", vocab=256, width=w, norm=dict(eps=1e-5), layers=[layer], loop=None)
    if kind == "mlstm":
        layer = dict(type="mlstm", mixer=dict(heads=heads, dim=128, vdim=128, gate_cap=15.0), mlp=None)
        return dict(architecture="Pebodra", vocab=256, width=w, norm=dict(eps=1e-5, groups=8), logit_softcap=50.0, layers=[layer])
    if kind == "mamba2":
        g = max(1, heads // 8)
        layer = dict(type="mamba2", mixer=dict(heads=heads, vdim=128, state=128, groups=g, conv=4, norm_groups=g), mlp=None)
        return dict(architecture="Pebodra", vocab=256, width=w, norm=dict(eps=1e-5, groups=8), logit_softcap=50.0, layers=[layer])
    layer = dict(type="hgrn2", mixer=dict(heads=heads, dim=128, vdim=128), mlp=None)
    return dict(architecture="Fezavik", vocab=256, width=w, norm=dict(eps=1e-5), layers=[layer])


def _generator(seed, what):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1000003 + sum(ord(c) * (i + 7) for i, c in enumerate(what))) & 0x7FFFFFFF)
    return g


def _weights(case, seed, declared):
    """Random weights at the scale of the random-weights mode, with the gates of the recurrent mixers where trained ones lie."""
    t = random_tensors_on_device(declared, DTYPES[case["dtype"]], "cuda", seed=seed, init_std=0.02, norm_std=0.1)
    g = _generator(seed, "gates")
    uniform = lambda name, low, high: torch.rand(t[name].shape, generator=g, device="cuda") * (high - low) + low
    for name in list(t):
        if name.endswith(".A_log"):
            t[name] = uniform(name, 1.0, 16.0).log()
        elif name.endswith(".dt_bias"):                 # softplus(dt_bias) between 0.001 and 0.1
            t[name] = torch.expm1(torch.exp(uniform(name, math.log(1e-3), math.log(0.1)))).log()
        elif name.endswith(".conv") or name.endswith("_conv"):
            t[name] = uniform(name, -0.5, 0.5)
        elif name.endswith(".f.b") and case.get("mixer") == "mlstm":
            t[name] = uniform(name, 3.0, 6.0)
    return t


class State:
    """What a program holds before the step."""


def _model(case, seed):
    arch = get_architecture(architecture_name(_config(case)))
    spec = arch.build_spec(arch.config_class.from_dict(_config(case)))
    model = CausalLM(spec, DTYPES[case["dtype"]], "cuda:0")
    return model, _weights(case, seed, model.declared())


def _inputs(case, seed):
    """Everything that is drawn from the seed beside the weights: tokens or rows, what the cache and the state slots hold."""
    news, held = _lengths(case)
    T, dtype = sum(news), DTYPES[case["dtype"]]
    hidden = SHAPES[case["shape"]][0] if "shape" in case else case["width"]
    g = _generator(seed, "inputs")
    normal = lambda *shape: torch.randn(shape, generator=g, device="cuda")
    d = {"ids": torch.randint(0, VOCAB, (T,), generator=g, device="cuda", dtype=torch.int32)}
    if case["kind"] == "layer":
        d["x"], d["delta"] = normal(T, hidden), (0.5 * normal(T, hidden)).to(dtype)
    elif case["kind"] != "model":
        d["h"] = normal(T, hidden).to(dtype)
    if "shape" in case:
        _, _, kv, hd, _, _, _ = SHAPES[case["shape"]]
        pages = sum(-(-(a + b) // PAGE) for a, b in zip(news, held)) + 1
        L = case.get("layers", 1)
        kvs = torch.empty((L, 2, pages, kv, PAGE, hd), dtype=dtype, device="cuda")
        kvs.normal_(0.0, 0.9, generator=g)              # what these projections give normed rows
        d["kv"] = kvs
        order = torch.randperm(pages - 1, generator=g, device="cuda").cpu().tolist()
        d["tables"], at = [], 0
        for a, b in zip(news, held):
            n = -(-(a + b) // PAGE)
            d["tables"].append(order[at:at + n])
            at += n
    if case["kind"] == "mixer":
        d["state"] = _start_state(case, g)
    return d


def _start_state(case, g):
    """The state slots: zero for a new request; after some context the size that a running state has."""
    n, w = case["requests"], case["width"]
    H = w // 128
    normal = lambda *shape: torch.randn(shape, generator=g, device="cuda")
    kind = case["mixer"]
    rows = {"gla": 0, "delta": 3 * (2 * (H // 2) * 128 + H * 128), "mlstm": 0, "mamba2": 3 * (H * 128 + 2 * max(1, H // 8) * 128), "hgrn2": 0}[kind]
    parts = [0.3 * normal(n, H * 128 * 128)]
    if kind == "mlstm":
        parts += [0.3 * normal(n, H * 128), torch.rand((n, H), generator=g, device="cuda")]
    if rows:
        parts.append(normal(n, rows))
    s = torch.cat(parts, dim=1)
    if not case["context"]:
        s.zero_()
    return s.view(n, H, 128, 128) if kind == "gla" else s


def _context(case, d, flag):
    news, held = _lengths(case)
    S, T = len(news), sum(news)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32).to("cuda")
    pos = [b + i for a, b in zip(news, held) for i in range(a)]
    seq = [s for s, a in enumerate(news) for _ in range(a)]
    cu = [sum(news[:s]) for s in range(S + 1)]
    groups, bound = [], max(a + b for a, b in zip(news, held))
    if "tables" in d:
        width = max(len(t) for t in d["tables"])
        if _captured(case):                             # a graph serves until a request outgrows its table
            b = 8
            while b < width:
                b *= 2
            width, bound = b, b * PAGE
        table = [t + [-1] * (width - len(t)) for t in d["tables"]]
        slots = [d["tables"][s][p // PAGE] * PAGE + p % PAGE for s, p in zip(seq, pos)]
        groups = [GroupView(block_table=i32(table), slot_mapping=i32(slots), page_size=PAGE, num_pages=d["kv"].shape[2],
                            max_pages_per_seq=width)]
    return StepContext(num_tokens=T, num_seqs=S, dtype=DTYPES[case["dtype"]], token_ids=d["ids"], positions=i32(pos), token_seq=i32(seq),
                       cu_tokens=i32(cu), context_lens=i32([a + b for a, b in zip(news, held)]), state_slots=i32(list(range(S))),
                       groups=groups, host_query_lens=news, host_context_lens=[a + b for a, b in zip(news, held)],
                       host_start_positions=held, max_query_len=max(news), max_context_len=bound, error_flag=flag,
                       host_state_slots=list(range(S)))


def prepare(case, seed):
    s = State()
    s.case = case
    s.model, tensors = _model(case, seed)
    ensure_built(s.model.kernel_modules())
    s.model.load(tensors)
    del tensors
    d = _inputs(case, seed)
    s.flag = torch.zeros(4, dtype=torch.int32, device="cuda")
    ops.set_error_word(s.flag)
    s.ctx = _context(case, d, s.flag)
    s.kv, s.x, s.delta, s.h = d.get("kv"), d.get("x"), d.get("delta"), d.get("h")
    s.start, s.state = d.get("state"), None
    if s.start is not None:
        s.state = s.start.clone()
    s.caches = []
    for i in range(case.get("layers", 1)):
        c = LayerCache(state=s.state)
        if s.kv is not None:
            c = LayerCache(group=0, k=s.kv[i, 0], v=s.kv[i, 1])
        s.caches.append(c)
    s.rows = torch.arange(s.ctx.num_tokens, dtype=torch.int32, device="cuda")
    s.graph = None
    if _captured(case):
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            _step(s)                                    # once outside the capture, as the engine does
        torch.cuda.current_stream().wait_stream(side)
        torch.cuda.synchronize()
        s.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(s.graph):
            s.out = _step(s)
        if s.state is not None:
            s.state.copy_(s.start)                      # the step above moved the state on
    return s


def _step(s):
    kind = s.case["kind"]
    if kind == "model":
        return [s.model.forward(s.ctx, s.caches, s.rows), s.kv]
    block = s.model.blocks[0]
    if kind == "layer":
        residual, delta = block.forward(s.x.clone(), s.delta, s.ctx, s.caches[0])
        return [residual, delta, s.kv]
    if kind == "mixer":
        return [block.mixer().forward(s.h, s.ctx, s.caches[0]), s.state]
    return [block.parts()["feed_forward"].forward(s.h, s.ctx)]


def run(s):
    if s.graph is not None:
        s.graph.replay()                                # decoded tokens: the state moves on with every step
        return s.out
    if s.state is not None:
        s.state.copy_(s.start)                          # a slot is handed over with what its request left there
    return _step(s)


# ----------------------------------------------------------------------------- what a pass cannot do without

def work(case):
    news, held = _lengths(case)
    T, S = sum(news), len(news)
    e = 2 if case["dtype"] == "bf16" else 4
    if "shape" in case:
        H, nq, nkv, d, ff, _, _ = SHAPES[case["shape"]]
        L = case.get("layers", 1)
        w = (nq + 2 * nkv) * d * H + H * nq * d + 3 * H * ff
        pairs = sum(a * b + a * (a + 1) // 2 for a, b in zip(news, held))
        kv = sum(2 * nkv * d * e * (a + b) for a, b in zip(news, held)) + T * 2 * nkv * d * e
        flops = L * (2 * T * w + 4 * nq * d * pairs)
        moved = L * (w * e + kv)
        if case["kind"] == "model":
            return {"bytes": moved + VOCAB * H * e + 4 * T * VOCAB, "flops": flops + 2 * T * H * VOCAB}
        return {"bytes": moved + T * H * (4 + 4 + 2 * e), "flops": flops}
    W = case["width"]
    heads = W // 128
    io = 2 * T * W * e
    if case["kind"] == "experts":
        expert, shared, router = 3 * W * W, 6 * W * W, 16 * W
        used = 16 * (1.0 - (1.0 - 1.0 / 16) ** (2 * T))             # experts that the step's pairs meet, if the choice is even
        return {"bytes": (used * expert + shared + router) * e + io, "flops": 2.0 * T * (2 * expert + shared + router)}
    inner = {"gla": 4 * W * W + 16 * W + 16 * W, "delta": 3 * W * W + 2 * heads * W, "mlstm": 4 * W * W + 2 * heads * W,
             "mamba2": 2 * W * W + 2 * max(1, heads // 8) * 128 * W + heads * W, "hgrn2": 3 * W * W}[case["mixer"]] + W * W
    per = {"gla": 5, "delta": 7, "mlstm": 5, "mamba2": 5, "hgrn2": 5}[case["mixer"]]
    state = S * heads * 128 * 128 * 4
    return {"bytes": inner * e + 2 * state + io, "flops": 2.0 * T * inner + per * T * heads * 128 * 128}


def tolerance(case):
    # bfloat16: about four times the error against 64 bits, which is that of rounding the operands of each product once
    # (a layer's residual rows, its pending output, and the cache's new rows); a whole model adds up sixteen layers of it
    if case["dtype"] == "f32":
        return {"rel": 1e-5, "max": 1e-3}
    if case["kind"] == "model":
        return {"rel": 0.03, "max": 0.5}
    return {"rel": 0.02, "max": 0.5}


# ----------------------------------------------------------------------------- the same in 64 bits

def _f(t):
    return t.to(torch.float64)


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _frequencies(d, theta, factor):
    out = []
    for j in range(d // 2):
        f = theta ** (-2.0 * j / d)
        lam = 2.0 * math.pi / f
        if lam > 8192 / 1.0:
            f = f / factor
        elif lam >= 8192 / 4.0:
            s = (8192 / lam - 1.0) / 3.0
            f = (1.0 - s) * f / factor + s * f
        out.append(f)
    return torch.tensor(out, dtype=torch.float64, device="cuda")


def _exact_layer(case, t, prefix, x, kv, news, held, tables):
    """One Llama layer on the stream ``x``; ``kv [2, pages, heads, slots, d]`` gets the new rows.  Returns the stream after
    attention and the feed-forward's output."""
    H, nq, nkv, d, _, factor, _ = SHAPES[case["shape"]]
    w = lambda name: _f(t[prefix + name])
    h = _rms(x, 1e-5) * w("input_layernorm.weight")
    # partners of the rotation lie side by side in the cache
    order = torch.stack([torch.arange(d // 2), torch.arange(d // 2) + d // 2], 1).reshape(-1).cuda()
    T = x.shape[0]
    q = (h @ w("self_attn.q_proj.weight").t()).view(T, nq, d)[:, :, order]
    k = (h @ w("self_attn.k_proj.weight").t()).view(T, nkv, d)[:, :, order]
    v = (h @ w("self_attn.v_proj.weight").t()).view(T, nkv, d)
    pos = torch.cat([torch.arange(b, a + b, device="cuda") for a, b in zip(news, held)])
    angle = pos.double()[:, None] * _frequencies(d, 500000.0, factor)
    c, s = angle.cos()[:, None], angle.sin()[:, None]
    turn = lambda z: torch.stack([z[..., 0::2] * c - z[..., 1::2] * s, z[..., 0::2] * s + z[..., 1::2] * c], -1).flatten(-2)
    q, k = turn(q), turn(k)
    attn = torch.empty(T, nq, d, dtype=torch.float64, device="cuda")
    at = 0
    for a, b, table in zip(news, held, tables):
        n = a + b
        idx = torch.arange(n, device="cuda")
        page, slot = torch.tensor(table, device="cuda")[idx // PAGE], idx % PAGE
        kv[0][page[b:], :, slot[b:]] = k[at:at + a]
        kv[1][page[b:], :, slot[b:]] = v[at:at + a]
        keys, values = kv[0][page, :, slot], kv[1][page, :, slot]                   # [n, nkv, d]
        ahead = idx[None, :] > (b + torch.arange(a, device="cuda"))[:, None]
        for g in range(nkv):
            for j in range(nq // nkv):
                head = g * (nq // nkv) + j
                scores = (q[at:at + a, head] @ keys[:, g].t()) * d ** -0.5
                attn[at:at + a, head] = torch.softmax(scores.masked_fill_(ahead, -math.inf), -1) @ values[:, g]
        at += a
    x = x + attn.view(T, nq * d) @ w("self_attn.o_proj.weight").t()
    h = _rms(x, 1e-5) * w("post_attention_layernorm.weight")
    gate = h @ w("mlp.gate_proj.weight").t()
    return x, (gate * torch.sigmoid(gate) * (h @ w("mlp.up_proj.weight").t())) @ w("mlp.down_proj.weight").t()


def _convolved(rows, old, taps, bias):
    """Causal convolution per channel and silu; ``old [taps - 1, C]`` are the rows before the first.  Returns (result, new old rows)."""
    n, K = rows.shape[0], taps.shape[1]
    full = torch.cat([old, rows])
    y = sum(full[j:j + n] * taps[:, j] for j in range(K))
    if bias is not None:
        y = y + bias
    return y * torch.sigmoid(y), full[n:]


def _exact_mixer(case, t, h, start):
    kind, W = case["mixer"], case["width"]
    H, D = W // 128, 128
    w = lambda name: _f(t["l0.mix." + name])
    news, _ = _lengths(case)
    sig, softplus = torch.sigmoid, torch.nn.functional.softplus
    state = _f(start).reshape(len(news), -1).clone()
    SZ = H * D * D
    outs, at = [], 0
    for r, n in enumerate(news):
        x = h[at:at + n]
        at += n
        S = state[r, :SZ].view(H, D, D).clone()
        o = torch.empty(n, H, D, dtype=torch.float64, device="cuda")
        heads = lambda z, c=H: z.view(n, c, D)
        if kind == "gla":
            q, k, v = heads(x @ w("q").t()) * D ** -0.5, heads(x @ w("k").t()), heads(x @ w("v").t())
            a = heads(torch.exp(torch.nn.functional.logsigmoid((x @ w("a1").t()) @ w("a2").t() + w("a2.b")) / 16.0))
            for i in range(n):
                S = a[i][:, :, None] * S + k[i][:, :, None] * v[i][:, None, :]
                o[i] = torch.einsum("hkv,hk->hv", S, q[i])
            gate = x @ w("g").t()
            y = (_rms(o, 1e-5) * w("norm")).reshape(n, W) * gate * sig(gate)
        elif kind == "hgrn2":
            q = x @ w("q").t()
            q = heads(q * sig(q))
            k = heads((1.0 - w("lower")) * sig(-(x @ w("f").t() + w("f.b"))))
            v = heads(x @ w("v").t())
            for i in range(n):
                S = S + k[i][:, :, None] * (v[i][:, None, :] - S)
                o[i] = torch.einsum("hkv,hk->hv", S, q[i])
            y = (_rms(o, 1e-5) * w("norm")).reshape(n, W)
        elif kind == "mlstm":
            q, k, v = heads(x @ w("q").t()) * D ** -0.5, heads(x @ w("k").t()), heads(x @ w("v").t())
            gi = 15.0 * torch.tanh((x @ w("i").t() + w("i.b")) / 15.0)
            gf = torch.nn.functional.logsigmoid(15.0 * torch.tanh((x @ w("f").t() + w("f.b")) / 15.0))
            N, m = state[r, SZ:SZ + H * D].view(H, D).clone(), state[r, SZ + H * D:].clone()
            for i in range(n):
                new = torch.maximum(gf[i] + m, gi[i])
                keep, take = torch.exp(gf[i] + m - new), torch.exp(gi[i] - new)
                m = new
                S = keep[:, None, None] * S + take[:, None, None] * k[i][:, :, None] * v[i][:, None, :]
                N = keep[:, None] * N + take[:, None] * k[i]
                den = torch.maximum((N * q[i]).sum(-1).abs(), torch.exp(-m)) + 1e-6
                o[i] = torch.einsum("hkv,hk->hv", S, q[i]) / den[:, None]
            state[r, SZ:SZ + H * D], state[r, SZ + H * D:] = N.reshape(-1), m
            y = _rms(o, 1e-5).reshape(n, W) * w("norm") * sig(x @ w("g").t())
        elif kind == "delta":
            G = H // 2
            rows = torch.cat([x @ w("q").t(), x @ w("k").t(), x @ w("v").t()], 1)
            y, old = _convolved(rows, state[r, SZ:].view(3, -1), torch.cat([w("q.conv"), w("k.conv"), w("v.conv")]), None)
            state[r, SZ:] = old.reshape(-1)
            unit = lambda z: z / torch.sqrt((z * z).sum(-1, keepdim=True) + 1e-6)
            q = unit(heads(y[:, :G * D], G)).repeat_interleave(2, 1) * D ** -0.5
            k = unit(heads(y[:, G * D:2 * G * D], G)).repeat_interleave(2, 1)
            v = heads(y[:, 2 * G * D:])
            beta = sig(x @ w("b").t())
            g = torch.exp(-torch.exp(w("A_log")) * softplus(x @ w("a").t() + w("dt_bias")))
            for i in range(n):
                S = g[i][:, None, None] * S
                u = beta[i][:, None] * (v[i] - torch.einsum("hkv,hk->hv", S, k[i]))
                S = S + k[i][:, :, None] * u[:, None, :]
                o[i] = torch.einsum("hkv,hk->hv", S, q[i])
            z = x @ w("g").t()
            y = (_rms(o, 1e-5) * w("norm")).reshape(n, W) * z * sig(z)
        else:
            G = max(1, H // 8)
            rows = x @ w("in").t()
            z, dt = rows[:, :W], softplus(rows[:, 2 * W + 2 * G * D:] + w("dt_bias"))
            y, old = _convolved(rows[:, W:2 * W + 2 * G * D], state[r, SZ:].view(3, -1), w("conv"), w("conv.b"))
            state[r, SZ:] = old.reshape(-1)
            v = heads(y[:, :W])
            k = heads(y[:, W:W + G * D], G).repeat_interleave(H // G, 1)
            q = heads(y[:, W + G * D:], G).repeat_interleave(H // G, 1)
            keep = torch.exp(-torch.exp(w("A_log")) * dt)
            for i in range(n):
                S = keep[i][:, None, None] * S + dt[i][:, None, None] * k[i][:, :, None] * v[i][:, None, :]
                o[i] = torch.einsum("hkv,hk->hv", S, q[i])
            o = o + w("D")[:, None] * v
            y = o.reshape(n, W) * z * sig(z)
            y = _rms(y.view(n, G, W // G), 1e-5).reshape(n, W) * w("norm")
        state[r, :SZ] = S.reshape(-1)
        outs.append(y @ w("o").t())
    return [torch.cat(outs), state.view(start.shape)]


def exact(case, seed):
    model, t = _model(case, seed)
    del model
    d = _inputs(case, seed)
    news, held = _lengths(case)
    if case["kind"] == "layer":
        kv = _f(d["kv"])
        x, y = _exact_layer(case, t, "model.layers.0.", _f(d["x"]) + _f(d["delta"]), kv[0], news, held, d["tables"])
        return [x, y, kv]
    if case["kind"] == "model":
        kv = _f(d["kv"])
        x = _f(t["model.embed_tokens.weight"])[d["ids"].long()]
        for i in range(case["layers"]):
            x, y = _exact_layer(case, t, "model.layers.%d." % i, x, kv[i], news, held, d["tables"])
            x = x + y
        return [(_rms(x, 1e-5) * _f(t["model.norm.weight"])) @ _f(t["model.embed_tokens.weight"]).t(), kv]
    if case["kind"] == "mixer":
        return _exact_mixer(case, t, _f(d["h"]), d["state"])
    w = lambda name: _f(t["l0.mlp." + name])
    h = _f(d["h"])
    values, chosen = torch.topk(h @ w("router").t() + w("router.b"), 2, dim=-1)
    weight = torch.softmax(values, -1)

    def unit(x, name):
        gate = x @ w(name + "gate").t()
        return (gate * torch.sigmoid(gate) * (x @ w(name + "up").t())) @ w(name + "down").t()

    y = unit(h, "shared.")
    for e in range(16):
        at, place = (chosen == e).nonzero(as_tuple=True)
        y[at] += weight[at, place][:, None] * unit(h[at], "e%d." % e)
    return [y]
