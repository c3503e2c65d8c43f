"""What is measured when this framework is made faster: calls that a user's program makes, over the sizes it makes them at.

Four kinds of pass, named by a case's "kind":

  prompt   `Model.step` on a batch of whole prompts of a whole model, replayed from its graph as a serving program that has
           seen the rounded shape before has it; the logits of every prompt's last token
  decode   a session of single-token steps of a whole model: `DecodeGraph.load`, then `DecodeGraph.run` for a few steps;
           the last step's logits and the tokens read back
  layer    one decoder layer on a step of several tokens (prompts, or a portion that goes on behind earlier tokens):
           `block.forward` on the float32 stream; the stream and the pending output of the feed-forward
  mixer    one recurrent mixer on such a step: `mixer.forward`; its output and every sequence's new state

Sizes are those of the presets; prompt lengths are those of the published request sets (183 to 275 tokens for chat, 1,000 to
7,069 for long prompts) and the benchmark's 2,048 tokens and 4,096 positions of context. Weights are drawn so that
activations stay of order one through a layer and attention is peaked (scores of standard deviation about 2), as in a
trained model; the embedding is wide enough that the next token is chosen by a clear margin, again as in a trained model.
"""
import math

import numpy as np
import torch
import torch.nn.functional as F

from qwenforge_b200.cache import SequenceCache
from qwenforge_b200.config import config_from_dict, preset_config
from qwenforge_b200.engine import Model, build_context
from qwenforge_b200.engine.graphs import DecodeGraph
from qwenforge_b200.sampling import Sampler
from qwenforge_b200.weights import random_state_on_device

DEVICE = "cuda"
VOCAB_OF_A_LAYER = 128          # a model that is built for one of its layers keeps a token table of this many rows
EXACT_FLOPS = 1.2e14            # no 64-bit reference beyond this much work (several seconds on the device)

QWEN = {"qwen2.5-0.5b": dict(width=896, inter=4864, layers=24, heads=14, kv_heads=2, dim=64, vocab=151936),
        "qwen2.5-3b": dict(width=2048, inter=11008, layers=36, heads=16, kv_heads=2, dim=128, vocab=151936),
        "qwen2.5-7b": dict(width=3584, inter=18944, layers=28, heads=28, kv_heads=4, dim=128, vocab=152064)}
THETA, EPS = 1e6, 1e-6
MIXERS = {"mlstm": {"zebovik-0.5b": dict(width=896, heads=7, dim=64, vdim=128), "zebovik-3b": dict(width=2048, heads=16, dim=64, vdim=128)},
          "mamba2": {"zebovik-0.5b": dict(width=896, heads=28, dim=128, vdim=64), "zebovik-3b": dict(width=2048, heads=32, dim=128, vdim=128)},
          "gla": {"gatosun-0.5b": dict(width=896, heads=7, dim=64, vdim=128), "gatosun-3b": dict(width=2048, heads=16, dim=64, vdim=128)}}
GATE_CAP, DENOMINATOR_FLOOR, TAPS, RANK, TAU = 15.0, 1e-6, 4, 64, 8.0


def listed():
    return [
        # one user waits for every token: the smallest call there is, a chain of short kernels
        {"name": "decode-0.5b-1", "kind": "decode", "model": "qwen2.5-0.5b", "seqs": 1, "context": 1024, "steps": 8},
        # the benchmark's headline: batch 8, 4,096 positions of context
        {"name": "decode-0.5b-8", "kind": "decode", "model": "qwen2.5-0.5b", "seqs": 8, "context": 4096, "steps": 8},
        # a filled batch of the middle size: weights and cache both count
        {"name": "decode-3b-16", "kind": "decode", "model": "qwen2.5-3b", "seqs": 16, "context": 2048, "steps": 4},
        # four chat turns that start together
        {"name": "prompt-0.5b-chat", "kind": "prompt", "model": "qwen2.5-0.5b", "lengths": "183,275,201,246"},
        # the benchmark's prompt, one layer of it
        {"name": "layer-0.5b-2048", "kind": "layer", "model": "qwen2.5-0.5b", "dtype": "bfloat16", "before": 0, "lengths": "2048"},
        # unequal long prompts that start together
        {"name": "layer-3b-ragged", "kind": "layer", "model": "qwen2.5-3b", "dtype": "bfloat16", "before": 0, "lengths": "2175,3152,1000,1031"},
        # the largest: the two longest published prompts at the largest size
        {"name": "layer-7b-long", "kind": "layer", "model": "qwen2.5-7b", "dtype": "bfloat16", "before": 0, "lengths": "4719,7069"},
        # a document's next portion: attention far back dominates
        {"name": "layer-3b-portion", "kind": "layer", "model": "qwen2.5-3b", "dtype": "bfloat16", "before": 15360, "lengths": "1024"},
        # the exact path (`dtype="float32"`), as a reference run uses it
        {"name": "layer-0.5b-float32", "kind": "layer", "model": "qwen2.5-0.5b", "dtype": "float32", "before": 0, "lengths": "1031"},
        # recurrent mixers: the matrix memory on the benchmark's prompt, the state space on unequal prompts that go on behind
        # an earlier portion, the gated linear attention on two prompts
        {"name": "mlstm-0.5b-2048", "kind": "mixer", "mixer": "mlstm", "model": "zebovik-0.5b", "before": 0, "lengths": "2048"},
        {"name": "mamba2-3b-ragged", "kind": "mixer", "mixer": "mamba2", "model": "zebovik-3b", "before": 64, "lengths": "2175,1000,1031"},
        {"name": "gla-3b", "kind": "mixer", "mixer": "gla", "model": "gatosun-3b", "before": 0, "lengths": "2048,1031"},
    ]


def _between(rng, low, high):
    """A whole number between the two, spread over its logarithm."""
    return max(low, min(high, round(math.exp(rng.uniform(math.log(low), math.log(high))))))


def _lengths(rng, most_tokens, most_seqs, least=33):
    """Unequal prompts of up to `most_tokens` tokens in all."""
    total, n = _between(rng, 4 * least, most_tokens), rng.randint(1, most_seqs)
    shares = [rng.uniform(0.3, 1.0) for _ in range(n)]
    return ",".join(str(max(least, int(total * s / sum(shares)))) for s in shares)


def draw(rng):
    kind = rng.choice(["decode", "prompt", "layer", "layer", "layer32", "mixer", "mixer"])
    if kind == "decode":
        model = rng.choice(["qwen2.5-0.5b", "qwen2.5-0.5b", "qwen2.5-3b"])
        seqs = _between(rng, 1, 16)
        return {"kind": "decode", "model": model, "seqs": seqs, "context": _between(rng, 200, 4096 if seqs <= 8 else 2048), "steps": 4}
    if kind == "prompt":
        return {"kind": "prompt", "model": "qwen2.5-0.5b", "lengths": _lengths(rng, 4096, 8)}
    if kind == "layer":
        model = rng.choice(sorted(QWEN))
        before = rng.choice([0, 0, _between(rng, 200, 12000)])
        return {"kind": "layer", "model": model, "dtype": "bfloat16", "before": before, "lengths": _lengths(rng, 2048 if before else 8192, 6)}
    if kind == "layer32":
        return {"kind": "layer", "model": rng.choice(["qwen2.5-0.5b", "qwen2.5-3b"]), "dtype": "float32", "before": 0, "lengths": _lengths(rng, 2048, 4)}
    mixer = rng.choice(sorted(MIXERS))
    return {"kind": "mixer", "mixer": mixer, "model": rng.choice(sorted(MIXERS[mixer])), "before": rng.choice([0, _between(rng, 5, 300)]),
            "lengths": _lengths(rng, 6144, 6)}


# ------------------------------------------------------------------------------------------------------------ inputs
def _numbers(case):
    return [int(n) for n in case["lengths"].split(",")]


def _generator(seed):
    return torch.Generator(device=DEVICE).manual_seed(int(seed))


class _Draw:
    """Tensors of one generator, in the order in which they are asked for; a matrix maps its inputs to numbers of order `gain`."""

    def __init__(self, seed, dtype):
        self.g, self.dtype = _generator(seed), dtype

    def normal(self, *shape, std=1.0, mean=0.0, dtype=None):
        out = torch.empty(shape, dtype=dtype or self.dtype, device=DEVICE)
        flat = out.view(-1)
        for at in range(0, flat.numel(), 1 << 27):
            n = min(1 << 27, flat.numel() - at)
            flat[at:at + n] = torch.randn(n, generator=self.g, device=DEVICE).mul_(std).add_(mean)
        return out

    def matrix(self, rows, cols, gain=1.0):
        return self.normal(rows, cols, std=gain * cols ** -0.5)

    def uniform(self, *shape, low=0.0, high=1.0):
        return torch.rand(shape, generator=self.g, device=DEVICE) * (high - low) + low

    def tokens(self, count, vocab):
        return torch.randint(0, vocab, (count,), generator=self.g, device=DEVICE)


def _qwen_weights(size, layers, vocab, d, tied):
    """Tensors by their names in a model's files."""
    w, nh, kvh, dim, inter = size["width"], size["heads"], size["kv_heads"], size["dim"], size["inter"]
    t = {"model.embed_tokens.weight": d.normal(vocab, w, std=0.8), "model.norm.weight": d.normal(w, std=0.1, mean=1.0)}
    if not tied:
        t["lm_head.weight"] = d.matrix(vocab, w)
    for i in range(layers):
        p = f"model.layers.{i}."
        for name, rows, gain in (("q", nh * dim, 1.5), ("k", kvh * dim, 1.5), ("v", kvh * dim, 1.0)):
            t[p + f"self_attn.{name}_proj.weight"] = d.matrix(rows, w, gain)
            t[p + f"self_attn.{name}_proj.bias"] = d.normal(rows, std=0.2)
        t[p + "self_attn.o_proj.weight"] = d.matrix(w, nh * dim, 0.5)
        t[p + "mlp.gate_proj.weight"], t[p + "mlp.up_proj.weight"] = d.matrix(inter, w), d.matrix(inter, w)
        t[p + "mlp.down_proj.weight"] = d.matrix(w, inter, 0.5)
        for name in ("input_layernorm", "post_attention_layernorm"):
            t[p + name + ".weight"] = d.normal(w, std=0.1, mean=1.0)
    return t


def _whole_inputs(case, seed):
    """Weights of the whole model and the prompts' tokens."""
    size, d = QWEN[case["model"]], _Draw(seed, torch.bfloat16)
    weights = _qwen_weights(size, size["layers"], size["vocab"], d, True)
    lengths = _numbers(case) if case["kind"] == "prompt" else [case["context"]] * case["seqs"]
    return weights, [d.tokens(n, size["vocab"]).tolist() for n in lengths]


def _layer_inputs(case, seed):
    """Weights of one layer (inside a model of that layer alone) and the float32 stream, the earlier tokens' rows first."""
    size, d = QWEN[case["model"]], _Draw(seed, getattr(torch, case["dtype"]))
    weights = _qwen_weights(size, 1, VOCAB_OF_A_LAYER, d, case["model"] != "qwen2.5-7b")
    early = d.normal(len(_numbers(case)) * case["before"], size["width"], dtype=torch.float32)
    return weights, early, d.normal(sum(_numbers(case)), size["width"], dtype=torch.float32)


def _mixer_inputs(case, seed):
    """The mixer's tensors by its own names, and what it reads (bfloat16 rows of order one), the earlier tokens' rows first."""
    s, d = MIXERS[case["mixer"]][case["model"]], _Draw(seed, torch.bfloat16)
    w, h, dim, vdim = s["width"], s["heads"], s["dim"], s["vdim"]
    t = {"o_weight": d.matrix(w, h * vdim)}
    if case["mixer"] == "mamba2":
        channels = h * vdim + 2 * dim
        dt = torch.exp(d.uniform(h, low=math.log(1e-3), high=math.log(0.1)))
        t.update(in_weight=d.matrix(h * vdim + channels + h, w), conv_weight=d.uniform(channels, TAPS, low=-0.5, high=0.5),
                 conv_bias=d.normal(channels, std=0.1, dtype=torch.float32), dt_bias=dt + torch.log(-torch.expm1(-dt)),
                 rate_log=torch.log(d.uniform(h, low=1.0, high=16.0)), skip=d.normal(h, std=0.1, mean=1.0, dtype=torch.float32),
                 norm=d.normal(h * vdim, std=0.1, mean=1.0))
    else:
        t.update(q_weight=d.matrix(h * dim, w), k_weight=d.matrix(h * dim, w), v_weight=d.matrix(h * vdim, w), g_weight=d.matrix(h * vdim, w))
        if case["mixer"] == "mlstm":
            t.update(norm=d.normal(h * vdim, std=0.1, mean=1.0), i_weight=d.matrix(h, w), f_weight=d.matrix(h, w),
                     i_bias=d.normal(h, std=0.1, dtype=torch.float32), f_bias=d.uniform(h, low=3.0, high=6.0))
        else:
            t.update(norm=d.normal(vdim, std=0.1, mean=1.0), a1=d.matrix(RANK, w), a2=d.matrix(h * dim, RANK),
                     a2_bias=d.normal(h * dim, dtype=torch.float32))
    return t, d.normal(len(_numbers(case)) * case["before"], w), d.normal(sum(_numbers(case)), w)


# ------------------------------------------------------------------------------------------------------------ states
def _open(model, totals):
    """A cache with one live sequence per total length, all pages granted."""
    cache = SequenceCache(model.cache_needs(), sum(-(-n // 64) * 64 for n in totals), len(totals), model.spec.max_positions,
                          model.dtype, model.device)
    slots = [cache.open() for _ in totals]
    cache.reserve(list(zip(slots, totals)))
    cache.flush()
    return cache, slots


def _contexts(model, slots, lengths, before):
    """The step that brings the earlier tokens (None without any) and the step that is measured."""
    ids = lambda n: np.zeros(n, dtype=np.int32)
    make = lambda entries: build_context(entries, None, model.err, model.dtype, model.device, model.attention, model.decode_scratch)
    early = make([(slot, 0, ids(before)) for slot in slots]) if before else None
    return early, make([(slot, before, ids(n)) for slot, n in zip(slots, lengths)])


@torch.inference_mode()
def prepare(case, seed):
    if case["kind"] in ("prompt", "decode"):
        weights, prompts = _whole_inputs(case, seed)
        model = Model(preset_config(case["model"]).model_spec(), torch.bfloat16, DEVICE).bind(weights)
        if case["kind"] == "prompt":
            cache = model.new_cache(sum(-(-len(p) // 64) * 64 for p in prompts), len(prompts))
            model.enable_prefill_graphs()
            state = {"case": case, "model": model, "cache": cache, "prompts": prompts}
            for _ in range(2):   # a serving program has met the shape
                run(state)
            return state
        steps = case["steps"]
        cache = model.new_cache(sum(-(-(len(p) + steps) // 64) * 64 for p in prompts), len(prompts))
        slots = [cache.open() for _ in prompts]
        first = []
        for at in range(0, len(prompts), 8):
            first += Sampler()(model.step(cache, list(zip(slots[at:at + 8], prompts[at:at + 8])))).tolist()
        cache.reserve([(s, case["context"] + steps) for s in slots])
        cache.flush()
        graph = DecodeGraph(model, cache, len(slots), case["context"] + steps, Sampler())
        graph.capture()
        return {"case": case, "graph": graph, "slots": slots, "first": first}
    lengths = _numbers(case)
    if case["kind"] == "layer":
        weights, early, stream = _layer_inputs(case, seed)
        tied = case["model"] != "qwen2.5-7b"
        config = preset_config(case["model"], num_hidden_layers=1, vocab_size=VOCAB_OF_A_LAYER, tie_word_embeddings=tied)
        model = Model(config.model_spec(), getattr(torch, case["dtype"]), DEVICE).bind(weights)
        cache, slots = _open(model, [n + case["before"] for n in lengths])
        before, ctx = _contexts(model, slots, lengths, case["before"])
        state = {"case": case, "block": model.blocks[0], "site": cache.site(0), "ctx": ctx, "stream": stream, "cache": cache}
        if before is not None:
            before.step_memo = {}
            state["block"].forward(early, None, before, state["site"], True)
        return state
    tensors, early, x = _mixer_inputs(case, seed)
    kept = preset_config(case["model"]).to_dict()
    kept["layers"] = [dict(next(layer for layer in kept["layers"] if layer["type"] == case["mixer"]), mlp=None)]
    kept["vocab"] = VOCAB_OF_A_LAYER
    model = Model(config_from_dict(kept).model_spec(), torch.bfloat16, DEVICE)
    mixer = model.blocks[0].mixer
    weights = random_state_on_device(model.tensor_specs(), 0, torch.bfloat16, DEVICE)   # (the rest of the model: not run)
    weights.update({mixer.file_name(name): value for name, value in tensors.items()})
    model.bind(weights)
    cache, slots = _open(model, [n + case["before"] for n in lengths])
    before, ctx = _contexts(model, slots, lengths, case["before"])
    site = cache.site(0)
    if before is not None:
        before.step_memo = {}
        mixer.forward(early, before, site, True)
    return {"case": case, "mixer": mixer, "site": site, "slots": slots, "start": site.storage.clone(), "ctx": ctx, "x": x, "cache": cache}


@torch.inference_mode()
def run(state):
    kind = state["case"]["kind"]
    if kind == "prompt":
        cache = state["cache"]
        slots = [cache.open() for _ in state["prompts"]]
        logits = state["model"].step(cache, list(zip(slots, state["prompts"])))
        for slot in slots:
            cache.close(slot)
        return {"logits": logits}
    if kind == "decode":
        graph, n, case = state["graph"], len(state["slots"]), state["case"]
        graph.load(state["slots"], state["first"], [case["context"]] * n, [1] * n, [1 << 20] * n, list(range(n)), [])
        tokens = graph.run(case["steps"])
        return {"logits": graph.last_logits, "tokens": np.array(tokens)}
    ctx = state["ctx"]
    ctx.step_memo = {}
    if kind == "layer":
        stream = state["stream"].clone()   # the layer adds into the stream in place
        delta = state["block"].forward(stream, None, ctx, state["site"], True)
        return {"stream": stream, "delta": delta}
    storage = state["site"].storage
    storage.copy_(state["start"])          # the sequences as the earlier tokens left them
    out = state["mixer"].forward(state["x"], ctx, state["site"], True)
    return {"out": out, "state": [storage[slot] for slot in state["slots"]]}


# ------------------------------------------------------------------------------------------------------------ work
def _pairs(lengths, before=0):
    """(query, key) pairs of causal attention."""
    return sum(n * before + n * (n + 1) // 2 for n in lengths)


def _qwen_layer_work(size, tokens, pairs, keys, item):
    w, nh, kvh, dim, inter = size["width"], size["heads"], size["kv_heads"], size["dim"], size["inter"]
    params = w * (nh + 2 * kvh) * dim + w * nh * dim + 3 * w * inter
    return {"weights": item * params, "flops": 2 * tokens * params + 4 * nh * dim * pairs, "cache": 2 * kvh * dim * keys * item}


def work(case):
    if case["kind"] == "mixer":
        s, lengths = MIXERS[case["mixer"]][case["model"]], _numbers(case)
        w, h, dim, vdim, t = s["width"], s["heads"], s["dim"], s["vdim"], sum(_numbers(case))
        rows = h * vdim * 2 + (2 * dim + h if case["mixer"] == "mamba2" else 2 * h * dim)
        params = w * rows + w * h * vdim + (RANK * (w + h * dim) if case["mixer"] == "gla" else 0)
        state = h * dim * vdim * 4 * len(lengths)
        return {"bytes": 2 * params + 4 * t * w + 2 * state, "flops": 2 * t * params + 4 * t * h * dim * vdim}
    size = QWEN[case["model"]]
    if case["kind"] == "layer":
        lengths, item = _numbers(case), 2 if case["dtype"] == "bfloat16" else 4
        t = sum(lengths)
        one = _qwen_layer_work(size, t, _pairs(lengths, case["before"]), sum(lengths) + case["before"] * len(lengths), item)
        return {"bytes": one["weights"] + one["cache"] + t * size["width"] * (4 + 4 + item), "flops": one["flops"]}
    head = 2 * size["vocab"] * size["width"]
    if case["kind"] == "prompt":
        lengths = _numbers(case)
        one = _qwen_layer_work(size, sum(lengths), _pairs(lengths), sum(lengths), 2)
        return {"bytes": size["layers"] * (one["weights"] + one["cache"]) + head + 4 * size["vocab"] * len(lengths),
                "flops": size["layers"] * one["flops"] + head * len(lengths)}
    n, steps = case["seqs"], case["steps"]
    one = _qwen_layer_work(size, n, n * case["context"], n * case["context"], 2)
    return {"bytes": steps * (size["layers"] * (one["weights"] + one["cache"]) + head + 4 * size["vocab"] * n),
            "flops": steps * (size["layers"] * one["flops"] + head * n)}


def tolerance(case):
    if case["kind"] in ("prompt", "decode"):
        return {"rel": 2e-2, "max": 0.2}
    if case["kind"] == "layer" and case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 1e-4}
    return {"rel": 1e-2, "max": 0.1}


# ------------------------------------------------------------------------------------------------------------ 64 bits
def _rms64(x, weight):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + EPS) * weight.double()


def _rotated(x, positions):
    """x [T, heads, dim], component j paired with j + dim / 2."""
    dim = x.shape[-1]
    angle = positions.double()[:, None] * THETA ** (-torch.arange(0, dim, 2, device=x.device, dtype=torch.float64) / dim)
    cos, sin = angle.cos()[:, None], angle.sin()[:, None]
    a, b = x[..., :dim // 2], x[..., dim // 2:]
    return torch.cat((a * cos - b * sin, b * cos + a * sin), dim=-1)


def _attend64(q, k, v, first):
    """q [n, heads, dim] at positions first ..; k, v [m, kv heads, dim] from position 0."""
    n, nh, dim = q.shape
    out, group = torch.empty_like(q), nh // k.shape[1]
    keys = torch.arange(k.shape[0], device=q.device)
    for at in range(0, n, 512):
        rows = torch.arange(at, min(n, at + 512), device=q.device)
        for head in range(nh):
            score = q[rows, head] @ k[:, head // group].T * dim ** -0.5
            score = score.masked_fill(keys[None] > (rows + first)[:, None], -math.inf)
            out[rows, head] = torch.softmax(score, dim=-1) @ v[:, head // group]
    return out


def _qwen_layer64(stream, t, prefix, size, lengths, kept=None, first=0):
    """One layer on the float64 rows of several sequences; `kept`: per sequence the keys and values of the `first` tokens before.
    Returns the stream before the feed-forward's output, that output, and the sequences' keys and values."""
    g = lambda name: t[prefix + name].double()
    nh, kvh, dim = size["heads"], size["kv_heads"], size["dim"]
    x = _rms64(stream, t[prefix + "input_layernorm.weight"])
    q, k, v = (F.linear(x, g(f"self_attn.{n}_proj.weight"), g(f"self_attn.{n}_proj.bias")) for n in "qkv")
    at, mixed, held = 0, [], []
    for i, n in enumerate(lengths):
        rows = slice(at, at + n)
        positions = torch.arange(first, first + n, device=stream.device)
        keys, values = _rotated(k[rows].view(n, kvh, dim), positions), v[rows].view(n, kvh, dim)
        if kept is not None:
            keys, values = torch.cat((kept[i][0], keys)), torch.cat((kept[i][1], values))
        held.append((keys, values))
        mixed.append(_attend64(_rotated(q[rows].view(n, nh, dim), positions), keys, values, first).reshape(n, -1))
        at += n
    stream = stream + F.linear(torch.cat(mixed), g("self_attn.o_proj.weight"))
    x = _rms64(stream, t[prefix + "post_attention_layernorm.weight"])
    delta = F.linear(F.silu(F.linear(x, g("mlp.gate_proj.weight"))) * F.linear(x, g("mlp.up_proj.weight")), g("mlp.down_proj.weight"))
    return stream, delta, held


def _whole64(case, seed):
    weights, prompts = _whole_inputs(case, seed)
    size, table = QWEN[case["model"]], weights["model.embed_tokens.weight"]
    kept, first, made, tokens = None, 0, [], prompts
    for _ in range(1 + case.get("steps", 0)):
        lengths = [len(p) for p in tokens]
        stream = table[torch.tensor([i for p in tokens for i in p], device=DEVICE)].double()
        held_all = []
        for i in range(size["layers"]):
            stream, delta, held = _qwen_layer64(stream, weights, f"model.layers.{i}.", size, lengths, kept and kept[i], first)
            stream = stream + delta
            held_all.append(held)
        ends = torch.tensor(lengths, device=DEVICE).cumsum(0) - 1
        logits = _rms64(stream[ends], weights["model.norm.weight"]) @ table.double().T
        chosen = logits.argmax(-1).tolist()
        kept, first, tokens = held_all, first + max(lengths), [[c] for c in chosen]
        made.append(chosen)
    return logits, np.array(made[1:])


def _silu64(x):
    return x * torch.sigmoid(x)


def _mixer64(case, t, x):
    """One sequence's rows from its start: (outputs, state as the cache keeps it)."""
    s = MIXERS[case["mixer"]][case["model"]]
    h, dim, vdim, n = s["heads"], s["dim"], s["vdim"], x.shape[0]
    t = {name: value.double() for name, value in t.items()}
    x = x.double()
    f64 = dict(dtype=torch.float64, device=x.device)
    state, y = torch.zeros(h, dim, vdim, **f64), torch.empty(n, h, vdim, **f64)
    if case["mixer"] == "mamba2":
        z, u, dt = F.linear(x, t["in_weight"]).split([h * vdim, h * vdim + 2 * dim, h], dim=1)
        past = torch.cat((u.new_zeros(TAPS - 1, u.shape[1]), u))
        mixed = _silu64(sum(past[j:j + n] * t["conv_weight"][:, j] for j in range(TAPS)) + t["conv_bias"])
        v, k, q = mixed.split([h * vdim, dim, dim], dim=1)
        v, dt = v.reshape(n, h, vdim), F.softplus(dt + t["dt_bias"])
        decay = torch.exp(-torch.exp(t["rate_log"]) * dt)
        for i in range(n):
            state = state * decay[i][:, None, None] + k[i][None, :, None] * (dt[i][:, None] * v[i])[:, None]
            y[i] = torch.einsum("hdv,d->hv", state, q[i])
        y = (y + t["skip"][:, None] * v).reshape(n, -1) * _silu64(z)
        return F.linear(_rms64(y, t["norm"]), t["o_weight"]), torch.cat((state.flatten(), past[-(TAPS - 1):].flatten()))
    q, k, v, gate = (F.linear(x, t[name + "_weight"]) for name in "qkvg")
    q, k, v = q.view(n, h, dim) * dim ** -0.5, k.view(n, h, dim), v.view(n, h, vdim)
    if case["mixer"] == "gla":
        decay = torch.exp(F.logsigmoid(F.linear(F.linear(x, t["a1"]), t["a2"], t["a2_bias"])) / TAU).view(n, h, dim)
        for i in range(n):
            state = state * decay[i][:, :, None] + k[i][:, :, None] * v[i][:, None]
            y[i] = torch.einsum("hdv,hd->hv", state, q[i])
        return F.linear(_rms64(y, t["norm"]).reshape(n, -1) * _silu64(gate), t["o_weight"]), state.flatten()
    capped = lambda name: GATE_CAP * torch.tanh(F.linear(x, t[name + "_weight"], t[name + "_bias"]) / GATE_CAP)
    add, forget = capped("i"), F.logsigmoid(capped("f"))
    norm, m = torch.zeros(h, dim, **f64), torch.zeros(h, **f64)
    for i in range(n):
        higher = torch.maximum(forget[i] + m, add[i])
        decay, take, m = torch.exp(forget[i] + m - higher), torch.exp(add[i] - higher), higher
        state = state * decay[:, None, None] + (take[:, None] * k[i])[:, :, None] * v[i][:, None]
        norm = norm * decay[:, None] + take[:, None] * k[i]
        size = torch.maximum((norm * q[i]).sum(-1).abs(), torch.exp(-m)) + DENOMINATOR_FLOOR
        y[i] = torch.einsum("hdv,hd->hv", state, q[i]) / size[:, None]
    y = y * torch.rsqrt(y.square().mean(-1, keepdim=True) + EPS)
    out = F.linear(y.reshape(n, -1) * t["norm"] * torch.sigmoid(gate), t["o_weight"])
    return out, torch.cat((state.flatten(), norm.flatten(), m))


@torch.inference_mode()
def exact(case, seed):
    """What `run` returns, from the formulas in float64."""
    if case["kind"] in ("prompt", "decode"):
        size, lengths = QWEN[case["model"]], _numbers(case) if case["kind"] == "prompt" else [case["context"]] * case["seqs"]
        one = _qwen_layer_work(size, sum(lengths), _pairs(lengths), 0, 2)
        if size["layers"] * one["flops"] > EXACT_FLOPS:
            return None
        logits, tokens = _whole64(case, seed)
        return {"logits": logits} if case["kind"] == "prompt" else {"logits": logits, "tokens": tokens}
    lengths, before = _numbers(case), case["before"]
    if case["kind"] == "layer":
        weights, early, stream = _layer_inputs(case, seed)
        size, kept = QWEN[case["model"]], None
        if before:   # only the earlier tokens' keys and values count for a single layer
            x = _rms64(early.double(), weights["model.layers.0.input_layernorm.weight"]).view(len(lengths), before, -1)
            k, v = (F.linear(x, *(weights[f"model.layers.0.self_attn.{n}_proj.{part}"].double() for part in ("weight", "bias"))) for n in "kv")
            shape = (before, size["kv_heads"], size["dim"])
            positions = torch.arange(before, device=DEVICE)
            kept = [(_rotated(k[i].view(shape), positions), v[i].view(shape)) for i in range(len(lengths))]
        stream, delta, _ = _qwen_layer64(stream.double(), weights, "model.layers.0.", size, lengths, kept, before)
        return {"stream": stream, "delta": delta}
    tensors, early, x = _mixer_inputs(case, seed)
    outs, states, at = [], [], 0
    for i, n in enumerate(lengths):
        out, state = _mixer64(case, tensors, torch.cat((early[i * before:(i + 1) * before], x[at:at + n])))
        outs.append(out[before:])
        states.append(state)
        at += n
    return {"out": torch.cat(outs), "state": states}
