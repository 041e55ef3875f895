"""Performance cases of the framework: what its users run through the public entry points, over the sizes they run it at.

Kinds of work:

  prefill   a batch of prompts of equal length through a stack (hybrid, Nuzopel or Gutenex design)
  serve     a batch of prompts, then decode steps through the captured step, every step's tokens given (as a host-side sampler does);
            the hybrid stack, whose decode step gives back tokens alone, then takes a second turn of prompt tokens behind them
  trace     one request through the continuous-batching rows: a prompt, then single tokens, logits of each (bin/trace_run)
  fa, la    one attention layer as an engine of the reference's shape drives it: a ragged batch of prompts, then decode rows
  decode    the split-KV decode attention over long, ragged caches

The stacks have the widths of bench.py and model_bench.py (width 1024, feed-forward 3584, vocabulary 32768) and one period of layers:
three recurrent ones and one attention layer.  Weights are random at the scales of a trained model and, as in a model file, bf16
numbers.  `exact` restates every path in float64 torch.
"""
from __future__ import annotations

import importlib
import math

import numpy as np
import torch

import __graft_entry__ as entry

W, FF, VOCAB, LAYERS = 1024, 3584, 32768, 4
FA_H, FA_G, FA_D, FA_ROT, THETA = 8, 2, 256, 64, 1e7
LA_H, LA_D, TAPS = 16, 128, 4
HEADS, RANK, ROT, WINDOW, KEEP, GATE_RANK = 16, 512, 64, 1024, 64, 128
EPS = 1e-6


# ---- cases ------------------------------------------------------------------------------------------------------------------
def listed():
    return [
        # the prompt phase of a full serving batch (bench.py's prompt length), a whole pass of scratch at once
        dict(name="hybrid prefill 64x1024", kind="prefill", model="hybrid", batch=64, prompt=1024),
        # a few short prompts arriving together: launches and small tiles count
        dict(name="hybrid prefill 3x333", kind="prefill", model="hybrid", batch=3, prompt=333),
        # a full batch of chat turns: short prompts, then tokens for all of them
        dict(name="hybrid serve 128", kind="serve", model="hybrid", batch=128, prompt=128, gen=16, turn=16, kv="fp16"),
        # a small batch with the quantised cache
        dict(name="hybrid serve 8 int8", kind="serve", model="hybrid", batch=8, prompt=500, gen=24, turn=9, kv="int8"),
        # one user: time to the next token
        dict(name="hybrid trace", kind="trace", model="hybrid", prompt=45, gen=8),
        # documents of a kilotoken and their continuation, on the layer-described designs
        dict(name="nuzopel serve 16", kind="serve", model="nuzopel", batch=16, prompt=1024, gen=16, kv="fp16"),
        dict(name="gutenex serve 16", kind="serve", model="gutenex", batch=16, prompt=1024, gen=16, kv="fp16"),
        # prompts of an odd length
        dict(name="nuzopel prefill 5x771", kind="prefill", model="nuzopel", batch=5, prompt=771),
        # one user on the looped design's layers
        dict(name="gutenex trace", kind="trace", model="gutenex", prompt=77, gen=6),
        # one layer under a host engine that owns the rest: ragged prompts, quantise-on-append, then decode rows
        dict(name="attention layer int8", kind="fa", n=7, longest=1000, gen=6, kv="int8", proj="fp16"),
        dict(name="DeltaNet layer", kind="la", n=9, longest=700, gen=6, proj="fp16"),
        # decode attention alone, a full batch in the middle of its generation
        dict(name="decode attention 128x1536", kind="decode", n=128, longest=1536, kv="fp16"),
    ]


def draw(rng):
    def log(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    kind = rng.choice(["prefill", "prefill", "serve", "serve", "trace", "fa", "la", "decode"])
    if kind in ("prefill", "serve", "trace"):
        model = rng.choice(["hybrid", "hybrid", "nuzopel", "gutenex"])
        most = 32768 if model == "hybrid" else 16384
        if kind == "trace":
            return dict(kind=kind, model=model, prompt=log(2, 600), gen=rng.randint(2, 12))
        prompt = log(20, 1500)
        batch = log(1, min(128, most // prompt))
        if kind == "prefill":
            return dict(kind=kind, model=model, batch=batch, prompt=prompt)
        case = dict(kind=kind, model=model, batch=batch, prompt=prompt, gen=rng.randint(4, 32), kv="fp16")
        return dict(case, turn=rng.randint(2, 32), kv=rng.choice(["fp16", "int8"])) if model == "hybrid" else case
    if kind == "fa":
        return dict(kind=kind, n=rng.randint(1, 12), longest=log(30, 1400), gen=rng.randint(1, 8), kv=rng.choice(["fp16", "int8"]),
                    proj=rng.choice(["fp16", "fp16", "fp32"]))
    if kind == "la":
        return dict(kind=kind, n=rng.randint(1, 12), longest=log(30, 1400), gen=rng.randint(1, 8), proj=rng.choice(["fp16", "fp16", "fp32"]))
    return dict(kind=kind, n=log(1, 128), longest=log(64, 4096), kv=rng.choice(["fp16", "int8"]))


def ragged(n, longest):
    """n lengths from about a third of `longest` to all of it."""
    return [max(1, longest - (longest * 2 // 3) * ((5 * i + 2) % n) // n if i else longest) for i in range(n)]


# ---- weights and inputs -------------------------------------------------------------------------------------------------------
class Draws:
    """Random tensors on the GPU, in the order they are asked for."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda").manual_seed(int(seed) * 2654435761 % (1 << 62) + 7)

    def normal(self, *shape, std=1.0):
        return torch.randn(shape, device="cuda", generator=self.g) * std

    def weight(self, *shape, std=0.02):
        return self.normal(*shape, std=std).bfloat16()

    def uniform(self, *shape, low=0.0, high=1.0):
        return torch.rand(shape, device="cuda", generator=self.g) * (high - low) + low

    def tokens(self, *shape):
        return torch.randint(0, VOCAB, shape, dtype=torch.int32, device="cuda", generator=self.g)


def ffn_weights(d):
    return dict(gate=d.weight(FF, W), up=d.weight(FF, W), down=d.weight(W, FF))


def fa_weights(d):
    kv = FA_G * FA_D
    return dict(wq=d.weight(FA_H * FA_D * 2, W), wk=d.weight(kv, W), wv=d.weight(kv, W), q_norm=d.normal(FA_D, std=0.05), k_norm=d.normal(FA_D, std=0.05),
                wo=d.weight(W, FA_H * FA_D))


def la_weights(d):
    c = LA_H * LA_D
    return dict(w_qkv=d.weight(3 * c, W), w_a=d.weight(LA_H, W), w_b=d.weight(LA_H, W), w_z=d.weight(c, W), conv_w=d.normal(3 * c, TAPS, std=0.3),
                a_log=d.uniform(LA_H, high=2.7), dt_bias=d.normal(LA_H, std=0.1), norm_w=1.0 + d.normal(LA_D, std=0.05), w_out=d.weight(W, c))


def hybrid_weights(d):
    layers = []
    for i in range(LAYERS):
        layers.append(dict(input_norm=d.normal(W, std=0.05), post_norm=d.normal(W, std=0.05), ffn=ffn_weights(d),
                           **(dict(fa=fa_weights(d)) if i % 4 == 3 else dict(la=la_weights(d)))))
    return dict(layers=layers, embed=d.weight(VOCAB, W), final_norm=d.normal(W, std=0.05))


def block_config(model):
    """One period of the layers model_bench.py runs."""
    mlp, layers = dict(kind="dense", ff=FF), []
    for i in range(LAYERS):
        if model == "nuzopel" and i % 4 == 3:
            layers.append(dict(type="latent_attention", mlp=mlp, mixer=dict(heads=HEADS, dim=128, rot_dim=ROT, vdim=128, kv_rank=RANK, mask=dict(size=WINDOW),
                                                                            rot=dict(base=1e4, dims=ROT), scale=192 ** -0.5)))
        elif model == "nuzopel":
            layers.append(dict(type="mlstm", mlp=mlp, mixer=dict(heads=HEADS, dim=128, vdim=128, gate_cap=15.0)))
        elif i % 4 == 3:
            layers.append(dict(type="attention", mlp=mlp, mixer=dict(heads=HEADS, kv_heads=HEADS // 4, dim=64, vdim=128, scale=64 ** -0.5, diff=0.5,
                                                                     mask=dict(size=WINDOW, keep_first=KEEP), rot=dict(base=1e4, dims=32))))
        elif i % 4 == 1:
            layers.append(dict(type="lightning", mlp=mlp, mixer=dict(heads=HEADS, dim=128, vdim=128, decay=[1.0 - 2.0 ** (-3 - h % 8) for h in range(HEADS)])))
        else:
            layers.append(dict(type="channel_delta", mlp=mlp, mixer=dict(heads=HEADS, kv_heads=HEADS, dim=128, vdim=128, conv=TAPS)))
    if model == "nuzopel":
        return dict(architecture="Nuzopel", width=W, vocab=VOCAB, layers=layers, norm=dict(eps=EPS), embedding=dict(scale=1.0), logit_scale=1.0)
    return dict(architecture="Gutenex", width=W, vocab=VOCAB, layers=layers, norm=dict(eps=EPS), logit_softcap=30.0)


def block_weights(d, config):
    """Tensors under the names of a model file: matrices in bf16, vectors in float32."""
    t = {"embed": d.weight(VOCAB, W), "final.norm": 1.0 + d.normal(W, std=0.05)}
    if config["architecture"] == "Gutenex":
        t["head"] = d.weight(VOCAB, W)
    for i, layer in enumerate(config["layers"]):
        m, p = layer["mixer"], f"l{i}.mix."
        qk, v = m["heads"] * m["dim"], m["heads"] * m["vdim"]
        t[p + "o"] = d.weight(W, v)
        if layer["type"] == "mlstm":
            t.update({p + "q": d.weight(qk, W), p + "k": d.weight(qk, W), p + "v": d.weight(v, W), p + "g": d.weight(v, W), p + "i": d.weight(HEADS, W),
                      p + "f": d.weight(HEADS, W), p + "i.b": d.normal(HEADS, std=0.1), p + "f.b": 3.0 + d.normal(HEADS, std=0.5),
                      p + "norm": 1.0 + d.normal(v, std=0.05)})
        elif layer["type"] == "latent_attention":
            t.update({p + "q": d.weight(m["heads"] * (m["dim"] + ROT), W), p + "uk": d.weight(qk, RANK), p + "uv": d.weight(v, RANK),
                      p + "dkv": d.weight(RANK + ROT, W), p + "dkv.norm": 1.0 + d.normal(RANK, std=0.05)})
        elif layer["type"] == "lightning":
            t.update({p + "q": d.weight(qk, W), p + "k": d.weight(qk, W), p + "v": d.weight(v, W), p + "g": d.weight(v, W), p + "norm": 1.0 + d.normal(v, std=0.05)})
        elif layer["type"] == "channel_delta":
            t.update({p + "q": d.weight(qk, W), p + "k": d.weight(qk, W), p + "v": d.weight(v, W), p + "b": d.weight(HEADS, W), p + "a1": d.weight(GATE_RANK, W),
                      p + "a2": d.weight(qk, GATE_RANK), p + "g1": d.weight(GATE_RANK, W), p + "g2": d.weight(v, GATE_RANK),
                      p + "A_log": d.normal(HEADS, std=0.2), p + "dt_bias": -3.0 + d.normal(qk, std=0.5), p + "norm": 1.0 + d.normal(m["vdim"], std=0.05)})
            t.update({p + f"{n}.conv": d.normal(qk if n != "v" else v, TAPS, std=0.5) for n in "qkv"})
        else:
            g = m["kv_heads"]
            t.update({p + "q": d.weight(2 * qk, W), p + "k": d.weight(2 * g * m["dim"], W), p + "v": d.weight(g * m["vdim"], W),
                      p + "q.norm": 1.0 + d.normal(m["dim"], std=0.05), p + "k.norm": 1.0 + d.normal(m["dim"], std=0.05)})
            t.update({p + n: d.normal(m["dim"], std=0.05) for n in ("lq1", "lk1", "lq2", "lk2")})
        t.update({f"l{i}.norm1": 1.0 + d.normal(W, std=0.05), f"l{i}.norm2": 1.0 + d.normal(W, std=0.05)})
        t.update({f"l{i}.mlp.{k}": w for k, w in ffn_weights(d).items()})
    return t


def host(t):
    return t.float().cpu().numpy()


def file_array(t):
    return t.view(torch.int16).cpu().numpy().view(np.uint16) if t.dtype == torch.bfloat16 else t.cpu().numpy()


def model_weights(case, seed):
    d = Draws(seed)
    return (hybrid_weights(d) if case["model"] == "hybrid" else block_weights(d, block_config(case["model"]))), d


def model_inputs(case, d):
    if case["kind"] == "trace":
        return dict(prompt=d.tokens(case["prompt"]), steps=d.tokens(case["gen"], 1))
    return dict(prompt=d.tokens(case["batch"], case["prompt"]), steps=d.tokens(case.get("gen", 0), case["batch"]), turn=d.tokens(case["batch"], case.get("turn", 0)))


# ---- states and passes ----------------------------------------------------------------------------------------------------------
def serving_stream():
    """The stream of the serving loop: captured steps need one that is not the default stream."""
    if not hasattr(serving_stream, "s"):
        serving_stream.s = torch.cuda.Stream()
    return serving_stream.s


def build_stack(case, weights):
    ops = entry.load_ops()
    batch, length = case.get("batch", 4), case["prompt"] + case.get("gen", 0) + case.get("turn", 0)
    if case["model"] == "hybrid":
        st = ops.HybridStack(LAYERS, FF, VOCAB, batch, length, batch, ops.KV_INT8 if case.get("kv") == "int8" else ops.KV_FP16, True, EPS)
        for i, lw in enumerate(weights["layers"]):
            parts = {k: {n: host(t) for n, t in lw[k].items()} for k in ("ffn", "fa", "la") if k in lw}
            st.set_layer_weights(i, dict(input_norm=host(lw["input_norm"]), post_norm=host(lw["post_norm"])), parts["ffn"], fa=parts.get("fa"), la=parts.get("la"))
        st.set_embedding(host(weights["embed"]), host(weights["final_norm"]))
        return st
    models = importlib.import_module(entry.PKG_NAME + ".models")
    st = models.build_model(block_config(case["model"]), models.Limits(batch, length, 0, max(batch * case["prompt"], batch), "bfloat16"),
                            {k: tuple(t.shape) for k, t in weights.items()})
    models.load_tensors(st, {k: file_array(t) for k, t in weights.items()})
    return st


def layer_inputs(case, d):
    counts = ragged(case["n"], case["longest"])
    return counts, d.normal(sum(counts), W), [d.normal(case["n"], W) for _ in range(case["gen"])]


def cache_inputs(case, d):
    counts = ragged(case["n"], case["longest"])
    rows = sum(counts)
    return counts, d.normal(rows, FA_G * FA_D), d.normal(rows, FA_G * FA_D, std=0.6), d.normal(case["n"], FA_H, FA_D)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("prefill", "serve", "trace"):
        weights, d = model_weights(case, seed)
        st = build_stack(case, weights)
        s = dict(case=case, stack=st, **model_inputs(case, d))
        torch.cuda.synchronize()
        with torch.cuda.stream(serving_stream()):
            if kind == "trace":
                st.begin_batching()
            if kind == "serve":
                st.forward_batch_decode(st.forward_batch_prefill(s["prompt"]))
                st.capture_decode(case["batch"])
        return s
    ops, d = entry.load_ops(), Draws(seed)
    if kind == "decode":
        counts, k, v, q = cache_inputs(case, d)
        fa = ops.FullAttention(ops.PROJ_FP16, max_batch=case["n"], max_prefill_rows=64)
        kv = ops.KVCache(1, case["n"], case["longest"], ops.KV_INT8 if case["kv"] == "int8" else ops.KV_FP16)
        slots = [kv.allocate_sequence(n) for n in counts]
        kv.append(0, slots, counts, k, v)
        return dict(case=case, op=fa, cache=kv, q=q, d_slots=torch.tensor(slots, dtype=torch.int32, device="cuda"))
    weights = fa_weights(d) if kind == "fa" else la_weights(d)
    counts, x, steps = layer_inputs(case, d)
    op = (ops.FullAttention if kind == "fa" else ops.LinearAttention)(ops.PROJ_FP16 if case["proj"] == "fp16" else ops.PROJ_FP32, max_batch=case["n"],
                                                                      max_prefill_rows=sum(counts))
    op.set_weights({k: host(t) for k, t in weights.items()})
    slots = list(range(case["n"]))
    if kind == "fa":
        cache = ops.KVCache(1, case["n"], case["longest"] + case["gen"], ops.KV_INT8 if case["kv"] == "int8" else ops.KV_FP16)
        slots = [cache.allocate_sequence(n + case["gen"]) for n in counts]
    else:
        cache = ops.LinearAttnState(1, case["n"])
    return dict(case=case, op=op, cache=cache, x=x, steps=steps, counts=counts, slots=slots, d_slots=torch.tensor(slots, dtype=torch.int32, device="cuda"))


def run(s):
    kind = s["case"]["kind"]
    if kind == "decode":
        return s["op"].decode_core(s["q"], s["cache"], 0, s["d_slots"])
    if kind in ("fa", "la"):
        op, cache = s["op"], s["cache"]
        cache.clear()
        prefill = op.forward_batch_prefill if kind == "fa" else op.forward_batch
        out = [prefill(s["x"], cache, 0, s["slots"], s["counts"])]
        for x in s["steps"]:
            out.append(op.forward(x, cache, 0, s["d_slots"]))
        return out
    st, case = s["stack"], s["case"]
    with torch.cuda.stream(serving_stream()):
        if kind == "trace":
            row = st.open(case["prompt"] + case["gen"])
            out = [st.extend(row, s["prompt"], [case["prompt"] - 1])]
            for token in s["steps"]:
                out.append(st.extend(row, token, [0]))
            st.retire(row)
            return out
        st.reset_cache()
        hybrid = case["model"] == "hybrid"
        if hybrid:
            out = st.forward_batch_prefill(s["prompt"], want_hidden=True)[1]
        else:
            st.forward_batch_prefill(s["prompt"])
            out = st.residual(case["batch"] * case["prompt"])
        if kind == "prefill":
            return out
        rows = []
        for tokens in s["steps"]:
            st.set_tokens(tokens)
            st.launch_decode(1)
            if not hybrid:
                rows.append(st.residual(case["batch"]))
        return out, st.forward_batch_prefill(s["turn"], want_hidden=True)[1] if hybrid else torch.stack(rows)


# ---- what a pass cannot do without ------------------------------------------------------------------------------------------------
def chunked(length, heads, inner, state):
    """Operations of a chunk-64 recurrence: `inner` products of 64 x 64 x 128 and `state` of 64 x 128 x 128 per chunk and head."""
    return heads * -(-length // 64) * (inner * 2 * 64 * 64 * 128 + state * 2 * 64 * 128 * 128)


def pairs(length, window=None, before=0):
    w = min(window or 1 << 30, length + before)
    return sum(min(t + 1, w) for t in (before, before + length - 1)) / 2 * length


def model_work(case):
    """(matrix weights of the layers, state bytes of a sequence, cache bytes of a token, prefill operations of a sequence beside the projections)."""
    model, p = case["model"], case["prompt"]
    if model == "hybrid":
        token = 2 * FA_G * FA_D * 2 if case.get("kv") != "int8" else 2 * FA_G * (FA_D + 4)
        return (W * (3 * (8224 + 2048) + 5120 + 2048 + LAYERS * 3 * FF), 3 * 4 * (LA_H * LA_D * LA_D + 3 * 6144), token,
                3 * chunked(p, LA_H, 5, 3) + 4 * FA_H * FA_D * pairs(p))
    state = 4 * HEADS * 128 * 128
    if model == "nuzopel":
        weights = W * (3 * (5 * 2048 + 32) + HEADS * 192 + RANK + ROT + 2048 + LAYERS * 3 * FF) + 2 * RANK * 2048
        return weights, 3 * state, (RANK + ROT) * 2, 3 * chunked(p, HEADS, 2, 2) + 2 * HEADS * (192 + 128) * pairs(p, WINDOW)
    weights = W * (2 * (4 * 2048 + 16 + 256) + 5 * 2048 + 2 * 2048 + 1024 + 2048 + LAYERS * 3 * FF) + 2 * 2 * 2048 * GATE_RANK
    return weights, 3 * state + 2 * 3 * 3 * 2048 * 4, (HEADS // 4) * 256 * 2, 2 * chunked(p, HEADS, 5, 3) + chunked(p, HEADS, 2, 2) + 4 * HEADS * (64 + 128) * pairs(p, WINDOW)


def work(case):
    kind = case["kind"]
    if kind == "decode":
        keys = sum(ragged(case["n"], case["longest"]))
        token = 2 * FA_G * FA_D * 2 if case["kv"] == "fp16" else 2 * FA_G * (FA_D + 4)
        return dict(bytes=keys * token + case["n"] * 2 * FA_H * FA_D * 4, flops=4 * FA_H * FA_D * keys)
    if kind in ("fa", "la"):
        counts, gen = ragged(case["n"], case["longest"]), case["gen"]
        rows = sum(counts) + gen * case["n"]
        weights = W * (5120 + 2048 if kind == "fa" else 8224 + 2048)
        size = 2 if case["proj"] == "fp16" else 4
        if kind == "fa":
            token = 2 * FA_G * FA_D * 2 if case["kv"] == "fp16" else 2 * FA_G * (FA_D + 4)
            moved = rows * token + sum(gen * n for n in counts) * token
            inner = 4 * FA_H * FA_D * (sum(pairs(n) for n in counts) + sum(gen * n for n in counts))
        else:
            moved = case["n"] * 4 * LA_H * LA_D * LA_D * (1 + 2 * gen)
            inner = sum(chunked(n, LA_H, 5, 3) for n in counts) + gen * case["n"] * 6 * LA_H * LA_D * LA_D
        return dict(bytes=weights * size * (1 + gen) + rows * W * 8 + moved, flops=2 * rows * weights + inner)
    weights, state, token, inner = model_work(case)
    batch, prompt, gen = case.get("batch", 1), case["prompt"], case.get("gen", 0)
    rows, heads = batch * (prompt + case.get("turn", 0)), batch * (1 + gen)
    seen = batch * sum(min(WINDOW, prompt + i) if case["model"] != "hybrid" else prompt + i for i in range(gen))
    total = dict(bytes=2 * weights * (1 + gen) + 2 * VOCAB * W * (1 + gen) + rows * (token + 4) + batch * state * (1 + 2 * gen) + seen * token,
                 flops=2 * weights * (rows + batch * gen) + 2 * VOCAB * W * heads + batch * inner)
    if case["model"] != "hybrid" and kind != "trace":
        total["bytes"] += 4 * W * (rows + batch * gen)
    return total


def tolerance(case):
    kind = case["kind"]
    if kind == "decode":
        return dict(rel=1.2e-3, max=0.05)            # fp16 products: 2.7e-4 off float64
    if kind in ("fa", "la"):
        return dict(rel=2.5e-3, max=0.1)             # 5e-4 to 6e-4 off
    if case["model"] == "hybrid":
        return dict(rel=0.018, max=0.4)              # four layers in fp16: 4e-3 to 8e-3 off
    return dict(rel=0.03, max=0.8)                   # four layers in bf16: 7e-3 to 2.4e-2 off


# ---- the same in float64 ------------------------------------------------------------------------------------------------------------
def rms(x, w=None, eps=EPS):
    y = x / torch.sqrt(x.square().mean(-1, keepdim=True) + eps)
    return y if w is None else y * w


def silu(x):
    return x * torch.sigmoid(x)


def turn(x, pos, base, dims, adjacent):
    """x [B, T, ..., D]: the first `dims` values turned in pairs, neighbours or halves, by pos * base^(-2i / dims)."""
    ang = pos.double()[:, None] * base ** (-2.0 * torch.arange(dims // 2, device=x.device, dtype=torch.float64) / dims)
    ang = ang.reshape((1, len(pos)) + (1,) * (x.ndim - 3) + (dims // 2,))
    out = x.clone()
    a, b = (slice(0, dims, 2), slice(1, dims, 2)) if adjacent else (slice(0, dims // 2), slice(dims // 2, dims))
    u, v = x[..., a], x[..., b]
    out[..., a], out[..., b] = u * ang.cos() - v * ang.sin(), v * ang.cos() + u * ang.sin()
    return out


def attend(q, k, v, scale, window=None, keep=0):
    """q [B, T, H, D], k [B, T, H or fewer, D], v alike: causal softmax attention within a window and the first `keep` positions."""
    t, per = q.shape[1], q.shape[2] // k.shape[2]
    i = torch.arange(t, device=q.device)
    see = i[:, None] >= i[None, :]
    if window:
        see &= (i[:, None] - i[None, :] < window) | (i[None, :] < keep)
    out = torch.empty(q.shape[:3] + v.shape[-1:], device=q.device, dtype=q.dtype)
    for b in range(q.shape[0]):
        for h in range(q.shape[2]):
            s = (q[b, :, h] @ k[b, :, h // per].T * scale).masked_fill(~see, -math.inf)
            out[b, :, h] = torch.softmax(s, -1) @ v[b, :, h // per]
    return out


def memory(q, k, v, step):
    """Walks a matrix memory S [B*H, D, V] over the tokens; step(t, S, k_t, v_t) -> S; out_t = q_t S.  q, k [B, T, H, D]."""
    b, t, h, dim = q.shape
    flat = [x.transpose(0, 1).reshape(t, b * h, -1).contiguous() for x in (q, k, v)]
    s = torch.zeros((b * h, dim, v.shape[-1]), device=q.device, dtype=q.dtype)
    out = torch.empty((t, b * h, v.shape[-1]), device=q.device, dtype=q.dtype)
    for i in range(t):
        s = step(i, s, flat[1][i], flat[2][i])
        out[i] = torch.bmm(flat[0][i][:, None], s)[:, 0]
    return out.reshape(t, b, h, -1).transpose(0, 1)


def delta_step(decay, beta):
    """decay [T, B*H, D or 1], beta [T, B*H]."""
    def step(i, s, k, v):
        s = s.mul_(decay[i][:, :, None])
        u = beta[i][:, None] * (v - torch.bmm(k[:, None], s)[:, 0])
        return s.baddbmm_(k[:, :, None], u[:, None])
    return step


def by_token(x):
    """[B, T, H, ...] -> [T, B*H, ...]"""
    return x.transpose(0, 1).reshape((x.shape[1], x.shape[0] * x.shape[2]) + x.shape[3:]).contiguous()


def unit(x):
    return x / torch.sqrt(x.square().sum(-1, keepdim=True) + 1e-6)


def causal_conv(x, w, order):
    """x [B, T, C], w [C, taps]; order[j]: how many tokens back tap j looks."""
    out = torch.zeros_like(x)
    for j, back in enumerate(order):
        out[:, back:] += x[:, :x.shape[1] - back] * w[:, j]
    return out


def fa_exact(x, w, quantised):
    b, t, _ = x.shape
    qg = (x @ w["wq"].T).reshape(b, t, FA_H, 2, FA_D)
    k, v = ((x @ w[n].T).reshape(b, t, FA_G, FA_D) for n in ("wk", "wv"))
    pos = torch.arange(t, device=x.device)
    q, k = (turn(rms(y, 1.0 + w[n]), pos, THETA, FA_ROT, True) for y, n in ((qg[..., 0, :], "q_norm"), (k, "k_norm")))
    if quantised:
        k, v = codes(k), codes(v)
    o = attend(q, k, v, FA_D ** -0.5)
    o = o * torch.sigmoid(qg[..., 1, :])
    return o.reshape(b, t, -1) @ w["wo"].T


def codes(x):
    """Values as the quantised cache holds them: 8-bit codes and a scale per token and head."""
    s = x.float().abs().amax(-1, keepdim=True) / 127.0
    s = torch.where(s > 1e-8, s, torch.ones_like(s))
    y = x.float() / s
    return (torch.sign(y) * torch.floor(y.abs() + 0.5)).clamp(-127, 127).double() * s.double()


def la_exact(x, w):
    b, t, _ = x.shape
    c = LA_H * LA_D
    mixed = silu(causal_conv(x @ w["w_qkv"].T, w["conv_w"], (1, 2, 3, 0)))
    q, k, v = (y.reshape(b, t, LA_H, LA_D) for y in mixed.split(c, -1))
    beta = torch.sigmoid(x @ w["w_b"].T)
    g = torch.exp(-torch.exp(w["a_log"]) * torch.nn.functional.softplus(x @ w["w_a"].T + w["dt_bias"]))
    o = memory(unit(q) * LA_D ** -0.5, unit(k), v, delta_step(by_token(g)[:, :, None], by_token(beta)))
    o = rms(o, w["norm_w"]).reshape(b, t, c) * silu(x @ w["w_z"].T)
    return o @ w["w_out"].T


def quantised_rows(m):
    s = m.float().abs().amax(1, keepdim=True) / 127.0
    s = torch.where(s > 1e-8, s, torch.ones_like(s))
    y = m.float() / s
    return ((torch.sign(y) * torch.floor(y.abs() + 0.5)).clamp(-127, 127) * s).double()


def hybrid_exact(weights, tokens, quantised):
    """Normed hidden rows [B, T, W] and the embedding; `quantised`: attention over 8-bit keys and values."""
    q8 = {"wq", "wk", "wv", "wo", "w_qkv", "w_a", "w_b", "w_z", "w_out", "gate", "up", "down"}
    emb = quantised_rows(weights["embed"])
    x = emb[tokens.long()]
    for lw in weights["layers"]:
        parts = {k: {n: quantised_rows(t) if n in q8 else t.double() for n, t in lw[k].items()} for k in ("ffn", "fa", "la") if k in lw}
        h = rms(x, 1.0 + lw["input_norm"].double())
        x = x + (fa_exact(h, parts["fa"], quantised) if "fa" in parts else la_exact(h, parts["la"]))
        h, f = rms(x, 1.0 + lw["post_norm"].double()), parts["ffn"]
        x = x + (silu(h @ f["gate"].T) * (h @ f["up"].T)) @ f["down"].T
    return rms(x, 1.0 + weights["final_norm"].double()), emb


def mlstm_exact(h, w, m):
    b, t, _ = h.shape
    q, k, v = ((h @ w[n].T).reshape(b, t, m["heads"], -1) for n in "qkv")
    cap = m["gate_cap"]
    ig, fg = (cap * torch.tanh((h @ w[n].T + w[n + ".b"]) / cap) for n in "if")
    ig, fg = by_token(ig), by_token(torch.nn.functional.logsigmoid(fg))
    mx = torch.zeros_like(ig[0])
    ones = torch.ones_like(v[..., :1])
    scale, floor = [], []
    for i in range(t):
        new = torch.maximum(fg[i] + mx, ig[i])
        scale.append((torch.exp(fg[i] + mx - new), torch.exp(ig[i] - new)))
        floor.append(torch.exp(-new))
        mx = new

    def step(i, s, k_t, v_t):
        keep, add = scale[i]
        return s.mul_(keep[:, None, None]).baddbmm_((add[:, None] * k_t)[:, :, None], v_t[:, None])
    o = memory(q * m["dim"] ** -0.5, k, torch.cat([v, ones], -1), step)            # the last column is the normaliser
    den = torch.maximum(o[..., -1].abs(), torch.stack(floor).reshape(t, b, -1).transpose(0, 1)) + 1e-6
    o = rms(o[..., :-1] / den[..., None]).reshape(b, t, -1) * w["norm"] * torch.sigmoid(h @ w["g"].T)
    return o @ w["o"].T


def latent_exact(h, w, m):
    b, t, _ = h.shape
    pos, heads, dim, rot = torch.arange(t, device=h.device), m["heads"], m["dim"], m["rot_dim"]
    y = h @ w["dkv"].T
    lat, r = rms(y[..., :RANK], w["dkv.norm"]), turn(y[..., RANK:], pos, m["rot"]["base"], rot, False)
    q = (h @ w["q"].T).reshape(b, t, heads, dim + rot)
    q = torch.cat([q[..., :dim], turn(q[..., dim:].contiguous(), pos, m["rot"]["base"], rot, False)], -1)
    k = torch.cat([(lat @ w["uk"].T).reshape(b, t, heads, dim), r[:, :, None].expand(b, t, heads, rot)], -1)
    o = attend(q, k, (lat @ w["uv"].T).reshape(b, t, heads, -1), m["scale"], m["mask"]["size"])
    return o.reshape(b, t, -1) @ w["o"].T


def lightning_exact(h, w, m):
    b, t, _ = h.shape
    q, k, v = (silu(h @ w[n].T).reshape(b, t, m["heads"], -1) for n in "qkv")
    decay = torch.tensor(m["decay"], device=h.device, dtype=torch.float64).repeat(b)[:, None, None]
    o = memory(q, k, v, lambda i, s, k_t, v_t: s.mul_(decay).baddbmm_(k_t[:, :, None], v_t[:, None]))
    return (rms(o.reshape(b, t, -1), w["norm"]) * torch.sigmoid(h @ w["g"].T)) @ w["o"].T


def channel_delta_exact(h, w, m):
    b, t, _ = h.shape
    q, k, v = (silu(causal_conv(h @ w[n].T, w[n + ".conv"], range(TAPS - 1, -1, -1))).reshape(b, t, m["heads"], -1) for n in "qkv")
    a = (h @ w["a1"].T @ w["a2"].T + w["dt_bias"]).reshape(b, t, m["heads"], -1)
    g = torch.exp(-torch.exp(w["A_log"])[:, None] * torch.nn.functional.softplus(a))
    o = memory(unit(q) * m["dim"] ** -0.5, unit(k), v, delta_step(by_token(g), by_token(torch.sigmoid(h @ w["b"].T))))
    o = rms(o, w["norm"]).reshape(b, t, -1) * torch.sigmoid(h @ w["g1"].T @ w["g2"].T)
    return o @ w["o"].T


def diff_exact(h, w, m):
    b, t, _ = h.shape
    pos = torch.arange(t, device=h.device)
    q = turn(rms((h @ w["q"].T).reshape(b, t, m["heads"], 2, m["dim"]), w["q.norm"]), pos, m["rot"]["base"], m["rot"]["dims"], True)
    k = turn(rms((h @ w["k"].T).reshape(b, t, m["kv_heads"], 2, m["dim"]), w["k.norm"]), pos, m["rot"]["base"], m["rot"]["dims"], True)
    v = (h @ w["v"].T).reshape(b, t, m["kv_heads"], m["vdim"])
    one, two = (attend(q[..., i, :], k[..., i, :], v, m["scale"], m["mask"]["size"], m["mask"]["keep_first"]) for i in (0, 1))
    lam = torch.exp((w["lq1"] * w["lk1"]).sum()) - torch.exp((w["lq2"] * w["lk2"]).sum()) + m["diff"]
    return (rms(one - lam * two) * (1.0 - m["diff"])).reshape(b, t, -1) @ w["o"].T


MIXERS = dict(mlstm=mlstm_exact, latent_attention=latent_exact, lightning=lightning_exact, channel_delta=channel_delta_exact, attention=diff_exact)


def block_exact(weights, config, tokens):
    """Residual rows [B, T, W]."""
    x = weights["embed"].double()[tokens.long()]
    gutenex = config["architecture"] == "Gutenex"
    act = silu if gutenex else lambda z: 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))
    for i, layer in enumerate(config["layers"]):
        w = {k[len(f"l{i}."):]: t.double() for k, t in weights.items() if k.startswith(f"l{i}.")}
        mix = {k[4:]: t for k, t in w.items() if k.startswith("mix.")}

        def ff(h):
            return (act(h @ w["mlp.gate"].T) * (h @ w["mlp.up"].T)) @ w["mlp.down"].T
        if gutenex:
            x = x + MIXERS[layer["type"]](rms(x, w["norm1"]), mix, layer["mixer"])
            x = x + ff(rms(x, w["norm2"]))
        else:
            x = x + rms(MIXERS[layer["type"]](x, mix, layer["mixer"]), w["norm1"])
            x = x + rms(ff(x), w["norm2"])
    return x


def exact(case, seed):
    with torch.no_grad():
        return exact_of(case, seed)


def exact_of(case, seed):
    kind = case["kind"]
    if kind in ("prefill", "serve", "trace"):
        weights, d = model_weights(case, seed)
        inp = model_inputs(case, d)
        prompt, steps, p = inp["prompt"].reshape(-1, case["prompt"]), inp["steps"], case["prompt"]
        if case["model"] == "hybrid":
            hid, emb = hybrid_exact(weights, torch.cat([prompt, steps.T] + ([inp["turn"]] if "turn" in inp else []), 1), case.get("kv") == "int8")
            if kind == "trace":
                return [(hid[:, t] @ emb.T) for t in range(p - 1, p + case["gen"])]
            return hid[:, p - 1] if kind == "prefill" else (hid[:, p - 1], hid[:, -1])
        config = block_config(case["model"])
        x = block_exact(weights, config, torch.cat([prompt, steps.T], 1))
        if kind == "trace":
            logits = rms(x[:, p - 1:], weights["final.norm"].double()) @ weights["head" if case["model"] == "gutenex" else "embed"].double().T
            if case["model"] == "gutenex":
                logits = config["logit_softcap"] * torch.tanh(logits / config["logit_softcap"])
            return [logits[:, t] for t in range(1 + case["gen"])]
        out = x[:, :p].reshape(-1, W)
        return out if kind == "prefill" else (out, x[:, p:].transpose(0, 1))
    d = Draws(seed)
    if kind == "decode":
        counts, k, v, q = cache_inputs(case, d)
        k, v = ((codes(y) if case["kv"] == "int8" else y.half().double()) for y in (y.reshape(-1, FA_G, FA_D) for y in (k, v)))
        out, at = [], 0
        for i, n in enumerate(counts):
            kk, vv = (y[at:at + n].repeat_interleave(FA_H // FA_G, 1) for y in (k, v))
            s = torch.einsum("hd,nhd->hn", q[i].double(), kk) * FA_D ** -0.5
            out.append(torch.einsum("hn,nhd->hd", torch.softmax(s, -1), vv))
            at += n
        return torch.stack(out)
    weights = {k: t.double() for k, t in (fa_weights(d) if kind == "fa" else la_weights(d)).items()}
    counts, x, steps = layer_inputs(case, d)
    first, later, at = [], [], 0
    for i, n in enumerate(counts):
        rows = torch.cat([x[at:at + n]] + [y[i:i + 1] for y in steps])[None].double()
        y = (fa_exact(rows, weights, case["kv"] == "int8") if kind == "fa" else la_exact(rows, weights))[0]
        first.append(y[:n])
        later.append(y[n:])
        at += n
    return [torch.cat(first)] + [torch.stack([y[j] for y in later]) for j in range(case["gen"])]
