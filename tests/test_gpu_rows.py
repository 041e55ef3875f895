"""GPU: the few-row projections of a decode step against the library GEMMs and the plain implementations, at the edges of their row tile (8 / 9,
16 / 17 rows) and of their column tiles: feed-forward widths of one gate / up group, of a ragged last batch and of more than one wave; vocabularies that one
slab per CTA holds and, above 64 columns per SM (9472 on 148), streamed ones."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
import test_gpu_gutenex as gutenex  # noqa: E402
import test_gpu_nuzopel as nuzopel  # noqa: E402
import test_gpu_stack as stack_tests  # noqa: E402
from test_gpu_nuzopel import models, wts  # noqa: E402,F401

pytestmark = pytest.mark.gpu

L, T, STEPS = 4, 6, 3


def _weights(synth, seed, inter, vocab):
    from oracle import cpu_stack
    return cpu_stack.make_stack_weights(synth, seed, L, inter, vocab, int8=False, norm_std=0.1)


def _stack(ops, weights, inter, vocab, rows):
    st = ops.HybridStack(num_layers=L, intermediate_size=inter, vocab_size=vocab, max_seqs=rows, max_seq_len=64, prefill_chunk_seqs=rows, kv_dtype=1,
                         int8_weights=False)
    for i, lw in enumerate(weights["layers"]):
        st.set_layer_weights(i, lw, lw["ffn"], fa=lw.get("fa"), la=lw.get("la"))
    st.set_embedding(weights["embed"], weights["final_norm"])
    return st


def _decode(torch, ops, weights, inter, vocab, rows, tokens):
    """Tokens of every step, and the normed hidden rows of a second prompt behind the steps: they see every step's cache and state."""
    st = _stack(ops, weights, inter, vocab, rows)
    picks = [st.forward_batch_prefill(tokens[:, :T].contiguous()).clone()]
    for d in range(STEPS):
        picks.append(st.forward_batch_decode(tokens[:, T + d].contiguous()).clone())
    hidden = st.forward_batch_prefill(tokens[:, :4].contiguous(), want_hidden=True)[1].clone()
    torch.cuda.synchronize()
    assert st.device_status() == 0
    return torch.stack(picks), hidden


def _logits(torch, ops, weights, inter, vocab, tokens):
    """The trace path: logits of single tokens behind a prompt."""
    st = _stack(ops, weights, inter, vocab, 2)
    st.begin_batching()
    row = st.open(T + STEPS)
    out = [st.extend(row, tokens[0, :T].contiguous(), [T - 1]).clone()]
    for d in range(STEPS):
        out.append(st.extend(row, tokens[0, T + d:T + d + 1].contiguous(), [0]).clone())
    return torch.cat([x.reshape(1, -1) for x in out])


# The two sides round the same values to fp16 at the same places; their sums differ in order only, so a rounding differs now and then by one
# unit, 2^-10 of a value.  Over 4 layers of about 8 rounded vectors each that stays under sqrt(32) * 2^-10 = 6e-3 of the result.
REL = 6e-3


@pytest.mark.parametrize("rows,inter,vocab", [(1, 64, 41), (8, 256, 1003), (9, 1088, 512), (16, 3584, 512), (17, 192, 6000), (32, 4096, 2051), (33, 256, 512)])
def test_decode_rows_against_library_gemms(ops, cuda, synth, monkeypatch, rows, inter, vocab):
    torch = cuda
    weights = _weights(synth, 70 + rows, inter, vocab)
    tokens = torch.from_numpy(synth.rng(70 + rows, "tokens").integers(0, vocab, (rows, T + STEPS)).astype(np.int32)).cuda()
    monkeypatch.setenv("B200ATTN_DECODE_GEMM", "cublas")
    want_t, want_h = _decode(torch, ops, weights, inter, vocab, rows, tokens)
    want_l = _logits(torch, ops, weights, inter, vocab, tokens)
    monkeypatch.delenv("B200ATTN_DECODE_GEMM")
    got_t, got_h = _decode(torch, ops, weights, inter, vocab, rows, tokens)
    got_l = _logits(torch, ops, weights, inter, vocab, tokens)
    assert (got_h - want_h).norm() <= REL * want_h.norm()
    assert (got_l - want_l).norm() <= REL * want_l.norm()
    # a pick may differ where two logits are closer than the error: a few per cent at these vocabularies
    assert (got_t == want_t).float().mean() >= 0.9
    assert ((got_t >= 0) & (got_t < vocab)).all()


@pytest.mark.parametrize("rows", [17, 32])
def test_more_rows_than_one_tile_take_the_library_gemms(ops, cuda, synth, monkeypatch, rows):
    """Above 16 rows the library GEMMs are the faster ones: the step is theirs, bit for bit."""
    torch = cuda
    weights = _weights(synth, 70 + rows, 256, 512)
    tokens = torch.from_numpy(synth.rng(70 + rows, "tokens").integers(0, 512, (rows, T + STEPS)).astype(np.int32)).cuda()
    got = _decode(torch, ops, weights, 256, 512, rows, tokens)
    monkeypatch.setenv("B200ATTN_DECODE_GEMM", "cublas")
    want = _decode(torch, ops, weights, 256, 512, rows, tokens)
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


def test_few_row_steps_against_cpu_composition(ops, cuda, oracle, synth, monkeypatch):
    monkeypatch.delenv("B200ATTN_DECODE_GEMM", raising=False)
    stack_tests.test_prefill_and_decode_against_cpu_composition(ops, cuda, oracle, synth, None)


# ---- vocabularies that are streamed ------------------------------------------------------------------------------------------------
def _head_limits(torch, hidden, embed):
    """float64 logits of normed rows; what sums of 1024 products in fp32 may be off (2^-23 of their absolute sum each); that sum itself."""
    x = hidden.half().double()
    absolute = x.abs() @ embed.abs().T
    return x @ embed.T, 1024 * 2.0 ** -23 * absolute, absolute


@pytest.mark.parametrize("vocab", [9473, 20001, 32768])
def test_streamed_head(ops, cuda, synth, vocab):
    """Picks over one column of a last tile, over ragged and over whole tiles, several tiles a warp: maximal under float64 logits of the same rows."""
    torch = cuda
    weights = _weights(synth, 33, 64, vocab)
    embed = torch.from_numpy(weights["embed"]).cuda().half().double()
    for rows in (1, 8, 9, 16, 17):
        tokens = torch.from_numpy(synth.rng(33, f"tokens{rows}").integers(0, vocab, (rows, T + 1)).astype(np.int32)).cuda()
        st = _stack(ops, weights, 64, vocab, rows)
        prompt = tokens[:, :T].contiguous()
        with_hidden, hidden = st.forward_batch_prefill(prompt, want_hidden=True)
        st.reset_cache()
        alone = st.forward_batch_prefill(prompt)
        stepped = st.forward_batch_decode(tokens[:, T].contiguous())
        st.reset_cache()
        then = st.forward_batch_prefill(tokens, want_hidden=True)[1]
        assert st.device_status() == 0
        logits, limit, absolute = _head_limits(torch, hidden, embed)
        at = torch.arange(rows, device="cuda")
        assert (logits[at, with_hidden.long()] >= logits.amax(1) - 2 * limit.amax(1)).all()
        # the norm on the way in may round a value to its neighbour, 2^-10 of it
        assert (logits[at, alone.long()] >= logits.amax(1) - 2 * (limit + 2.0 ** -10 * absolute).amax(1)).all()
        # a step against a prompt of the same tokens: other products in the layers, four of them
        logits = _head_limits(torch, then, embed)[0]
        assert (logits[at, stepped.long()] >= logits.amax(1) - 0.05 * (logits.amax(1) - logits.mean(1))).all()


@pytest.mark.parametrize("vocab", [9473, 20001, 32768])
def test_streamed_logits(ops, cuda, synth, monkeypatch, vocab):
    """Logits of 1 to 17 places of a prompt: the last place against float64 from its normed row, all of them against the library GEMM's."""
    torch = cuda
    n = 20
    weights = _weights(synth, 34, 64, vocab)
    embed = torch.from_numpy(weights["embed"]).cuda().half().double()
    tokens = torch.from_numpy(synth.rng(34, "tokens").integers(0, vocab, (1, n)).astype(np.int32)).cuda()
    hidden = _stack(ops, weights, 64, vocab, 2).forward_batch_prefill(tokens, want_hidden=True)[1]
    logits, limit, absolute = _head_limits(torch, hidden, embed)

    def run(places):
        st = _stack(ops, weights, 64, vocab, 2)
        st.begin_batching()
        out = st.extend(st.open(n), tokens[0].contiguous(), range(n - places, n)).clone().reshape(places, vocab)
        assert st.device_status() == 0
        return out
    for places in (1, 8, 9, 16, 17):
        got = run(places)
        assert ((got[-1].double() - logits[0]).abs() <= (limit + 2.0 ** -10 * absolute)[0]).all()
        monkeypatch.setenv("B200ATTN_DECODE_GEMM", "cublas")
        want = run(places)
        monkeypatch.delenv("B200ATTN_DECODE_GEMM")
        assert (got - want).norm() <= 2.0 ** -11 * want.norm()         # the same rows: a rounding of the norm now and then


@pytest.mark.parametrize("design", [0, 1])
def test_wide_layers_and_streamed_logits_of_block_stacks(cuda, models, wts, design):
    """A feed-forward width of two waves with a ragged end, a vocabulary that is streamed, and (Gutenex) its soft cap."""
    mod, make = ((nuzopel, nuzopel.make), (gutenex, gutenex.make))[design]
    layers = [nuzopel.mlstm(2, 32, 48, ff=4802)] if design == 0 else [gutenex.lightning(2, 32, 48, ff=4802)]
    c = mod.Case(models, wts, *make(layers, width=64, vocab=20001, seed=35), "bfloat16")
    toks = c.tokens(34)
    want = c.expect(toks)
    with nuzopel.on_stream(cuda):
        c.stack.begin_batching()
        for cuts in ([1], [9, 1, 16]):
            row = c.stack.open()
            c.judge(c.run(cuda, row, toks, cuts), want, f"cuts {cuts}")
            c.stack.retire(row)


# ---- layer-described stacks (bf16) -------------------------------------------------------------------------------------------------
def _gutenex_layers():
    return [gutenex.lightning(2, 32, 48, ff=96), gutenex.delta(4, 2, 32, 32, conv=4, a_rank=20, g_rank=12, ff=70), gutenex.diff(4, 2, 32, 64, 16, 30, 5, ff=64),
            gutenex.delta(2, 2, 16, 24, ff=None)]


def _designs():
    return [(nuzopel, nuzopel.make, nuzopel.whole_layers(), {}), (gutenex, gutenex.make, _gutenex_layers(), {}),
            (gutenex, gutenex.make, _gutenex_layers(), dict(loop=(0, 2, 3)))]


@pytest.mark.parametrize("width", [32, 96, 1024])
@pytest.mark.parametrize("design", [0, 1, 2])
def test_block_rows_against_the_plain_implementation(cuda, models, wts, design, width):
    """Single tokens behind a portion: every product over the width on the few-row kernels, and behind them what their K does not fit."""
    mod, make, layers, more = _designs()[design]
    c = mod.Case(models, wts, *make(layers, width=width, seed=40 + width, **more), "bfloat16")
    toks = c.tokens(60)
    want = c.expect(toks)
    with nuzopel.on_stream(cuda):
        c.stack.begin_batching()
        for cuts in ([1], [20, 1]):
            row = c.stack.open()
            c.judge(c.run(cuda, row, toks, cuts), want, f"cuts {cuts}")
            c.stack.retire(row)


@pytest.mark.parametrize("rows", [9, 17, 32, 33])
@pytest.mark.parametrize("design", [0, 1])
def test_block_rows_of_a_batch(cuda, models, wts, design, rows):
    """Residual rows of batched steps against the plain implementation, some rows of the batch."""
    mod, make, layers, more = _designs()[design]
    c = mod.Case(models, wts, *make(layers, width=256, seed=60, **more), "bfloat16", max_seqs=rows, max_seq_len=64)
    tokens = np.stack([c.tokens(24, 5 + k) for k in range(rows)])
    t = cuda.tensor(tokens, dtype=cuda.int32, device="cuda")
    with nuzopel.on_stream(cuda):
        c.stack.forward_batch_prefill(t[:, :20].contiguous())
        got = []
        for d in range(20, 24):
            c.stack.forward_batch_decode(t[:, d].contiguous())
            got.append(c.stack.residual(rows).clone())
        assert c.stack.device_status() == 0
    got = cuda.stack(got, 1).cpu().numpy()
    for k in (0, 8, rows - 1):
        _, residual, limit = c.expect(tokens[k])
        off = np.sqrt(np.mean(((got[k] - residual[20:]) / c.residual_unit(residual)) ** 2, axis=-1))
        assert (off <= limit[1][20:]).all(), f"row {k}: {off / limit[1][20:]} of the limits"


# ---- layers of their own -------------------------------------------------------------------------------------------------------------
@pytest.mark.parametrize("rows", [1, 8, 9, 17, 32, 33])
@pytest.mark.parametrize("kind", ["fa16", "fa8", "la"])
def test_layer_decode_against_library_gemms(ops, cuda, synth, monkeypatch, kind, rows):
    """Decode steps of one layer back to back, nothing between the calls; fp32 activations, fp16 projections."""
    torch = cuda
    w = synth.la_weights(95) if kind == "la" else synth.fa_weights(95)
    xs = torch.from_numpy(np.stack([synth.hidden_states(95, f"step{d}", rows) for d in range(6)])).cuda()
    slots = torch.arange(rows, dtype=torch.int32, device="cuda")

    def run():
        op = (ops.LinearAttention if kind == "la" else ops.FullAttention)(ops.PROJ_FP16, max_batch=rows, max_prefill_rows=64)
        op.set_weights(w)
        if kind == "la":
            cache = ops.LinearAttnState(1, rows)
        else:
            cache = ops.KVCache(1, rows, 16, ops.KV_FP16 if kind == "fa16" else ops.KV_INT8)
            for _ in range(rows):
                cache.allocate_sequence(16)
        return torch.stack([op.forward(x, cache, 0, slots) for x in xs])

    monkeypatch.setenv("B200ATTN_DECODE_GEMM", "cublas")
    want = run()
    monkeypatch.delenv("B200ATTN_DECODE_GEMM")
    got = run()
    # one layer: three rounded vectors on the way, sqrt(3) * 2^-10 where every rounding differs by a unit
    assert (got - want).norm() <= 2e-3 * want.norm()


@pytest.mark.parametrize("kind", ["fa16", "fa8", "la"])
@pytest.mark.parametrize("rows", [1, 8, 17])
def test_layer_calls_on_unaligned_rows(ops, cuda, synth, kind, rows):
    """Inputs that start one, two and three floats behind a 16-byte boundary, prompts and decode rows: the products of before the few-row kernels."""
    torch = cuda
    w = synth.la_weights(98) if kind == "la" else synth.fa_weights(98)
    xs = torch.from_numpy(np.stack([synth.hidden_states(98, f"step{d}", rows) for d in range(4)])).cuda()
    slots = torch.arange(rows, dtype=torch.int32, device="cuda")

    def at(x, shift):
        base = torch.empty(x.numel() + shift, device="cuda")
        out = base[shift:].view(x.shape)
        assert (out.data_ptr() - base.data_ptr()) == 4 * shift
        return out.copy_(x)

    def run(shift):
        op = (ops.LinearAttention if kind == "la" else ops.FullAttention)(ops.PROJ_FP16, max_batch=rows, max_prefill_rows=64)
        op.set_weights(w)
        if kind == "la":
            cache = ops.LinearAttnState(1, rows)
        else:
            cache = ops.KVCache(1, rows, 16, ops.KV_FP16 if kind == "fa16" else ops.KV_INT8)
            for _ in range(rows):
                cache.allocate_sequence(16)
        prefill = op.forward_batch if kind == "la" else op.forward_batch_prefill
        return torch.stack([prefill(at(xs[0], shift), cache, 0, list(range(rows)), [1] * rows)] + [op.forward(at(x, shift), cache, 0, slots) for x in xs])
    want = run(0)
    for shift in (1, 2, 3):
        got = run(shift)
        assert torch.equal(got[0], want[0])                        # a prompt takes the same products
        assert (got - want).norm() <= 2e-3 * want.norm()           # as test_layer_decode_against_library_gemms


# ---- steps whose rows are all without a sequence ------------------------------------------------------------------------------------
@pytest.mark.parametrize("kind", ["fa16", "fa8", "la"])
def test_layer_calls_of_inactive_rows(ops, cuda, synth, kind):
    """Calls of slots -1 alone between calls of active rows, nothing else between them: the active ones give what they give without."""
    torch = cuda
    rows = 8
    w = synth.la_weights(96) if kind == "la" else synth.fa_weights(96)
    xs = torch.from_numpy(np.stack([synth.hidden_states(96, f"step{d}", rows) for d in range(8)])).cuda()
    slots, none = torch.arange(rows, dtype=torch.int32, device="cuda"), torch.full((rows,), -1, dtype=torch.int32, device="cuda")

    def run(idle):
        op = (ops.LinearAttention if kind == "la" else ops.FullAttention)(ops.PROJ_FP16, max_batch=rows, max_prefill_rows=64)
        op.set_weights(w)
        if kind == "la":
            cache = ops.LinearAttnState(1, rows)
        else:
            cache = ops.KVCache(1, rows, 16, ops.KV_FP16 if kind == "fa16" else ops.KV_INT8)
            for _ in range(rows):
                cache.allocate_sequence(16)
        out = []
        for x in xs:
            for _ in range(idle):
                op.forward(x, cache, 0, none)
            out.append(op.forward(x, cache, 0, slots))
        return torch.stack(out)
    want = run(0)
    assert torch.equal(run(1), want) and torch.equal(run(3), want)


@pytest.mark.parametrize("captured", [False, True])
def test_steps_of_inactive_rows(ops, cuda, synth, captured):
    """Steps behind the last sequence's end, then new sequences: their tokens are those of a stack that ran no such steps."""
    torch = cuda
    weights = _weights(synth, 97, 256, 512)
    prompts = torch.from_numpy(synth.rng(97, "prompts").integers(0, 512, (4, T)).astype(np.int32)).cuda()

    def run(idle):
        st = _stack(ops, weights, 256, 512, 2)
        st.begin_batching()
        if captured:
            st.capture_decode(2)
        picks = []
        for a in (0, 2):
            for p in prompts[a:a + 2]:
                st.admit(p.contiguous(), T + STEPS + 1)
            for _ in range(STEPS):
                st.step(2)
                picks.append(st.get_tokens(2).clone())
            st.retire(1)
            st.retire(0)
            for _ in range(idle):
                st.step(2)
        torch.cuda.synchronize()
        assert st.device_status() == 0
        return torch.stack(picks)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        assert torch.equal(run(3), run(0))
    torch.cuda.synchronize()
