"""GPU: prompt-sized products on pairs of CTAs with their successor in the epilogue, at the edges of their tiles (feed-forward: 256 rows, 128 outputs, parts
of 32; DeltaNet projection: 253 tokens behind 3 that only serve as taps, 32 at a time) and of their dispatch (feed-forward: more than 128 rows; DeltaNet
projection: one sequence, or from 300 rows and 36 more for each sequence on, at most 3000, and 24 rows a sequence)."""
import ctypes as C
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
import test_gpu_nuzopel as nuzopel  # noqa: E402
from test_gpu_nuzopel import models, wts  # noqa: E402,F401

pytestmark = pytest.mark.gpu

# Rounding to fp16 at the same places on both sides, sums in another order and gate / up rounded on one side only: a unit of 2^-10 of a value now and
# then.  Over 4 layers of about 8 rounded vectors each that stays under sqrt(32) * 2^-10 = 6e-3 of the result.
REL = 6e-3


@pytest.mark.parametrize("seqs,tokens,inter", [(2, 65, 64), (3, 85, 192), (4, 64, 1088), (7, 37, 128), (9, 57, 3584), (2, 128, 2048 + 64),
                                               (4, 2048, 64), (4, 2049, 64)])
def test_prompts_in_one_pass_against_one_by_one(ops, cuda, synth, seqs, tokens, inter):
    """Rows of one pass: 130, 255, 256, 259, 513, 256; one by one they are at most 128, on the library products.  8192 is the most whose kernels are launched
    as programmatic dependents, 8196 is past it; one by one these are."""
    from oracle import cpu_stack
    torch, vocab = cuda, 512
    weights = cpu_stack.make_stack_weights(synth, 90 + seqs, 4, inter, vocab, int8=False, norm_std=0.1)
    toks = torch.from_numpy(synth.rng(90 + seqs, "tokens").integers(0, vocab, (seqs, tokens)).astype(np.int32)).cuda()
    hidden = []
    for chunk in (1, seqs):
        st = ops.HybridStack(num_layers=4, intermediate_size=inter, vocab_size=vocab, max_seqs=seqs, max_seq_len=tokens, prefill_chunk_seqs=chunk, kv_dtype=1,
                             int8_weights=False)
        for i, lw in enumerate(weights["layers"]):
            st.set_layer_weights(i, lw, lw["ffn"], fa=lw.get("fa"), la=lw.get("la"))
        st.set_embedding(weights["embed"], weights["final_norm"])
        hidden.append(st.forward_batch_prefill(toks, want_hidden=True)[1].clone())
        torch.cuda.synchronize()
        assert st.device_status() == 0
    assert (hidden[1] - hidden[0]).norm() <= REL * hidden[0].norm()


@pytest.mark.parametrize("ff,width,rows", [(8, 80, 129), (72, 72, 255), (136, 64, 257), (1000, 136, 300), (264, 2304, 513)])
def test_feed_forward_widths(cuda, models, wts, ff, width, rows):      # noqa: F811
    """Gate rows in front of up rows, widths that end inside a tile and inside a 64-deep slice."""
    c = nuzopel.Case(models, wts, *nuzopel.make([nuzopel.mlstm(1, 8, 8, ff=ff)], width=width, seed=7), "bfloat16")
    toks = c.tokens(rows)
    want = c.expect(toks)
    with nuzopel.on_stream(cuda):
        c.stack.begin_batching()
        row = c.stack.open(rows)
        c.judge(c.run(cuda, row, toks, [rows]), want, f"ff {ff} width {width}")


# fp16 operands against fp32 ones: each of the about 10 roundings between a row's input and its output moves it by up to 2^-11, 5e-3 in all; a tap taken
# from the wrong place moves the row by a good part of itself.
ROW_REL = 5e-3


def fused_rows(n):
    """From so many rows on, a pass of n sequences takes the projection with the convolution in its epilogue."""
    return max(min(300 + 36 * n, 3000), 24 * n) if n > 1 else 1


@pytest.mark.parametrize("fused", [False, True])
@pytest.mark.parametrize("counts", [
    [1], [2, 1, 3], [31, 1, 33, 64], [247, 16, 5], [248, 2, 3, 1, 20], [249, 1, 40], [250, 3, 252, 7], [251, 2, 1, 1, 1, 90], [252, 260], [253, 253, 4], [254, 0, 40, 0],
    [16] * 40, [1] * 70, [506, 33], [600],
])
def test_convolution_at_the_edges_of_tiles_and_sequences(ops, cuda, synth, counts, fused):
    """Sequence starts and ends at every place around a tile's first tokens, in the middle of its chunks, several to a chunk; two calls, the second with
    the state that the first left behind, against the layer with fp32 projections (convolution in a kernel of its own).  fused: with one more sequence
    behind them, which brings the pass to the fewest rows that the fused projection takes; without it most of them are below."""
    if fused:
        counts = counts + [max(1, fused_rows(len(counts) + 1) - sum(counts))]
    torch, n = cuda, len(counts)
    w = synth.la_weights(77)
    out, conv = [], []
    for proj in (ops.PROJ_FP32, ops.PROJ_FP16):
        la = ops.LinearAttention(proj, max_batch=n, max_prefill_rows=sum(counts))
        la.set_weights(w)
        st = ops.LinearAttnState(1, n + 1)
        slots = [n - i for i in range(n)]
        y = []
        for call in range(2):
            x = torch.from_numpy(synth.hidden_states(77, f"edges.{call}", sum(counts))).cuda()
            y.append(la.forward_batch(x, st, 0, slots, counts))
        assert la.device_status() == 0
        out.append(torch.cat(y))
        conv.append(torch.stack([st.export_state(0, s)[1] for s in slots]))
    worst = ((out[1] - out[0]).norm(dim=1) / out[0].norm(dim=1)).max()
    assert worst <= ROW_REL, worst
    assert (conv[1] - conv[0]).norm() <= ROW_REL * conv[0].norm()


def test_more_sequences_than_the_tables_on_chip_hold(ops, cuda, synth):
    """Above 512 sequences their first rows and slots are read from memory.  The last one is as long as the fused projection needs."""
    torch, n = cuda, 514
    w = synth.la_weights(78)
    counts = [1 + i % 3 for i in range(n - 1)]
    counts.append(fused_rows(n) - sum(counts))
    x = torch.from_numpy(synth.hidden_states(78, "many", sum(counts))).cuda()
    out = []
    for proj in (ops.PROJ_FP32, ops.PROJ_FP16):
        la = ops.LinearAttention(proj, max_batch=n, max_prefill_rows=sum(counts))
        la.set_weights(w)
        st = ops.LinearAttnState(1, n)
        out.append([la.forward_batch(x, st, 0, list(range(n)), counts) for _ in range(2)][1])
    assert ((out[1] - out[0]).norm(dim=1) / out[0].norm(dim=1)).max() <= ROW_REL


@pytest.mark.parametrize("rows,fp16_kv", [(14 * 256, 1), (14 * 256 + 1, 0), (38 * 256 - 1, 1), (75 * 256 + 3, 1)])
def test_large_products_of_a_layer_equal_smaller_ones(ops, cuda, synth, rows, fp16_kv):
    """Attention layer on both sides of where its products move to the pairs (296 tiles are four rounds: the input projection above 14 x 256 rows, the output
    projection above 74 x 256), in one call and a sequence at a time: the same sums in the same order, whatever the kernel, so outputs agree to the bit."""
    torch = cuda
    w, per = synth.fa_weights(79), 1024
    counts = [per] * (rows // per) + ([rows % per] if rows % per else [])
    x = torch.from_numpy(synth.hidden_states(79, "large", rows)).cuda()
    out = []
    for chunk in (len(counts), 1):
        fa = ops.FullAttention(ops.PROJ_FP16, max_batch=len(counts), max_prefill_rows=rows)
        fa.set_weights(w)
        kv = ops.KVCache(1, len(counts), per, ops.KV_FP16 if fp16_kv else ops.KV_INT8)
        slots = [kv.allocate_sequence(per) for _ in counts]
        y, at = [], 0
        for i in range(0, len(counts), chunk):
            n = sum(counts[i:i + chunk])
            y.append(fa.forward_batch_prefill(x[at:at + n].contiguous(), kv, 0, slots[i:i + chunk], counts[i:i + chunk]))
            at += n
        out.append(torch.cat(y))
    assert torch.equal(out[0], out[1])


@pytest.mark.parametrize("kind,out_kind,rows,out,depth,taken", [
    (0, 2, 15 * 256, 5120, 1024, True), (0, 2, 14 * 256, 5120, 1024, False), (1, 1, 75 * 256, 1024, 2048, True), (1, 1, 74 * 256, 1024, 2048, False),
    (1, 1, 65536, 2048, 128, False), (1, 2, 65536, 2048, 504, False), (1, 2, 65536, 2048, 512, True), (1, 2, 65536, 2048, 4096, False),
    (0, 0, 65536, 2048, 1024, False), (2, 2, 65536, 2048, 1024, False), (1, 2, 65536, 2048, 1028, False),
])
def test_large_products_go_to_the_pairs_where_these_are_faster(ops, cuda, kind, out_kind, rows, out, depth, taken):
    """Kinds 0 fp16, 1 bf16, 2 fp32; four rounds of tiles on this device, depths 512 to 3584."""
    f = C.CDLL(ops.LIB_PATH)["_ZN4b20015gemm_pair_takesEPKviS1_S1_iNS_8ElemTypeES2_iii"]
    f.restype, f.argtypes = C.c_bool, [C.c_void_p, C.c_int, C.c_void_p, C.c_void_p, C.c_int, C.c_int, C.c_int, C.c_int, C.c_int, C.c_int]
    assert cuda.cuda.get_device_properties(0).multi_processor_count == 148
    assert f(16, depth, 32, 48, out, kind, out_kind, rows, out, depth) == taken


# ---- the kernel's forms one by one, against float64 of the same operands: tiles whole, halved and quartered (74 pairs: as many to a round) ------------------
def _operands(torch, rows, cols, dtype, seed, scale, pitch=None):
    g = torch.Generator(device="cuda").manual_seed(seed)
    whole = (torch.randn(rows, pitch or cols, device="cuda", generator=g) * scale).to(dtype)
    return whole, whole[:, :cols].double()


def _call(ops, torch, name, *args):
    """A launcher of the library on the current stream; its device word must stay clean."""
    word = torch.zeros(1, dtype=torch.int32, device="cuda")
    conv = [C.c_void_p(a.data_ptr()) if torch.is_tensor(a) else C.c_bool(a) if isinstance(a, bool) else C.c_int(a) for a in args]
    f = C.CDLL(ops.LIB_PATH)[name]
    assert f(C.c_void_p(torch.cuda.current_stream().cuda_stream), *conv, C.c_void_p(word.data_ptr())) == 0
    torch.cuda.synchronize()
    assert int(word) == 0


# Sums of K fp32 products: within 2^-18 of the sum of their magnitudes (K <= 4096 roundings of 2^-24 in some order, at most sqrt(K) of them in one direction).
SUM = 2.0 ** -18


@pytest.mark.parametrize("form", ["fp16 silu", "bf16 silu", "bf16 gelu"])
@pytest.mark.parametrize("rows,ff,depth", [
    (130, 64, 64), (257, 264, 72),              # one tile, five: quarters
    (130, 4712, 136),                           # 37 tiles: halves
    (600, 2400, 1024),                          # 57: one part-empty round of whole tiles
    (2304, 1160, 136), (2305, 1304, 72), (2600, 1384, 200),          # 90, 110, 121: a whole round, then quarters, halves, whole ones
    (4099, 2424, 520),                          # 323: four rounds and halves
])
def test_feed_forward_forms(ops, cuda, form, rows, ff, depth):
    """Gate rows in front of up rows (bf16) and groups of 32 of each (fp16).  Rounding to 11 (fp16) or 8 bits (bf16) moves a value by up to 2^-11 or 2^-8 of it.
    bf16 products are rounded in front of the activation: gate, up and the result by so much each, where the activations' slopes are at most 1.13."""
    torch = cuda
    half, silu = form.startswith("fp16"), form.endswith("silu")
    dtype, unit = (torch.float16, 2.0 ** -11) if half else (torch.bfloat16, 2.0 ** -8)
    if half:
        ff = -(-ff // 32) * 32
    x, xd = _operands(torch, rows, depth, dtype, 1, 1.0)
    w, wd = _operands(torch, 2 * ff, depth, dtype, 2, 1.5 / depth ** 0.5)
    gate, up = (wd.view(-1, 2, 32, depth)[:, i].reshape(ff, depth) for i in (0, 1)) if half else (wd[:ff], wd[ff:])
    y = torch.full((rows + 2, ff), 7.0, dtype=dtype, device="cuda")
    _call(ops, torch, "_ZN4b2008gemm_gluEP11CUstream_stNS_8ElemTypeEiPKvS4_PviiibPi", 0 if half else 1, 1 if silu else 0, x, w, y, rows, ff, depth, not half)
    assert (y[rows:] == 7.0).all()
    g, u = xd @ gate.t(), xd @ up.t()
    f = g * torch.sigmoid(g) if silu else torch.nn.functional.gelu(g, approximate="tanh")
    want = f * u
    sums = SUM * (1.13 * (xd.abs() @ gate.abs().t()) * u.abs() + (xd.abs() @ up.abs().t()) * f.abs())
    rounded = unit * want.abs() + (0.0 if half else unit * (1.13 * (g * u).abs() + want.abs()))
    excess = (y[:rows].double() - want).abs() - 1.05 * (rounded + sums) - 1e-5       # two roundings compound; the special functions are good to 2^-20
    assert excess.max() <= 0, float(excess.max())


@pytest.mark.parametrize("kind,out_kind", [(0, 2), (1, 1), (1, 2)])
@pytest.mark.parametrize("rows,out,depth,x_more,y_more", [
    (255, 264, 72, 0, 0), (1025, 264, 520, 8, 16),                   # one and two columns of tiles, quarters
    (9 * 256 + 1, 4 * 256 - 8, 128, 0, 8),                           # 40: whole
    (8 * 256 + 3, 10 * 256, 512, 24, 0), (9 * 256, 11 * 256 + 40, 200, 0, 24),       # 90: a round and quarters; 108: and halves
    (15 * 256 - 5, 20 * 256, 1024, 0, 0),                            # 300
])
def test_plain_forms(ops, cuda, kind, out_kind, rows, out, depth, x_more, y_more):
    """fp16 to fp32, bf16 to bf16 and fp32, with row pitches on either side; what lies outside the matrix is left alone."""
    torch = cuda
    dtype, out_dtype = (torch.float16 if kind == 0 else torch.bfloat16), (torch.float32 if out_kind == 2 else torch.bfloat16)
    x, xd = _operands(torch, rows, depth, dtype, 3, 1.0, depth + x_more)
    w, wd = _operands(torch, out, depth, dtype, 4, 1.0)
    y = torch.full((rows + 1, out + y_more), 7.0, dtype=out_dtype, device="cuda")
    _call(ops, torch, "_ZN4b2009gemm_pairEP11CUstream_stPKviS3_PviNS_8ElemTypeES5_iiiPi", x, depth + x_more, w, y, out + y_more, kind, out_kind, rows, out, depth)
    assert (y[rows:] == 7.0).all() and (y[:, out:] == 7.0).all()
    want, sums = xd @ wd.t(), SUM * (xd.abs() @ wd.abs().t())
    excess = (y[:rows, :out].double() - want).abs() - sums - (2.0 ** -8 * want.abs() * 1.01 if out_kind == 1 else 0.0)       # 8 bits
    assert excess.max() <= 0, float(excess.max())
