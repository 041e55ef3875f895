"""GPU: prompt-sized products on pairs of CTAs with their successor in the epilogue, at the edges of their tiles (256 rows, 128 outputs, parts of 32) and of
their dispatch (more than 128 rows)."""
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


@pytest.mark.parametrize("seqs,tokens,inter", [(2, 65, 64), (3, 85, 192), (4, 64, 1088), (7, 37, 128), (9, 57, 3584), (2, 128, 2048 + 64)])
def test_prompts_in_one_pass_against_one_by_one(ops, cuda, synth, seqs, tokens, inter):
    """Rows of one pass: 130, 255, 256, 259, 513, 256; one by one they are at most 128, on the library products."""
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
