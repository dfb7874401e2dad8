"""GPU parity of the product of few rows against a matrix that streams from HBM (gemm_stream_kernel), through the
de-embedding of a batch, at the edges of its tiles, runs and row counts."""
import numpy as np
import pytest

from conftest import rel_err
from webgpt_b200 import synth

pytestmark = pytest.mark.gpu

# Two pieces of 32 features for each of 148 CTAs and one more feature; a run's last tile of 32, 64 or 96 features and of a
# single live one; runs of up to five tiles, so that both accumulators come round to both parities; K of 1, 2.5, 3, 6, 12 and 25
# k-blocks, more than a ring holds; rows off 16 and the largest row tile; vocabularies of fewer pieces than SMs, and of one to two.
SHAPES = [(64, 1, 50, 6), (384, 6, 65, 96), (64, 1, 9472, 6), (64, 1, 9473, 16), (160, 5, 9503, 17), (192, 3, 18977, 33), (192, 3, 19000, 64), (384, 6, 14209, 48),
          (192, 3, 33001, 65), (384, 6, 50257, 128), (160, 5, 50257, 113),
          (64, 1, 95011, 24), (768, 12, 9473, 7), (768, 12, 14209, 128), (1600, 25, 9601, 33), (512, 8, 1000, 96), (384, 6, 4733, 80)]


@pytest.mark.parametrize("E,H,V,rows", SHAPES)
def test_logits_of_a_batch(oracle, E, H, V, rows):
    """Logits of every sequence of a batch against the oracle, whole rows of them: behind a prompt, behind one decode step, and
    the ids that a greedy completion takes from both (the second from a captured step). The bound is that of the other batch
    tests: operands exact to 2^-22 and FP32 sums that truncate, K / 16 steps, come to 5e-6 of the largest logit at K = 1600; the
    block ahead of the product brings as much again."""
    from webgpt_b200 import GPT
    params = dict(n_layer=1, n_head=H, n_embd=E, n_ctx=8, vocab_size=V)
    w = synth.make_weights(params, seed=rows, std=0.05, ln_random=True)
    prompts = np.stack([synth.make_tokens(V, 2, seed=5, stream=i) for i in range(rows)])
    gpt = GPT(None, params=params, weights=w)
    gpt.initialize()
    try:
        s = gpt.session(rows)
        s.reset()
        got = s.forward(prompts)
        m = oracle.Model(params, synth.weight_list(params, w))
        ref = np.stack([m.run(p) for p in prompts])
        for i in range(rows):
            assert rel_err(got[i], ref[i]) < 5e-5, i
        first = np.argmax(got, 1).astype(np.uint32)
        got2 = s.forward(first[:, None])
        ref2 = np.stack([m.run(np.append(p, t)) for p, t in zip(prompts, first)])
        for i in range(rows):
            assert rel_err(got2[i], ref2[i]) < 5e-5, i
        s.reset()
        ids = s.generate_greedy(prompts, 2)
        for i in range(rows):
            for k, r in enumerate((ref[i], ref2[i])):
                best = np.sort(r)[-2:]
                if best[1] - best[0] <= 5e-5 * np.abs(r).max():
                    break  # the completion may go on from another token
                assert ids[i, k] == int(np.argmax(r)), (i, k)
    finally:
        gpt.destroy()
