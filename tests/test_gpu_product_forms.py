"""GPU parity of prompts whose products take each kernel and shape that the rule for prompts gives them (csrc/pair_plan.h,
product_shape): test_product_plan.py checks that these do."""
import pytest

from conftest import rel_err
from webgpt_b200 import synth

pytestmark = pytest.mark.gpu

PROMPTS = [(384, 70), (384, 700), (768, 420), (768, 1023), (1216, 250), (1600, 70), (1600, 200), (1600, 333), (1600, 700)]


@pytest.mark.parametrize("E,n", PROMPTS)
def test_prompt(oracle, E, n):
    """Logits behind a prompt and of one more token over the cache it left; bound as for other prompts on pairs."""
    import numpy as np
    from webgpt_b200 import GPT
    params = dict(n_layer=1, n_head=E // 64, n_embd=E, n_ctx=n + 1, vocab_size=264)
    w = synth.make_weights(params, seed=n, std=0.05, ln_random=True)
    ids = synth.make_tokens(264, n + 1, seed=7)
    gpt = GPT(None, params=params, weights=w)
    gpt.initialize()
    try:
        m = oracle.Model(params, synth.weight_list(params, w))
        s = gpt.session()
        s.reset()
        assert rel_err(s.forward(ids[:n])[0], m.run(ids[:n])) < 5e-5
        assert rel_err(s.forward(ids[n:])[0], m.run(np.array(ids))) < 5e-5
    finally:
        gpt.destroy()
