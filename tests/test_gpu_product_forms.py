"""GPU parity of prompts whose products take each kernel and shape that the rule for prompts gives them (csrc/pair_plan.h,
product_shape): test_product_plan.py checks that these do."""
import numpy as np
import pytest

from conftest import rel_err
from webgpt_b200 import synth

pytestmark = pytest.mark.gpu

PROMPTS = [(384, 70), (384, 700), (768, 420), (768, 1023), (1216, 250), (1600, 70), (1600, 200), (1600, 333), (1600, 700), (1600, 800)]


@pytest.mark.parametrize("E,n", PROMPTS)
def test_prompt(oracle, E, n):
    """Logits behind a prompt and of one more token over the cache it left; bound as for other prompts on pairs."""
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


# n_embd, tokens, truncating additions to one large sum of the up and of the down projection, by the shapes that these products take
# outside a prompt (test_product_plan.py): rows at which the cheapest shape by estimate has three times as many for the down projection
TRUNCATIONS = [(768, 1000, 144, 96), (1024, 700, 192, 128), (1280, 600, 240, 160), (1600, 420, 300, 200), (1600, 512, 300, 200),
               (2048, 300, 384, 256)]


def block64(w, E, H, ids):
    """The rows behind one block in float64."""
    f = lambda k: w["transformer." + k].astype(np.float64)  # noqa: E731
    ln = lambda x, k: ((x - x.mean(-1, keepdims=True)) / np.sqrt(x.var(-1, keepdims=True) + 1e-5)  # noqa: E731
                       * f(k + ".weight") + f(k + ".bias"))
    n = len(ids)
    x = f("wte.weight")[ids] + f("wpe.weight")[:n]
    qkv = ln(x, "h.0.ln_1") @ f("h.0.attn.c_attn.weight") + f("h.0.attn.c_attn.bias")
    q, k, v = (a.reshape(n, H, -1).transpose(1, 0, 2) for a in np.split(qkv, 3, 1))
    s = np.where(np.tril(np.ones((n, n), bool)), q @ k.transpose(0, 2, 1) / np.sqrt(E / H), -np.inf)
    s = np.exp(s - s.max(-1, keepdims=True))
    o = ((s / s.sum(-1, keepdims=True)) @ v).transpose(1, 0, 2).reshape(n, E)
    x = x + o @ f("h.0.attn.c_proj.weight") + f("h.0.attn.c_proj.bias")
    u = ln(x, "h.0.ln_2") @ f("h.0.mlp.c_fc.weight") + f("h.0.mlp.c_fc.bias")
    g = 0.5 * u * (1 + np.tanh(np.sqrt(2 / np.pi) * (u + 0.044715 * u ** 3)))
    return x + g @ f("h.0.mlp.c_proj.weight") + f("h.0.mlp.c_proj.bias")


@pytest.mark.parametrize("E,n,up,down", TRUNCATIONS)
def test_sums_truncate_no_more_often(E, n, up, down):
    """The rows behind a block whose down projection prevails (some fifteen times what it is added to), in 2-norm. A truncation takes at
    most 2^-23 of the partial sum and half of that in the mean, a partial sum of m of N random terms is sqrt(m / N) of the whole
    and the mean square over m a third: 2^-24 / sqrt(3) for each. The up projection's own sums are a fifth of what GELU gets,
    the rest being its bias: a fifth of its losses. Pairs are exact to 2^-22, three products; FP32 between the kernels as
    much again."""
    from webgpt_b200 import GPT
    H = E // 64
    params = dict(n_layer=1, n_head=H, n_embd=E, n_ctx=n, vocab_size=264)
    w = synth.make_weights(params, seed=n, std=0.05, ln_random=True)
    w["transformer.h.0.attn.c_proj.weight"] *= np.float32(0.1)
    w["transformer.h.0.mlp.c_fc.weight"] *= np.float32(4 / E ** 0.5)
    w["transformer.h.0.mlp.c_fc.bias"] *= np.float32(20)
    ids = synth.make_tokens(264, n, seed=8)
    ref = block64(w, E, H, ids)
    gpt = GPT(None, params=params, weights=w)
    gpt.initialize()
    try:
        s = gpt.session()
        s.reset()
        s.forward(ids, want_logits=False)
        got = s.tap()[:n].astype(np.float64)
    finally:
        gpt.destroy()
    assert np.linalg.norm(got - ref) < (2 ** -24 / 3 ** 0.5 * (down + up / 5) + 6 * 2 ** -22) * np.linalg.norm(ref)
