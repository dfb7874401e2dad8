"""GPU parity of LayerNorm at the edges of its forms: one, two or four warps a row, and how many values a lane holds."""
import numpy as np
import pytest

from conftest import rel_err
from webgpt_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", (4, 124, 384, 388, 768, 772, 1600, 1664, 1668, 2044, 2048, 2052))
def test_operator_rows(N):
    """The operator's form against float64. A row's mean and deviations are sums of N FP32 terms, at most 64 per lane and a
    butterfly: 75 roundings at most of terms that are at most the largest value, 75 x 2^-24 of that for the mean, as much relative
    for the variance, and five more roundings behind it."""
    from webgpt_b200 import Device, _lib
    rng = np.random.default_rng(N)
    dev = Device(0)
    try:
        g, b = rng.standard_normal(N, dtype=np.float32), rng.standard_normal(N, dtype=np.float32)
        g_d, b_d = dev.tensor(g), dev.tensor(b)
        for rows in (1, 3, 4, 5, 130):
            x = (rng.standard_normal((rows, N)) * 2 + rng.uniform(-3, 3, (rows, 1))).astype(np.float32)
            x_d, o_d = dev.tensor(x), dev.buffer(rows * N * 4)
            _lib.call("wgpt_layernorm", dev.handle, rows, N, x_d.ptr, g_d.ptr, b_d.ptr, o_d.ptr)
            got = o_d.read(np.float32, rows * N).reshape(rows, N)
            x_d.destroy(), o_d.destroy()
            z = x.astype(np.float64)
            d = z - z.mean(1, keepdims=True)
            sd = np.sqrt((d * d).mean(1, keepdims=True) + 1e-5)
            top = np.abs(z).max(1, keepdims=True)
            bound = 2.0 ** -24 * ((75 * top + 80 * np.abs(d)) / sd * np.abs(g) + np.abs(d / sd * g) + np.abs(b) + np.abs(d / sd * g + b))
            assert (np.abs(got - (d / sd * g + b)) <= bound).all(), rows
    finally:
        dev.destroy()


# n_embd, heads: values per lane at four and two warps a row (1, 2, 3, 4, 7) and past what two warps hold
WIDTHS = [(64, 1), (384, 6), (512, 8), (576, 9), (768, 12), (1024, 16), (1088, 17), (1600, 25), (1856, 29), (2048, 32)]


@pytest.mark.parametrize("E,H", WIDTHS)
def test_rows_of_a_prompt(oracle, E, H):
    """The form that writes pairs, inside a model: prompts either side of 1536 and of 4096 rows (four, two, one warp a row), so
    that the last token of every sequence has passed each form. Bound as for other prompts on pairs."""
    from webgpt_b200 import GPT
    V = 72
    params = dict(n_layer=1, n_head=H, n_embd=E, n_ctx=128, vocab_size=V)
    w = synth.make_weights(params, seed=E, std=0.05, ln_random=True)
    gpt = GPT(None, params=params, weights=w)
    gpt.initialize()
    try:
        m = oracle.Model(params, synth.weight_list(params, w))
        for n_seq, n_tok in ((1, 70), (12, 128), (13, 119), (32, 128), (33, 125)):  # 70, 1536, 1547, 4096, 4125 rows
            prompts = np.stack([synth.make_tokens(V, n_tok, seed=6, stream=i) for i in range(n_seq)])
            s = gpt.session(n_seq)
            s.reset()
            got = s.forward(prompts)
            for i in {0, n_seq // 2, n_seq - 1}:
                assert rel_err(got[i], m.run(prompts[i])) < 5e-5, (n_seq, n_tok, i)
    finally:
        gpt.destroy()
