"""GPU parity of the kernels on half-precision pairs, of the ring GEMV and of the cluster sampling kernel, at the sizes
where their tiles, slices and dispatch rules have edges."""
import ctypes as C

import numpy as np
import pytest

from conftest import rel_err
from webgpt_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    from webgpt_b200 import Device
    d = Device(0)
    yield d
    d.destroy()


def matmul(dev, A, W, b=None):
    from webgpt_b200 import _lib
    M, K = A.shape
    N = W.shape[1]
    a_d, w_d, o_d = dev.tensor(A), dev.tensor(W), dev.buffer(M * N * 4)
    b_d = dev.tensor(b) if b is not None else None
    _lib.call("wgpt_matmul", dev.handle, M, N, K, a_d.ptr, w_d.ptr, b_d.ptr if b_d else None, o_d.ptr)
    _lib.call("wgpt_device_check", dev.handle)
    return o_d.read(np.float32, M * N).reshape(M, N)


# (rows, K, N): one row tile and its neighbours, 256-row tiles, N off every tile width, K off 16, 64 and the cluster's
# slices (a strip of more than 8 x 192 rows of K, fewer k-blocks than slices)
SHAPES = [(32, 8, 8), (33, 72, 40), (64, 768, 136), (65, 200, 264), (127, 1600, 128), (128, 3072, 8), (129, 64, 4800),
          (255, 1544, 520), (257, 768, 768), (513, 136, 2312), (1100, 768, 3072)]


@pytest.mark.parametrize("M,K,N", SHAPES)
def test_product_of_pairs_error_bound(dev, M, K, N):
    """Elementwise bound from the representation. Per product: each operand is off by at most 2^-22 of itself, the dropped
    h1 g1 is at most 2^-22, so 3 * 2^-22. Per accumulation: the FP32 accumulator of an MMA step is truncated, 2^-23 of the
    sum so far, 3 K / 16 steps. Both against sum |x w|; 2^-23 more for what is stored. (Operands below 2^-17 of their row's
    largest carry the absolute error 2^-40 of it, K terms of that at most.)"""
    rng = np.random.default_rng(M + 7 * K + N)
    A = rng.standard_normal((M, K), dtype=np.float32)
    W = (rng.standard_normal((K, N), dtype=np.float32) * np.exp2(rng.integers(-6, 7, N))).astype(np.float32)
    ref = A.astype(np.float64) @ W.astype(np.float64)
    mag = np.abs(A).astype(np.float64) @ np.abs(W).astype(np.float64)
    top = np.abs(A).max(1)[:, None].astype(np.float64) * np.abs(W).max(0)[None, :] * K
    bound = (3 * 2.0 ** -22 + (3 * K / 16 + 2) * 2.0 ** -23) * mag + 2.0 ** -39 * top
    got = matmul(dev, A, W)
    assert (np.abs(got - ref) <= bound).all()
    assert np.array_equal(matmul(dev, A, W), got)  # deterministic
    # powers of two per row and per column pass through exactly
    r, c = np.exp2(rng.integers(-30, 31, M)), np.exp2(rng.integers(-30, 31, N))
    scaled = matmul(dev, (A * r[:, None]).astype(np.float32), (W * c[None, :]).astype(np.float32))
    assert np.array_equal(scaled, (got * r[:, None] * c[None, :]).astype(np.float32))


K_OVER_TWO_PAIRS = [(700, 1608, 1608), (900, 1160, 1304), (250, 1160, 3080), (700, 1544, 1608), (512, 3080, 2312)]
WIDTH_OVER_TWO_PAIRS = [("up", 1216, (238, 250, 256)), ("qkv", 1600, (238, 250, 256))]  # the product, n_embd and tokens


@pytest.mark.parametrize("M,K,N", K_OVER_TWO_PAIRS)
def test_product_of_pairs_with_k_over_two_pairs(dev, M, K, N):
    """Fewer tiles than CTA pairs: two pairs share a tile's K (26 k-blocks, 19, 25 and 49), ragged rows and columns, one row tile
    and several. test_pair_plan.py follows the rule; (900, 1160, 1304) takes this form on 36 clusters of four or more only."""
    test_product_of_pairs_error_bound(dev, M, K, N)


@pytest.mark.parametrize("E,n", [(E, n) for _, E, tokens in WIDTH_OVER_TWO_PAIRS for n in tokens])
def test_model_products_with_k_over_two_pairs(oracle, E, n):
    """K over two pairs with what a model's products do at their end: q, k and v as pairs and into the cache, GELU and pairs. The
    logits behind the prompt, and of two more tokens over the cache it left; bound as in test_prompt_lengths."""
    from webgpt_b200 import GPT
    from webgpt_b200.model import Session
    p = dict(n_layer=1, n_head=E // 64, n_embd=E, n_ctx=260, vocab_size=512)
    w = synth.make_weights(p, seed=61, std=0.04, ln_random=True)
    gpt, m = GPT(None, params=p, weights=w), oracle.Model(p, synth.weight_list(p, w))
    gpt.initialize()
    s = Session(gpt, 1)
    try:
        ids = synth.make_tokens(512, n + 2, seed=62)
        for a, b in ((0, n), (n, n + 1), (n + 1, n + 2)):
            assert rel_err(s.forward(ids[a:b])[0], m.run(ids[:b])) < 2e-5, b
    finally:
        s.destroy()
        gpt.destroy()


def test_deembedding_of_a_small_odd_vocabulary(oracle):
    """Two pairs a tile again, rows that are no multiple of 16 bytes."""
    from webgpt_b200 import GPT
    from webgpt_b200.model import Session
    p = dict(n_layer=1, n_head=12, n_embd=768, n_ctx=32, vocab_size=515)
    w = synth.make_weights(p, seed=23, std=0.05, ln_random=True)
    gpt, m = GPT(None, params=p, weights=w), oracle.Model(p, synth.weight_list(p, w))
    gpt.initialize()
    s = Session(gpt, 7)
    try:
        ids = np.stack([synth.make_tokens(p["vocab_size"], 9, seed=24, stream=i) for i in range(7)])
        lg = s.forward(ids)
        for i in range(7):
            assert rel_err(lg[i], m.run(ids[i])) < 2e-5
    finally:
        s.destroy()
        gpt.destroy()


@pytest.mark.parametrize("M,N,a,w", [(40, 72, 128, -124), (40, 72, -124, 128), (600, 520, 128, -124), (40, 72, 114, 10),
                                     (40, 72, -60, -60)])
def test_product_of_pairs_at_the_ends_of_the_exponent_range(dev, M, N, a, w):
    """Operands of up to 2^a and 2^w, the largest FP32 number among them, whose products are finite: bound as above. The
    largest values fit the scaled form, and a row's and a column's power of two come back without passing infinity."""
    rng = np.random.default_rng(M + N + abs(a))
    K, one = 136, 1 - 2.0 ** -24
    A, W = (rng.standard_normal((M, K)) / 8).clip(-one, one), (rng.standard_normal((K, N)) / 8).clip(-one, one)
    A[3, 5], W[7, 6] = one, -one
    A, W = (A * 2.0 ** a).astype(np.float32), (W * 2.0 ** w).astype(np.float32)
    assert np.isfinite(A).all() and np.isfinite(W).all()
    ref = A.astype(np.float64) @ W.astype(np.float64)
    mag = np.abs(A).astype(np.float64) @ np.abs(W).astype(np.float64)
    top = np.abs(A).max(1)[:, None].astype(np.float64) * np.abs(W).max(0)[None, :].astype(np.float64) * K
    got = matmul(dev, A, W)
    assert (np.abs(got - ref) <= (3 * 2.0 ** -22 + (3 * K / 16 + 2) * 2.0 ** -23) * mag + 2.0 ** -39 * top).all()


@pytest.mark.parametrize("M,K,N", [(9, 768, 136), (12, 3072, 768), (13, 72, 40), (16, 40, 2304), (17, 1600, 128), (24, 8, 8),
                                   (25, 768, 768), (31, 3080, 72)])
def test_product_of_9_to_31_rows_is_fp32(dev, M, K, N):
    """One or two row groups of 12 or 16, the last one ragged, K slices of uneven length. FP32 sums: at most one rounding of
    2^-24 per term and per addition of a partial sum."""
    rng = np.random.default_rng(M + K + N)
    A = rng.standard_normal((M, K), dtype=np.float32)
    W = rng.standard_normal((K, N), dtype=np.float32)
    b = rng.standard_normal(N, dtype=np.float32)
    ref = A.astype(np.float64) @ W.astype(np.float64) + b
    bound = (K + 20) * 2.0 ** -24 * (np.abs(A).astype(np.float64) @ np.abs(W).astype(np.float64) + np.abs(b))
    got = matmul(dev, A, W, b)
    assert (np.abs(got - ref) <= bound).all()
    assert rel_err(got, ref) < 4e-6  # and not a product of split operands: sqrt(K / 3) 2^-24 of a sum, four times over


@pytest.mark.parametrize("M,K,N", [(9, 64, 72), (31, 96, 264), (40, 96, 264), (300, 776, 200)])
def test_products_of_integers_are_exact(dev, M, K, N):
    """Integers of at most 11 bits are exact in the first plane and their sums in FP32: any misplaced element shows."""
    A = ((np.arange(M)[:, None] * 7 + np.arange(K)[None, :] * 3) % 11 - 5).astype(np.float32)
    W = ((np.arange(K)[:, None] * 5 + np.arange(N)[None, :]) % 13 - 6).astype(np.float32)
    b = np.arange(N, dtype=np.float32)
    assert np.array_equal(matmul(dev, A, W, b).astype(np.float64), A.astype(np.float64) @ W + b)


@pytest.mark.parametrize("M,K,N", [(33, 3072, 136), (64, 6400, 136), (128, 6400, 264), (257, 3080, 72), (600, 1600, 520)])
def test_products_of_long_integers_are_exact(dev, M, K, N):
    """Thirteen-bit integers take both planes and their sums against -1, 0 and 1 stay exact in FP32: a correction product
    that goes missing in any stage of the ring, k-block or slice of a long K shows, from either side."""
    rng = np.random.default_rng(M + K)
    big = lambda *s: (rng.integers(4097, 4103, s) * rng.choice((-1, 1), s)).astype(np.float32)  # noqa: E731
    unit = lambda *s: rng.integers(-1, 2, s).astype(np.float32)  # noqa: E731
    for A, W in ((big(M, K), unit(K, N)), (unit(M, K), big(K, N))):
        assert np.array_equal(matmul(dev, A, W).astype(np.float64), A.astype(np.float64) @ W)
    # the same rows against codes of one plane
    from webgpt_b200 import _lib
    A, q = big(M, K), unit(K, N).astype(np.int8)
    if K % 16 == 0:
        h = C.c_void_p()
        p_d, s_d = dev.tensor(q.view(np.uint32)), dev.tensor(np.ones(N, np.float32))
        a_d, o_d = dev.tensor(A), dev.buffer(M * N * 4)
        _lib.call("wgpt_int8_weight_create", dev.handle, K, N, p_d.ptr, s_d.ptr, C.byref(h))
        _lib.call("wgpt_int8_matmul_w", dev.handle, M, h, a_d.ptr, o_d.ptr)
        got = o_d.read(np.float32, M * N).reshape(M, N)
        _lib.call("wgpt_int8_weight_destroy", h)
        assert np.array_equal(got.astype(np.float64), A.astype(np.float64) @ q)


@pytest.mark.parametrize("T,E,H", [(32, 128, 2), (63, 64, 1), (65, 128, 2), (128, 192, 3), (129, 128, 2), (200, 128, 4),
                                   (321, 64, 1)])
def test_attention_operator_on_pairs(dev, oracle, T, E, H):
    """Query tiles of 64, key tiles shared by two warp groups, head sizes with and without the pair attention."""
    from webgpt_b200 import _lib
    rng = np.random.default_rng(T + E)
    x = rng.standard_normal((T, E), dtype=np.float32)
    ws = [(rng.standard_normal((E, E), dtype=np.float32) * 0.15).astype(np.float32) for _ in range(4)]
    bs = [rng.standard_normal(E, dtype=np.float32) for _ in range(4)]
    scale = float(np.float32(1 / np.sqrt(E // H)))
    d = [dev.tensor(a) for pair in zip(ws, bs) for a in pair]
    x_d, o_d = dev.tensor(x), dev.buffer(T * E * 4)
    _lib.call("wgpt_attention", dev.handle, T, E, scale, H, E // H, x_d.ptr, *[t.ptr for t in d], o_d.ptr)
    _lib.call("wgpt_device_check", dev.handle)
    ref = oracle.attention(x, H, scale, ws[0], bs[0], ws[1], bs[1], ws[2], bs[2], ws[3], bs[3])
    # three products behind one another, each within ~1e-6 of its largest value at these K; 2e-5 is the operators' bound
    assert rel_err(o_d.read(np.float32, T * E).reshape(T, E), ref) < 2e-5


def attention64(x, H, scale, wq, wk, wv, wo):
    """Causal attention of one window in double precision, no biases."""
    T, E = x.shape
    q, k, v = ((x @ w).reshape(T, H, E // H).transpose(1, 0, 2) for w in (wq, wk, wv))
    s = np.where(np.tri(T, dtype=bool), q @ k.transpose(0, 2, 1) * scale, -np.inf)
    p = np.exp(s - s.max(-1, keepdims=True))
    return ((p / p.sum(-1, keepdims=True)) @ v).transpose(1, 0, 2).reshape(T, E) @ wo


@pytest.mark.parametrize("T,E,H", [(64, 64, 1), (130, 128, 2), (200, 192, 3), (450, 128, 2)])
@pytest.mark.parametrize("rows,b", [("last", 24), ("first", 24), ("one in seven", 24), ("any", 14), ("last", 62)])
def test_attention_operator_rows_of_any_size(dev, T, E, H, rows, b):
    """Each row against its own magnitude, beside rows 2^b times its size: before it, behind it and between. The scale keeps
    the largest scores near one, so that no row's softmax amplifies its operands' last bits. Bound as in
    test_attention_operator_on_pairs; later rows leave no trace in earlier ones."""
    from webgpt_b200 import _lib
    rng = np.random.default_rng(T + E + b)
    x = rng.standard_normal((T, E))
    at = {"last": [T - 1], "first": [0], "one in seven": range(3, T, 7), "any": range(T)}[rows]
    x[at] *= 2.0 ** (rng.integers(-b, b + 1, len(at)) if rows == "any" else np.full(len(at), b))[:, None]
    x = x.astype(np.float32)
    ws = [(rng.standard_normal((E, E)) * 0.15).astype(np.float32) for _ in range(4)]
    scale = 2.0 ** -(2 * b + 1)
    zero = dev.tensor(np.zeros(E, np.float32))
    d = [dev.tensor(w) for w in ws]

    def run(rows_in):
        x_d, o_d = dev.tensor(rows_in), dev.buffer(T * E * 4)
        _lib.call("wgpt_attention", dev.handle, T, E, scale, H, E // H, x_d.ptr, *[p for w in d for p in (w.ptr, zero.ptr)], o_d.ptr)
        _lib.call("wgpt_device_check", dev.handle)
        return o_d.read(np.float32, T * E).reshape(T, E)

    got, ref = run(x), attention64(x.astype(np.float64), H, scale, *(w.astype(np.float64) for w in ws))
    err = np.abs(got - ref).max(1) / np.abs(ref).max(1)
    assert err.max() < 2e-5, (int(err.argmax()), float(err.max()))
    other = x.copy()
    other[T - 1] *= np.float32(0.5)
    assert np.array_equal(run(other)[:T - 1], got[:T - 1])


@pytest.fixture(scope="module")
def model64(oracle):
    """Head size 64, two layers: every prefill and decode path of the model takes it."""
    from webgpt_b200 import GPT
    params = dict(n_layer=2, n_head=3, n_embd=192, n_ctx=384, vocab_size=4104)
    w = synth.make_weights(params, seed=17, std=0.08, ln_random=True)
    gpt = GPT(None, params=params, weights=w)
    gpt.initialize()
    yield gpt, oracle.Model(params, synth.weight_list(params, w)), params
    gpt.destroy()


@pytest.mark.parametrize("n", [8, 9, 16, 63, 64, 65, 128, 129, 300, 384])
def test_prompt_lengths(model64, n):
    gpt, m, p = model64
    ids = synth.make_tokens(p["vocab_size"], n, seed=n)
    assert rel_err(gpt.run(ids), m.run(ids)) < 2e-5  # two layers of the products above


@pytest.mark.parametrize("n", [65, 96, 128, 129, 193])
def test_prompts_of_many_sequences(model64, n):
    """More query tiles than SMs: one group of softmax warps per CTA, key tiles from the first to the diagonal, ragged last
    tiles beside the next sequence's rows; a second chunk meets the cache that the first one left."""
    from webgpt_b200.model import Session
    gpt, m, p = model64
    n_seq = 52
    ids = np.stack([synth.make_tokens(p["vocab_size"], n + 70, seed=54, stream=i) for i in range(n_seq)])
    s = Session(gpt, n_seq)
    try:
        for a, b in ((0, n), (n, n + 70)):
            lg = s.forward(ids[:, a:b])
            for i in (0, 1, n_seq - 1):
                assert rel_err(lg[i], m.run(ids[i, :b])) < 2e-5, (i, b)
    finally:
        s.destroy()


@pytest.mark.parametrize("n,n_seq", [(65, 1), (130, 1), (256, 1), (129, 52)])
def test_prefill_attention_keeps_small_probabilities(oracle, n, n_seq):
    """The first key takes a row's probability and its values are zero, so the output is what the other keys add with
    probabilities of about 2^-24.5; everything behind the attention is linear or a normalisation.

    Bound, relative: a probability is off by 2^-40 of the largest at most, n of them in one direction against a sum of n random
    ones are sqrt(n) 2^-15.5 (3.4e-4 at 256 keys); the output's own pair, 2^-40 of a bound that is 34 times the values' size at
    most, adds 9e-5 at 64 keys."""
    from webgpt_b200 import GPT
    from webgpt_b200.model import Session
    E, rng = 128, np.random.default_rng(31)
    p = dict(n_layer=1, n_head=2, n_embd=E, n_ctx=256, vocab_size=520)
    w = {k: np.zeros(synth.tensor_shape(p, k), np.float32) for k in synth.tensor_names(p)}
    for k in ("ln_f", "h.0.ln_1", "h.0.ln_2"):
        w[f"transformer.{k}.weight"][:] = 1
    wte, wpe = w["transformer.wte.weight"], w["transformer.wpe.weight"]
    wte[1:, 1:] = rng.standard_normal((519, E - 1))
    wpe[0, 0] = 100  # token 0 at position 0: normalised to 11.3 in dimension 0, equal values in all others
    qkv, bias = w["transformer.h.0.attn.c_attn.weight"], w["transformer.h.0.attn.c_attn.bias"]
    qkv[1:, :2 * E] = rng.standard_normal((E - 1, 2 * E)) * 0.05
    for h in (0, 64):
        qkv[1:, h] = 0
        bias[h], qkv[0, E + h] = 4, 3.02  # 4 x 3.02 x 11.27 / 8 = 17.0, e^-17.0 = 2^-24.5
    for d in range(E):  # differences of two dimensions: exactly zero at position 0
        m, v = 1 + d % 63, rng.uniform(0.5, 1.5)
        qkv[2 * m, 2 * E + d], qkv[2 * m + 1, 2 * E + d] = v, -v
    w["transformer.h.0.attn.c_proj.weight"][:] = rng.standard_normal((E, E)) * 2.0 ** 26 / np.sqrt(E)
    ids = np.concatenate([np.zeros((n_seq, 1)), rng.integers(1, 520, (n_seq, n - 1))], 1).astype(np.uint32)
    gpt, m = GPT(None, params=p, weights=w), oracle.Model(p, synth.weight_list(p, w))
    gpt.initialize()
    s = Session(gpt, n_seq)
    try:
        lg = s.forward(ids)
        for i in {0, n_seq - 1}:
            assert rel_err(np.asarray(lg).reshape(n_seq, -1)[i], m.run(ids[i])) < 1e-3
    finally:
        s.destroy()
        gpt.destroy()


@pytest.mark.parametrize("n_seq", [2, 5, 6, 16, 17, 48, 49, 64, 65, 70])
def test_decode_rows(model64, n_seq):
    """Row tiles of 16, 32, 48 and 64, the step to the planes of more rows, ragged last tiles; greedy ids of the first and
    last sequence, and logits of one more step behind a chunked prompt."""
    gpt, m, p = model64
    prompts = np.stack([synth.make_tokens(p["vocab_size"], 9, seed=90, stream=i) for i in range(n_seq)])
    s = gpt.session(n_seq)
    got = s.generate_greedy(prompts, 6)
    for i in (0, n_seq - 1):
        assert np.array_equal(got[i], m.kv_generate_greedy(prompts[i], 6)), i
    s.reset()
    s.forward(prompts[:, :4], want_logits=False)
    s.forward(prompts[:, 4:], want_logits=False)
    lg = s.forward(got[:, :1])
    for i in (0, n_seq - 1):
        assert rel_err(lg[i], m.run(np.concatenate([prompts[i], got[i, :1]]))) < 2e-5


@pytest.mark.parametrize("halves,per_code", [("1", 4), ("0", 2)])
def test_int8_handle_memory(dev, monkeypatch, halves, per_code):
    """Four bytes per code, or two without the half-precision copy, for any number of rows; all of it comes back, and both
    forms agree with the codes (bounds as in test_int8_handle_rows, of the less precise of two splits)."""
    from webgpt_b200 import _lib
    monkeypatch.setenv("WGPT_INT8_HALVES", halves)
    K, N, M = 4096, 16384, 40
    rng = np.random.default_rng(4)
    q, scale = rng.integers(-127, 128, (K, N), dtype=np.int8), np.full(N, 0.5, np.float32)
    A = rng.standard_normal((M, K), dtype=np.float32)
    p_d, s_d, a_d, o_d = dev.tensor(q.view(np.uint32)), dev.tensor(scale), dev.tensor(A), dev.buffer(M * N * 4)
    h = C.c_void_p()
    for rows in (1, M):  # workspaces and code are in place from here on
        _lib.call("wgpt_int8_weight_create", dev.handle, K, N, p_d.ptr, s_d.ptr, C.byref(h))
        _lib.call("wgpt_int8_matmul_w", dev.handle, rows, h, a_d.ptr, o_d.ptr)
        _lib.call("wgpt_int8_weight_destroy", h)
    free = dev.mem_info()[0]
    _lib.call("wgpt_int8_weight_create", dev.handle, K, N, p_d.ptr, s_d.ptr, C.byref(h))
    slack = 4 << 20
    for rows in (1, M):
        _lib.call("wgpt_int8_matmul_w", dev.handle, rows, h, a_d.ptr, o_d.ptr)
        _lib.call("wgpt_device_check", dev.handle)
        assert abs(free - dev.mem_info()[0] - per_code * K * N) < slack, rows
    got = o_d.read(np.float32, M * N).reshape(M, N)
    _lib.call("wgpt_int8_weight_destroy", h)
    assert abs(free - dev.mem_info()[0]) < slack
    cols = slice(0, N, 37)
    Wf = q[:, cols].astype(np.float64) * 0.5
    assert (np.abs(got[:, cols] - A.astype(np.float64) @ Wf) <= (2.0 ** -20 + K / 4 * 2.0 ** -23) * (np.abs(A).astype(np.float64) @ np.abs(Wf))).all()


@pytest.fixture(scope="module")
def model8(oracle):
    """Head size 8: a head's output is a quarter of a warp."""
    from webgpt_b200 import GPT
    params = dict(n_layer=2, n_head=8, n_embd=64, n_ctx=96, vocab_size=264)
    w = synth.make_weights(params, seed=19, std=0.1, ln_random=True)
    gpt = GPT(None, params=params, weights=w)
    gpt.initialize()
    yield gpt, oracle.Model(params, synth.weight_list(params, w)), params
    gpt.destroy()


@pytest.mark.parametrize("n_seq", [2, 6])
@pytest.mark.parametrize("slices", [2, 4, 8])
@pytest.mark.parametrize("fixture", ["model64", "model8"])
def test_decode_attention_slices(request, monkeypatch, fixture, slices, n_seq):
    """The cluster merge of 2, 4 and 8 slices, f32 output (2 sequences) and pairs (6), at contexts from one position on:
    up to seven slices without a position, slices of unequal length, and one that takes several steps."""
    gpt, m, p = request.getfixturevalue(fixture)
    monkeypatch.setenv("WGPT_ATTN_SPLIT", str(slices))
    ids = np.stack([synth.make_tokens(p["vocab_size"], 90, seed=51, stream=i) for i in range(n_seq)])
    from webgpt_b200.model import Session
    s = Session(gpt, n_seq)
    try:
        for t in range(13):
            lg = s.forward(ids[:, t:t + 1])
            for i in (0, n_seq - 1):
                assert rel_err(lg[i], m.run(ids[i, :t + 1])) < 2e-5, t
        s.forward(ids[:, 13:88], want_logits=False)
        for t in (88, 89):
            lg = s.forward(ids[:, t:t + 1])
            for i in (0, n_seq - 1):
                assert rel_err(lg[i], m.run(ids[i, :t + 1])) < 2e-5, t
    finally:
        s.destroy()


@pytest.mark.parametrize("n_seq", [2, 150])
def test_decode_attention_steps(model64, monkeypatch, n_seq):
    """One slice of every head: the newest position as the first or last of a step of 32, in a step copied ahead of the wait
    (two steps of many sequences, four of few) and in one copied later; all stages in use and used again."""
    from webgpt_b200.model import Session
    gpt, m, p = model64
    monkeypatch.setenv("WGPT_ATTN_SPLIT", "1")
    ids = np.stack([synth.make_tokens(p["vocab_size"], 300, seed=53, stream=i) for i in range(n_seq)])
    s = Session(gpt, n_seq)
    try:
        at = 0
        for t in (31, 32, 33, 63, 64, 127, 128, 129, 160, 192, 299):
            if t > at:
                s.forward(ids[:, at:t], want_logits=False)
            lg = s.forward(ids[:, t:t + 1])
            at = t + 1
            for i in (0, n_seq - 1):
                assert rel_err(lg[i], m.run(ids[i, :t + 1])) < 2e-5, t
    finally:
        s.destroy()


@pytest.mark.parametrize("slices", ["1", "4"])
@pytest.mark.parametrize("n_seq", [6, 16, 64])
def test_decode_steps_behind_one_another(model64, monkeypatch, n_seq, slices):
    """Steps launched one behind the other without a graph: the first layer's attention starts while the step before has yet to
    advance the position, so it has asked for rows of another slice (seen in nearly every CTA of that layer at 6 and 16
    sequences, in most at 64). Captured steps follow one another whole. Same ids, and the same caches bit for bit."""
    from webgpt_b200 import GPT
    from webgpt_b200.model import Session
    gpt, m, p = model64
    monkeypatch.setenv("WGPT_ATTN_SPLIT", slices)
    monkeypatch.setenv("WGPT_GRAPH", "0")
    eager = GPT(None, params=p, weights=synth.make_weights(p, seed=17, std=0.08, ln_random=True))
    eager.initialize()
    prompts = np.stack([synth.make_tokens(p["vocab_size"], 29, seed=57, stream=i) for i in range(n_seq)])
    s, t = Session(gpt, n_seq), Session(eager, n_seq)
    try:
        a, b = s.generate_greedy(prompts, 110), t.generate_greedy(prompts, 110)
        assert np.array_equal(a, b)
        assert np.array_equal(a[0], m.kv_generate_greedy(prompts[0], 110))
        assert np.array_equal(s.forward(a[:, 109:]), t.forward(b[:, 109:]))
    finally:
        s.destroy()
        t.destroy()
        eager.destroy()


def test_decode_slices_follow_the_context(model64, monkeypatch):
    """Sums over another number of slices differ in their last bits, so equal logits show which number ran: one-token
    forwards take it from the context they meet, and a captured completion changes it as it grows (at 64 and 192 positions
    for these sizes), so that both leave the same cache."""
    from webgpt_b200.model import Session
    gpt, _, p = model64
    ids = np.stack([synth.make_tokens(p["vocab_size"], 301, seed=52, stream=i) for i in range(2)])

    def logits(n, slices):
        monkeypatch.setenv("WGPT_ATTN_SPLIT", slices)
        s = Session(gpt, 2)
        s.forward(ids[:, :n], want_logits=False)
        out = s.forward(ids[:, n:n + 1])
        s.destroy()
        return out

    for n, want in ((30, "1"), (100, "2"), (300, "4")):
        by_context = logits(n, "0")
        assert [k for k in "1248" if np.array_equal(logits(n, k), by_context)] == [want], n
    monkeypatch.setenv("WGPT_ATTN_SPLIT", "0")
    s, t = Session(gpt, 2), Session(gpt, 2)
    try:
        new = s.generate_greedy(ids[:, :16], 300)
        t.forward(ids[:, :16], want_logits=False)
        for i in range(299):
            t.forward(new[:, i:i + 1], want_logits=False)
        assert np.array_equal(s.forward(new[:, 299:]), t.forward(new[:, 299:]))
    finally:
        s.destroy()
        t.destroy()


@pytest.mark.parametrize("n_seq", [1, 2, 3, 5, 7, 8])
def test_ring_gemv_rows(oracle, n_seq):
    """Layers that do not fit shared memory (n_embd 1600): FP32 through the ring for up to five sequences, and for eight
    in FP32 mode; K = 1600 is no multiple of a stage's 256.

    Bound: the reference adds each product's K terms one after another in FP32. For terms of random sign a rounding is at
    most 2^-24 of a running sum that grows like sqrt(k), uniformly spread (1/sqrt(3)), so the error of a sum is about
    sqrt(K / 2) 2^-24 / sqrt(3) of its size, 1.9e-6 at the longest K of 6400; four of these is 8e-6. The kernel's own sums,
    split over lanes and warps, add far less."""
    from webgpt_b200 import GPT, _lib
    params = dict(n_layer=1, n_head=25, n_embd=1600, n_ctx=24, vocab_size=512)
    w = synth.make_weights(params, seed=41, std=0.04, ln_random=True)
    m = oracle.Model(params, synth.weight_list(params, w))
    gpt = GPT(None, params=params, weights=w)
    gpt.initialize()
    try:
        if n_seq == 8:
            gpt.device.set_precision(_lib.PRECISION_FP32)
        prompts = np.stack([synth.make_tokens(512, 5, seed=5, stream=i) for i in range(n_seq)])
        s = gpt.session(n_seq)
        for t in range(5):  # token by token: every pass is a decode pass
            lg = s.forward(prompts[:, t:t + 1])
        for i in (0, n_seq - 1):
            assert rel_err(lg[i], m.run(prompts[i])) < 8e-6
        # the same rows as a prompt of n_seq tokens, in two passes (from six rows on these are products of pairs)
        s1 = gpt.session(1)
        s1.reset()  # the session of one sequence is the one above when n_seq is 1
        s1.forward(prompts[0], want_logits=False)
        ids = np.concatenate([prompts[0], synth.make_tokens(512, n_seq, seed=6)])
        assert rel_err(s1.forward(ids[5:])[0], m.run(ids)) < 8e-6
    finally:
        gpt.destroy()


def test_decode_rows_of_a_wide_model(oracle):
    """n_embd 3072: LayerNorm scale, shift and row statistics leave the normalising product fewer ring stages than its slice
    of K asks for, at 32 and at 64 rows. Two tokens as decode passes; bound as in test_decode_rows."""
    from webgpt_b200 import GPT
    params = dict(n_layer=1, n_head=48, n_embd=3072, n_ctx=8, vocab_size=256)
    w = synth.make_weights(params, seed=23, std=0.02, ln_random=True)
    m = oracle.Model(params, synth.weight_list(params, w))
    gpt = GPT(None, params=params, weights=w)
    gpt.initialize()
    try:
        for n_seq in (24, 64):
            prompts = np.stack([synth.make_tokens(256, 2, seed=8, stream=i) for i in range(n_seq)])
            s = gpt.session(n_seq)
            s.forward(prompts[:, :1], want_logits=False)
            lg = s.forward(prompts[:, 1:])
            for i in (0, n_seq - 1):
                assert rel_err(lg[i], m.run(prompts[i])) < 2e-5, n_seq
    finally:
        gpt.destroy()


@pytest.mark.parametrize("K,N", [(48, 40), (768, 136), (1616, 152), (3072, 768)])
def test_int8_handle_rows(dev, oracle, K, N):
    """Up to eight rows in the block kernel (columns per item 1-4, K slices 1-8), above 16 rows as pairs against the exact
    codes: error bound as above with one inexact operand and two MMAs per step."""
    from webgpt_b200 import _lib
    h = C.c_void_p()
    _, q, packed, scale = synth.make_int8_case(1, K, N)
    p_d, s_d = dev.tensor(packed), dev.tensor(scale)
    _lib.call("wgpt_int8_weight_create", dev.handle, K, N, p_d.ptr, s_d.ptr, C.byref(h))
    try:
        for M in (1, 2, 3, 4, 5, 7, 8, 9, 16, 17, 33, 129, 257):
            A = np.random.default_rng(M).standard_normal((M, K), dtype=np.float32)
            a_d, o_d = dev.tensor(A), dev.buffer(M * N * 4)
            _lib.call("wgpt_int8_matmul_w", dev.handle, M, h, a_d.ptr, o_d.ptr)
            _lib.call("wgpt_device_check", dev.handle)
            Wf = q.astype(np.float64) * scale.astype(np.float64)
            ref, mag = A.astype(np.float64) @ Wf, np.abs(A).astype(np.float64) @ np.abs(Wf)
            steps = K if M <= 16 else 2 * K / 16 + 2  # CUDA cores: one rounding per term at most
            bound = (2.0 ** -22 + (steps + 2) * 2.0 ** -23) * mag + 2.0 ** -39 * np.abs(A).max() * np.abs(Wf).max() * K
            assert (np.abs(o_d.read(np.float32, M * N).reshape(M, N) - ref) <= bound).all(), M
    finally:
        _lib.call("wgpt_int8_weight_destroy", h)


@pytest.mark.parametrize("M,K,N", [(323, 16, 8), (129, 16, 6400), (206, 336, 768), (323, 208, 768), (1024, 464, 256)])
def test_int8_handle_one_k_block_per_slice(dev, M, K, N):
    """Row tiles of more than 64 rows with one k-block per CTA of the cluster: the FP32 partial tile is larger than the one
    stage it lies over. Bound as in test_int8_handle_rows."""
    from webgpt_b200 import _lib
    h = C.c_void_p()
    A, q, packed, scale = synth.make_int8_case(M, K, N)
    p_d, s_d, a_d, o_d = dev.tensor(packed), dev.tensor(scale), dev.tensor(A), dev.buffer(M * N * 4)
    _lib.call("wgpt_int8_weight_create", dev.handle, K, N, p_d.ptr, s_d.ptr, C.byref(h))
    try:
        _lib.call("wgpt_int8_matmul_w", dev.handle, M, h, a_d.ptr, o_d.ptr)
        _lib.call("wgpt_device_check", dev.handle)
        got = o_d.read(np.float32, M * N).reshape(M, N)
    finally:
        _lib.call("wgpt_int8_weight_destroy", h)
    Wf = q.astype(np.float64) * scale.astype(np.float64)
    ref, mag = A.astype(np.float64) @ Wf, np.abs(A).astype(np.float64) @ np.abs(Wf)
    bound = (2.0 ** -22 + (2 * K / 16 + 4) * 2.0 ** -23) * mag + 2.0 ** -39 * np.abs(A).max() * np.abs(Wf).max() * K
    assert (np.abs(got - ref) <= bound).all()


@pytest.mark.parametrize("V", [48, 4096, 4097, 50257, 65536, 65540])
def test_sampling_kernel_edges(dev, oracle, V):
    """One CTA or a cluster, the largest vocabulary its registers hold and the one beyond, top_k at its limit and beyond;
    an all-equal row has more values at the bound than a list holds, a falling one has them all in one CTA."""
    from webgpt_b200 import _lib
    rng = np.random.default_rng(V)
    rows = np.stack([rng.standard_normal(V).astype(np.float32), np.zeros(V, np.float32),
                     -np.arange(V, dtype=np.float32), np.where(np.arange(V) % 128 < 8, 5.0, -5.0).astype(np.float32)])
    u = rng.random(len(rows))
    r_d, u_d, o_d = dev.tensor(rows), dev.tensor(u), dev.buffer(4 * len(rows))
    for top_k in (1, 2, 31, 47, 48, 49):
        if top_k > V:
            continue
        _lib.call("wgpt_sample_topk", dev.handle, r_d.ptr, len(rows), V, top_k, 1.3, u_d.ptr, o_d.ptr)
        got = o_d.read(np.uint32, len(rows))
        assert [int(t) for t in got] == [oracle.sample_topk(rows[i], top_k, 1.3, u[i]) for i in range(len(rows))], top_k


@pytest.mark.parametrize("n_rows,V,ks", [(12, 8192, (32, 33)), (13, 8191, (8, 9)), (32, 32000, (32, 33)), (33, 50257, (20, 21)),
                                         (49, 50257, (1,)), (2, 257, (32, 33, 40)), (2, 383, (47, 48)), (2, 384, (48,))])
def test_sampling_on_both_sides_of_the_cluster_rule(dev, oracle, n_rows, V, ks):
    """Rows, vocabularies and kept logits at which one kernel hands over to the other: the same picks."""
    from webgpt_b200 import _lib
    rng = np.random.default_rng(V + n_rows)
    rows, u = rng.standard_normal((n_rows, V), dtype=np.float32), rng.random(n_rows)
    r_d, u_d, o_d = dev.tensor(rows), dev.tensor(u), dev.buffer(4 * n_rows)
    for top_k in ks:
        _lib.call("wgpt_sample_topk", dev.handle, r_d.ptr, n_rows, V, top_k, 0.8, u_d.ptr, o_d.ptr)
        got = o_d.read(np.uint32, n_rows)
        assert [int(t) for t in got] == [oracle.sample_topk(rows[i], top_k, 0.8, u[i]) for i in range(n_rows)], top_k
