"""The work that users of webgpt_b200 have it do, as cases that can be timed.

Every case goes through the package's public entry points: GPT.generate and Session.generate_* (the KV-cached token
loop, greedy or top-k sampled, one sequence or a batch), GPT.run (logits of one window), the pass-list route of the
instruction classes (GPT(fused=False)), and the int8 weight handles of the C ABI. Models are the package's own
configurations (synth.CONFIGS) with seeded random weights: the loaded model is what a user's program keeps, the
prompts, windows and activations are what it gets anew, and those are made from the seed.
"""
import ctypes as C
import math
import random

import numpy as np
import torch

from webgpt_b200 import GPT, Device, _lib, synth
from webgpt_b200.model import Session

INT8_SHAPES = ((768, 3072), (3072, 768), (1600, 6400), (6400, 1600))  # (K, N): the two MLP products of gpt2 and gpt2-xl


def listed():
    return [
        # the char-level model on one prompt: the smallest decode step, its weights stay in L2
        {"name": "char greedy", "kind": "generate", "model": "char", "n_seq": 1, "n_prompt": 32, "n_new": 200, "top_k": 1},
        # one user's completion on gpt2, greedy: the benchmark's workload
        {"name": "gpt2 greedy", "kind": "generate", "model": "gpt2", "n_seq": 1, "n_prompt": 64, "n_new": 256, "top_k": 1},
        # the reference page's defaults: a short prompt, 30 tokens, top_k 3, temperature 1
        {"name": "gpt2 sampled", "kind": "generate", "model": "gpt2", "n_seq": 1, "n_prompt": 21, "n_new": 30, "top_k": 3},
        # logits of one window of odd length: scoring, or a host loop with its own sampler
        {"name": "gpt2 run 333", "kind": "run", "model": "gpt2", "n_tok": 333},
        # a few sequences at once: what one GPU holds of 64 sequences spread over eight
        {"name": "gpt2 batch 8", "kind": "generate", "model": "gpt2", "n_seq": 8, "n_prompt": 64, "n_new": 64, "top_k": 1},
        # a full serving batch: an 8192-row prefill, then 64-row decode steps
        {"name": "gpt2 batch 64", "kind": "generate", "model": "gpt2", "n_seq": 64, "n_prompt": 128, "n_new": 64, "top_k": 1},
        # the largest model, a full context of prefill
        {"name": "gpt2-xl run 1024", "kind": "run", "model": "gpt2-xl", "n_tok": 1024},
        # the largest model, one user's completion
        {"name": "gpt2-xl greedy", "kind": "generate", "model": "gpt2-xl", "n_seq": 1, "n_prompt": 200, "n_new": 32, "top_k": 1},
        # the largest model serving several users
        {"name": "gpt2-xl batch 16", "kind": "generate", "model": "gpt2-xl", "n_seq": 16, "n_prompt": 96, "n_new": 24, "top_k": 1},
        # a host program written against the instruction classes: one enqueue per operator, weights in the reference's layout
        {"name": "gpt2 passes 128", "kind": "passes", "model": "gpt2", "n_tok": 128},
        # int8 weight-only product of one decode token
        {"name": "int8 1 row", "kind": "int8", "M": 1, "K": 1600, "N": 6400},
        # the same operator over a prefill chunk
        {"name": "int8 256 rows", "kind": "int8", "M": 256, "K": 3072, "N": 768},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def _draw_once(rng):
    kind = rng.choice(("generate", "generate", "generate", "generate", "run", "run", "passes", "int8", "int8"))
    if kind == "int8":
        K, N = rng.choice(INT8_SHAPES)
        return {"kind": kind, "M": _log_int(rng, 1, 256), "K": K, "N": N}
    if kind == "passes":
        return {"kind": kind, "model": "gpt2", "n_tok": _log_int(rng, 1, 256)}
    model = rng.choice(("char", "gpt2", "gpt2", "gpt2-xl", "gpt2-xl"))
    n_ctx = synth.CONFIGS[model]["n_ctx"]
    if kind == "run":
        return {"kind": kind, "model": model, "n_tok": _log_int(rng, 1, n_ctx)}
    n_seq = 1 if rng.random() < 0.4 else _log_int(rng, 2, 16 if model == "gpt2-xl" else 64)
    n_prompt = _log_int(rng, 1, 256)
    n_new = _log_int(rng, 8, 32 if model == "gpt2-xl" else 160)
    # mostly completions that fit the context; the char model's is short enough for its window to slide now and then
    if n_prompt + n_new > n_ctx and rng.random() < 0.7:
        n_prompt = n_ctx - n_new
    return {"kind": kind, "model": model, "n_seq": n_seq, "n_prompt": n_prompt, "n_new": n_new,
            "top_k": 1 if rng.random() < 0.6 else rng.randint(2, 40)}


def draw(rng):
    cost = lambda c: max(work(c)["bytes"], work(c)["flops"] / 50)  # noqa: E731
    most = max(cost(c) for c in listed())
    while True:
        c = _draw_once(rng)
        if cost(c) <= most:
            return c


# ------------------------------------------------------------------------------------------ what a program keeps
_models = {}


def _weights(params, seed=1234):
    """Seeded weights of the model's shapes, four distinct blocks repeated over the layers (each layer has its own
    copy on the device). The spread is such that a product of normalised rows comes out of order one, as in a trained
    model, so that completions do not settle on one token; LayerNorm gains and shifts are random too."""
    n = min(params["n_layer"], 4)
    w = synth.make_weights(dict(params, n_layer=n), seed=seed, std=1.4 / math.sqrt(params["n_embd"]), ln_random=True)
    for l in range(n, params["n_layer"]):
        for k in synth.LAYER_KEYS:
            w[f"transformer.h.{l}.{k}"] = w[f"transformer.h.{l % n}.{k}"]
    return w


def _model(name, fused=True):
    if (name, fused) not in _models:
        params = synth.CONFIGS[name]
        gpt = GPT(None, params=params, weights=_weights(params), fused=fused)
        gpt.initialize()
        gpt._weights = None  # the host copy has been uploaded
        _models[name, fused] = gpt
    return _models[name, fused]


def _device():
    if "device" not in _models:
        _models["device"] = Device()
    return _models["device"]


class _Batch:
    """A program's session of n_seq sequences, given back with the state."""

    def __init__(self, gpt, n_seq):
        self.session = Session(gpt, n_seq)

    def __del__(self):
        self.session.destroy()


class _Int8:
    """An int8 weight handle, its activations and result, given back with the state."""

    def __init__(self, case, seed):
        M, K, N = case["M"], case["K"], case["N"]
        g = torch.Generator(device="cuda").manual_seed(seed)
        q = torch.randint(-127, 128, (K, N), generator=g, device="cuda", dtype=torch.int8)
        scale = torch.rand(N, generator=g, device="cuda") * 0.019 + 0.001
        self.A = torch.randn(M, K, generator=g, device="cuda")
        self.out = torch.empty(M, N, device="cuda")
        self.dev, self.M, self.handle = _device(), M, C.c_void_p()
        torch.cuda.synchronize()  # the framework's stream does not wait for torch's
        _lib.call("wgpt_int8_weight_create", self.dev.handle, K, N, q.data_ptr(), scale.data_ptr(), C.byref(self.handle))

    def __del__(self):
        _lib.call("wgpt_int8_weight_destroy", self.handle)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "int8":
        return {"kind": kind, "int8": _Int8(case, seed)}
    params = synth.CONFIGS[case["model"]]
    gpt = _model(case["model"], fused=kind != "passes")
    if kind != "generate":
        return {"kind": kind, "gpt": gpt, "idx": synth.make_tokens(params["vocab_size"], case["n_tok"], seed=seed)}
    n_seq, n_prompt, n_new = case["n_seq"], case["n_prompt"], case["n_new"]
    prompts = synth.make_tokens(params["vocab_size"], n_seq * n_prompt, seed=seed).reshape(n_seq, n_prompt)
    state = {"kind": kind, "gpt": gpt, "prompts": prompts, "n_new": n_new, "top_k": case["top_k"], "seed": seed}
    if n_seq > 1:
        state["batch"] = _Batch(gpt, n_seq)
        state["uniforms"] = np.random.default_rng(seed).random((n_new, n_seq))
    return state


# ------------------------------------------------------------------------------------------ one pass
def run(state):
    if state["kind"] == "int8":
        s = state["int8"]
        _lib.call("wgpt_int8_matmul_w", s.dev.handle, s.M, s.handle, s.A.data_ptr(), s.out.data_ptr())
        return s.out
    gpt = state["gpt"]
    if state["kind"] in ("run", "passes"):
        return gpt.run(state["idx"])
    if "batch" in state:
        session = state["batch"].session
        if state["top_k"] == 1:
            return session.generate_greedy(state["prompts"], state["n_new"])
        return session.generate_sample(state["prompts"], state["n_new"], state["top_k"], 1.0, state["uniforms"])
    rand = random.Random(state["seed"]).random  # in place of Math.random(), so that a pass can be repeated
    return np.array(list(gpt.generate(state["prompts"][0], state["n_new"], state["top_k"], 1.0, rand)), np.uint32)


# ------------------------------------------------------------------------------------------ what a pass cannot do without
def _forward_work(p, n_seq, n_old, n_tok):
    """One forward pass of n_tok new tokens per sequence behind n_old cached ones: every weight once, the cached K and
    V rows read and the new ones written, the logits of each sequence's newest position."""
    E, L, V, rows = p["n_embd"], p["n_layer"], p["vocab_size"], n_seq * n_tok
    weights = L * (12 * E * E + 13 * E) + 2 * E + V * E
    kv = L * 2 * E * n_seq * (n_old + n_tok)
    pairs = n_seq * (n_tok * n_old + n_tok * (n_tok + 1) / 2)  # (query, visible key)
    return (4.0 * (weights + kv + 2 * rows * E + n_seq * V),
            2.0 * rows * L * 12 * E * E + 4.0 * L * E * pairs + 2.0 * n_seq * V * E)


def work(case):
    if case["kind"] == "int8":
        M, K, N = case["M"], case["K"], case["N"]
        return {"bytes": float(K * N + 4 * N + 4 * M * (K + N)), "flops": 2.0 * M * K * N}
    p = synth.CONFIGS[case["model"]]
    if case["kind"] != "generate":
        b, f = _forward_work(p, 1, 0, case["n_tok"])
        return {"bytes": b, "flops": f}
    n_seq, n_ctx = case["n_seq"], p["n_ctx"]
    n = case["n_prompt"]
    b, f = _forward_work(p, n_seq, 0, min(n, n_ctx))
    for i in range(1, case["n_new"]):
        # one token behind the cache, or the whole window again once it slides (every position index has shifted)
        db, df = _forward_work(p, n_seq, n + i - 1, 1) if n + i <= n_ctx else _forward_work(p, n_seq, 0, n_ctx)
        b, f = b + db, f + df
    return {"bytes": b, "flops": f}


def tolerance(case):
    """f32 in and out. One product's sum of a few thousand terms is good to about 1e-5 whatever the order; through a
    whole model the same roundings pass every later layer. Token ids are whole values: one may differ where the two
    best logits are as close as that, and then that sequence goes on from another token."""
    if case["kind"] == "int8":
        return {"rel": 1e-5}
    if case["kind"] == "generate":
        return {"rel": 1e-5, "differ": 0.01}
    return {"rel": 5e-5}
