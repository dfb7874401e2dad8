"""CPU checks of the rule that gives a prompt's products their kernel and shape (csrc/pair_plan.h, product_shape): every shape
that it can return can be launched, and the prompts that the GPU test names take every form."""
import ctypes as C
import os
import subprocess

import pytest

from conftest import ROOT
from test_gpu_product_forms import PROMPTS, TRUNCATIONS
from test_split_plan import SMEM

DRIVER = r"""
#include "pair_plan.h"
using namespace wgpt;
extern "C" void shape(const int *clusters, long long smem, int M, int K, int N, long long *out) {
  const ProductShape s = product_shape(SplitLimits{clusters, (size_t)smem}, 74, M, N, K, N % 4 == 0, 2, true);
  const long long v[] = {s.split, s.pair.bn, s.pair.KS, s.sh.row_tiles, s.sh.rn, s.sh.S, s.sh.stages, (long long)s.sh.smem};
  for (int i = 0; i < 8; i++) out[i] = v[i];
}
extern "C" int ln_warps(int rows, int N) { return layernorm_warps(rows, N); }
extern "C" int streams(int M, int K, int N) { return stream_fits(148, M, K, N); }
extern "C" void general(const int *clusters, long long smem, int M, int K, int N, int *out) {  // the route of other callers
  const ProductShape s = product_shape(SplitLimits{clusters, (size_t)smem}, 74, M, N, K, N % 4 == 0, 2, false);
  out[0] = s.split, out[1] = s.sh.S, out[2] = s.pair.KS;
}
"""
B200 = (0, 148, 74, 45, 33, 26, 22, 15, 15)


@pytest.fixture(scope="module")
def shape(tmp_path_factory):
    d = tmp_path_factory.mktemp("product_plan")
    src, lib = d / "plan.cpp", d / "plan.so"
    src.write_text(DRIVER)
    subprocess.run(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-I", os.path.join(ROOT, "webgpt_b200", "csrc"),
                    str(src), "-o", str(lib)], check=True)
    so = C.CDLL(str(lib))

    def call(M, K, N, clusters=B200):
        out = (C.c_longlong * 8)()
        so.shape((C.c_int * 9)(*clusters), C.c_longlong(SMEM), M, K, N, out)
        return dict(zip(("split", "bn", "KS", "row_tiles", "rn", "S", "stages", "smem"), out))

    def general(M, K, N, clusters=B200):
        out = (C.c_int * 3)()
        so.general((C.c_int * 9)(*clusters), C.c_longlong(SMEM), M, K, N, out)
        return dict(zip(("split", "S", "KS"), out))

    call.general = general
    call.ln_warps, call.streams = so.ln_warps, so.streams
    return call


def truncations(s, K):
    """Truncating additions to the large sum: four per k-block and slice in the split form, twelve in the pair form."""
    kb = (K + 63) // 64
    return 4 * -(-kb // s["S"]) if s["split"] else 12 * -(-kb // s["KS"])


@pytest.mark.parametrize("E", [64, 256, 384, 768, 1024, 1280, 1600, 2048, 3072])
def test_no_prompt_truncates_more_often(shape, E):
    """Against the shape that the same product takes outside a prompt, whose sums are what a prompt's have to be at least."""
    for K, N in ((E, 3 * E), (E, E), (E, 4 * E), (4 * E, E)):
        for M in range(9, 1025):
            s, g = shape(M, K, N), shape.general(M, K, N)
            assert truncations(s, K) <= truncations(g, K), (M, K, N, s, g)


@pytest.mark.parametrize("rows", range(129, 161))
def test_shapes_within_the_estimates_error_stay(shape, rows):
    """XL's up projection at 144 to 160 rows: the shape that the estimate has 5 % ahead makes a pass up to 3 % longer."""
    s, g = shape(rows, 1600, 6400), shape.general(rows, 1600, 6400)
    assert s["split"] == g["split"] == 0 and s["KS"] == g["KS"]


def test_deembeddings_that_stream(shape):
    """Two pieces of 32 features an SM: at exactly that, one full round of the pair kernel, a long K stays with it (1 to 2 %)."""
    for M in (6, 128):
        for K in (768, 2048, 3072, 4096):
            assert [shape.streams(M, K, N) for N in (9471, 9472, 9473, 50257)] == [0, K <= 2048, 1, 1]
    assert [shape.streams(M, 512, 65) for M in (6, 96, 97)] == [1, 1, 0] and not shape.streams(129, 64, 50257)


def test_warps_of_a_narrow_row(shape):
    """Rows that one warp holds in a float4 a lane: past 1024 of them more warps make a pass up to 4 % longer."""
    for N in (32, 64, 128):
        assert [shape.ln_warps(rows, N) for rows in (1, 1024, 1025, 4096)] == [4, 4, 1, 1]
    for N in (132, 384, 768, 1600, 2048):
        assert [shape.ln_warps(rows, N) for rows in (1, 1536, 1537, 4096, 4097)] == [4, 4, 2, 2, 1]


@pytest.mark.parametrize("E,n,up,down", TRUNCATIONS)
def test_truncations_of_the_gpu_test(shape, E, n, up, down):
    assert truncations(shape.general(n, E, 4 * E), E) == up and truncations(shape.general(n, 4 * E, E), 4 * E) == down


@pytest.mark.parametrize("clusters", [B200, (0, 148, 74, 48, 36, 28, 23, 20, 16), (0, 140, 66, 40, 28, 0, 0, 0, 0)])
@pytest.mark.parametrize("E", [8, 64, 200, 384, 768, 1160, 1600, 3072])
def test_shapes_can_be_launched(shape, E, clusters):
    for K, N in ((E, 3 * E), (E, E), (E, 4 * E), (4 * E, E)):
        for M in (9, 16, 17, 63, 64, 65, 100, 128, 129, 255, 256, 257, 300, 333, 384, 385, 511, 512, 513, 700, 768, 769, 1000, 1024):
            s = shape(M, K, N, clusters)
            if s["split"]:
                assert s["rn"] % 16 == 0 and 16 <= s["rn"] <= 128 and s["row_tiles"] * s["rn"] >= M, (M, K, N, s)
                assert 1 <= s["S"] <= min(8, (K + 63) // 64) and clusters[s["S"]] > 0 and s["stages"] >= 1, (M, K, N, s)
                ring = max(s["stages"] * (32768 + s["rn"] * 256), s["rn"] * 512)
                assert 1024 + ring <= s["smem"] <= SMEM, (M, K, N, s)
            else:
                assert s["bn"] % 32 == 0 and 64 <= s["bn"] <= 256 and s["KS"] in (1, 2), (M, K, N, s)
                if s["KS"] == 2:
                    assert K > 64 and ((M + 255) // 256) * -(-N // s["bn"]) <= clusters[4], (M, K, N, s)


def form(s):
    return ("split", min(s["S"], 2)) if s["split"] else ("pair", s["KS"])


def test_prompts_of_the_gpu_test_take_every_form(shape):
    """Each epilogue (q | k | v, output, GELU, down) with each form that the rule gives it at any width up to XL's."""
    seen = set()
    for E, M in PROMPTS:
        for name, K, N in (("qkv", E, 3 * E), ("o", E, E), ("up", E, 4 * E), ("down", 4 * E, E)):
            seen.add((name, form(shape(M, K, N))))
    want = set()
    for E in (384, 768, 1024, 1216, 1280, 1600):
        for M in range(65, 1025, 9):  # where the rule applies
            for name, K, N in (("qkv", E, 3 * E), ("o", E, E), ("up", E, 4 * E), ("down", 4 * E, E)):
                want.add((name, form(shape(M, K, N))))
    assert want - seen == set()
