"""CPU checks of the routes that products of pairs take (csrc/pair_plan.h): that the shapes which GPU tests name for K split over
two CTA pairs do take it, on a B200 (33 clusters of four CTAs, one per SM) and with a few clusters fewer or more."""
import ctypes as C
import os
import subprocess

import pytest

from conftest import ROOT
from test_gpu_pairs import K_OVER_TWO_PAIRS, WIDTH_OVER_TWO_PAIRS
from test_split_plan import SMEM

DRIVER = r"""
#include "pair_plan.h"
using namespace wgpt;
extern "C" int slices(const int *clusters, long long smem, int pairs, int M, int K, int N, int prompt) {  // 0: gemm_split_kernel
  const ProductShape s = product_shape(SplitLimits{clusters, (size_t)smem}, pairs, M, N, K, N % 4 == 0, 2, prompt != 0);
  if (s.split) return 0;
  const PairShape ps = s.pair;
  if (ps.bn % 32 != 0 || ps.bn < 64 || ps.bn > 256) return -1;
  if (ps.KS == 2 && ((M + 255) / 256) * ((N + ps.bn - 1) / ps.bn) > clusters[4]) return -2;
  return ps.KS;
}
"""


@pytest.fixture(scope="module")
def slices(tmp_path_factory):
    d = tmp_path_factory.mktemp("pair_plan")
    src, lib = d / "plan.cpp", d / "plan.so"
    src.write_text(DRIVER)
    subprocess.run(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-I", os.path.join(ROOT, "webgpt_b200", "csrc"),
                    str(src), "-o", str(lib)], check=True)
    so = C.CDLL(str(lib))

    def call(M, K, N, of_four=33, prompt=False):
        clusters = (C.c_int * 9)(0, 148, 74, 45, of_four, 26, 22, 15, 15)
        return so.slices(clusters, C.c_longlong(SMEM), 74, M, K, N, int(prompt))

    return call


@pytest.mark.parametrize("of_four", range(31, 38))
def test_shapes_of_the_gpu_tests(slices, of_four):
    for M, K, N in K_OVER_TWO_PAIRS:
        if (M, K, N) != (900, 1160, 1304):  # 36 tiles with the split: not on 33 clusters, where it is one more shape without
            assert slices(M, K, N, of_four) == 2, (M, K, N)
    for name, E, tokens in WIDTH_OVER_TWO_PAIRS:
        for n in tokens:
            assert slices(n, E, {"qkv": 3, "up": 4}[name] * E, of_four, True) == 2, (name, n)


@pytest.mark.parametrize("prompt", [False, True])
def test_products_of_gpt2_and_xl(slices, prompt):
    """Rows at which K is split over two pairs, as the rule's comment lists them, of operators and of prompts."""
    def rows(K, N):
        return [M for M in range(65, 1025) if slices(M, K, N, prompt=prompt) == 2]

    for K, N in ((768, 2304), (768, 768), (768, 3072), (3072, 768), (1600, 6400)):
        assert rows(K, N) == []
    assert rows(1600, 4800) == list(range(145, 257))
    assert rows(1600, 1600) == list(range(641, 769))
    assert rows(6400, 1600) == list(range(641, 1025))


def test_every_shape_is_in_range(slices):
    for M in (1, 64, 65, 255, 256, 257, 700, 1024, 8192):
        for K in (8, 64, 72, 768, 1608, 6400):
            for N in (8, 40, 768, 2056, 50257):
                for of_four in (0, 1, 33):
                    for prompt in (False, True):
                        assert slices(M, K, N, of_four, prompt) in (0, 1, 2)
