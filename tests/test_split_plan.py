"""CPU checks of the launch shapes of the cluster split-K product (csrc/split_plan.h): what a CTA keeps in shared memory
fits what is asked for, and what is asked for fits an SM. The limits are a B200's: 227 KB per CTA, of which 2 KB are left
to the kernel's static arrays, and clusters of one to eight CTAs, one per SM, on 148 SMs in groups of 16 or fewer."""
import ctypes as C
import os
import subprocess

import pytest

from conftest import ROOT

SMEM = 232448 - 2048
CLUSTERS = (0, 148, 74, 48, 36, 28, 23, 20, 16)

DRIVER = r"""
#include "split_plan.h"
using namespace wgpt;
static void put(const SplitShape &sh, long long *out) {
  out[0] = sh.row_tiles; out[1] = sh.rn; out[2] = sh.S; out[3] = sh.stages; out[4] = (long long)sh.smem;
}
extern "C" void decode(const int *clusters, long long smem, int M, int K, int N, int norm, long long *out) {
  put(split_shape_decode(SplitLimits{clusters, (size_t)smem}, M, K, N, norm != 0), out);
}
extern "C" void rows(const int *clusters, long long smem, int M, int K, int N, int w_planes, long long *out) {
  double cycles;
  put(split_shape_rows(SplitLimits{clusters, (size_t)smem}, M, K, N, w_planes, &cycles), out);
}
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("split_plan")
    src, lib = d / "plan.cpp", d / "plan.so"
    src.write_text(DRIVER)
    subprocess.run(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-I", os.path.join(ROOT, "webgpt_b200", "csrc"),
                    str(src), "-o", str(lib)], check=True)
    so = C.CDLL(str(lib))
    clusters = (C.c_int * 9)(*CLUSTERS)

    def call(fn, *args):
        out = (C.c_longlong * 5)()
        getattr(so, fn)(clusters, C.c_longlong(SMEM), *args, out)
        return dict(zip(("row_tiles", "rn", "S", "stages", "smem"), out))

    return call


def ring_bytes(sh, w_planes):
    return sh["stages"] * (w_planes * 16384 + sh["rn"] * 256)


@pytest.mark.parametrize("w_planes", [1, 2])
@pytest.mark.parametrize("N", [8, 256, 768, 3072, 6400])
def test_partial_tile_fits_the_ring(plan, w_planes, N):
    """The FP32 partial tile of rn x 128 lies over the ring; 1024 bytes go to its alignment. Every K of 16 to 640 (one to
    ten k-blocks, so up to one k-block per CTA of a cluster), rows around every row tile."""
    for K in range(16, 641, 16):
        for M in (9, 17, 32, 63, 64, 65, 80, 96, 127, 128, 129, 206, 256, 257, 323, 384, 385, 700, 1024):
            sh = plan("rows", M, K, N, w_planes)
            assert sh["stages"] >= 1 and sh["rn"] % 16 == 0 and sh["rn"] <= 128 and sh["row_tiles"] * sh["rn"] >= M
            assert sh["smem"] <= SMEM
            assert sh["smem"] >= 1024 + max(ring_bytes(sh, w_planes), sh["rn"] * 512), (M, K, N, sh)


@pytest.mark.parametrize("M", [9, 16, 17, 32, 33, 48, 49, 64])
def test_normalising_form_fits_or_is_refused(plan, M):
    """Scale, shift and row statistics lie behind the ring; a width at which nothing fits is refused (smem 0) and the
    caller takes another path. Everything up to 8192 has to fit."""
    for E in list(range(64, 1665, 32)) + [2048, 2560, 2688, 2880, 3072, 3200, 4096, 5120, 8192, 12288, 16384]:
        kb = (E + 63) // 64
        for N in (3 * E, 4 * E):
            sh = plan("decode", M, E, N, 1)
            if sh["smem"] == 0:
                assert E > 8192
                continue
            behind = -(-kb // sh["S"]) * 512 + sh["rn"] * ((E + 127) // 128) * 8
            assert sh["stages"] >= 1 and sh["smem"] <= SMEM
            assert sh["smem"] >= 1024 + max(ring_bytes(sh, 2), sh["rn"] * 512) + behind
        for K, N in ((E, E), (4 * E, E)):
            sh = plan("decode", M, K, N, 0)
            assert sh["stages"] >= 1 and 1024 + max(ring_bytes(sh, 2), sh["rn"] * 512) <= sh["smem"] <= SMEM


def test_ring_keeps_its_share_where_everything_fits(plan):
    """At the widths of GPT-2 and GPT-2 XL neither limit bites: 200 KB of stages, or the whole slice of K."""
    for E in (768, 1600):
        for M in (6, 16, 17, 48, 64):
            for K, N, norm in ((E, 3 * E, 1), (E, E, 0), (E, 4 * E, 1), (4 * E, E, 0)):
                sh = plan("decode", M, K, N, norm)
                need = -(-((K + 63) // 64) // sh["S"])
                assert sh["stages"] == min(need, 204800 // (32768 + sh["rn"] * 256), 6)
