// Launch shapes of gemm_split_kernel (gemm_split.cuh): row tile, K slices, ring stages and dynamic shared memory.
// Plain C++, so that the arithmetic a shared-memory layout rests on can be swept on the host.
#pragma once
#include <algorithm>
#include <cmath>
#include <cstddef>

namespace wgpt {

constexpr int GS_MAX_STAGES = 6;
constexpr int GS_BK = 64;               // K per stage
constexpr int GS_PLANE_BYTES = 16384;   // one plane of a 128 x 64 weight tile
constexpr size_t GS_RING_BYTES = size_t(200) << 10;

struct SplitShape {
  int row_tiles, rn, S, stages;
  size_t smem;  // dynamic; 0: does not fit
};

// What the shapes depend on: clusters of S CTAs that are resident at once with one CTA per SM, and the dynamic shared
// memory that a CTA may ask for.
struct SplitLimits {
  const int *max_clusters;  // [9]
  size_t smem;
};

// Bytes of one ring stage: w_planes planes of a weight tile and both planes of rn activation rows.
inline size_t split_stage_bytes(int rn, int w_planes) { return (size_t)w_planes * GS_PLANE_BYTES + (size_t)rn * (GS_BK * 4); }

// What the normalising form keeps behind the ring: LayerNorm scale and shift of the CTA's slice of K, and the statistics of
// every row's 128-column tiles.
inline size_t split_norm_bytes(int K, int rn, int S) {
  const int kb = (K + GS_BK - 1) / GS_BK;
  return (size_t)((kb + S - 1) / S) * GS_BK * 8 + (size_t)rn * ((K + 127) / 128) * 8;
}

// As many stages as a CTA's slice of K has k-blocks, as the ring's share of shared memory holds, and as the whole fits.
// The partial tile [rn][128] lies over the ring once that has been read, so the ring is never smaller than it: a slice of
// one k-block against a one-plane weight has a stage of 16 KB + 256 rn and a tile of 512 rn.
inline void split_place(SplitShape &sh, const SplitLimits &lim, int K, int w_planes, bool norm) {
  const int kb = (K + GS_BK - 1) / GS_BK;
  const size_t stage = split_stage_bytes(sh.rn, w_planes), part = (size_t)sh.rn * 512;
  const size_t fixed = 1024 + (norm ? split_norm_bytes(K, sh.rn, sh.S) : 0);
  sh.stages = 0;
  sh.smem = 0;
  if (fixed >= lim.smem) return;
  const size_t room = std::min(lim.smem - fixed, GS_RING_BYTES);
  sh.stages = (int)std::min<size_t>({(size_t)((kb + sh.S - 1) / sh.S), room / stage, (size_t)GS_MAX_STAGES});
  const size_t ring = std::max(sh.stages * stage, part);
  if (sh.stages < 1 || fixed + ring > lim.smem) return;
  sh.smem = fixed + ring;
}

// One row tile of RN rows (kNorm / decode): the smallest number of K slices with the shortest longest slice, among those
// whose clusters are all resident at once with one CTA per SM (a second round would double the product's time).
inline SplitShape split_shape_decode(const SplitLimits &lim, int M, int K, int N, bool norm) {
  SplitShape sh = {};
  sh.row_tiles = 1;
  sh.rn = (M + 15) & ~15;
  const int ft = (N + 127) / 128, kb = (K + GS_BK - 1) / GS_BK;
  sh.S = 1;
  for (int S = 2; S <= 8 && S <= kb; S++)
    if (ft <= lim.max_clusters[S] && (kb + S - 1) / S < (kb + sh.S - 1) / sh.S) sh.S = S;
  split_place(sh, lim, K, 2, norm);
  return sh;
}

// Any number of rows, activations as planes: row tiles of up to 128 and K slices by the same kind of estimate
// (pair_plan.h): a k-block costs max(6 RN tensor-core cycles, 32 KB + 256 RN bytes from L2 at 40 a cycle), a round
// 9000 cycles of start, exchange and store and 60 more per row of the tile. A model's prompts of up to 1024 rows depart from it where
// product_shape has another shape well ahead.
inline SplitShape split_shape_rows(const SplitLimits &lim, int M, int K, int N, int w_planes, double *cycles) {
  SplitShape best = {};
  const int ft = (N + 127) / 128, kb = (K + GS_BK - 1) / GS_BK, rt0 = (M + 127) / 128;
  *cycles = 1e30;
  for (int rt = rt0; rt <= rt0 + 2; rt++) {
    const int rn = (((M + rt - 1) / rt) + 15) & ~15;
    for (int S = 1; S <= 8 && S <= kb; S++) {
      if (lim.max_clusters[S] < 1) continue;
      const int rounds = (ft * rt + lim.max_clusters[S] - 1) / lim.max_clusters[S];
      const double c = rounds * (((kb + S - 1) / S) * std::fmax(6.0 * rn, 820 + 6.4 * rn) + 9000 + 60.0 * rn);
      if (c < *cycles) {
        *cycles = c;
        best.row_tiles = (M + rn - 1) / rn; best.rn = rn; best.S = S;
      }
    }
  }
  if (best.S > 0) split_place(best, lim, K, w_planes, false);
  return best;
}

}  // namespace wgpt
