// Launch shapes of the products of pairs: gemm_pair_kernel's tile width and CTA pairs per tile (gemm_pair.cuh), and which
// products gemm_split_kernel takes (gemm_split.cuh); and of the LayerNorm ahead of them. Plain C++, so that the routes can be
// followed on the host.
#pragma once
#include <cmath>

#include "split_plan.h"

namespace wgpt {

// Warps that share a row of a LayerNorm whose result leaves as pairs (layernorm_kernel). One warp a row is a long chain on few warps:
// up to 1536 rows four share one, up to 4096 two; beyond that every SM has warps enough and the barriers cost more. Rows of up to 128
// values are one float4 a lane of one warp: the other three have nothing to do, and that a CTA holds one row in place of four, so that
// few rows spread over more SMs, stops paying at 1024 rows.
// us per pass, 1 / 2 / 4 warps: GPT-2 70 / 333 tokens 559 / 544 / 538, 789 / 772 / 763, 16 / 32 / 64 sequences of 128 1749 / 1728 / 1736, 2912 / 2869 /
// 2897, 5269 / 5281 / 5306. One warp / this rule: n_embd 1600, 48 layers, 129 / 200 / 333 / 513 / 1024 tokens 4460 / 4089, 4774 / 4502, 5919 / 5696,
// 7869 / 7706, 11271 / 11022 (power cap: runs of one side differ by 1.4 %); 384, 6 layers, 100 / 576 / 1536 / 4096 rows 244 / 240, 427 / 425, 452 / 438,
// 690 / 688; 256, 12 layers, 100 / 1600 / 4096 412 / 407, 768 / 740, 975 / 981; 128, 12 layers, 150 / 512 / 1024 414 / 407, 573 / 555, 623 / 612, and were
// 3200 / 4096 rows 696 / 707, 728 / 739 with two warps; 64, 1200 / 2048 / 4096 rows 563 / 569, 576 / 587, 612 / 623 with four, two and two.
inline int layernorm_warps(int rows, int N) {
  if (N <= 128) return rows <= 1024 ? 4 : 1;
  return rows <= 1536 ? 4 : rows <= 4096 ? 2 : 1;
}

// Where gemm_stream_kernel (gemm_stream.cuh) takes a product of few rows from gemm_pair_kernel, whose 256-row tile is mostly padding
// there: from two pieces of features for every SM on, or where K is so short that the pair kernel's start and its epilogue are most of it.
// At exactly two pieces (9472 on 148 SMs) the pair kernel's tiles are one full round, which a long K makes the better one. us per decode
// pass of one block, pair / stream: n_embd 768, vocabulary 50257, 6 / 16 / 64 / 128 rows 92 / 67, 111 / 70, 172 / 98, 196 / 124; 4104, 6 / 128 rows 46.2 /
// 42.5, 94.6 / 94.3; 1000, 64 rows 64.8 / 67.0. n_embd 1600, 4104, 64 rows 107 / 111. Vocabulary 9472, 6 / 64 / 128 rows, n_embd 1024 57.1 / 52.1, 95.6 /
// 91.4, 133 / 129; 2048 97.1 / 90.0, 147 / 145, 184 / 184; 3072 164 / 157, 228 / 229, 291 / 294; 4096 240 / 229, 325 / 330, 393 / 400, 33 rows 275 / 281; one
// feature more, 3072 168 / 159, 250 / 231, 314 / 296; 4096 247 / 231, 349 / 332, 416 / 400. n_embd 384, 64 / 96 rows, vocabulary 65 82.4 / 73.8, 95.8 / 88.0; 2000 69.4 /
// 66.1, 79.0 / 76.8; 9400 75.6 / 70.9, 87.4 / 83.8. n_embd 512, 64 / 80 / 96 rows, 1000 70.8 / 67.9, 73.9 / 73.7, 80.1 / 79.9; 4104 74.9 / 72.2, 80.1 / 79.1, 87.3 /
// 86.2; 4700 75.0 / 72.3, 79.8 / 79.3, 87.8 / 88.2; 9400 78.2 / 73.8, 82.9 / 80.1, 90.2 / 88.4. 640, 1000, 64 / 96 rows 65.6 / 63.4, 69.5 / 69.7.
constexpr int GT_MAX_ROWS = 128;
constexpr int GT_PIECE = 32;  // features per copy of a run's last tile, and the granularity of the runs
inline bool stream_fits(int sms, int M, int K, int N) {
  const int two = 2 * GT_PIECE * sms;
  return M <= GT_MAX_ROWS && (N > two || (N == two && K <= 2048) || (K <= 512 && M <= 96));
}

struct PairShape {
  int bn, KS;  // tile columns, CTA pairs that share a tile's K
};

// A tile's cycles per k-block of GS_BK: max(tensor pipe, shared memory).
inline int pair_kb_cycles(int bn) { return 6 * bn > 640 + 5 * bn / 2 ? 6 * bn : 640 + 5 * bn / 2; }

// Tile width of gemm_pair_kernel without a split: the multiple of 32 whose rounds over the pairs cost least. *cycles: the
// estimate with 40 bytes per cycle from L2 as a third bound and 12 000 cycles for the first copies and the last epilogue.
inline int pair_tile_columns(int pairs, int M, int N, int K = 0, double *cycles = nullptr) {
  const int m_tiles = (M + 255) / 256;
  int best = 256;
  long long best_cost = -1;
  for (int bn = 256; bn >= 64; bn -= 32) {
    const long long rounds = ((long long)m_tiles * ((N + bn - 1) / bn) + pairs - 1) / pairs;
    const long long cost = rounds * pair_kb_cycles(bn);
    if (best_cost < 0 || cost < best_cost) {
      best = bn;
      best_cost = cost;
      const double per_kb = std::fmax((double)cost / rounds, 820 + 3.2 * bn);
      if (cycles) *cycles = rounds * per_kb * ((K + GS_BK - 1) / GS_BK) + 12000;
    }
  }
  return best;
}

// The same with K split over clusters of two pairs where that is shorter: a tile each, half the k-blocks, and for the exchange
// 4000 cycles and 12 per column; the last epilogue, 70 cycles a column, is shared too. Of GPT-2's and XL's products it is q | k | v
// of XL at 145 to 256 rows, XL's down projection from 641 on and its output projection to 768 (33 clusters of four); product_shape
// leaves those as they are in prompts. us per pass without / with, when this alone chose: XL 145 / 175 / 200 tokens 4818 / 4658, 4985 / 4822, 4961 / 4918, but 210 / 235 / 255 4860 / 4927, 4920 / 5026,
// 4858 / 4983; 645 / 700 / 765 9194 / 8816, 9398 / 9017, 9699 / 9307; 800 to 1024 the same. Sums of half as many steps: logits of
// three XL layers at 200 / 700 / 1024 tokens 7.4e-6 / 1.59e-5 / 1.64e-5 from float64, 1.20e-5 / 2.13e-5 / 2.18e-5 without. Six
// layers of other widths: n_embd 1216 and 1408 at 180 to 256 rows 1 to 2.5 % faster, 1344 to 1856 at 600 to 768 1 to 3, 2432 at 400
// and 512 4 to 6, 1792 and 1856 at 200 to 256 1 to 2 % slower. So the estimate is off for one row tile of many columns; 35 cycles
// a column in place of 12 put XL at 205 to 256 right, and cost XL 0.9 % at 641 to 768 and n_embd 1216 to 1408 what they had gained.
inline PairShape pair_shape(const SplitLimits &lim, int pairs, int M, int N, int K) {
  const int kb = (K + GS_BK - 1) / GS_BK, m_tiles = (M + 255) / 256, bn1 = pair_tile_columns(pairs, M, N);
  PairShape best = {bn1, 1};
  double least = (double)(((long long)m_tiles * ((N + bn1 - 1) / bn1) + pairs - 1) / pairs) * pair_kb_cycles(bn1) * kb + 70.0 * bn1;
  for (int bn = 256; kb >= 2 && bn >= 64; bn -= 32) {
    if ((long long)m_tiles * ((N + bn - 1) / bn) > lim.max_clusters[4]) continue;
    const double c = (double)((kb + 1) / 2) * pair_kb_cycles(bn) + 4000 + 12.0 * bn + 70.0 * ((bn / 32 + 1) / 2 * 32);
    if (c < least) {
      least = c;
      best = {bn, 2};
    }
  }
  return best;
}

// Whether gemm_split_kernel should be the faster one, by the estimates of both; *sh: its shape. The form without the K split
// stands for gemm_pair_kernel here: with the better estimate plus 10 000 cycles XL at 200 tokens took 4949 -> 4730 us, but 333
// 6085 -> 6514 and GPT-2 512 969 -> 1004 (prompts that went by this alone then).
inline bool pair_product_splits(const SplitLimits &lim, int pairs, int M, int K, int N, int w_planes, SplitShape *sh) {
  double big = 0, split = 0;
  pair_tile_columns(pairs, M, N, K, &big);
  *sh = split_shape_rows(lim, M, K, N, w_planes, &split);
  return sh->smem > 0 && split < big;
}

struct ProductShape {
  bool split;
  SplitShape sh;   // split
  PairShape pair;  // otherwise
};
// Additions to the large sum of one output over K, each of which the tensor core truncates (gemm_pair.cuh): the pair form adds
// all three products of a 16-deep step to it, the split form the large one alone; slices of K are sums of their own.
inline int product_truncations(const ProductShape &s, int K) {
  const int kb = (K + GS_BK - 1) / GS_BK;
  return s.split ? 4 * ((kb + s.sh.S - 1) / s.sh.S) : 12 * ((kb + s.pair.KS - 1) / s.pair.KS);
}

// Cycles of a product in a prompt (weights known ahead, both planes, no row factors), fitted to 55 prompts of 70 to 1024 rows at
// n_embd 768, 1024, 1280 and 1600 of which every shape of each of the four products was timed inside whole passes. Against the
// estimates above: an MMA step of the split form waits less for L2 than 40 bytes a cycle, its start and exchange are 2400 cycles
// and not 9000, and one CTA without a cluster pays more, not less, for it stores its rows alone; the pair form's epilogue grows
// with its columns. Good to about a tenth.
inline double product_cycles(const SplitLimits &lim, int pairs, int M, int N, int K, const ProductShape &s) {
  const int kb = (K + GS_BK - 1) / GS_BK;
  if (s.split) {
    const int rn = s.sh.rn, S = s.sh.S, rounds = ((N + 127) / 128 * s.sh.row_tiles + lim.max_clusters[S] - 1) / lim.max_clusters[S];
    return rounds * (((kb + S - 1) / S) * std::fmax(6.0 * rn, 620 + 1.35 * rn) + (S == 1 ? 5000 : 2400) + 68.0 * rn);
  }
  const int bn = s.pair.bn, tiles = (M + 255) / 256 * ((N + bn - 1) / bn);
  const double per_kb = std::fmax(4.6 * bn, 408 + 1.5 * bn);
  return s.pair.KS == 1 ? (double)((tiles + pairs - 1) / pairs) * kb * per_kb + 8050 + 86.0 * bn
                        : (double)((kb + 1) / 2) * per_kb + 8050 + 51.0 * bn;
}

// The kernel and shape of a product of pairs. split_ok: rows that gemm_split_kernel can store (N and the row stride multiples of four
// floats). Operators, exact codes (w_planes 1) and more than kFittedRows rows, to none of which product_cycles was fitted: by the
// estimates above. A prompt's product in a model: the cheapest of all shapes of both kernels by product_cycles, if that has it ahead of
// the former by 3 % with the same kernel or by 6 % with the other, and if it truncates no more often.
//
// The margins: within a kernel the estimate orders shapes well, between the two it errs by up to a tenth. With 3 % for both XL at 144 to 160
// rows takes its up projection in CTAs without a cluster, 4173 -> 4221 and 4235 -> 4378 us a pass; with 6 % for both XL loses 2 % at 257 to 512.
//
// The truncations: without that limit the down projection went to two pairs a tile at n_embd 768 from 897 rows on, 1024 from 641, 1280
// from 561, 1600 at 401 to 512; 2-norm from float64 of the rows behind one block whose down projection prevails, estimates above / without /
// with the limit: 768 x 1000 rows 7.92e-6 / 8.42e-6 / 5.15e-6, 1024 x 700 9.13e-6 / 1.06e-5 / 6.39e-6, 1280 x 600 1.10e-5 / 1.53e-5 / 1.10e-5,
// 1600 x 512 1.37e-5 / 1.91e-5 / 1.37e-5, 2048 x 300 1.76e-5 / 2.10e-5 / 1.24e-5. Without it GPT-2's 1024 tokens would take 1268 us in place of 1291,
// XL's 416 / 512 6.24 / 6.53 ms in place of 6.38 / 6.73.
//
// us per pass, the estimates above / this rule (n_embd, layers):
//   384, 6: 200 / 416 / 512 / 700 / 1024 tokens 291 / 292, 344 / 345, 423 / 386, 466 / 436, 532 / 515
//   512, 8: 352 / 512 / 880 / 1000 tokens 481 / 451, 560 / 506, 690 / 668, 720 / 707
//   768, 12: 352 / 450 / 544 / 700 / 900 / 1024 tokens 787 / 729, 861 / 810, 963 / 883, 1039 / 1014, 1231 / 1233, 1320 / 1291
//   1024, 24: 240 / 320 / 500 / 700 / 1024 tokens 1481 / 1402, 1725 / 1582, 2074 / 1987, 2528 / 2490, 3168 / 2962
//   1280, 24: 160 / 288 / 385 / 416 / 576 / 769 / 1024 tokens 1629 / 1630, 2255 / 1888, 2385 / 2414, 2468 / 2436, 2982 / 2871, 3580 / 3417, 4214 / 3976
//   1600, 48: 160 / 333 / 416 / 512 / 576 / 700 / 850 / 1024 tokens 4218 / 4252, 5803 / 5328, 6503 / 6380, 6794 / 6734, 8109 / 7807, 8842 / 8593, 10520 / 10357, 11156 / 10991
//   2048, 12: 136 / 176 / 288 / 450 / 576 / 768 / 1024 tokens 1243 / 1160, 1355 / 1304, 2048 / 1818, 2284 / 2239, 2938 / 2795, 3223 / 3055, 3937 / 3916
//   3072, 4: 96 / 160 / 288 / 480 / 641 / 1024 tokens 720 / 657, 922 / 924, 1282 / 1204, 1509 / 1473, 1994 / 1966, 2656 / 2667
//   4096, 2: 100 / 200 / 300 / 1024 tokens 601 / 528, 737 / 739, 1116 / 1118, 2227 / 2238
// Of 108 prompts only 1280 x 385 is slower by more than two runs of one side differ (1.2 %, 416 rows 1.4 % faster). Not beyond 1024 rows,
// which were not fitted: by product_cycles alone, without margins and limit, GPT-2 16 / 32 / 64 sequences of 128 took 1753 / 1722, 2989 / 2904,
// 5412 / 5641, XL 12 / 16 of 96 11873 / 12045, 14336 / 14528.
constexpr int kFittedRows = 1024;
inline ProductShape product_shape(const SplitLimits &lim, int pairs, int M, int N, int K, bool split_ok, int w_planes, bool prompt) {
  const int kb = (K + GS_BK - 1) / GS_BK, rt0 = (M + 127) / 128;
  ProductShape best = {}, t = {};
  best.split = pair_product_splits(lim, pairs, M, K, N, w_planes, &best.sh) && split_ok;
  if (!best.split) best.pair = pair_shape(lim, pairs, M, N, K);
  if (!prompt || w_planes != 2 || M > kFittedRows) return best;
  const int most = product_truncations(best, K);
  const bool general = best.split;
  double least = product_cycles(lim, pairs, M, N, K, best);
  for (t.pair.bn = 256; t.pair.bn >= 64; t.pair.bn -= 32) {
    const int tiles = (M + 255) / 256 * ((N + t.pair.bn - 1) / t.pair.bn);
    for (t.pair.KS = 1; t.pair.KS <= 2; t.pair.KS++) {
      if ((t.pair.KS == 2 && (kb < 2 || tiles > lim.max_clusters[4])) || product_truncations(t, K) > most) continue;
      const double c = (general ? 1.06 : 1.03) * product_cycles(lim, pairs, M, N, K, t);
      if (c < least) {
        least = c;
        best = t;
      }
    }
  }
  if (!split_ok) return best;
  t.split = true;
  for (int rt = rt0; rt <= rt0 + 2; rt++) {
    t.sh = {};
    t.sh.rn = (((M + rt - 1) / rt) + 15) & ~15;
    t.sh.row_tiles = (M + t.sh.rn - 1) / t.sh.rn;
    for (t.sh.S = 1; t.sh.S <= 8 && t.sh.S <= kb; t.sh.S++) {
      if (lim.max_clusters[t.sh.S] < 1 || product_truncations(t, K) > most) continue;
      const double c = (general ? 1.03 : 1.06) * product_cycles(lim, pairs, M, N, K, t);
      if (c >= least) continue;
      ProductShape placed = t;
      split_place(placed.sh, lim, K, 2, false);
      if (placed.sh.smem == 0) continue;
      least = c;
      best = placed;
    }
  }
  return best;
}

}  // namespace wgpt
