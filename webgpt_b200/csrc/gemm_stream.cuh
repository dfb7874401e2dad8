// C[M,N] = X[M,K] . Wt[N,K]^T on pairs (pair.cuh) for up to 128 rows against a matrix that is a stream from HBM: the
// de-embedding of a batch (GPT-2: 50257 x 768, 154 MB).
//
// One CTA per SM stays for the whole product and owns a contiguous run of output features, so the weights' stream through
// its ring never stops between tiles: the features are the accumulator's lanes (tcgen05.mma with the weight tile as A, 128 at
// a time), the rows the instruction's N, and two accumulators alternate, so that a tile is stored while the next one is
// multiplied. Rows cost what they are (RN = M rounded up to 16), in tensor-core time and in stored bytes alike.
//
//   weights     : tiles of {64 of K, 128 features} per plane; a run's last tile in pieces of 32 features, so that at most 31
//                 rows are read that no feature of the run needs (past N: the second plane's first, or zeros; lanes that are never
//                 stored); the ring's first tiles ahead of the dependency wait;
//   activations : {64 of K, RN rows, 2 planes} by TMA with every weight tile, out of L2;
//   products    : as in gemm_split_kernel: the weights' first plane with both planes of the rows (2 RN columns), the second
//                 with the first, so that the large and the small sums have accumulators of their own;
//   store       : a lane is a feature, so a warp stores 32 neighbouring values of a row (128 bytes; a row of 50257 floats is
//                 aligned to four bytes only).
//
// What bounds it: HBM in a decode step, where the first tiles arrive beside the kernel before: one more launch of it costs GPT-2's step of
// 8 / 16 / 64 / 128 sequences 27.6 / 27.6 / 28.5 / 35.7 us for 154 MB, 0.85 of the copy rate up to 64 (some of it perhaps out of L2, behind a launch
// that has just read the same). Cold and alone 33 us at 8 rows and 35 at 64, 0.7 of it, the rest start and the ring's latency; the
// tensor pipe is busy for 6 and 22 % of that. A step with 8 / 64 sequences 362 -> 335 / 636 -> 561 us against gemm_pair_kernel (cold 54 and 107 us:
// 256 rows of the pair's tile are multiplied and read back whatever the batch is), XL with 16 2.56 -> 2.52 ms. See stream_fits in
// pair_plan.h for where it takes over.
// Every wait is bounded; on expiry *err = 3, the copies in flight get another bounded wait, and the result is void.
#pragma once
#include "gemm_split.cuh"
#include "pair_plan.h"

namespace wgpt {

constexpr int GT_THREADS = 192;      // warp 0 TMA, warp 1 MMA, warps 2-5 accumulator read-back and store
constexpr int GT_MAX_STAGES = 6;

struct StreamArgs {
  int M, K, N, rn, stages;
  const float *colscale;  // [N]
  float *out;             // [M][ld]
  int ld;
  int *err;
};

inline size_t stream_stage_bytes(int rn) { return (size_t)GS_W_BYTES + (size_t)rn * (GP_BK * 4); }

// map_w / map_wp: the two weight planes one below the other as 2 N rows, boxes of 128 / GT_PIECE rows; map_x: rn rows, 2 planes.
__global__ void __launch_bounds__(GT_THREADS, 1)
gemm_stream_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_wp,
                   const __grid_constant__ CUtensorMap map_x, const __grid_constant__ StreamArgs p) {
  extern __shared__ uint8_t gt_smem_raw[];
  uint8_t *tiles = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(gt_smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ uint64_t full_w[GT_MAX_STAGES], full_x[GT_MAX_STAGES], empty[GT_MAX_STAGES], acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_word, requested_w, requested_x;
  volatile int *abort_flag = &abort_word;
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int rn = p.rn, S = p.stages;
  const int pieces = (p.N + GT_PIECE - 1) / GT_PIECE;
  const int f_beg = (int)((long long)pieces * blockIdx.x / gridDim.x) * GT_PIECE;
  const int f_end = min(p.N, (int)((long long)pieces * (blockIdx.x + 1) / gridDim.x) * GT_PIECE);
  const int n_tiles = (f_end - f_beg + 127) / 128, kb_all = (p.K + GP_BK - 1) / GP_BK, total = n_tiles * kb_all;
  const uint32_t stage_bytes = GS_W_BYTES + (uint32_t)rn * (GP_BK * 4);
  const uint32_t need = 4u * (uint32_t)rn, tmem_cols = need <= 64 ? 64u : need <= 128 ? 128u : need <= 256 ? 256u : 512u;

  // weight tile `q` of this CTA's sequence (k-blocks of its tiles in order) into its stage
  auto load_w = [&](int q) {
    const int t = q / kb_all, x = (q - t * kb_all) * GP_BK, f = f_beg + 128 * t, left = f_end - f;
    uint64_t *bar = &full_w[q % S];
    uint8_t *st = tiles + (size_t)(q % S) * stage_bytes;
    if (left > 128 - GT_PIECE) {
      mbar_expect_tx(bar, GS_W_BYTES);
      tma_load_3d(st, &map_w, x, f, bar);
      tma_load_3d(st + GS_W_BYTES / 2, &map_w, x, p.N + f, bar);
    } else {
      const int n = (left + GT_PIECE - 1) / GT_PIECE;
      mbar_expect_tx(bar, (uint32_t)n * (2 * GT_PIECE * GP_BK * 2));
      for (int i = 0; i < n; i++) {
        tma_load_3d(st + i * (GT_PIECE * GP_BK * 2), &map_wp, x, f + GT_PIECE * i, bar);
        tma_load_3d(st + GS_W_BYTES / 2 + i * (GT_PIECE * GP_BK * 2), &map_wp, x, p.N + f + GT_PIECE * i, bar);
      }
    }
  };

  if (threadIdx.x == 0) {
    for (int i = 0; i < S; i++) {
      mbar_init(&full_w[i], 1);
      mbar_init(&full_x[i], 1);
      mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < 2; i++) {
      mbar_init(&acc_full[i], 1);
      mbar_init(&acc_empty[i], 4);
    }
    abort_word = 0;
    requested_w = requested_x = total;
    fence_async_smem();
    for (int q = 0; q < min(S, total); q++) load_w(q);  // no kernel writes the weights: ahead of the dependency wait
  }
  if (warp == 1) tmem_alloc(&tmem_slot, tmem_cols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_acc = tmem_slot;
  pdl_launch_dependents();
  pdl_wait();

  if (warp == 0) {
    if (lane == 0) {
      for (int q = 0; q < total; q++) {
        const int s = q % S, use = q / S;
        if (q >= S) {
          if (*abort_flag || !mbar_wait(&empty[s], (use & 1) ^ 1, TC_POLLS)) {
            *abort_flag = 1;
            requested_w = requested_x = q;
            break;
          }
          load_w(q);
        }
        mbar_expect_tx(&full_x[s], (uint32_t)rn * (GP_BK * 4));
        tma_load_3d(tiles + (size_t)s * stage_bytes + GS_W_BYTES, &map_x, (q % kb_all) * GP_BK, 0, &full_x[s]);
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // the whole warp runs this loop and one elected lane issues (see umma1_f16)
    const uint32_t idesc = f16_idesc(128, rn), idesc2 = f16_idesc(128, 2 * rn), desc0 = umma_desc_lo(smem_addr(tiles));
    int s = 0, ph = 0;
    for (int t = 0; t < n_tiles; t++) {
      const uint32_t acc = tmem_acc + (uint32_t)(t & 1) * 2u * (uint32_t)rn;
      if (!mbar_wait(&acc_empty[t & 1], ((t >> 1) & 1) ^ 1, TC_POLLS)) *abort_flag = 1;
      tc_fence_after();
      for (int kb = 0; kb < kb_all; kb++) {
        if (!mbar_wait(&full_w[s], ph, TC_POLLS) || !mbar_wait(&full_x[s], ph, TC_POLLS)) *abort_flag = 1;
        if (__any_sync(0xffffffffu, *abort_flag)) break;
        tc_fence_after();
        const uint32_t w0 = desc0 + (uint32_t)s * (stage_bytes >> 4), w1 = w0 + (GS_W_BYTES >> 5), x0 = w0 + (GS_W_BYTES >> 4);
#pragma unroll
        for (int k = 0; k < GP_BK / 16; k++) {
          umma1_f16(acc, w0 + 2 * k, x0 + 2 * k, idesc2, (kb > 0 || k > 0) ? 1u : 0u);
          umma1_f16(acc + (uint32_t)rn, w1 + 2 * k, x0 + 2 * k, idesc, 1u);
        }
        umma_commit_elect(&empty[s]);
        if (++s == S) { s = 0; ph ^= 1; }
      }
      umma_commit_elect(&acc_full[t & 1]);  // (also after an abort)
    }
  } else {
    const int quad = warp & 3;
    for (int t = 0; t < n_tiles; t++) {
      const int f = f_beg + 128 * t + quad * 32 + lane;
      const bool live = f < f_end;
      const float cs = live ? __ldg(p.colscale + f) : 0.f;
      if (!mbar_wait(&acc_full[t & 1], (t >> 1) & 1, TC_POLLS << 2)) *abort_flag = 1;
      tc_fence_after();
      const uint32_t acc = tmem_acc + (uint32_t)(t & 1) * 2u * (uint32_t)rn + ((uint32_t)(quad * 32) << 16);
      float *o = p.out + f;
#pragma unroll 1
      for (int c = 0; c < rn; c += 16) {
        float v[16], w[16];
        tmem_ld_2x16(acc + (uint32_t)c, acc + (uint32_t)(rn + c), v, w);
#pragma unroll
        for (int j = 0; j < 16; j++)
          if (live && c + j < p.M) o[(size_t)(c + j) * p.ld] = (v[j] + w[j]) * cs;
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[t & 1]);
    }
  }
  __syncthreads();
  if (threadIdx.x == 0 && *abort_flag) {
    atomicExch(p.err, 3);
    ring_drain(full_w, S, requested_w, TC_POLLS);
    ring_drain(full_x, S, requested_x, TC_POLLS);
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_acc, tmem_cols);
  }
}

}  // namespace wgpt
