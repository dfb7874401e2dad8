// C[M,N] = X[M,K] . Wt[N,K]^T (+ epilogue) on pairs (pair.cuh) for few to some hundred rows: batched decode and short
// prefills, where a 256-row tile would be mostly padding and the product is a stream of weights.
//
// A CTA owns 128 output features (the 128 lanes of the accumulator: tcgen05.mma with the weight tile as A), a tile of RN
// activation rows (the instruction's N) and a slice of K. The S CTAs of a cluster share one output tile, each taking a
// slice of K, and add their partial tiles through distributed shared memory, so the product is finished in one launch:
// the kernel it replaces (gemm_tc_kernel, operands exchanged) left split-K slices in HBM for a second kernel, and eight
// dependent launches per transformer block at 5-8 us each were what a 64-row decode pass took its time for.
//
//   weights   : both planes of a {64 of K, 128 rows} tile per TMA box (32 KB) into a ring, requested before the
//               dependency wait (they are written by no kernel);
//   activations: MODE kPlanes - both planes by TMA;
//               MODE kNorm   - FP32 rows, normalised on the way in (LayerNorm, instructions.js:451-550) by six warps:
//               their producer left (mean, sum of squared deviations) of every row and 128-column tile, which are
//               merged here, so that neither a LayerNorm pass nor a grid-wide exchange stands between two products;
//   reduction : every CTA puts its [RN][128] partial tile into its own shared memory (the ring's, by then read), the
//               cluster synchronises once, and CTA r finishes rows r RN/S ..: it reads the S partial rows in rank order
//               (results do not depend on timing), applies scale, bias, GELU / residual, and stores 512 contiguous
//               bytes per row. stats != nullptr: also this tile's (mean, squared deviations) of each finished row.
//
// The activations' two planes lie one behind the other, so one MMA multiplies the weights' first plane with both (2 RN
// columns: the main products and the first correction side by side) and a second one adds the other correction to the
// latter: two instructions per 16 of K instead of three, and the large and the small sums have accumulators of their own.
// The slices of K are added in FP32, rounding to nearest.
// Every wait is bounded; on expiry the CTA sets *err = 3, gives its copies in flight another bounded wait and carries on
// through its cluster barriers (the result is void).
#pragma once
#include "gemm_pair.cuh"
#include "split_plan.h"

namespace wgpt {

constexpr int GS_THREADS = 256;        // warp 0 TMA, warp 1 MMA, warps 2-7 staging, warps 4-7 accumulator read-back
constexpr int GS_STAGERS = 192;
constexpr int GS_W_BYTES = GP_A_BYTES;  // both planes of a 128 x 64 weight tile
static_assert(GS_W_BYTES == 2 * GS_PLANE_BYTES && GP_BK == GS_BK, "the launch shapes are planned for these tiles");

struct SplitArgs {
  int M, K, N;
  int rn;              // activation rows per CTA: a multiple of 16, at most 128 (kPlanes) / RN (kNorm)
  int f_tiles;         // ceil(N / 128)
  int stages;          // ring stages (<= GS_MAX_STAGES); max(stages * stage_bytes, rn * 512) bytes of ring (split_plan.h)
  Epilogue epi;
  float2 *stats;       // [M][f_tiles] or nullptr
  int dyn;             // the weight and its scales were written by the previous kernel: nothing is read ahead of the wait
  int w_planes;        // 2, or 1 for a weight that is exact in one plane (small integers)
  // kNorm
  const float *x;      // [M][K] FP32
  const float2 *x_stats;  // [M][x_tiles]: mean and sum of squared deviations of columns 128 t ..
  int x_tiles;
  const float *gamma, *beta;
  float x_scale;
  int *err;
};

__device__ __forceinline__ void umma1_f16(uint32_t tmem_d, uint32_t alo, uint32_t blo, uint32_t idesc,
                                          uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, e;\n\t.reg .b64 da, db;\n\t"
      "mov.b64 da, {%1, %5};\n\tmov.b64 db, {%2, %5};\n\t"
      "setp.ne.b32 p, %4, 0;\n\telect.sync _|e, 0xffffffff;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, p;\n\t}" ::"r"(tmem_d),
      "r"(alo), "r"(blo), "r"(idesc), "r"(accumulate), "r"(kUmmaDescHi)
      : "memory");
}
// Twice 32 lanes x 16 consecutive 32-bit columns, both loads in flight together.
__device__ __forceinline__ void tmem_ld_2x16(uint32_t t0, uint32_t t1, float (&v)[16], float (&w)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%32];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%33];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=&f"(v[0]), "=&f"(v[1]), "=&f"(v[2]), "=&f"(v[3]), "=&f"(v[4]), "=&f"(v[5]), "=&f"(v[6]), "=&f"(v[7]), "=&f"(v[8]), "=&f"(v[9]), "=&f"(v[10]), "=&f"(v[11]), "=&f"(v[12]), "=&f"(v[13]), "=&f"(v[14]), "=&f"(v[15]),
        "=&f"(w[0]), "=&f"(w[1]), "=&f"(w[2]), "=&f"(w[3]), "=&f"(w[4]), "=&f"(w[5]), "=&f"(w[6]), "=&f"(w[7]), "=&f"(w[8]), "=&f"(w[9]), "=&f"(w[10]), "=&f"(w[11]), "=&f"(w[12]), "=&f"(w[13]), "=&f"(w[14]), "=&f"(w[15])
      : "r"(t0), "r"(t1)
      : "memory");
}
// umma_commit by one elected lane of a converged warp.
__device__ __forceinline__ void umma_commit_elect(uint64_t *bar) {
  asm volatile(
      "{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\t"
      "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(smem_addr(bar))
      : "memory");
}
__device__ __forceinline__ void sts64(uint32_t saddr, uint2 v) {
  asm volatile("st.shared.v2.u32 [%0], {%1,%2};" ::"r"(saddr), "r"(v.x), "r"(v.y) : "memory");
}

// Mean and 1/sqrt(var + eps) of a row of K values from the (mean, sum of squared deviations) of its 128-column tiles.
__device__ __forceinline__ float2 merge_row_stats(const float2 *st, int tiles, int K) {
  float m = 0.f, q = 0.f;
#pragma unroll 4
  for (int t = 0; t < tiles; t++) m += st[t].x * (float)min(128, K - 128 * t);
  m /= (float)K;
#pragma unroll 4
  for (int t = 0; t < tiles; t++) q += st[t].y + (float)min(128, K - 128 * t) * (st[t].x - m) * (st[t].x - m);
  return make_float2(m, 1.0f / sqrtf(q / (float)K + 1e-5f));
}

// grid.x = row tiles x feature tiles x S, cluster (S, 1, 1). map_w: box of 128 rows; map_x (RN == 0): box of rn rows.
// RN == 0: activations as planes by TMA, rn at run time. RN > 0: normalised on the way in, rn == RN. OP: a per-operator
// product, with row factors and, where p.dyn says so, a weight that the previous kernel wrote.
template <int RN, bool OP>
__global__ void __launch_bounds__(GS_THREADS, 2)
gemm_split_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                  const __grid_constant__ SplitArgs p) {
  extern __shared__ uint8_t gs_smem_raw[];
  uint8_t *tiles = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(gs_smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ uint64_t full_w[GS_MAX_STAGES], full_x[GS_MAX_STAGES], empty[GS_MAX_STAGES], acc_full;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_word, requested;  // requested: k-blocks, as the producer leaves it
  __shared__ float2 row_norm[RN > 0 ? RN : 1];
  volatile int *abort_flag = &abort_word;
  float *part = reinterpret_cast<float *>(tiles);  // [rn][128], over the ring once its last tile has been read
  // LayerNorm scale and shift of this CTA's slice of K (times x_scale), behind the ring

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int rn = RN > 0 ? RN : p.rn;
  uint32_t S;
  asm volatile("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(S));
  const int rank = (int)cluster_ctarank();
  const int tile = blockIdx.x / S, ft = tile % p.f_tiles, row0 = (tile / p.f_tiles) * rn, f0 = ft * 128;
  const int total_kb = (p.K + GP_BK - 1) / GP_BK;
  const int kb0 = (int)((long long)total_kb * rank / S), nkb = (int)((long long)total_kb * (rank + 1) / S) - kb0;
  const int stages = p.stages, w_bytes = p.w_planes * (GS_W_BYTES / 2);
  const int stage_bytes = w_bytes + rn * (GP_BK * 4);
  float4 *gam = reinterpret_cast<float4 *>(tiles + (size_t)stages * stage_bytes), *bet = gam + nkb * (GP_BK / 4);
  float2 *tile_st = reinterpret_cast<float2 *>(bet + nkb * (GP_BK / 4));  // [rows][x_tiles], as their producers left them
  const uint32_t tmem_cols = rn <= 16 ? 32u : (rn <= 32 ? 64u : (rn <= 64 ? 128u : 256u));

  if (threadIdx.x == 0) {
    for (int i = 0; i < stages; i++) {
      mbar_init(&full_w[i], 1);
      mbar_init(&full_x[i], RN > 0 ? GS_STAGERS / 32 : 1);
      mbar_init(&empty[i], 1);
    }
    mbar_init(&acc_full, 1);
    abort_word = 0;
    fence_async_smem();
    if (OP && p.dyn) pdl_wait();
    const int pre = min(stages, nkb);
    requested = nkb;
    for (int j = 0; j < pre; j++) {  // weights: ahead of the dependency wait
      mbar_expect_tx(&full_w[j], (uint32_t)w_bytes);
      tma_load_3d(tiles + (size_t)j * stage_bytes, &map_w, (kb0 + j) * GP_BK, f0, &full_w[j]);
    }
  }
  if (warp == 1) tmem_alloc(&tmem_slot, tmem_cols);
  if (RN > 0) {
    for (int i = threadIdx.x; i < nkb * (GP_BK / 4); i += GS_THREADS) {
      const int col = kb0 * GP_BK + 4 * i;
      const bool in = col < p.K;  // past the end both are zero, and so is what is multiplied
      gam[i] = in ? scale4(__ldg(reinterpret_cast<const float4 *>(p.gamma + col)), p.x_scale) : make_float4(0.f, 0.f, 0.f, 0.f);
      bet[i] = in ? scale4(__ldg(reinterpret_cast<const float4 *>(p.beta + col)), p.x_scale) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_acc = tmem_slot;
  Epilogue e = p.epi;
  // this lane's four columns of the tile: their constants ahead of the wait too
  const int n = f0 + lane * 4;
  const bool n_live = n < p.N;
  float4 cs = make_float4(1.f, 1.f, 1.f, 1.f), bs = make_float4(0.f, 0.f, 0.f, 0.f);
  pdl_launch_dependents();
  if (OP && p.dyn) pdl_wait();
  if (n_live && e.colscale != nullptr) cs = __ldcg(reinterpret_cast<const float4 *>(e.colscale + n));
  if (n_live && e.bias != nullptr) bs = __ldcg(reinterpret_cast<const float4 *>(e.bias + n));
  pdl_wait();  // the activations come from the previous kernel
  if (e.kc != nullptr && e.pos != nullptr) {
    e.pos_base = __ldcg(e.pos);
    e.pos = nullptr;
  }
  const int r_beg = rn * rank / (int)S, r_end = rn * (rank + 1) / (int)S;
  // the residual of this warp's first two rows: a round trip to L2 that would otherwise follow the exchange
  float4 res_first[2] = {make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f)};
#pragma unroll
  for (int u = 0; u < 2; u++) {
    const int r = r_beg + warp + u * (GS_THREADS / 32);
    if (e.residual != nullptr && n_live && r < r_end && row0 + r < p.M)
      res_first[u] = __ldcg(reinterpret_cast<const float4 *>(e.residual + (size_t)(row0 + r) * e.ld + n));
  }

  if (warp == 0) {
    if (lane == 0) {
      for (int j = 0; j < nkb; j++) {
        const int s = j % stages, use = j / stages;
        uint8_t *st = tiles + (size_t)s * stage_bytes;
        if (j >= stages) {
          if (*abort_flag || !mbar_wait(&empty[s], (use & 1) ^ 1, TC_POLLS)) { *abort_flag = 1; requested = j; break; }
          mbar_expect_tx(&full_w[s], (uint32_t)w_bytes);
          tma_load_3d(st, &map_w, (kb0 + j) * GP_BK, f0, &full_w[s]);
        }
        if (RN == 0) {
          mbar_expect_tx(&full_x[s], (uint32_t)rn * (GP_BK * 4));
          tma_load_3d(st + w_bytes, &map_x, (kb0 + j) * GP_BK, row0, &full_x[s]);
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // the whole warp runs this loop and one elected lane issues (see umma1_f16)
    const uint32_t idesc = f16_idesc(128, rn), idesc2 = f16_idesc(128, 2 * rn), desc0 = umma_desc_lo(smem_addr(tiles));
    for (int j = 0; j < nkb; j++) {
      const int s = j % stages, use = j / stages;
      if (!mbar_wait(&full_w[s], use & 1, TC_POLLS) || !mbar_wait(&full_x[s], use & 1, TC_POLLS)) *abort_flag = 1;
      if (__any_sync(0xffffffffu, *abort_flag)) break;
      tc_fence_after();
      const uint32_t w0 = desc0 + (uint32_t)s * ((uint32_t)stage_bytes >> 4), w1 = w0 + (GS_W_BYTES >> 5);
      const uint32_t x0 = w0 + ((uint32_t)w_bytes >> 4);
#pragma unroll
      for (int k = 0; k < GP_BK / 16; k++) {
        umma1_f16(tmem_acc, w0 + 2 * k, x0 + 2 * k, idesc2, (j > 0 || k > 0) ? 1u : 0u);
        if (p.w_planes == 2) umma1_f16(tmem_acc + (uint32_t)rn, w1 + 2 * k, x0 + 2 * k, idesc, 1u);
      }
      umma_commit_elect(&empty[s]);
    }
    umma_commit_elect(&acc_full);  // (also reached after an abort)
  } else if (RN > 0) {
    // ---------------- activations: 16 lanes per row (one float4 each), 12 rows per step ----------------
    constexpr int ITERS = RN > 0 ? (RN + 11) / 12 : 1, G = 12 / ITERS;  // G k-blocks of loads in flight together
    const int t = threadIdx.x - 64, k4 = t & 15, mrow = t >> 4;
    const int rows = min(RN, p.M - row0);
    // the statistics first (every thread a few of them), then the rows: both are in flight together
    constexpr int NST = 4;
    const int n_st = rows * p.x_tiles;
    const float2 *st_src = p.x_stats + (size_t)row0 * p.x_tiles;
    float2 st_pre[NST];
#pragma unroll
    for (int i = 0; i < NST; i++) st_pre[i] = t + GS_STAGERS * i < n_st ? __ldcg(st_src + t + GS_STAGERS * i) : make_float2(0.f, 0.f);
    for (int j0 = 0; j0 < nkb; j0 += G) {
      float4 v[G][ITERS];
#pragma unroll
      for (int g = 0; g < G; g++) {
        const int col = (kb0 + j0 + g) * GP_BK + 4 * k4;
        const bool in = j0 + g < nkb && col < p.K;
#pragma unroll
        for (int i = 0; i < ITERS; i++) {
          const int m = mrow + 12 * i;
          v[g][i] = in && m < rows ? __ldcg(reinterpret_cast<const float4 *>(p.x + (size_t)(row0 + m) * p.K + col))
                                   : make_float4(0.f, 0.f, 0.f, 0.f);
        }
      }
      if (j0 == 0) {
#pragma unroll
        for (int i = 0; i < NST; i++)
          if (t + GS_STAGERS * i < n_st) tile_st[t + GS_STAGERS * i] = st_pre[i];
        for (int i = t + GS_STAGERS * NST; i < n_st; i += GS_STAGERS) tile_st[i] = __ldcg(st_src + i);
        asm volatile("bar.sync 1, %0;" ::"n"(GS_STAGERS) : "memory");
        if (t < rows) row_norm[t] = merge_row_stats(tile_st + t * p.x_tiles, p.x_tiles, p.K);
        asm volatile("bar.sync 1, %0;" ::"n"(GS_STAGERS) : "memory");
      }
#pragma unroll
      for (int g = 0; g < G; g++) {
        const int j = j0 + g;
        if (j >= nkb) break;
        const int s = j % stages, use = j / stages;
        if (j >= stages && (*abort_flag || !mbar_wait(&empty[s], (use & 1) ^ 1, TC_POLLS))) { *abort_flag = 1; break; }
        const uint32_t xt = smem_addr(tiles + (size_t)s * stage_bytes) + (uint32_t)w_bytes;
        const float4 ga = gam[j * (GP_BK / 4) + k4], be = bet[j * (GP_BK / 4) + k4];
#pragma unroll
        for (int i = 0; i < ITERS; i++) {
          const int m = mrow + 12 * i;
          if (m < rows) {  // other columns of the accumulator are never read
            const float2 mr = row_norm[m];
            const float4 a = v[g][i];
            uint2 h0, h1;
            pair_split4(make_float4(ga.x * ((a.x - mr.x) * mr.y) + be.x, ga.y * ((a.y - mr.x) * mr.y) + be.y,
                                    ga.z * ((a.z - mr.x) * mr.y) + be.z, ga.w * ((a.w - mr.x) * mr.y) + be.w), h0, h1);
            // 128-byte swizzle: 16-byte chunk c of row m sits at chunk c ^ (m % 8)
            const uint32_t at = xt + (uint32_t)m * 128u + ((uint32_t)((k4 >> 1) ^ (m & 7)) << 4) + (uint32_t)(k4 & 1) * 8u;
            sts64(at, h0);
            sts64(at + (uint32_t)RN * 128u, h1);
          }
        }
        fence_async_smem();  // visible to the tensor core's reads
        __syncwarp();
        if (lane == 0) mbar_arrive(&full_x[s]);
      }
    }
  }
  if (warp >= 4) {  // accumulator -> this CTA's partial tile; lane = feature, one shared-memory row per activation row
    if (!mbar_wait(&acc_full, 0, TC_POLLS << 2)) *abort_flag = 1;
    tc_fence_after();
    const int quad = warp & 3;
    const uint32_t lanes = tmem_acc + ((uint32_t)(quad * 32) << 16);
#pragma unroll 1
    for (int c = 0; c < rn; c += 16) {
      float v[16], w[16];
      tmem_ld_2x16(lanes + (uint32_t)c, lanes + (uint32_t)(rn + c), v, w);
#pragma unroll
      for (int j = 0; j < 16; j++) part[(c + j) * 128 + quad * 32 + lane] = v[j] + w[j];
    }
    tc_fence_before();
  }
  if (S > 1) {
    cluster_arrive();
    cluster_wait();
  } else {
    __syncthreads();
  }
  if (threadIdx.x == 0 && *abort_flag) atomicExch(p.err, 3);

  const int cnt = min(128, p.N - f0);
  const uint32_t pbase = smem_addr(part) + (uint32_t)lane * 16u;
  constexpr int NW = GS_THREADS / 32;
  for (int r = r_beg + warp; r < r_end; r += 2 * NW) {  // two rows at a time: their remote reads are in flight together
    const int m0 = row0 + r, m1 = m0 + NW;
    if (m0 >= p.M) break;
    const bool two = r + NW < r_end && m1 < p.M;
    float4 res[2] = {res_first[0], res_first[1]};
    if (e.residual != nullptr && n_live && r != r_beg + warp) {
      res[0] = __ldcg(reinterpret_cast<const float4 *>(e.residual + (size_t)m0 * e.ld + n));
      if (two) res[1] = __ldcg(reinterpret_cast<const float4 *>(e.residual + (size_t)m1 * e.ld + n));
    }
    float4 q[2][8];
    const uint32_t at = pbase + (uint32_t)r * 512u;
#pragma unroll
    for (int s = 0; s < 8; s++)
      if (s < (int)S) {
        uint32_t ra;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(at), "r"(s));
        q[0][s] = dsmem_ld4(ra);
        if (two) q[1][s] = dsmem_ld4(ra + NW * 512u);
      }
#pragma unroll
    for (int u = 0; u < 2; u++) {
      if (u == 1 && !two) break;
      const int m = u == 0 ? m0 : m1;
      float4 v = q[u][0];
#pragma unroll
      for (int s = 1; s < 8; s++)
        if (s < (int)S) v = add4(v, q[u][s]);
      if (n_live) {
        v = pair_epi_value4(e, v, cs, bs, res[u], m, OP);
        pair_epi_store4(e, v, m, n);
      }
      if (p.stats != nullptr) {
        const float2 st = tile_row_stats(v, n_live, cnt);
        if (lane == 0) p.stats[(size_t)m * p.f_tiles + ft] = st;
      }
    }
  }
  if (S > 1) {  // no CTA leaves while another may still read its partial tile (nothing is published by this barrier)
    cluster_arrive_relaxed();
    cluster_wait();
  } else {
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_acc, tmem_cols);
  }
  // here, where nothing else is in registers (ahead of the epilogue: prompts of 21 tokens 431 -> 446 us, XL 64 3.06 -> 3.18 ms)
  if (threadIdx.x == 0 && *abort_flag) {
    ring_drain(full_w, stages, requested, TC_POLLS);
    if (RN == 0) ring_drain(full_x, stages, requested, TC_POLLS);
  }
}

}  // namespace wgpt
