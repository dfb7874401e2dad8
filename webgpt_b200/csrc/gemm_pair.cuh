// C[M,N] = A[M,K] . Wt[N,K]^T (+ epilogue) for operands stored as pairs of half-precision planes (pair.cuh), many rows.
//
// Two CTAs of a cluster (two SMs) share one 256 x BN output tile through tcgen05 cta_group::2 (kind::f16, FP32
// accumulation). Per 64-deep k-block each CTA fetches its 128 rows of both planes of A (32 KB) and its BN/2 rows of both
// planes of Wt (one 3-D TMA box each, 128-byte swizzle), and the leader issues twelve MMAs: four 16-deep steps of
// h0 g0, h0 g1, h1 g0. Nothing passes through registers on the way in: both planes come ready from the producer of the
// matrix, so the only signals are TMA -> MMA -> TMA, and both CTAs' copies are counted on the leader's barrier.
//
// What bounds it: the tensor pipe, 6 BN cycles per k-block and pair; shared memory (operand reads of the MMAs, 4 KB + 16
// BN bytes each, plus the copies coming in) needs 640 + 2.5 BN cycles at 128 bytes a cycle, so a tile of fewer than
// about 180 columns is bound by shared memory instead. BN is a run-time multiple of 32 chosen by the host (pair_plan.h) so that
// rounds x max(6 BN, 640 + 2.5 BN) is smallest, in a model's prompts of up to 1024 rows by product_cycles, which knows the epilogue
// too: products of a few tiles per pair would
// otherwise leave a nearly empty last round (8192 x 768: 96 tiles of 256 columns on 74 pairs take two rounds, 128 of
// 192 columns take two shorter ones). 8192 x 8192 x 8192 runs at 470 TFLOP/s = 1410 issued, the rate a plain
// half-precision product sustains under the power cap.
//
// Accumulation: one FP32 accumulator in tensor memory over the whole of K. The tensor core truncates each time it adds to
// it, always towards zero, so the error grows with the number of MMAs: 12 per 64 of K here, 24 in the 3xTF32 kernel
// (GPT-2 XL logits of a 1024-token window, against FP32 mode: 2.3e-5 in 2-norm, 4.7e-5 in 3xTF32). Two accumulators
// alternate by tile, so a tile's epilogue (18 000 cycles for 128 x 256 FP32 values, most of it waiting for stores that
// L2 takes at about 2.2 TB/s when every SM stores at once) runs beside the next tile's MMAs. Summing shorter pieces
// of K into registers instead leaves the MMAs no room to run ahead: pieces of 128 / 256 / 384 took 109 / 91 / 79 us for
// 8192 x 2304 x 768 (3xTF32: 135 us).
//
// K split (clusters of 2 KS CTAs): where a product has fewer tiles than pairs, KS pairs share a tile, each with a slice of K, as
// their own accumulators; every CTA leaves its FP32 tile in its ring, the cluster synchronises once, and each pair finishes
// every KS-th 32-column block of the tile, adding the KS partial sums in slice order. One tile per cluster.
//
// Roles: warp 0 TMA producer, warp 1 MMA issuer (leader CTA only), warps 2-9 epilogue, two per quarter of the
// accumulator lanes. Every wait is bounded; on expiry the CTA sets *err = 3, drains and exits.
#pragma once
#include "gemm_tc2.cuh"
#include "pair.cuh"

namespace wgpt {

constexpr int GP_BM = 128, GP_BK = 64;             // rows of A per CTA; 64 halves = one 128-byte swizzle row
constexpr int GP_MAX_STAGES = 4;
constexpr int GP_A_BYTES = 2 * GP_BM * GP_BK * 2;  // both planes
constexpr int GP_RING_BYTES = 3 * 2 * GP_A_BYTES;  // stages of A, then Wt: three of a 256-column tile
constexpr int GP_EPI_WARPS = 8;
constexpr int GP_THREADS = 32 * (2 + GP_EPI_WARPS);
constexpr int GP_PAD = 32 * 33;
constexpr int GP_PART_LD = 36;                     // floats per row of a 32-column block of a partial tile: 16-byte rows, all banks
static_assert(8 * GP_BM * GP_PART_LD * 4 <= GP_RING_BYTES, "a 256-column partial tile lies over the ring");
constexpr size_t GP_SMEM_BYTES = 1024 + (size_t)GP_RING_BYTES + 256;

// One box of both planes of a pair matrix: {64 halves, box rows, 2 planes}.
__device__ __forceinline__ void tma_load_3d(void *dst, const CUtensorMap *map, int x, int y, uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
          smem_addr(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(0), "r"(smem_addr(bar))
      : "memory");
}
__device__ __forceinline__ void tma_load_3d_pair(void *dst, const CUtensorMap *map, int x, int y, uint32_t bar_addr) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%2, %3, %4}], [%5];" ::"r"(smem_addr(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(0), "r"(bar_addr)
      : "memory");
}
// Low word of umma_desc_sw128 (start address) and its constant high word. One lane issues every MMA of an SM, so what an
// instruction costs to issue bounds the narrow tiles: the descriptors' low words are sums of a per-stage base and a
// constant, and the loop around them is run by the whole warp, the lane being elected inside the instruction. Issued
// from a branch that one lane had taken, an MMA took about 98 cycles whatever its size (operands have to be moved to
// the uniform registers it reads, one by one); a decode product of 128 x 16 x 832 took 8.4 us, elected 5.5.
__device__ __forceinline__ uint32_t umma_desc_lo(uint32_t saddr) { return (saddr & 0x3FFFFu) >> 4; }
constexpr uint32_t kUmmaDescHi = (1024u >> 4) | (1u << 14) | (2u << 29);
__device__ __forceinline__ void umma2_f16(uint32_t tmem_d, uint32_t alo, uint32_t blo, uint32_t idesc,
                                          uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, e;\n\t.reg .b64 da, db;\n\t"
      "mov.b64 da, {%1, %5};\n\tmov.b64 db, {%2, %5};\n\t"
      "setp.ne.b32 p, %4, 0;\n\telect.sync _|e, 0xffffffff;\n\t"
      "@e tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %3, p;\n\t}" ::"r"(tmem_d),
      "r"(alo), "r"(blo), "r"(idesc), "r"(accumulate), "r"(kUmmaDescHi)
      : "memory");
}
// umma2_commit by one elected lane of a converged warp.
__device__ __forceinline__ void umma2_commit_elect(uint32_t cluster_addr) {
  asm volatile(
      "{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\t"
      "@e tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(cluster_addr)
      : "memory");
}
// Instruction descriptor of kind::f16: FP32 accumulate, half A and B, both K-major.
__host__ __device__ constexpr uint32_t f16_idesc(int m, int n) {
  return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// gridDim.x = 2 KS x clusters, cluster (2 KS,1,1). Cluster p walks the 256 x bn tiles p, p + clusters, ... (row tile fastest);
// with KS > 1 there are as many clusters as tiles.
// map_a: box of 128 rows; map_b: box of bn/2 rows. bn % 32 == 0, bn <= 256.
// b_exact: the weight is exact in one plane (integers of at most 11 bits) and has no second one (map_b: one plane).
__global__ void __launch_bounds__(GP_THREADS, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, int M, int K,
                 int N, int bn, int b_exact, Epilogue epi, int *err) {
  // narrower tiles leave room for a fourth stage (a copy takes about 3000 cycles to arrive under load)
  const int stage_bytes = GP_A_BYTES + bn * (b_exact ? GP_BK : GP_BK * 2);
  const int S = 4 * stage_bytes <= GP_RING_BYTES ? 4 : 3;
  extern __shared__ uint8_t gp_smem_raw[];
  uint8_t *tiles = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(gp_smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t *bars = reinterpret_cast<uint64_t *>(tiles + GP_RING_BYTES);
  uint64_t *full = bars, *empty = bars + GP_MAX_STAGES, *acc_full = bars + 2 * GP_MAX_STAGES;
  uint64_t *acc_empty = acc_full + 2;  // the leader's: an arrival of every epilogue warp of both CTAs
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(acc_empty + 2);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
  __shared__ float epi_pad[GP_EPI_WARPS * GP_PAD];

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  uint32_t cluster_size;
  asm volatile("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(cluster_size));
  const uint32_t crank = cluster_ctarank(), rank = crank & 1, lead = crank & ~1u;  // place in the pair, the pair's leader
  const bool leader = rank == 0;
  const int KS = (int)cluster_size >> 1, slice = (int)crank >> 1;
  const int all_kb = (K + GP_BK - 1) / GP_BK, kb0 = all_kb * slice / KS, total_kb = all_kb * (slice + 1) / KS - kb0;
  const int m_tiles = (M + 255) / 256, n_tiles = (N + bn - 1) / bn;
  const int n_work = m_tiles * n_tiles;
  const int pair = (int)(blockIdx.x / cluster_size), pairs = (int)(gridDim.x / cluster_size);

  if (threadIdx.x == 0) {
    for (int i = 0; i < S; i++) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < 2; i++) {
      mbar_init(&acc_full[i], 1);
      mbar_init(&acc_empty[i], 2 * GP_EPI_WARPS);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_async_smem();
  }
  if (warp == 1) tmem_alloc2(tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // both CTAs' barriers exist before anything is signalled across the pair
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  pdl_launch_dependents();
  pdl_wait();  // A (activations) comes from the previous kernel

  int issued = 0;  // stages that thread 0 has requested
  if (warp == 0) {
    if (lane == 0) {
      const uint32_t stage_tx = 2u * (uint32_t)stage_bytes;  // both CTAs
      int s = 0, phase = 0;  // ring position and the parity of the round through the ring
      for (int w = pair; w < n_work && !*abort_flag; w += pairs) {
        const int nt = w / m_tiles, mt = w - nt * m_tiles;
        const int m0 = mt * 256 + (int)rank * GP_BM, nb0 = nt * bn + (int)rank * (bn >> 1);
        for (int kb = 0; kb < total_kb; kb++) {
          uint8_t *st = tiles + (size_t)s * stage_bytes;
          if (*abort_flag || !mbar_wait(&empty[s], phase ^ 1, TC_POLLS)) { *abort_flag = 1; break; }
          const uint32_t lead_full = peer_smem_addr(&full[s], lead);
          if (leader) mbar_expect_tx(&full[s], stage_tx);
          tma_load_3d_pair(st, &map_a, (kb0 + kb) * GP_BK, m0, lead_full);
          tma_load_3d_pair(st + GP_A_BYTES, &map_b, (kb0 + kb) * GP_BK, nb0, lead_full);
          issued++;
          if (++s == S) { s = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    if (leader) {
      const uint32_t idesc = f16_idesc(256, bn);
      const uint32_t b_plane = ((uint32_t)(bn >> 1) * (GP_BK * 2)) >> 4, desc0 = umma_desc_lo(smem_addr(tiles));
      int s = 0, phase = 0, i = 0;  // i: tiles of this pair so far; accumulator = i & 1, its use count = i >> 1
      for (int w = pair; w < n_work; w += pairs, i++) {
        const int buf = i & 1, use = i >> 1;
        if (!mbar_wait(&acc_empty[buf], (use & 1) ^ 1, TC_POLLS << 4)) *abort_flag = 1;
        if (__any_sync(0xffffffffu, *abort_flag)) break;
        tc_fence_after();
        const uint32_t tmem_acc = tmem_base + (uint32_t)(buf * 256);
        for (int kb = 0; kb < total_kb; kb++) {
          if (!mbar_wait(&full[s], phase, TC_POLLS)) *abort_flag = 1;
          if (__any_sync(0xffffffffu, *abort_flag)) break;
          tc_fence_after();
          const uint32_t a0 = desc0 + (uint32_t)s * ((uint32_t)stage_bytes >> 4), a1 = a0 + (GP_A_BYTES >> 5);
          const uint32_t b0 = a0 + (GP_A_BYTES >> 4), b1 = b0 + b_plane;
#pragma unroll
          for (int k = 0; k < GP_BK / 16; k++) {
            umma2_f16(tmem_acc, a0 + 2 * k, b0 + 2 * k, idesc, (kb > 0 || k > 0) ? 1u : 0u);
            if (!b_exact) umma2_f16(tmem_acc, a0 + 2 * k, b1 + 2 * k, idesc, 1u);
            umma2_f16(tmem_acc, a1 + 2 * k, b0 + 2 * k, idesc, 1u);
          }
          umma2_commit_elect(smem_addr(&empty[s]));  // both CTAs may refill the stage once these MMAs have read it
          umma2_commit_elect(peer_smem_addr(&empty[s], lead + 1));
          if (++s == S) { s = 0; phase ^= 1; }
        }
        umma2_commit_elect(smem_addr(&acc_full[buf]));  // (also reached after an abort)
        umma2_commit_elect(peer_smem_addr(&acc_full[buf], lead + 1));
      }
    }
  } else {
    const int quad = warp & 3, half = (warp - 2) >> 2;  // two warps share a quarter of the lanes, alternate chunks
    float *pad = epi_pad + (warp - 2) * GP_PAD;
    const int sub_r = lane >> 3, col4 = (lane & 7) * 4;
    Epilogue e = epi;
    if (e.kc != nullptr && e.pos != nullptr) {  // one read of the position counter instead of one per store
      e.pos_base = __ldcg(e.pos);
      e.pos = nullptr;
    }
    const int chunks = bn >> 5;
    const bool vec_ok = ((N | e.ld) & 3) == 0;
    // a finished 32 x 32 block in `pad`: rows row0 .., columns nb ..
    auto out_block = [&](int row0, int nb) {
      const int n = nb + col4;
      if (vec_ok) {
        if (n < N) pair_epi_block(e, pad, row0, sub_r, col4, n, M);
      } else {
#pragma unroll 1
        for (int it = 0; it < 8; it++) {
          const int r = it * 4 + sub_r, m = row0 + r;
          if (m >= M) break;
#pragma unroll 1
          for (int k = 0; k < 4; k++)
            if (n + k < N) pair_epi1(e, pad[r * 33 + col4 + k], m, n + k);
        }
      }
    };
    int i = 0;
    if (KS > 1) {
      float *part = reinterpret_cast<float *>(tiles);
      if (!mbar_wait(&acc_full[0], 0, TC_POLLS << 4) || *abort_flag) *abort_flag = 1;
      tc_fence_after();
#pragma unroll 1
      for (int c = half; c < chunks; c += 2) {
        float v[32];
        tmem_ld_32x32(tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(c * 32), v);
        float4 *dst = reinterpret_cast<float4 *>(part + (size_t)(c * GP_BM + quad * 32 + lane) * GP_PART_LD);
#pragma unroll
        for (int j = 0; j < 8; j++) dst[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
      }
      tc_fence_before();
      cluster_arrive();
      cluster_wait();
      const int nt = pair / m_tiles, mt = pair - nt * m_tiles;
      const int row0 = mt * 256 + (int)rank * GP_BM + quad * 32;
#pragma unroll 1
      for (int c = slice + half * KS; c < chunks; c += 2 * KS) {
        const int nb = nt * bn + c * 32;
        if (row0 >= M || nb >= N) break;  // same for the whole warp
        const uint32_t at = smem_addr(part + (size_t)(c * GP_BM + quad * 32 + sub_r) * GP_PART_LD + col4);
        float4 t[8];
#pragma unroll 1
        for (int k = 0; k < KS; k++) {
          uint32_t ra;
          asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(at), "r"(2 * k + (int)rank));
          float4 q[8];
#pragma unroll
          for (int it = 0; it < 8; it++) q[it] = dsmem_ld4(ra + (uint32_t)(it * 4 * GP_PART_LD * 4));
#pragma unroll
          for (int it = 0; it < 8; it++) t[it] = k == 0 ? q[it] : add4(t[it], q[it]);
        }
#pragma unroll
        for (int it = 0; it < 8; it++) {
          float *d = pad + (it * 4 + sub_r) * 33 + col4;
          d[0] = t[it].x; d[1] = t[it].y; d[2] = t[it].z; d[3] = t[it].w;
        }
        __syncwarp();
        out_block(row0, nb);
        __syncwarp();
      }
    }
    for (int w = KS > 1 ? n_work : pair; w < n_work; w += pairs, i++) {
      const int nt = w / m_tiles, mt = w - nt * m_tiles;
      const int row0 = mt * 256 + (int)rank * GP_BM + quad * 32, n0 = nt * bn;
      const int buf = i & 1, use = i >> 1;
      if (!mbar_wait(&acc_full[buf], use & 1, TC_POLLS << 4) || *abort_flag) { *abort_flag = 1; break; }
      tc_fence_after();
      const uint32_t tmem_acc = tmem_base + (uint32_t)(buf * 256) + ((uint32_t)(quad * 32) << 16);
#pragma unroll 1
      for (int c = half; c < chunks; c += 2) {
        const int nb = n0 + c * 32;
        if (row0 >= M || nb >= N) break;  // same for the whole warp; nothing to read from here on
        float v[32];
        tmem_ld_32x32(tmem_acc + (uint32_t)(c * 32), v);
#pragma unroll
        for (int j = 0; j < 32; j++) pad[lane * 33 + j] = v[j];
        __syncwarp();
        out_block(row0, nb);
        __syncwarp();
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(peer_smem_addr(&acc_empty[buf], lead));
    }
    tc_fence_before();
  }

  if (KS > 1 && warp < 2) {  // the epilogue warps' barrier between partial tiles and sums
    cluster_arrive();
    cluster_wait();
  }
  __syncthreads();
  if (threadIdx.x == 0 && *abort_flag) {
    atomicExch(err, 3);
    pair_drain(full, S, issued, leader);
  }
  cluster_sync_all();  // neither CTA leaves (or frees tensor memory) while the other may still signal it
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc2(tmem_base, 512);
  }
}

}  // namespace wgpt
