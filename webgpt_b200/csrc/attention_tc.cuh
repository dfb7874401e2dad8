// Prefill attention of a model on pairs (pair.cuh) for head size 64 and more than one tile of queries, on tcgen05: the same
// mathematics as attn_prefill64_pair_kernel (instructions.js:1101-1214, :593-666), whose warp-level MMAs ran at 153 TFLOP/s
// issued, one CTA of eight warps per SM waiting for its own chain of key tiles.
//
// Queries, keys and values come as pairs from the product that made them (pair_epi_store4), by TMA: a prompt at the start of
// the context. (Keys and values staged from the FP32 cache by three warps, each query tile again, were the kernel's bound:
// 2.1 us per tile of 64 keys.) A CTA takes 128 queries of one head against key tiles of 64:
//   one warp   TMA: the queries, then two tiles of keys and of values in flight;
//   one warp   issues the MMAs: scores S = Q K^T (three products) from shared memory, values O = P V with the probabilities as
//              the operand in tensor memory and the values' tile as the MN-major operand, as it lies;
//   4 KG warps softmax, a thread a query row: no shuffles, the tile's 64 scores in registers (half as many at a time, read
//              twice, took 4500 cycles per 128 keys). The probabilities' pairs go back in the scores' place; a tile's O is
//              added to FP32 sums in registers, which are rescaled there when the maximum has grown, so that nothing is
//              accumulated across tiles in tensor memory.
// S and O have two buffers each, so that the scores of the next tile are there when a tile is done. 256 columns of tensor memory
// and 97 KB of shared memory. KG == 1: one group of four softmax warps, two CTAs an SM. KG == 2: two groups take alternate
// tiles and meet at the end, one CTA an SM (168 registers): for grids where the chain of a row's tiles is what the kernel takes.
// What bounds it: a softmax warp's own path, 0.75 us per tile of 64 keys (64 exponentials at eight cycles, seven instructions each
// around them, two trips to tensor memory) and 0.7 us until the tile's O is added; the tensor pipe needs 0.5. Alone and
// cold, that kernel / this one: a layer of GPT-2 at 333 / 1024 tokens 17.2 / 12.4 and 39.3 / 22.5 us, of XL at 1024 64 / 27 us.
// Against float64 the logits are nearer than with that kernel (exp2_approx).
// Every wait is bounded; on expiry *err = 3 and the result is void.
#pragma once
#include "attention.cuh"
#include "gemm_split.cuh"

namespace wgpt {

constexpr int AT_Q = 128, AT_K = 64;  // queries per CTA, keys per tile
constexpr uint32_t AT_QPLANE = AT_Q * 128, AT_KPLANE = AT_K * 128;  // bytes of one plane of a tile
constexpr float AT_P_EXP = 4.f, AT_P_UP = kPairTop / 16.f;  // 2^AT_P_EXP AT_P_UP = kPairTop
constexpr uint32_t AT_COLS = 256, AT_O = 128;  // tensor memory: S / P at 0 and 64, O at 128 and 192
constexpr size_t attn_tc_smem_bytes() { return 1024 + (size_t)2 * AT_QPLANE + 8 * AT_KPLANE; }

// Both planes of a box of rows of one sequence: {64 halves, box rows, 1 sequence, 2 planes}.
__device__ __forceinline__ void tma_load_4d(void *dst, const CUtensorMap *map, int x, int y, int z, uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(
          smem_addr(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(0), "r"(smem_addr(bar))
      : "memory");
}
// D (+)= A[tensor memory] B[smem], by one elected lane of a converged warp.
__device__ __forceinline__ void umma1_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint32_t blo, uint32_t idesc,
                                             uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, e;\n\t.reg .b64 db;\n\t"
      "mov.b64 db, {%2, %5};\n\t"
      "setp.ne.b32 p, %4, 0;\n\telect.sync _|e, 0xffffffff;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %3, p;\n\t}" ::"r"(tmem_d),
      "r"(tmem_a), "r"(blo), "r"(idesc), "r"(accumulate), "r"(kUmmaDescHi)
      : "memory");
}
// 32 registers per thread -> 32 lanes x 32 consecutive 32-bit columns.
__device__ __forceinline__ void tmem_st_32x32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31};" ::"r"(r[0]),
      "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
      "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]),
      "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]),
      "r"(r[29]), "r"(r[30]), "r"(r[31]), "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// Two units in the last place, as expf; 0 for -infinity. exp2f in its place leaves every logit as it is (it differs below 2^-126
// alone) and takes 1.2 % of a pass of 1024 GPT-2 tokens. Logits of one block that is mostly attention, against float64, 1 to 52
// prompts of 65 to 1024 tokens at GPT-2's and XL's widths: nearer than with attn_prefill64_pair_kernel's expf at every size (GPT-2
// 65 / 333 / 1024 tokens 7.6e-7 / 1.15e-6 / 7.37e-6, were 9.6e-7 / 1.39e-6 / 7.51e-6; XL 1.17e-6 / 1.107e-5 / 1.504e-5, were 1.32e-6
// / 1.115e-5 / 1.525e-5); with q and k 2.5 times as large 31 % nearer to 1.5 % further, 3 % nearer on average.
__device__ __forceinline__ float exp2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// 32 lanes x 64 consecutive 32-bit columns -> 64 registers per thread, both loads in flight together.
__device__ __forceinline__ void tmem_ld_32x64(uint32_t taddr, float (&v)[64]) {
#define AT_R8(b) "=f"(v[b]), "=f"(v[b + 1]), "=f"(v[b + 2]), "=f"(v[b + 3]), "=f"(v[b + 4]), "=f"(v[b + 5]), "=f"(v[b + 6]), "=f"(v[b + 7])
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x64.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, "
      "%32, %33, %34, %35, %36, %37, %38, %39, %40, %41, %42, %43, %44, %45, %46, %47, "
      "%48, %49, %50, %51, %52, %53, %54, %55, %56, %57, %58, %59, %60, %61, %62, %63}, [%64];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : AT_R8(0), AT_R8(8), AT_R8(16), AT_R8(24), AT_R8(32), AT_R8(40), AT_R8(48), AT_R8(56)
      : "r"(taddr)
      : "memory");
#undef AT_R8
}

// 2^d of a whole number d <= 0 (or -infinity), exactly; 0 below the normal range.
__device__ __forceinline__ float pow2_whole(float d) { return __int_as_float(max(0, 127 + (int)d) << 23); }

// gridDim.x = query tiles x heads x sequences. map_q, map_kv: planes [2][n_seq][n_tok][3 E] of q | k | v, boxes of 128 and 64
// rows, zeros beyond a sequence's tokens. Output planes [2][n_seq * n_tok][ldo].
template <int KG>
__global__ void __launch_bounds__(128 * KG + 64, KG == 1 ? 2 : 1)
attn_prefill64_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_kv, int n_tok, int H,
                         float to_exp2, __half *__restrict__ planes, size_t plane, int ldo, int *err) {
  extern __shared__ uint8_t at_smem_raw[];
  uint8_t *Qs = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(at_smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t *Ks = Qs + 2 * AT_QPLANE, *Vs = Ks + 4 * AT_KPLANE;  // [2 tiles][2 planes][64 keys][128 bytes]
  __shared__ uint64_t q_full, k_full[2], v_full[2], s_done[2], p_ready[2], o_done[2], drained;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_word;
  volatile int *abort_flag = &abort_word;
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  // The query tiles with the most keys first: an SM takes its next CTA when one of its own ends.
  const int order = (int)blockIdx.x, n_tiles = (n_tok + AT_Q - 1) / AT_Q, heads = (int)gridDim.x / n_tiles;
  const int hq = order % heads, h = hq % H, seq = hq / H, t0 = (n_tiles - 1 - order / heads) * AT_Q;
  const int nq = min(AT_Q, n_tok - t0);
  const int tiles = (t0 + nq - 1) / AT_K + 1;  // key tiles up to the newest key any query of this tile may see

  if (tid == 0) {
    mbar_init(&q_full, 1);
    for (int b = 0; b < 2; b++) {
      mbar_init(&k_full[b], 1);
      mbar_init(&v_full[b], 1);
      mbar_init(&p_ready[b], 4);
      mbar_init(&s_done[b], 1);
      mbar_init(&o_done[b], 1);
    }
    mbar_init(&drained, 1);
    abort_word = 0;
    fence_async_smem();
  }
  if (warp == 4 * KG) tmem_alloc(&tmem_slot, AT_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  if (tid == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&map_q)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&map_kv)) : "memory");
  }
  pdl_launch_dependents();  // behind the allocation: the next kernel's CTAs want tensor memory too
  pdl_wait();
  // Barriers of tile i: index i & 1, parity (i >> 1) & 1. False, for the whole warp: give up.
  auto waited = [&](uint64_t *bar, int i) -> bool {
    if (!mbar_wait(bar + (i & 1), (i >> 1) & 1, TC_POLLS)) *abort_flag = 1;
    return !__any_sync(0xffffffffu, *abort_flag);
  };

  if (warp < 4 * KG) {
    const int kg = warp >> 2, quad = warp & 3;
    const int prow = t0 + min(tid & 127, nq - 1);  // rows past the end shadow the last
    const int warp_first = t0 + min(32 * quad, nq - 1), warp_last = t0 + min(32 * quad + 31, nq - 1);
    const bool warp_live = 32 * quad < nq;
    const float c = to_exp2;  // raw score -> exponent of two; positive
    // Running maximum of this thread's row as a power of two, rounded up, and sum of the probabilities. With a whole number the
    // shift and every rescale are exact, and an exponent has the rounding of one multiply-add. A probability is held times
    // kPairTop, as every value that becomes a pair: 2^AT_P_EXP of it in the exponent, where the ones that count are then small
    // numbers, the rest by an exact multiplication. (With all of it in the exponent the logits of XL at 1024 tokens were 2 %
    // further from float64; with 2^AT_P_EXP alone a pair ends at 2^-29 of its row's largest instead of 2^-40, and GPT-2 prompts
    // of 333 / 1024 tokens take 801 / 1400 us instead of 803 / 1406.)
    float m = -INFINITY, l = 0.f;
    float o[64];
#pragma unroll
    for (int d = 0; d < 64; d++) o[d] = 0.f;
    const uint32_t lanes = tmem + ((uint32_t)(32 * quad) << 16);
    for (int i = kg; i < tiles; i += KG) {
      const int j0 = i * AT_K;
      const bool seen = warp_live && j0 <= warp_last;  // otherwise nothing of the tile concerns this warp's rows
      float corr = 1.f;
      if (!waited(s_done, i)) break;
      if (seen) {
        tc_fence_after();
        const uint32_t sp = lanes + (uint32_t)((i & 1) * AT_K);
        float v[64];
        tmem_ld_32x64(sp, v);
        if (j0 + AT_K - 1 > warp_first) {  // some key is beyond some row
#pragma unroll
          for (int u = 0; u < 64; u++) v[u] = j0 + u <= prow ? v[u] : -INFINITY;
        }
        float x0 = v[0], x1 = v[1], x2 = v[2], x3 = v[3];
#pragma unroll
        for (int u = 4; u < 64; u += 4) {
          x0 = fmaxf(x0, v[u]);
          x1 = fmaxf(x1, v[u + 1]);
          x2 = fmaxf(x2, v[u + 2]);
          x3 = fmaxf(x3, v[u + 3]);
        }
        // finite: a row of a warp that a tile concerns sees that tile's first key (rows in groups of 32, tiles of 64)
        const float mn = fmaxf(m, ceilf(fmaxf(fmaxf(x0, x1), fmaxf(x2, x3)) * c));
        corr = pow2_whole(m - mn);
        m = mn;
        const float shift = AT_P_EXP - mn;
        float p0 = 0.f, p1 = 0.f, p2 = 0.f, p3 = 0.f;
#pragma unroll
        for (int half = 0; half < 2; half++) {
          uint32_t r[32];  // sixteen columns of the first plane, sixteen of the second
#pragma unroll
          for (int u = 0; u < 32; u += 4) {
            float *e = v + 32 * half + u;
#pragma unroll
            for (int k = 0; k < 4; k++) e[k] = exp2_approx(fmaf(e[k], c, shift)) * AT_P_UP;
            p0 += e[0]; p1 += e[1]; p2 += e[2]; p3 += e[3];
            r[u / 2] = pair_word(e[0], e[1], r[16 + u / 2]);
            r[u / 2 + 1] = pair_word(e[2], e[3], r[17 + u / 2]);
          }
          tmem_st_32x32(sp + 32u * half, r);  // over the scores they came from
        }
        l = l * corr + ((p0 + p1) + (p2 + p3));
        tmem_wait_st();
        tc_fence_before();
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_ready[i & 1]);
      if (!waited(o_done, i)) break;
      if (seen) {
        tc_fence_after();
        float v[64];
        tmem_ld_32x64(lanes + AT_O + (uint32_t)((i & 1) * 64), v);
#pragma unroll
        for (int d = 0; d < 64; d++) o[d] = o[d] * corr + v[d];
        tc_fence_before();
      }
    }
    if (KG > 1) {  // the second group's sums to the first, over the tiles of keys and values: [66][128] floats
      float *rec = reinterpret_cast<float *>(Ks) + (tid & 127);
      asm volatile("bar.sync 1, %0;" ::"n"(128 * KG) : "memory");  // every product has read its tiles
      if (kg > 0) {
#pragma unroll
        for (int d = 0; d < 64; d++) rec[d * 128] = o[d];
        rec[64 * 128] = m;
        rec[65 * 128] = l;
      }
      asm volatile("bar.sync 1, %0;" ::"n"(128 * KG) : "memory");
      if (kg == 0) {
        const float n = rec[64 * 128], x = fmaxf(m, n);  // finite: the first group has seen key 0
        const float ca = pow2_whole(m - x), cb = pow2_whole(n - x);
        l = l * ca + rec[65 * 128] * cb;
#pragma unroll
        for (int d = 0; d < 64; d++) o[d] = o[d] * ca + rec[d * 128] * cb;
      }
    }
    // Out through shared memory (the queries' place; every product has read them), so that 128 bytes of a row leave
    // together; the probabilities' power of two is in l too, and the values' own scale is also the output pair's.
    if (kg == 0 && warp_live) {
      const float inv = 1.f / l;
      uint8_t *row = Qs + tid * 128;
#pragma unroll
      for (int d = 0; d < 8; d++) {
        uint4 a, b;
        a.x = pair_word(o[8 * d] * inv, o[8 * d + 1] * inv, b.x);
        a.y = pair_word(o[8 * d + 2] * inv, o[8 * d + 3] * inv, b.y);
        a.z = pair_word(o[8 * d + 4] * inv, o[8 * d + 5] * inv, b.z);
        a.w = pair_word(o[8 * d + 6] * inv, o[8 * d + 7] * inv, b.w);
        *reinterpret_cast<uint4 *>(row + ((d ^ (tid & 7)) << 4)) = a;
        *reinterpret_cast<uint4 *>(row + AT_QPLANE + ((d ^ (tid & 7)) << 4)) = b;
      }
      __syncwarp();
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const int r = 32 * warp + 4 * i + (lane >> 3), d = lane & 7;
        if (r < nq) {
          const uint8_t *src = Qs + r * 128 + ((d ^ (r & 7)) << 4);
          __half *at = planes + ((size_t)seq * n_tok + t0 + r) * ldo + h * 64 + 8 * d;
          *reinterpret_cast<uint4 *>(at) = *reinterpret_cast<const uint4 *>(src);
          *reinterpret_cast<uint4 *>(at + plane) = *reinterpret_cast<const uint4 *>(src + AT_QPLANE);
        }
      }
    }
  } else if (warp == 4 * KG + 1) {
    const int x = h * 64, E = H * 64;
    int issued = 0;  // tiles of keys and of values requested
    if (lane == 0) {
      mbar_expect_tx(&q_full, 2 * AT_QPLANE);
      tma_load_4d(Qs, &map_q, x, t0, seq, &q_full);
    }
    auto ask = [&](int i, uint8_t *dst, int col, uint64_t *bars) {
      if (lane == 0) {
        mbar_expect_tx(bars + (i & 1), 2 * AT_KPLANE);
        tma_load_4d(dst + (size_t)(i & 1) * 2 * AT_KPLANE, &map_kv, col, i * AT_K, seq, bars + (i & 1));
      }
    };
    for (int i = 0; i < tiles; i++) {
      if (i >= 2 && !waited(s_done, i - 2)) break;  // the MMAs have read what was there
      ask(i, Ks, x + E, k_full);
      if (i >= 2 && !waited(o_done, i - 2)) {  // (void: the keys' copy is waited for all the same)
        mbar_wait(&k_full[i & 1], (i >> 1) & 1, TC_POLLS);
        break;
      }
      ask(i, Vs, x + 2 * E, v_full);
      issued = i + 1;
    }
    if (__any_sync(0xffffffffu, *abort_flag)) {
      mbar_wait(&q_full, 0, TC_POLLS);
      ring_drain(k_full, 2, issued, TC_POLLS);
      ring_drain(v_full, 2, issued, TC_POLLS);
    }
  } else {
    // the whole warp runs this and one elected lane issues
    const uint32_t q0 = umma_desc_lo(smem_addr(Qs)), k0 = umma_desc_lo(smem_addr(Ks)), v0 = umma_desc_lo(smem_addr(Vs));
    const uint32_t idesc = f16_idesc(128, 64), idesc_o = idesc | (1u << 16);  // values: MN-major
    auto scores = [&](int i) {
      const uint32_t d = tmem + (uint32_t)((i & 1) * AT_K), kt = k0 + (uint32_t)(i & 1) * (2u * AT_KPLANE >> 4);
      // The corrections first: the accumulator truncates with every instruction, and is small until the main products come.
#pragma unroll
      for (int s = 0; s < 4; s++) {
        umma1_f16(d, q0 + 2 * s, kt + (AT_KPLANE >> 4) + 2 * s, idesc, s > 0 ? 1u : 0u);
        umma1_f16(d, q0 + (AT_QPLANE >> 4) + 2 * s, kt + 2 * s, idesc, 1u);
      }
#pragma unroll
      for (int s = 0; s < 4; s++) umma1_f16(d, q0 + 2 * s, kt + 2 * s, idesc, 1u);
      umma_commit_elect(&s_done[i & 1]);
    };
    bool ok = waited(&q_full, 0);
    for (int i = 0; ok && i < min(tiles, 2); i++) {
      ok = waited(k_full, i);
      if (!ok) break;
      tc_fence_after();
      scores(i);
    }
    for (int i = 0; ok && i < tiles; i++) {
      ok = waited(v_full, i) && waited(p_ready, i);
      if (!ok) break;
      tc_fence_after();
      const uint32_t d = tmem + AT_O + (uint32_t)((i & 1) * 64), p = tmem + (uint32_t)((i & 1) * AT_K);
      const uint32_t vt = v0 + (uint32_t)(i & 1) * (2u * AT_KPLANE >> 4);
      // 16 keys: 8 columns of each plane, 16 rows of the values' tile; the corrections first here too
#pragma unroll
      for (int s = 0; s < 4; s++) {
        const uint32_t p0 = p + 32u * (s >> 1) + 8u * (s & 1), vs = vt + (uint32_t)s * (2048u >> 4);
        umma1_f16_ts(d, p0, vs + (AT_KPLANE >> 4), idesc_o, s > 0 ? 1u : 0u);
        umma1_f16_ts(d, p0 + 16u, vs, idesc_o, 1u);
      }
#pragma unroll
      for (int s = 0; s < 4; s++)
        umma1_f16_ts(d, p + 32u * (s >> 1) + 8u * (s & 1), vt + (uint32_t)s * (2048u >> 4), idesc_o, 1u);
      umma_commit_elect(&o_done[i & 1]);
      if (i + 2 < tiles) {  // into the probabilities' place once they have been read
        ok = waited(k_full, i + 2) && waited(o_done, i);
        if (!ok) break;
        tc_fence_after();
        scores(i + 2);
      }
    }
    if (__any_sync(0xffffffffu, *abort_flag)) {  // what has been issued ends before its operands go
      umma_commit_elect(&drained);
      mbar_wait(&drained, 0, TC_POLLS);
    }
  }
  __syncthreads();
  if (tid == 0 && *abort_flag) atomicExch(err, 3);
  if (warp == 4 * KG) {
    tc_fence_after();
    tmem_dealloc(tmem, AT_COLS);
  }
}

}  // namespace wgpt
