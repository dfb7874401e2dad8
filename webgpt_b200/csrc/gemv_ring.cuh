// out[M,N] = x[M,K] . Wt[N,K]^T (+ epilogue) in FP32 on the CUDA cores for one to eight rows: the layer products of a decode
// step whose weights do not fit the SMs' shared memory (gemv_block_kernel) and are a stream from HBM.
//
// A CTA owns FT output columns (N / FT CTAs fill the SMs once) and pulls its rows of Wt through a ring of shared-memory
// stages by TMA ({256 of K, FT rows} per box, one producer warp). Eight warps share the columns (warp w: w, w + 8,
// ..), lanes share K: a step reads one float4 per column and one per row of x, which all of the warp's columns use. Sums
// stay in registers over the whole of K, so warps meet only at the ring's barriers.
//
// What bounds it: HBM, and the hand-off between dependent products (wait, read of x, LayerNorm, exchange: 3-4 us of a
// 10 us product). The ring is filled before the dependency wait, while the previous product finishes, so the stream stops
// for less than that. GPT-2 XL, one sequence, four products of a block: 51 us in the register-streaming kernel (2.4
// TB/s), 38 us here (3.2 TB/s); asking for the rest of the tile in L2 ahead of the wait gained nothing. Once its own last
// stage is requested, a CTA asks for its share of the next product's first 10 MB in L2 (RingArgs::ahead), so that HBM has
// something to do while the kernels change places: the next kernel's CTAs find no room before this one's leave.
//
//   x: gamma != nullptr: LayerNorm (instructions.js:451-550) of the rows by 8 / M warps each, the row in registers;
//      otherwise as it is. Rows of this CTA's slice of K live in shared memory.
//   S > 1 (long K with many rows, where every CTA staging all of x would cost more than the weights): the CTAs of a
//      cluster take slices of K and their sums are added in rank order through distributed shared memory.
// Every wait is bounded; on expiry *err = 2, the copies in flight get another bounded wait, and the result is void.
#pragma once
#include "gemm_tc.cuh"

namespace wgpt {

constexpr int GR_WARPS = 8;
constexpr int GR_THREADS = 32 * (GR_WARPS + 1);
constexpr int GR_MAX_STAGES = 16;
constexpr int GR_KT = 256;  // K values per stage: with 128 the warps spent more time at the barriers than reading
constexpr uint32_t GR_POLLS = 1u << 20;

struct RingArgs {
  const float *x;             // [rows][K]
  const float *gamma, *beta;  // LayerNorm of x, or nullptr (only then may S exceed 1)
  int rows, K, N, ft, stages;
  Epilogue epi;
  const char *ahead;          // the first bytes of the next product's weights, or nullptr
  unsigned int ahead_bytes;
  int *err;
};

// LayerNorm of the rows into shared memory by 8 / M warps each (M = 8, 4, 2, 1), a row of K <= 2048 values in registers
// throughout; gamma and beta are in shared memory already, or (ASYNC) on their way there by cp.async of these threads. red: 2 x
// 8 floats. With one warp for a row of 1600, fetching its scale and shift as it went, the stream waited 6 us.
template <int M, bool ASYNC>
__device__ __forceinline__ void ring_layernorm(const float *__restrict__ x, int rows, int K, const float4 *gam,
                                               const float4 *bet, float *xs, int xld, float *red, int warp, int lane) {
  constexpr int WPR = GR_WARPS / M, V = 16 / WPR > 1 ? 16 / WPR : 2;  // float4 per lane
  const int K4 = K >> 2, m = warp / WPR, part = warp % WPR;
  const bool live = m < rows;
  const float4 *src = reinterpret_cast<const float4 *>(x + (size_t)(live ? m : 0) * K);
  float4 v[V];
#pragma unroll
  for (int j = 0; j < V; j++) {
    const int i = (j * WPR + part) * 32 + lane;
    v[j] = live && i < K4 ? __ldcg(src + i) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  static_assert(!ASYNC || WPR > 1, "the barrier behind the first sum shows gamma and beta to everybody");
  if (ASYNC) cp_async_wait<0>();
  float s = 0.f;
#pragma unroll
  for (int j = 0; j < V; j++) s += (v[j].x + v[j].y) + (v[j].z + v[j].w);
  s = warp_sum(s);
  if (WPR > 1) {
    if (lane == 0) red[warp] = s;
    asm volatile("bar.sync 1, %0;" ::"n"(32 * GR_WARPS) : "memory");
    s = 0.f;
#pragma unroll
    for (int w = 0; w < WPR; w++) s += red[m * WPR + w];
  }
  const float mean = s / (float)K;
  float q = 0.f;
#pragma unroll
  for (int j = 0; j < V; j++)
    if ((j * WPR + part) * 32 + lane < K4) {
      const float a = v[j].x - mean, b = v[j].y - mean, c = v[j].z - mean, d = v[j].w - mean;
      q += (a * a + b * b) + (c * c + d * d);
    }
  q = warp_sum(q);
  if (WPR > 1) {
    if (lane == 0) red[8 + warp] = q;
    asm volatile("bar.sync 1, %0;" ::"n"(32 * GR_WARPS) : "memory");
    q = 0.f;
#pragma unroll
    for (int w = 0; w < WPR; w++) q += red[8 + m * WPR + w];
  }
  const float rsd = 1.0f / sqrtf(q / (float)K + 1e-5f);
  if (!live) return;
  float4 *dst = reinterpret_cast<float4 *>(xs + (size_t)m * xld);
#pragma unroll
  for (int j = 0; j < V; j++) {
    const int i = (j * WPR + part) * 32 + lane;
    if (i < K4) {
      const float4 g = gam[i], b = bet[i];
      dst[i] = make_float4(g.x * ((v[j].x - mean) * rsd) + b.x, g.y * ((v[j].y - mean) * rsd) + b.y,
                           g.z * ((v[j].z - mean) * rsd) + b.z, g.w * ((v[j].w - mean) * rsd) + b.w);
    } else if (i < (xld >> 2)) {
      dst[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
}

// grid = ceil(N / ft) * S, cluster (S,1,1). M: rows rounded up to 1, 2, 4, 5 or 8; FPW: columns per warp (ft <= 8 FPW).
// Dynamic shared memory: ring [stages][ft][kt] (128-byte aligned), x [M][K slice padded to kt], sums [ft][M] (padded to a
// multiple of 4), and with a LayerNorm gamma [K], beta [K].
template <int M, int FPW>
__global__ void __launch_bounds__(GR_THREADS, 1)
gemv_ring_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ RingArgs p) {
  extern __shared__ uint8_t gr_smem_raw[];
  __shared__ uint64_t full[GR_MAX_STAGES], empty[GR_MAX_STAGES];
  __shared__ int abort_word;
  __shared__ float ln_red[16];
  volatile int *abort_flag = &abort_word;
  float *ring = reinterpret_cast<float *>((reinterpret_cast<uintptr_t>(gr_smem_raw) + 127) & ~uintptr_t(127));
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  uint32_t S;
  asm volatile("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(S));
  const int rank = (int)cluster_ctarank();
  const int col0 = (int)(blockIdx.x / S) * p.ft, ncol = min(p.ft, p.N - col0);
  const int chunks_all = (p.K + GR_KT - 1) / GR_KT;
  const int ch0 = (int)((long long)chunks_all * rank / S), nch = (int)((long long)chunks_all * (rank + 1) / S) - ch0;
  const int stage_floats = p.ft * GR_KT;
  float *xs = ring + (size_t)p.stages * stage_floats;
  const int xld = ((chunks_all + (int)S - 1) / (int)S) * GR_KT;  // row stride of xs
  float *sums = xs + (size_t)M * xld;
  float4 *gam = reinterpret_cast<float4 *>(sums + ((p.ft * M + 3) & ~3)), *bet = gam + (p.K >> 2);

  // Scale and shift, up to two rows: asked for ahead of the weights and not waited for until the row is there. A CTA that
  // starts late, on an SM that its predecessor has just left, otherwise waits for them behind 148 rings of requests (3 us).
  // XL 1 x 200 + 32 / 2 x 300 + 24 tokens: 54.15 / 49.9 -> 53.75 / 49.1 ms; with four rows 54.9 -> 56.1.
  constexpr bool kAsyncNorm = M <= 2;
  if (kAsyncNorm && p.gamma != nullptr && warp < GR_WARPS) {
    for (int i = tid; i < (p.K >> 2); i += 32 * GR_WARPS) {
      cp_async16(smem_addr(gam + i), p.gamma + 4 * i);
      cp_async16(smem_addr(bet + i), p.beta + 4 * i);
    }
    cp_async_commit();
  }
  if (tid == 0) {
    for (int i = 0; i < p.stages; i++) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], GR_WARPS);
    }
    abort_word = 0;
    fence_async_smem();
  }
  __syncthreads();
  const uint32_t tx = (uint32_t)stage_floats * 4u;
  int issued = min(p.stages, nch);  // the producer thread's count
  if (warp == GR_WARPS && lane == 0) {
    const int pre = issued;
    for (int i = 0; i < pre; i++) {  // weights: ahead of the dependency wait
      mbar_expect_tx(&full[i], tx);
      tma_load_2d(ring + (size_t)i * stage_floats, &map_w, (ch0 + i) * GR_KT, col0, &full[i]);
    }
  }
  // the output this thread will finish (a second round of them is rare): its bias ahead of the wait, the rest right after
  Epilogue e = p.epi;
  const int o_first = rank * GR_THREADS + tid;
  const bool has = o_first < p.ft * p.rows && o_first % p.ft < ncol;
  const int m_first = o_first / p.ft, n_first = col0 + o_first % p.ft;
  float bias_v = 0.f, res_v = 0.f;
  if (has && e.bias != nullptr) bias_v = __ldg(e.bias + n_first);
  if (!kAsyncNorm && p.gamma != nullptr) {
    for (int i = tid; i < (p.K >> 2); i += GR_THREADS) {
      gam[i] = __ldg(reinterpret_cast<const float4 *>(p.gamma) + i);
      bet[i] = __ldg(reinterpret_cast<const float4 *>(p.beta) + i);
    }
    __syncthreads();
  }
  pdl_launch_dependents();
  pdl_wait();
  if (e.kc != nullptr && e.pos != nullptr) {
    e.pos_base = __ldcg(e.pos);
    e.pos = nullptr;
  }
  if (has && e.residual != nullptr) res_v = __ldcg(e.residual + (size_t)m_first * e.ld + n_first);

  if (warp == GR_WARPS) {
    if (lane == 0) {
      for (int i = p.stages, s = 0, ph = 0; i < nch; i++) {
        if (*abort_flag || !mbar_wait(&empty[s], ph, GR_POLLS)) { *abort_flag = 1; break; }
        mbar_expect_tx(&full[s], tx);
        tma_load_2d(ring + (size_t)s * stage_floats, &map_w, (ch0 + i) * GR_KT, col0, &full[s]);
        issued = i + 1;
        if (++s == p.stages) { s = 0; ph ^= 1; }
      }
      if (p.ahead != nullptr) {  // this CTA's share of what the next product is to find in L2
        const unsigned int n16 = p.ahead_bytes >> 4;
        const unsigned int beg = (unsigned int)((unsigned long long)n16 * blockIdx.x / gridDim.x);
        const unsigned int end = (unsigned int)((unsigned long long)n16 * (blockIdx.x + 1) / gridDim.x);
        for (unsigned int o = beg; o < end; o += 1024u) prefetch_l2(p.ahead + ((size_t)o << 4), min(end - o, 1024u) << 4);
      }
    }
    __syncwarp();
  } else {
    const int k_lo = ch0 * GR_KT, k_len = min(nch * GR_KT, p.K - k_lo);
    if (p.gamma != nullptr) {
      ring_layernorm<(M <= 2 ? M : (M <= 4 ? 4 : 8)), kAsyncNorm>(p.x, p.rows, p.K, gam, bet, xs, xld, ln_red, warp, lane);
    } else {
      // eight loads in flight per thread, whatever rows they fall into; every CTA reads the same rows at the same time,
      // so each starts at another place
      const int n4 = xld >> 2, live4 = k_len >> 2, total = p.rows * n4, K4 = p.K >> 2;
      const float4 *src = reinterpret_cast<const float4 *>(p.x + k_lo);
      const int rot = (int)((blockIdx.x * 52u) % (unsigned)total);
      for (int j0 = tid; j0 < total; j0 += 8 * 32 * GR_WARPS) {
        float4 v[8];
#pragma unroll
        for (int u = 0; u < 8; u++) {
          const int j = j0 + u * 32 * GR_WARPS;
          int idx = j + rot;
          idx = idx >= total ? idx - total : idx;
          const int m = (int)((unsigned)idx / (unsigned)n4), i = idx - m * n4;
          v[u] = j < total && i < live4 ? __ldcg(src + (size_t)m * K4 + i) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int u = 0; u < 8; u++) {
          const int j = j0 + u * 32 * GR_WARPS;
          int idx = j + rot;
          idx = idx >= total ? idx - total : idx;
          if (j < total) reinterpret_cast<float4 *>(xs)[idx] = v[u];
        }
      }
    }
    asm volatile("bar.sync 1, %0;" ::"n"(32 * GR_WARPS) : "memory");

    float acc[FPW][M];
#pragma unroll
    for (int f = 0; f < FPW; f++)
#pragma unroll
      for (int m = 0; m < M; m++) acc[f][m] = 0.f;
    int s = 0, ph = 0;
    for (int i = 0; i < nch; i++) {
      const bool ok = mbar_wait(&full[s], ph, GR_POLLS);
      if (!__all_sync(0xffffffffu, ok)) { *abort_flag = 1; break; }
      const float4 *w4 = reinterpret_cast<const float4 *>(ring + (size_t)s * stage_floats) + lane;
      const float4 *x4 = reinterpret_cast<const float4 *>(xs + (size_t)i * GR_KT) + lane;
#pragma unroll
      for (int t = 0; t < GR_KT / 128; t++) {
        float4 xv[M];
#pragma unroll
        for (int m = 0; m < M; m++) xv[m] = x4[(size_t)min(m, p.rows - 1) * (xld >> 2) + 32 * t];
#pragma unroll
        for (int f = 0; f < FPW; f++) {
          const float4 w = w4[min(warp + GR_WARPS * f, p.ft - 1) * (GR_KT >> 2) + 32 * t];
#pragma unroll
          for (int m = 0; m < M; m++) acc[f][m] += dot4(w, xv[m]);
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[s]);
      if (++s == p.stages) { s = 0; ph ^= 1; }
    }
#pragma unroll
    for (int f = 0; f < FPW; f++)
#pragma unroll
      for (int m = 0; m < M; m++) {
        const float v = warp_sum(acc[f][m]);
        if (lane == 0 && warp + GR_WARPS * f < p.ft) sums[(warp + GR_WARPS * f) * M + m] = v;
      }
  }
  if (S > 1) {
    cluster_arrive();
    cluster_wait();
  } else {
    __syncthreads();
  }
  if (tid == 32 * GR_WARPS && *abort_flag) {
    atomicExch(p.err, 2);
    ring_drain(full, p.stages, issued, GR_POLLS);
  }
  // outputs: column fastest, so that a warp stores runs of a row; a cluster's CTAs share them
  for (int o = o_first; o < p.ft * p.rows; o += (int)S * GR_THREADS) {
    const int m = o / p.ft, c = o - m * p.ft;
    if (c >= ncol) continue;
    float v = 0.f;
    if (S > 1) {
      for (int r = 0; r < (int)S; r++) {
        float t;
        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(t) : "r"(dsmem_addr(sums + c * M + m, (uint32_t)r)) : "memory");
        v += t;
      }
    } else {
      v = sums[c * M + m];
    }
    if (o == o_first) {
      v += bias_v;
      if (e.act == 1) v = gelu_f(v);
      *epi_addr(e, m, col0 + c) = v + res_v;
    } else {
      epi_store(e, v, m, col0 + c);
    }
  }
  if (S > 1) {  // no CTA leaves while another may still read its sums
    cluster_arrive_relaxed();
    cluster_wait();
  }
}

}  // namespace wgpt
