// Top-k sampling of the next token on the device: the reference's selectTopK -> cpuSoftmax ->
// sampleFromDistribution chain (globals.js:47-74, called at model.js:81-83) without reading the logits back.
// The reference draws Math.random() inside sampleFromDistribution; here the caller supplies one uniform
// number per (step, sequence), so a run is reproducible and can be compared token for token with a CPU run
// that uses the same numbers.
//
// One CTA of 1024 threads per sequence:
//   1. every thread folds its strided share of the logits into one 64-bit key (order-preserving float bits in
//      the high word, ~index in the low word, so larger key = earlier in the reference's stable descending sort);
//   2. a bitonic sort of the 1024 per-thread maxima gives tau, the top_k-th largest of them: a lower bound of
//      the true top_k-th key, reached by exactly top_k threads;
//   3. those threads rescan their share and append every key >= tau to a candidate list
//      (at most top_k * ceil(V / 1024) entries); a rank sort of the candidates yields the top_k keys in order;
//   4. exp((v - max) / temperature) in double precision, a left-to-right sum and running sum as in the
//      reference, and the first index whose running sum exceeds the uniform number is the pick.
// The kernel then writes the token and advances the session like argmax_kernel.
#pragma once
#include "common.cuh"

namespace wgpt {

constexpr int kSampleThreads = 1024;
constexpr int kMaxTopK = 128;

__device__ __forceinline__ unsigned long long sample_key(float v, int idx) {
  uint32_t u = __float_as_uint(v);
  if (u == 0x80000000u) u = 0u;  // -0 and +0 compare equal in the reference's sort
  uint32_t k = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
  return ((unsigned long long)k << 32) | (unsigned long long)(0xFFFFFFFFu - (uint32_t)idx);
}

__device__ __forceinline__ int sample_key_index(unsigned long long c) {
  return (int)(0xFFFFFFFFu - (uint32_t)(c & 0xFFFFFFFFull));
}

// Dynamic shared memory: (1024 + cap) 64-bit keys, cap = top_k * ceil(V / 1024).
// uniforms: [steps][gridDim.x] doubles in [0,1), indexed by the session's step counter.
// done_counter must be zero on entry and is left zero.
__global__ void __launch_bounds__(kSampleThreads)
sample_topk_kernel(const float *__restrict__ logits, int V, int top_k, double temperature,
                   const double *__restrict__ uniforms, int cap, uint32_t *__restrict__ next_ids,
                   uint32_t *__restrict__ out_ids, int out_stride, int *__restrict__ pos, int *__restrict__ step,
                   int n_tok, unsigned int *__restrict__ done_counter) {
  extern __shared__ __align__(16) unsigned long long skeys[];
  unsigned long long *srt = skeys;
  unsigned long long *cand = skeys + kSampleThreads;
  __shared__ unsigned long long top[kMaxTopK];
  __shared__ double ev[kMaxTopK];
  __shared__ double s_sum;
  __shared__ int s_cnt;
  pdl_launch_dependents();
  pdl_wait();
  const int seq = blockIdx.x, tid = threadIdx.x;
  const int my_step = __ldcg(step);
  const float *x = logits + (size_t)seq * V;

  unsigned long long best = 0ull;  // below every real key (their low word is never zero for idx < 2^32 - 1)
  {
    int i = tid;  // 16 loads in flight per thread: one CTA scans the row, so latency is what bounds it
    for (; i + 15 * kSampleThreads < V; i += 16 * kSampleThreads) {
      float f[16];
#pragma unroll
      for (int u = 0; u < 16; u++) f[u] = __ldcg(x + i + u * kSampleThreads);
#pragma unroll
      for (int u = 0; u < 16; u++) {
        unsigned long long c = sample_key(f[u], i + u * kSampleThreads);
        best = c > best ? c : best;
      }
    }
    for (; i + 3 * kSampleThreads < V; i += 4 * kSampleThreads) {
      float f[4];
#pragma unroll
      for (int u = 0; u < 4; u++) f[u] = __ldcg(x + i + u * kSampleThreads);
#pragma unroll
      for (int u = 0; u < 4; u++) {
        unsigned long long c = sample_key(f[u], i + u * kSampleThreads);
        best = c > best ? c : best;
      }
    }
    for (; i < V; i += kSampleThreads) {
      unsigned long long c = sample_key(__ldcg(x + i), i);
      best = c > best ? c : best;
    }
  }
  srt[tid] = best;
  if (tid == 0) s_cnt = 0;
  __syncthreads();
  // bitonic sort, descending
  for (int k2 = 2; k2 <= kSampleThreads; k2 <<= 1) {
    for (int j = k2 >> 1; j > 0; j >>= 1) {
      int other = tid ^ j;
      if (other > tid) {
        unsigned long long a = srt[tid], b = srt[other];
        bool desc = (tid & k2) == 0;
        if (desc ? (a < b) : (a > b)) { srt[tid] = b; srt[other] = a; }
      }
      __syncthreads();
    }
  }
  const unsigned long long tau = srt[top_k - 1];
  if (best >= tau && best != 0ull) {  // at most top_k threads: their share again, 16 loads at a time
    int i = tid;
    for (; i + 15 * kSampleThreads < V; i += 16 * kSampleThreads) {
      float f[16];
#pragma unroll
      for (int u = 0; u < 16; u++) f[u] = __ldcg(x + i + u * kSampleThreads);
#pragma unroll
      for (int u = 0; u < 16; u++) {
        unsigned long long c = sample_key(f[u], i + u * kSampleThreads);
        if (c >= tau) {
          int slot = atomicAdd(&s_cnt, 1);
          if (slot < cap) cand[slot] = c;
        }
      }
    }
    for (; i < V; i += kSampleThreads) {
      unsigned long long c = sample_key(__ldcg(x + i), i);
      if (c >= tau) {
        int slot = atomicAdd(&s_cnt, 1);
        if (slot < cap) cand[slot] = c;
      }
    }
  }
  __syncthreads();
  const int C = s_cnt < cap ? s_cnt : cap;
  for (int i = tid; i < C; i += kSampleThreads) {
    unsigned long long ci = cand[i];
    int rank = 0;
    for (int j = 0; j < C; j++) rank += cand[j] > ci ? 1 : 0;
    if (rank < top_k) top[rank] = ci;
  }
  __syncthreads();
  // softmax over the kept logits in double precision (JS numbers), globals.js:59-64
  const double vmax = (double)__ldcg(x + sample_key_index(top[0]));
  if (tid < top_k) ev[tid] = exp(((double)__ldcg(x + sample_key_index(top[tid])) - vmax) / temperature);
  __syncthreads();
  if (tid == 0) {
    double s = 0.0;
    for (int j = 0; j < top_k; j++) s += ev[j];
    s_sum = s;
  }
  __syncthreads();
  if (tid < top_k) ev[tid] = ev[tid] / s_sum;
  __syncthreads();
  if (tid == 0) {
    const double u = __ldcg(uniforms + (size_t)my_step * gridDim.x + seq);
    int pick = top_k - 1;
    double cum = 0.0;
    for (int j = 0; j < top_k; j++) {
      cum += ev[j];
      if (u < cum) { pick = j; break; }
    }
    uint32_t id = (uint32_t)sample_key_index(top[pick]);
    next_ids[seq] = id;
    if (out_ids) out_ids[(size_t)seq * out_stride + my_step] = id;
    __threadfence();
    unsigned int prev = atomicAdd(done_counter, 1u);
    if (prev == gridDim.x - 1) {
      *pos = __ldcg(pos) + n_tok;
      *step = my_step + 1;
      *done_counter = 0u;
    }
  }
}

// ------------------------------------------------------------------------------------------------
// The same pick for top_k <= 48 by a cluster of C CTAs per sequence, each holding its share of the logits in registers (for
// few rows; pick_in_cluster in api.cu has the limits). A
// decode step waits for this kernel, and what it takes is a chain of latencies: one CTA reading the row twice and sorting
// 1024 maxima (55 barriers) took 10.6 us per token at 50257 logits; this form takes 8 us off the step (GPT-2, top_k 3 / 20: 235.8 / 238.8 -> 221 / 223).
//   1. every thread reads its logits once, all loads in flight; the 64 groups of eight lanes leave their best keys in shared
//      memory and every warp finds the top_k-th largest of them: a bound that at least top_k values of this CTA's share reach;
//   2. values at or above it go straight to a list of this CTA in the first CTA's shared memory (more than kPickCap of them,
//      which takes a row made for it: this CTA's exact top_k instead, one block-wide maximum at a time);
//   3. after one cluster barrier the first CTA drops what is below the largest of the C bounds, ranks the rest, and goes on
//      as sample_topk_kernel does from its sorted list, with the logits taken out of the keys.
constexpr int kPickThreads = 512, kPickVals = 16, kPickCap = 256, kPickTopK = 48, kPickCluster = 8;

__device__ __forceinline__ float sample_key_value(unsigned long long c) {
  const uint32_t k = (uint32_t)(c >> 32);
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k);
}
__device__ __forceinline__ unsigned long long max64(unsigned long long a, unsigned long long b) { return a > b ? a : b; }

__global__ void __launch_bounds__(kPickThreads)
sample_pick_kernel(const float *__restrict__ logits, int V, int top_k, double temperature,
                   const double *__restrict__ uniforms, uint32_t *__restrict__ next_ids, uint32_t *__restrict__ out_ids,
                   int out_stride, int *__restrict__ pos, int *__restrict__ step, int n_tok,
                   unsigned int *__restrict__ done_counter) {
  __shared__ unsigned long long lists[kPickCluster][kPickCap];  // used in the first CTA
  __shared__ unsigned long long bounds[kPickCluster];
  __shared__ int counts[kPickCluster];
  __shared__ unsigned long long best_hw[64], kept[kPickCluster * kPickCap], top[kPickTopK];
  __shared__ double ev[kPickTopK];
  __shared__ double s_sum;
  __shared__ int s_cnt;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  uint32_t C;
  asm volatile("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(C));
  const int rank = (int)cluster_ctarank(), seq = blockIdx.x / C, rows = gridDim.x / C;
  cluster_arrive();  // pairs with the wait ahead of the first remote store
  if (tid == 0) s_cnt = 0;
  pdl_launch_dependents();
  pdl_wait();
  const int my_step = __ldcg(step);
  const int share = (V + (int)C - 1) / (int)C, beg = rank * share, end = min(V, beg + share);
  const float *x = logits + (size_t)seq * V;
  float f[kPickVals];
#pragma unroll
  for (int u = 0; u < kPickVals; u++) {
    const int i = beg + tid + u * kPickThreads;
    f[u] = i < end ? __ldcg(x + i) : 0.f;
  }
  double uni = 0.0;
  if (rank == 0 && tid == 0) uni = __ldcg(uniforms + (size_t)my_step * rows + seq);
  auto key_of = [&](int u) -> unsigned long long {
    const int i = beg + tid + u * kPickThreads;
    return i < end ? sample_key(f[u], i) : 0ull;
  };
  unsigned long long best = 0ull;
#pragma unroll
  for (int u = 0; u < kPickVals; u++) best = max64(best, key_of(u));
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) best = max64(best, __shfl_xor_sync(0xffffffffu, best, o));
  if ((lane & 7) == 0) best_hw[4 * warp + (lane >> 3)] = best;
  __syncthreads();
  unsigned long long tau;
  {
    const unsigned long long m0 = best_hw[lane], m1 = best_hw[lane + 32];
    int r0 = 0, r1 = 0;
#pragma unroll 8
    for (int j = 0; j < 64; j++) {
      const unsigned long long c = best_hw[j];
      r0 += c > m0 ? 1 : 0;
      r1 += c > m1 ? 1 : 0;
    }
    const unsigned int a0 = __ballot_sync(0xffffffffu, r0 == top_k - 1 && m0 != 0ull);
    const unsigned int a1 = __ballot_sync(0xffffffffu, r1 == top_k - 1 && m1 != 0ull);
    const unsigned long long t0 = __shfl_sync(0xffffffffu, m0, a0 ? __ffs(a0) - 1 : 0);
    const unsigned long long t1 = __shfl_sync(0xffffffffu, m1, a1 ? __ffs(a1) - 1 : 0);
    tau = a0 ? t0 : (a1 ? t1 : 1ull);  // fewer groups with a value than top_k: every value counts
  }
  cluster_wait();
#pragma unroll
  for (int u = 0; u < kPickVals; u++) {
    const unsigned long long c = key_of(u);
    if (c >= tau) {
      const int slot = atomicAdd(&s_cnt, 1);
      if (slot < kPickCap) dsmem_st64(dsmem_addr(&lists[rank][slot], 0), c);
    }
  }
  __syncthreads();
  int cnt = s_cnt;
  if (cnt > kPickCap) {
    unsigned long long last = ~0ull;
    for (cnt = 0; cnt < top_k; cnt++) {
      unsigned long long b = 0ull;
#pragma unroll
      for (int u = 0; u < kPickVals; u++) {
        const unsigned long long c = key_of(u);
        b = c < last ? max64(b, c) : b;
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) b = max64(b, __shfl_xor_sync(0xffffffffu, b, o));
      __syncthreads();
      if (lane == 0) best_hw[warp] = b;
      __syncthreads();
      b = 0ull;
      for (int w = 0; w < kPickThreads / 32; w++) b = max64(b, best_hw[w]);
      if (tid == 0) dsmem_st64(dsmem_addr(&lists[rank][cnt], 0), b);
      last = b;
    }
  }
  if (tid == 0) {
    dsmem_st64(dsmem_addr(&bounds[rank], 0), tau);
    dsmem_st(dsmem_addr(&counts[rank], 0), __int_as_float(cnt));
  }
  cluster_arrive();
  cluster_wait();
  if (rank != 0) return;
  if (tid == 0) s_cnt = 0;
  unsigned long long floor_key = 0ull;
  for (int r = 0; r < (int)C; r++) floor_key = max64(floor_key, bounds[r]);
  __syncthreads();
  for (int i = tid; i < (int)C * kPickCap; i += kPickThreads) {
    const int r = i / kPickCap, j = i % kPickCap;
    if (j < counts[r] && lists[r][j] >= floor_key) kept[atomicAdd(&s_cnt, 1)] = lists[r][j];
  }
  __syncthreads();
  const int n = s_cnt;
  for (int i = tid; i < n; i += kPickThreads) {
    const unsigned long long ci = kept[i];
    int r = 0;
#pragma unroll 4
    for (int j = 0; j < n; j++) r += kept[j] > ci ? 1 : 0;
    if (r < top_k) top[r] = ci;
  }
  __syncthreads();
  // softmax over the kept logits in double precision (JS numbers), globals.js:59-64
  if (tid < top_k) ev[tid] = exp(((double)sample_key_value(top[tid]) - (double)sample_key_value(top[0])) / temperature);
  __syncthreads();
  if (tid == 0) {
    double s = 0.0;
    for (int j = 0; j < top_k; j++) s += ev[j];
    s_sum = s;
  }
  __syncthreads();
  if (tid < top_k) ev[tid] = ev[tid] / s_sum;
  __syncthreads();
  if (tid == 0) {
    int pick = top_k - 1;
    double cum = 0.0;
    for (int j = 0; j < top_k; j++) {
      cum += ev[j];
      if (uni < cum) { pick = j; break; }
    }
    const uint32_t id = (uint32_t)sample_key_index(top[pick]);
    next_ids[seq] = id;
    if (out_ids) out_ids[(size_t)seq * out_stride + my_step] = id;
    __threadfence();
    const unsigned int prev = atomicAdd(done_counter, 1u);
    if (prev == (unsigned int)rows - 1) {
      *pos = __ldcg(pos) + n_tok;
      *step = my_step + 1;
      *done_counter = 0u;
    }
  }
}

}  // namespace wgpt
