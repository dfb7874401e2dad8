// FP32 matrices as pairs of half-precision planes, for products on the tensor cores at the half-precision rate.
//
// A value x of a row is written as x = 2^e (h0 + h1): h0 = half(x 2^-e), h1 = half(x 2^-e - h0), both rounded to
// nearest, e one exponent per row (weights) or per tensor (activations whose bound is known). A product of two such
// values is h0 g0 + h0 g1 + h1 g0, three half-precision products accumulated in FP32; the exponents come back as an
// exact multiplication in the epilogue. Precision against the three TF32 products it replaces (which truncate):
//   * representation: |x - 2^e(h0+h1)| <= 2^-22 |x| (TF32 hi + truncated lo: 2^-20 |x|), for every |x| down to 2^-17 of
//     the scaled range's top (2^15); smaller ones have the absolute error 2^-40 of that top, 2^16 below what one FP32
//     rounding of the row's largest term costs the sum;
//   * the dropped product h1 g1 is <= 2^-22 |x y| (TF32: 2^-20);
//   * an MMA adds 16 products at once instead of 8, so half as many FP32 accumulations are rounded.
// Both planes together are 4 bytes per value, as the FP32 value itself: nothing more is streamed from HBM, and no
// operand has to be split by CUDA threads between shared memory and the tensor core.
#pragma once
#include <cmath>
#include <cstring>

#include "common.cuh"

namespace wgpt {

constexpr float kPairTop = 32768.f;  // scaled values stay below this (the half format ends at 65504)

// The power of two that brings `bound` (> 0, finite) to (kPairTop / 2, kPairTop]; its reciprocal is exact too. A bound
// of zero, an infinity or a NaN gives 1 (an infinite or NaN element then turns the products it enters into NaN, as
// hi + lo = inf + (inf - inf) did).
__host__ __device__ inline float pair_scale_for(float bound) {
#ifdef __CUDA_ARCH__
  const uint32_t b = __float_as_uint(bound);
#else
  uint32_t b;
  memcpy(&b, &bound, 4);
#endif
  if (b == 0u || b >= 0x7F800000u) return 1.f;  // zero, negative, infinite, NaN
  int e = 141 - (int)(b >> 23) + ((b & 0x7FFFFFu) == 0u ? 1 : 0);  // bound 2^e <= 2^15; -113 at the largest number
  e = e > 126 ? 126 : e;  // 2^-e stays normal; even a row of 2^-126 keeps 25 bits
#ifdef __CUDA_ARCH__
  return __uint_as_float((uint32_t)(e + 127) << 23);
#else
  return std::ldexp(1.f, e);
#endif
}

// Four scaled values -> the four halves of each plane, packed for one 8-byte store.
__device__ __forceinline__ void pair_split4(float4 v, uint2 &p0, uint2 &p1) {
  const __half2 a0 = __floats2half2_rn(v.x, v.y), b0 = __floats2half2_rn(v.z, v.w);
  const float2 af = __half22float2(a0), bf = __half22float2(b0);
  const __half2 a1 = __floats2half2_rn(v.x - af.x, v.y - af.y), b1 = __floats2half2_rn(v.z - bf.x, v.w - bf.y);
  p0 = make_uint2(*reinterpret_cast<const uint32_t *>(&a0), *reinterpret_cast<const uint32_t *>(&b0));
  p1 = make_uint2(*reinterpret_cast<const uint32_t *>(&a1), *reinterpret_cast<const uint32_t *>(&b1));
}
__device__ __forceinline__ float4 scale4(float4 v, float s) { return make_float4(v.x * s, v.y * s, v.z * s, v.w * s); }

// A raw sum times the powers of two of its row and its column (or a column's scale), the smaller first: a row of 1e35 against
// a column of 1e-35 would pass infinity on the way to one.
__device__ __forceinline__ float pair_descale(float v, float rs, float cs) { return rs < cs ? v * rs * cs : v * cs * rs; }
__device__ __forceinline__ float4 pair_descale4(float4 v, float rs, float4 cs) {
  return make_float4(pair_descale(v.x, rs, cs.x), pair_descale(v.y, rs, cs.y), pair_descale(v.z, rs, cs.z), pair_descale(v.w, rs, cs.w));
}

// Epilogue of the kernels that multiply pairs: four raw sums of row m, columns n..n+3, with the columns' constants and
// the residual already in registers -> the finished values, and their store. `rows`: the product may have row factors (a
// model's have none, and kernels made for them leave the branch out).
__device__ __forceinline__ float4 pair_epi_value4(const Epilogue &e, float4 v, float4 cs, float4 bs, float4 res, int m, bool rows) {
  if (rows && e.rowscale != nullptr)
    v = add4(pair_descale4(v, __ldcg(e.rowscale + m), cs), bs);
  else
    v = make_float4(v.x * cs.x + bs.x, v.y * cs.y + bs.y, v.z * cs.z + bs.z, v.w * cs.w + bs.w);
  if (e.act == 1) v = make_float4(gelu_f(v.x), gelu_f(v.y), gelu_f(v.z), gelu_f(v.w));
  return make_float4(v.x + res.x, v.y + res.y, v.z + res.z, v.w + res.w);
}
__device__ __forceinline__ void pair_epi_store4(const Epilogue &e, float4 v, int m, int n) {
  if (e.pair != nullptr) {
    uint2 p0, p1;
    pair_split4(scale4(v, e.kc != nullptr && n >= 2 * e.E ? e.pair_scale_v : e.pair_scale), p0, p1);
    __half *o = e.pair + (size_t)m * e.ld + n;
    *reinterpret_cast<uint2 *>(o) = p0;
    *reinterpret_cast<uint2 *>(o + e.pair_plane) = p1;
    if (e.kc == nullptr || n < e.E) return;
  }
  *reinterpret_cast<float4 *>(epi_addr(e, m, n)) = v;
}
// The same for 32 rows of a 32-column block held in `pad` (row stride 33): this lane finishes columns n..n+3 (block
// columns col4..col4+3) of rows row0 + 4 it + sub_r. Without an activation the residuals of all its rows are requested
// together (one row at a time, the epilogue is a chain of L2 round trips longer than the MMAs it has to hide behind), or the
// row factors of a per-operator product, which has no residual (one loop for both took a model's products 0.5 to 1 %);
// with one, the loop stays rolled: 32 inlined GELUs per block made the kernel miss in the instruction cache at every
// step (36 000 cycles per tile instead of 18 000).
__device__ __forceinline__ void pair_epi_block(const Epilogue &e, const float *pad, int row0, int sub_r, int col4, int n,
                                               int M) {
  const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
  const float4 cs = e.colscale != nullptr ? __ldcg(reinterpret_cast<const float4 *>(e.colscale + n)) : make_float4(1.f, 1.f, 1.f, 1.f);
  const float4 bs = e.bias != nullptr ? __ldg(reinterpret_cast<const float4 *>(e.bias + n)) : zero4;
  if (e.act == 0 && e.pair == nullptr && e.rowscale == nullptr) {
    float4 res[8];
#pragma unroll
    for (int it = 0; it < 8; it++) {
      const int m = row0 + it * 4 + sub_r;
      res[it] = e.residual != nullptr && m < M
                    ? __ldcg(reinterpret_cast<const float4 *>(e.residual + (size_t)m * e.ld + n)) : zero4;
    }
#pragma unroll
    for (int it = 0; it < 8; it++) {
      const int r = it * 4 + sub_r, m = row0 + r;
      const float *src = pad + r * 33 + col4;
      float4 v = make_float4(src[0], src[1], src[2], src[3]);
      if (m >= M) continue;
      *reinterpret_cast<float4 *>(epi_addr(e, m, n)) =
          make_float4(v.x * cs.x + bs.x + res[it].x, v.y * cs.y + bs.y + res[it].y, v.z * cs.z + bs.z + res[it].z,
                      v.w * cs.w + bs.w + res[it].w);
    }
  } else if (e.act == 0 && e.kc != nullptr && e.rowscale == nullptr) {  // q | k | v as pairs, and to the cache
#pragma unroll
    for (int it = 0; it < 8; it++) {
      const int r = it * 4 + sub_r, m = row0 + r;
      const float *src = pad + r * 33 + col4;
      if (m >= M) continue;
      pair_epi_store4(e, make_float4(src[0] * cs.x + bs.x, src[1] * cs.y + bs.y, src[2] * cs.z + bs.z, src[3] * cs.w + bs.w), m, n);
    }
  } else if (e.act == 0 && e.pair == nullptr && e.residual == nullptr) {
    float rs[8];
#pragma unroll
    for (int it = 0; it < 8; it++) rs[it] = row0 + it * 4 + sub_r < M ? __ldcg(e.rowscale + row0 + it * 4 + sub_r) : 0.f;
#pragma unroll
    for (int it = 0; it < 8; it++) {
      const int r = it * 4 + sub_r, m = row0 + r;
      const float *src = pad + r * 33 + col4;
      if (m >= M) continue;
      *reinterpret_cast<float4 *>(epi_addr(e, m, n)) =
          add4(pair_descale4(make_float4(src[0], src[1], src[2], src[3]), rs[it], cs), bs);
    }
  } else {
#pragma unroll 1
    for (int it = 0; it < 8; it++) {
      const int r = it * 4 + sub_r, m = row0 + r;
      if (m >= M) break;
      const float *src = pad + r * 33 + col4;
      const float4 res = e.residual != nullptr ? __ldcg(reinterpret_cast<const float4 *>(e.residual + (size_t)m * e.ld + n)) : zero4;
      pair_epi_store4(e, pair_epi_value4(e, make_float4(src[0], src[1], src[2], src[3]), cs, bs, res, m, true), m, n);
    }
  }
}
__device__ __forceinline__ void pair_epi1(const Epilogue &e, float v, int m, int n) {  // N % 4 != 0: never a pair out
  if (e.rowscale) v *= __ldcg(e.rowscale + m);
  epi_store(e, v, m, n);
}

// Rows of an FP32 matrix [rows, K] -> planes [2][rows][K], one exponent per row: descale[row] = 2^e, and, where asked
// for, norm[row] = the row's 2-norm (the load step derives bounds of a product's outputs from it). One warp per row,
// two passes over the row (the second from L1/L2). HBM-bound: 8 bytes per value. K % 4 == 0.
__global__ void __launch_bounds__(256)
pair_rows_kernel(const float *__restrict__ in, size_t ld, int rows, int K, __half *__restrict__ planes,
                 float *__restrict__ descale, float *__restrict__ norm) {
  const int row = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  pdl_launch_dependents();
  pdl_wait();
  if (row >= rows) return;
  const float4 *x = reinterpret_cast<const float4 *>(in + (size_t)row * ld);
  const int K4 = K >> 2;
  float m = 0.f, q = 0.f;
#pragma unroll 8
  for (int i = lane; i < K4; i += 32) {
    const float4 v = __ldcg(x + i);
    m = fmaxf(m, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
    q += dot4(v, v);
  }
  m = warp_max(m);
  const float s = pair_scale_for(m);
  if (norm != nullptr) q = warp_sum(q);
  if (lane == 0) {
    descale[row] = 1.f / s;
    if (norm != nullptr) norm[row] = sqrtf(q);
  }
  uint2 *o0 = reinterpret_cast<uint2 *>(planes + (size_t)row * K);
  uint2 *o1 = reinterpret_cast<uint2 *>(planes + ((size_t)rows + row) * K);
#pragma unroll 8
  for (int i = lane; i < K4; i += 32) {
    uint2 a, b;
    pair_split4(scale4(__ldcg(x + i), s), a, b);
    o0[i] = a;
    o1[i] = b;
  }
}

// FP32 values -> planes, one exponent for the whole tensor (scale = the power of two it is multiplied by). n % 4 == 0.
__global__ void __launch_bounds__(256)
pair_convert_kernel(const float *__restrict__ in, size_t n, float scale, __half *__restrict__ planes) {
  pdl_launch_dependents();
  pdl_wait();
  const size_t n4 = n >> 2;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += (size_t)gridDim.x * blockDim.x) {
    uint2 a, b;
    pair_split4(scale4(__ldcg(reinterpret_cast<const float4 *>(in) + i), scale), a, b);
    reinterpret_cast<uint2 *>(planes)[i] = a;
    reinterpret_cast<uint2 *>(planes + n)[i] = b;
  }
}

// ------------------------------------------------------------------------------------------------
// Operands of one per-operator product (or the four of an attention) as pairs, in one launch: activations X[M,K] row by row,
// weights W[K,N] in the reference layout (instructions.js:219-224) transposed on the way, one exponent per column.
//
// A cluster of S CTAs takes 32 columns of a weight, each CTA a slice of K held in shared memory: the column maxima are
// exchanged through distributed shared memory, so the weight is read once, and it may be read before the dependency wait
// (parameter buffers are constants); only the writes wait. HBM-bound: 8 bytes per value. The transposition, split-K
// product and second stage this prepares for took 21-26 us for GPT-2's products at 128 rows; this pass and the product
// that finishes in its cluster take about half.
struct PairOperands {
  // activations
  const float *x;
  int M, K;
  __half *xp;         // [2][M][K]
  float *x_descale;   // [M]
  int x_ctas;         // a multiple of the cluster size
  int block_rows;     // 1: a CTA per row (K <= 8192), 0: a warp per row
  // weights [K,N]
  int n_w, N, klen;   // klen: rows of K per CTA of a cluster, a multiple of 8
  const float *w[4], *bias[4];
  __half *wp[4];      // plane 0 of the weight's first column, rows of K
  size_t plane[4];
  float *descale[4];  // [N]
  float *bias_out[4]; // [N] copy of bias (zero where there is none), or nullptr
};

__device__ __forceinline__ void pair_operand_rows(const PairOperands &p, int cta) {  // cta: of p.x_ctas
  __shared__ float red[8];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, K4 = p.K >> 2;
  if (p.block_rows) {
    constexpr int V = 8;
    for (int row = cta; row < p.M; row += p.x_ctas) {
      const float4 *x = reinterpret_cast<const float4 *>(p.x + (size_t)row * p.K);
      float4 v[V];
      float m = 0.f;
#pragma unroll
      for (int j = 0; j < V; j++) v[j] = tid + 256 * j < K4 ? __ldcg(x + tid + 256 * j) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int j = 0; j < V; j++) m = fmaxf(m, fmaxf(fmaxf(fabsf(v[j].x), fabsf(v[j].y)), fmaxf(fabsf(v[j].z), fabsf(v[j].w))));
      m = warp_max(m);
      if (lane == 0) red[warp] = m;
      __syncthreads();
#pragma unroll
      for (int w = 0; w < 8; w++) m = fmaxf(m, red[w]);
      __syncthreads();
      const float s = pair_scale_for(m);
      if (tid == 0) p.x_descale[row] = 1.f / s;
      uint2 *o0 = reinterpret_cast<uint2 *>(p.xp + (size_t)row * p.K);
      uint2 *o1 = reinterpret_cast<uint2 *>(p.xp + ((size_t)p.M + row) * p.K);
#pragma unroll
      for (int j = 0; j < V; j++)
        if (tid + 256 * j < K4) {
          uint2 a, b;
          pair_split4(scale4(v[j], s), a, b);
          o0[tid + 256 * j] = a;
          o1[tid + 256 * j] = b;
        }
    }
  } else {
    for (int row = cta * 8 + warp; row < p.M; row += p.x_ctas * 8) {
      const float4 *x = reinterpret_cast<const float4 *>(p.x + (size_t)row * p.K);
      float m = 0.f;
#pragma unroll 8
      for (int i = lane; i < K4; i += 32) {
        const float4 v = __ldcg(x + i);
        m = fmaxf(m, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
      }
      m = warp_max(m);
      const float s = pair_scale_for(m);
      if (lane == 0) p.x_descale[row] = 1.f / s;
      uint2 *o0 = reinterpret_cast<uint2 *>(p.xp + (size_t)row * p.K);
      uint2 *o1 = reinterpret_cast<uint2 *>(p.xp + ((size_t)p.M + row) * p.K);
#pragma unroll 8
      for (int i = lane; i < K4; i += 32) {
        uint2 a, b;
        pair_split4(scale4(__ldcg(x + i), s), a, b);
        o0[i] = a;
        o1[i] = b;
      }
    }
  }
}

// grid = n_w ceil(N / 32) S + x_ctas, cluster (S,1,1), 256 threads; dynamic shared memory klen x 33 floats. The weights' CTAs come
// first: they have work ahead of the dependency wait, and behind the rows' CTAs, which only wait, they found room 1.5 to 2.5 us
// later (pass list of GPT-2, us, rows first / weights first: 64 tokens 940 / 940, 128 1115 / 1056, 250 1329 / 1258). A thread has
// six rows in flight; with twelve, for slices of more than 192 rows, the kernel spills and the lists take 1.2 to 2 % longer.
__global__ void __launch_bounds__(256)
pair_operands_kernel(const __grid_constant__ PairOperands p) {
  extern __shared__ __align__(16) float po_tile[];  // [klen][33]
  __shared__ float own[32], stat[8][32], scl[32];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  pdl_launch_dependents();
  const int w_ctas = (int)gridDim.x - p.x_ctas;
  if ((int)blockIdx.x >= w_ctas) {  // whole clusters
    pdl_wait();
    pair_operand_rows(p, (int)blockIdx.x - w_ctas);
    return;
  }
  uint32_t S;
  asm volatile("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(S));
  const int rank = (int)cluster_ctarank(), cl = (int)(blockIdx.x / S);
  const int nblk = (p.N + 31) >> 5, wi = cl / nblk, blk = cl - wi * nblk, n0 = blk * 32;
  const int kb = min(p.K, rank * p.klen), kn = min(p.K, kb + p.klen) - kb;
  cluster_arrive();
  {
    const int c4 = (tid & 7) * 4, r0 = tid >> 3;
    const bool in = n0 + c4 < p.N;  // N % 4 == 0
    const float *src = p.w[wi] + (size_t)kb * p.N + n0 + c4;
    constexpr int U = 6;
    for (int r = r0; r < kn; r += 32 * U) {
      float4 v[U];
#pragma unroll
      for (int u = 0; u < U; u++)
        v[u] = in && r + 32 * u < kn ? ldg_stream4(reinterpret_cast<const float4 *>(src + (size_t)(r + 32 * u) * p.N))
                                     : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int u = 0; u < U; u++)
        if (r + 32 * u < kn) {
          float *t = po_tile + (r + 32 * u) * 33 + c4;
          t[0] = v[u].x; t[1] = v[u].y; t[2] = v[u].z; t[3] = v[u].w;
        }
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int c = 4 * warp + i;
    float m = 0.f;
#pragma unroll 4
    for (int r = lane; r < kn; r += 32) m = fmaxf(m, fabsf(po_tile[r * 33 + c]));
    m = warp_max(m);
    if (lane == 0) own[c] = m;
  }
  __syncthreads();
  cluster_wait();  // every CTA of the cluster is running
  if (tid < 32)
    for (int r = 0; r < (int)S; r++) dsmem_st(dsmem_addr(&stat[rank][tid], (uint32_t)r), own[tid]);
  cluster_arrive();
  cluster_wait();
  pdl_wait();  // what this kernel writes may still be read by earlier ones
  if (tid < 32) {
    float m = 0.f;
    for (int r = 0; r < (int)S; r++) m = fmaxf(m, stat[r][tid]);
    const float s = pair_scale_for(m);
    scl[tid] = s;
    if (rank == 0) {
      const int n = n0 + tid;
      const float b = n < p.N && p.bias[wi] != nullptr ? p.bias[wi][n] : 0.f;
      if (n < p.N) {
        p.descale[wi][n] = 1.f / s;
        if (p.bias_out[wi] != nullptr) p.bias_out[wi][n] = b;
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int c = 4 * warp + i;
    if (n0 + c >= p.N) continue;
    const float s = scl[c];
    __half2 *o0 = reinterpret_cast<__half2 *>(p.wp[wi] + (size_t)(n0 + c) * p.K + kb);
    __half2 *o1 = reinterpret_cast<__half2 *>(p.wp[wi] + p.plane[wi] + (size_t)(n0 + c) * p.K + kb);
#pragma unroll 2
    for (int k2 = lane; 2 * k2 < kn; k2 += 32) {  // K % 8 == 0 and klen % 8 == 0: pairs are whole
      const float x = po_tile[2 * k2 * 33 + c] * s, y = po_tile[(2 * k2 + 1) * 33 + c] * s;
      const __half2 a = __floats2half2_rn(x, y);
      const float2 f = __half22float2(a);
      o0[k2] = a;
      o1[k2] = __floats2half2_rn(x - f.x, y - f.y);
    }
  }
}

}  // namespace wgpt
