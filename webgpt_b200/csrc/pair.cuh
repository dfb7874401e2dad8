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
#include "common.cuh"

namespace wgpt {

constexpr float kPairTop = 32768.f;  // scaled values stay below this (the half format ends at 65504)

// The power of two that brings `bound` (> 0, finite) to (kPairTop / 2, kPairTop]; its reciprocal is exact too. A bound
// of zero, an infinity or a NaN gives 1 (an infinite or NaN element then turns the products it enters into NaN, as
// hi + lo = inf + (inf - inf) did).
__host__ __device__ inline float pair_scale_for(float bound) {
  if (!(bound > 0.f) || !(bound < 3.0e38f)) return 1.f;
  int ex;
  const float m = frexpf(bound, &ex);            // bound = m 2^ex, m in [1/2, 1)
  int e = 15 - (m == 0.5f ? ex - 1 : ex);        // bound 2^e <= 2^15
  e = e < -110 ? -110 : (e > 110 ? 110 : e);     // 2^e and 2^-e stay normal; rows below 2^-95 lose low bits only
  return ldexpf(1.f, e);
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

// Epilogue of the kernels that multiply pairs: four raw sums of row m, columns n..n+3, with the columns' constants and
// the residual already in registers -> the finished values, and their store.
__device__ __forceinline__ float4 pair_epi_value4(const Epilogue &e, float4 v, float4 cs, float4 bs, float4 res, int m) {
  if (e.rowscale != nullptr) v = scale4(v, __ldg(e.rowscale + m));
  v = make_float4(v.x * cs.x + bs.x, v.y * cs.y + bs.y, v.z * cs.z + bs.z, v.w * cs.w + bs.w);
  if (e.act == 1) v = make_float4(gelu_f(v.x), gelu_f(v.y), gelu_f(v.z), gelu_f(v.w));
  return make_float4(v.x + res.x, v.y + res.y, v.z + res.z, v.w + res.w);
}
__device__ __forceinline__ void pair_epi_store4(const Epilogue &e, float4 v, int m, int n) {
  if (e.pair != nullptr) {
    uint2 p0, p1;
    pair_split4(scale4(v, e.pair_scale), p0, p1);
    __half *o = e.pair + (size_t)m * e.ld + n;
    *reinterpret_cast<uint2 *>(o) = p0;
    *reinterpret_cast<uint2 *>(o + e.pair_plane) = p1;
  } else {
    *reinterpret_cast<float4 *>(epi_addr(e, m, n)) = v;
  }
}
// The same for 32 rows of a 32-column block held in `pad` (row stride 33): this lane finishes columns n..n+3 (block
// columns col4..col4+3) of rows row0 + 4 it + sub_r. Without an activation the residuals of all its rows are requested
// together (one row at a time, the epilogue is a chain of L2 round trips longer than the MMAs it has to hide behind);
// with one, the loop stays rolled: 32 inlined GELUs per block made the kernel miss in the instruction cache at every
// step (36 000 cycles per tile instead of 18 000).
__device__ __forceinline__ void pair_epi_block(const Epilogue &e, const float *pad, int row0, int sub_r, int col4, int n,
                                               int M) {
  const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
  const float4 cs = e.colscale != nullptr ? __ldg(reinterpret_cast<const float4 *>(e.colscale + n)) : make_float4(1.f, 1.f, 1.f, 1.f);
  const float4 bs = e.bias != nullptr ? __ldg(reinterpret_cast<const float4 *>(e.bias + n)) : zero4;
  if (e.act == 0 && e.pair == nullptr) {
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
      if (e.rowscale != nullptr) v = scale4(v, __ldg(e.rowscale + m));
      *reinterpret_cast<float4 *>(epi_addr(e, m, n)) =
          make_float4(v.x * cs.x + bs.x + res[it].x, v.y * cs.y + bs.y + res[it].y, v.z * cs.z + bs.z + res[it].z,
                      v.w * cs.w + bs.w + res[it].w);
    }
  } else {
#pragma unroll 1
    for (int it = 0; it < 8; it++) {
      const int r = it * 4 + sub_r, m = row0 + r;
      if (m >= M) break;
      const float *src = pad + r * 33 + col4;
      const float4 res = e.residual != nullptr ? __ldcg(reinterpret_cast<const float4 *>(e.residual + (size_t)m * e.ld + n)) : zero4;
      pair_epi_store4(e, pair_epi_value4(e, make_float4(src[0], src[1], src[2], src[3]), cs, bs, res, m), m, n);
    }
  }
}
__device__ __forceinline__ void pair_epi1(const Epilogue &e, float v, int m, int n) {  // N % 4 != 0: never a pair out
  if (e.rowscale) v *= __ldg(e.rowscale + m);
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

}  // namespace wgpt
