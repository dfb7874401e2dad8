// Causal attention over a KV cache, replacing the reference's formatQ + fusedWeights + softmax +
// attentionValues chain (instructions.js:1101-1214, :593-666) without materialising the [H*T, T] score and
// probability matrices. Masked scores are -1e9 in the reference (:1176) and exp(-1e9 - max) is exactly 0 in
// f32, so skipping masked keys gives the same probabilities.
//
// Layout: Q rows [rows, ldq] with head h in columns [h*HS, (h+1)*HS); K and V rows for sequence s, position
// j at base + (s*kv_seq_stride + j)*ldkv, same column convention (the reference's [T, E] K/V buffers).
#pragma once
#include "common.cuh"
#include "pair.cuh"

namespace wgpt {

// ------------------------------------------------------------------------------------------------
// Decode: one query row per sequence at position *pos (keys 0..*pos). grid = (H, n_seq, n_split): the CTAs along
// z share one (sequence, head) and each takes a slice of the positions. A CTA (8 warps) runs an online softmax
// over its slice; with n_split > 1 the slices' CTAs are a cluster and the first one merges their un-normalised results
// (acc, max, sum) in slice order. Left to the consumer, the merge cost every CTA of the output projection the partial
// results of every row (GPT-2 pass of 2 / 4 / 5 sequences 319 / 397 / 466 us, merged here 298 / 354 / 409).
// HBM-bound for many sequences: reads 2*HS*4 bytes per position per head; for few, the chain q -> scores -> merge behind the
// dependency wait. Cache rows of earlier steps do not depend on the previous kernel, only the newest one does: the first
// NST steps of a CTA's slice are copied to shared memory ahead of the wait (cp.async, each thread the pieces that it will
// use itself, so that no barrier is needed and no registers are held), the lines beyond them are asked for in L2. With eight
// rows in registers per thread instead, requested behind the wait, 768 CTAs were five to an SM and a few of them a second
// wave, and a CTA took 4 us from the wait. Whole completions in ms, that kernel / this one in one library: GPT-2 3 x 64 + 64
// tokens 20.4 / 20.2, 8 x 64 + 64 23.8 / 23.3, 64 x 128 + 64 46.2 / 44.6, 16 x 300 + 64 33.1 / 31.1; XL 1 x 200 + 32 56.3 / 53.6,
// 4 x 100 + 24 57.5 / 56.8, 16 x 96 + 24 67.5 / 64.7.
// Split-K partial tiles of the QKV product that feeds a decode attention (batched decode on the tensor cores):
// [slice][feature tile of 128][row = sequence][128], feature n of [0, 3E) = q | k | v. With FROM_QKV_PART the
// attention CTA is that product's second stage for its own (sequence, head): it adds the slices in order, adds the
// bias, keeps q, and writes the k and v rows of the newest position into the cache before it reads the cache.
struct QkvPartials {
  const float *part;
  const float *bias;  // [3E]
  int splits, n_rows, E;
};

// One output value, as FP32 or (planes != nullptr) as a pair (pair.cuh).
__device__ __forceinline__ void attn_put(float *out, __half *planes, size_t plane, float pair_scale, size_t at, float v) {
  if (planes == nullptr) {
    out[at] = v;
  } else {
    v *= pair_scale;
    const __half h0 = __float2half_rn(v);
    planes[at] = h0;
    planes[plane + at] = __float2half_rn(v - __half2float(h0));
  }
}

constexpr int kAttnDecodeU = 2;  // positions per lane group and step
constexpr size_t attn_decode_smem_bytes(int nst) { return (size_t)nst * kAttnDecodeU * 2 * 256 * 16; }

template <int HS, int NST, bool FROM_QKV_PART = false>
__global__ void __launch_bounds__(256, NST == 2 ? 6 : 3)
attn_decode_kernel(const float *__restrict__ q, int ldq, const float *__restrict__ kc, const float *__restrict__ vc,
                   int ldkv, size_t kv_seq_stride, float *__restrict__ out, int ldo, const int *__restrict__ pos,
                   float scale, QkvPartials qp, __half *__restrict__ planes, size_t plane, float pair_scale) {
  constexpr int LPP = HS / 4;      // lanes per position (one float4 each)
  constexpr int G = 32 / LPP;      // positions per warp iteration
  constexpr int NW = 8;
  const int h = blockIdx.x, seq = blockIdx.y, split = blockIdx.z, n_split = gridDim.z, H = gridDim.x;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane / LPP, lig = lane % LPP;
  const float *kb = kc + (size_t)seq * kv_seq_stride * ldkv + h * HS;
  const float *vb = vc + (size_t)seq * kv_seq_stride * ldkv + h * HS;
  TRACE_BEGIN(3);
  trace(3, 0);
  if (n_split > 1) cluster_arrive();  // pairs with the wait ahead of the first remote store
  pdl_launch_dependents();
  constexpr int U = kAttnDecodeU, STEP = NW * G * U;  // positions per step of the CTA
  extern __shared__ __align__(16) float4 kv_stage[];      // [NST][U][K, V][256]
  const uint32_t slot = smem_addr(kv_stage + tid);
  const float *kbl = kb + lig * 4, *vbl = vb + lig * 4;
  int beg = 0, end = 0;  // this CTA's slice of positions 0 .. p
  auto slice = [&](int p) {
    const int chunk = (p + n_split) / n_split;
    beg = split * chunk;
    end = min(p + 1, beg + chunk);
  };
  // Step i of the slice into stage i % NST: rows below `limit` only.
  auto request = [&](int i, int limit) {
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int j = beg + i * STEP + (warp + u * NW) * G + g;
      if (j < end && j < limit) {
        const uint32_t at = slot + (uint32_t)(((i % NST) * U + u) * 2) * 4096u;
        cp_async16(at, kbl + (size_t)j * ldkv);
        cp_async16(at + 4096u, vbl + (size_t)j * ldkv);
      }
    }
    cp_async_commit();
  };
  // Rows below *pos as it stands now were finished by the steps that advanced it there (common.cuh). It is one step old, or zero
  // ahead of a prompt's end, in most CTAs of a first layer whose step follows another without a graph launch in between.
  const int pos_s = __ldcg(pos);
  slice(pos_s);
#pragma unroll
  for (int i = 0; i < NST; i++) request(i, pos_s);
  {
    constexpr int LPR = HS * 4 >= 128 ? HS * 4 / 128 : 1;  // 128-byte lines per row slice
    const int first = beg + NST * STEP, total = max(end - first, 0) * 2 * LPR;
    for (int i = tid; i < total; i += 256) {
      const int r = first + i / (2 * LPR), w = i % (2 * LPR);
      prefetch_line_l2((w < LPR ? kb : vb) + (size_t)r * ldkv + (w % LPR) * 32);
    }
  }
  pdl_wait();  // q, the cache row of this step and *pos come from earlier kernels
  trace(3, 1);
  // The newest row, where its step is among those requested already: together with q and *pos, one round trip for all three.
  auto request_newest = [&] {
#pragma unroll
    for (int i = 0; i < NST; i++)
#pragma unroll
      for (int u = 0; u < U; u++)
        if (beg + i * STEP + (warp + u * NW) * G + g == pos_s && pos_s < end) {
          const uint32_t at = slot + (uint32_t)((i * U + u) * 2) * 4096u;
          cp_async16(at, kbl + (size_t)pos_s * ldkv);
          cp_async16(at + 4096u, vbl + (size_t)pos_s * ldkv);
        }
    cp_async_commit();
  };
  if (!FROM_QKV_PART) request_newest();
  const int L = __ldcg(pos) + 1;
  float4 q4;
  if (FROM_QKV_PART) {
    __shared__ __align__(16) float s_q[HS];
    if (tid < 3 * HS) {
      const int sec = tid / HS, d = tid - sec * HS;
      const int n = sec * qp.E + h * HS + d;
      const int n_tiles = (3 * qp.E + 127) >> 7, nt = n >> 7;
      const float *p0 = qp.part + ((size_t)nt * qp.n_rows + seq) * 128 + (n & 127);
      const size_t zstride = (size_t)n_tiles * qp.n_rows * 128;
      float a = 0.f;
#pragma unroll 8
      for (int z = 0; z < qp.splits; z++) a += __ldcg(p0 + (size_t)z * zstride);
      a += qp.bias[n];
      if (sec == 0) s_q[d] = a;
      // the newest position's row; kc/vc are written here and read below by this same CTA only
      else if (sec == 1) const_cast<float *>(kb)[(size_t)(L - 1) * ldkv + d] = a;
      else const_cast<float *>(vb)[(size_t)(L - 1) * ldkv + d] = a;
    }
    __syncthreads();
    request_newest();
    q4 = *reinterpret_cast<const float4 *>(&s_q[lig * 4]);
  } else {
    q4 = __ldcg(reinterpret_cast<const float4 *>(q + (size_t)seq * ldq + h * HS + lig * 4));
  }
  if (L - 1 != pos_s) {  // the position has moved since: another slice
    slice(L - 1);
    cp_async_wait<0>();
#pragma unroll
    for (int i = 0; i < NST; i++) request(i, L);
  }

  float m = -INFINITY, l = 0.f;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  // One maximum and one rescale for the U positions of a group's step. The trip count is the same for every lane of the warp
  // (the shuffles below name all 32 lanes); a position past the end of the slice contributes nothing.
  const int steps = (end - beg + STEP - 1) / STEP;
  for (int i = 0; i < steps; i++) {
    if (i + 1 < steps) cp_async_wait<NST - 1>();
    else cp_async_wait<0>();  // the newest row's copies are the last ones
    const float4 *st = kv_stage + (size_t)((i % NST) * U * 2) * 256 + tid;
    float s[U], mn = m;
#pragma unroll
    for (int u = 0; u < U; u++) {
      s[u] = dot4(q4, st[u * 512]);  // past the end the stage holds anything
#pragma unroll
      for (int o = LPP / 2; o > 0; o >>= 1) s[u] += __shfl_xor_sync(0xffffffffu, s[u], o);
      s[u] = beg + i * STEP + (warp + u * NW) * G + g < end ? s[u] * scale : -INFINITY;
      mn = fmaxf(mn, s[u]);
    }
    if (mn != -INFINITY) {  // otherwise this group has seen no position yet
      const float corr = expf(m - mn);  // m = -inf on the first step: 0
      l *= corr;
      acc.x *= corr; acc.y *= corr; acc.z *= corr; acc.w *= corr;
#pragma unroll
      for (int u = 0; u < U; u++)
        if (beg + i * STEP + (warp + u * NW) * G + g < end) {
          const float pr = expf(s[u] - mn);
          const float4 v = st[u * 512 + 256];
          l += pr;
          acc.x += pr * v.x; acc.y += pr * v.y; acc.z += pr * v.z; acc.w += pr * v.w;
        }
      m = mn;
    }
    request(i + NST, L);  // into the stage that has just been used
  }
  __syncwarp();
  // merge the G groups of the warp
#pragma unroll
  for (int o = LPP; o < 32; o <<= 1) {
    float mo = __shfl_xor_sync(0xffffffffu, m, o), lo = __shfl_xor_sync(0xffffffffu, l, o);
    float4 ao;
    ao.x = __shfl_xor_sync(0xffffffffu, acc.x, o); ao.y = __shfl_xor_sync(0xffffffffu, acc.y, o);
    ao.z = __shfl_xor_sync(0xffffffffu, acc.z, o); ao.w = __shfl_xor_sync(0xffffffffu, acc.w, o);
    float mn = fmaxf(m, mo);
    float c0 = (m == -INFINITY) ? 0.f : expf(m - mn), c1 = (mo == -INFINITY) ? 0.f : expf(mo - mn);
    l = l * c0 + lo * c1;
    acc.x = acc.x * c0 + ao.x * c1; acc.y = acc.y * c0 + ao.y * c1;
    acc.z = acc.z * c0 + ao.z * c1; acc.w = acc.w * c0 + ao.w * c1;
    m = mn;
  }
  trace(3, 2);
  __shared__ float sm_m[NW], sm_l[NW];
  __shared__ __align__(16) float sm_acc[NW][HS];
  if (g == 0) {
    *reinterpret_cast<float4 *>(&sm_acc[warp][lig * 4]) = acc;
    if (lig == 0) { sm_m[warp] = m; sm_l[warp] = l; }
  }
  __syncthreads();
  float keep_a = 0.f, keep_m = -INFINITY, keep_l = 0.f;
  if (tid < HS) {
    float mm = sm_m[0];
#pragma unroll
    for (int w = 1; w < NW; w++) mm = fmaxf(mm, sm_m[w]);
    float ll = 0.f, a = 0.f;
#pragma unroll
    for (int w = 0; w < NW; w++) {
      float c = (sm_m[w] == -INFINITY) ? 0.f : expf(sm_m[w] - mm);
      ll += sm_l[w] * c;
      a += sm_acc[w][tid] * c;
    }
    if (n_split == 1) {
      attn_put(out, planes, plane, pair_scale, (size_t)seq * ldo + h * HS + tid, a / ll);
    } else {
      keep_a = a;
      keep_m = mm;
      keep_l = ll;
    }
  }
  if (n_split > 1) {
    // The slices of a (sequence, head) are a cluster along z: every CTA hands its record to the first one, which merges
    // them in slice order and finishes the output, so no consumer has to (and no merge pass stands before it).
    __shared__ float mrg[8][HS + 2];
    cluster_wait();
    if (tid < HS) {
      dsmem_st(dsmem_addr(&mrg[split][tid], 0), keep_a);
      if (tid == 0) { dsmem_st(dsmem_addr(&mrg[split][HS], 0), keep_m); dsmem_st(dsmem_addr(&mrg[split][HS + 1], 0), keep_l); }
    }
    cluster_arrive();
    cluster_wait();
    if (split == 0 && tid < HS) {
      float mm = mrg[0][HS];
      for (int r = 1; r < n_split; r++) mm = fmaxf(mm, mrg[r][HS]);
      float ll = 0.f, a = 0.f;
      for (int r = 0; r < n_split; r++) {
        const float c = (mrg[r][HS] == -INFINITY) ? 0.f : expf(mrg[r][HS] - mm);
        ll += mrg[r][HS + 1] * c;
        a += mrg[r][tid] * c;
      }
      attn_put(out, planes, plane, pair_scale, (size_t)seq * ldo + h * HS + tid, a / ll);
    }
  }
  trace(3, 4);
}

// ------------------------------------------------------------------------------------------------
// Prefill: n_tok new query rows per sequence at positions *pos .. *pos+n_tok-1, keys 0..position.
// grid = (ceil(n_tok/32), H, n_seq), 128 threads: a 32-query tile against 32-key tiles held in shared
// memory, online softmax per query row. Thread (qi = tid/4, sub = tid%4) owns keys sub, sub+4, ... of the
// tile for the scores and dims sub, sub+4, ... of the output.
constexpr size_t attn_prefill_smem_bytes(int hs) { return (size_t)(96 * (hs + 1) + 32 * 33) * sizeof(float); }

template <int HS>
__global__ void __launch_bounds__(128)
attn_prefill_kernel(const float *__restrict__ q, int ldq, const float *__restrict__ kc, const float *__restrict__ vc,
                    int ldkv, size_t kv_seq_stride, float *__restrict__ out, int ldo, int n_tok,
                    const int *__restrict__ pos, float scale) {
  constexpr int TQ = 32, TK = 32, LD = HS + 1, DPT = HS / 4;
  extern __shared__ float attn_smem[];  // attn_prefill_smem_bytes(HS): above 48 KB for HS = 128
  float (*Qs)[LD] = reinterpret_cast<float (*)[LD]>(attn_smem);
  float (*Ks)[LD] = reinterpret_cast<float (*)[LD]>(attn_smem + TQ * LD);
  float (*Vs)[LD] = reinterpret_cast<float (*)[LD]>(attn_smem + (TQ + TK) * LD);
  float (*Ps)[TK + 1] = reinterpret_cast<float (*)[TK + 1]>(attn_smem + (TQ + 2 * TK) * LD);
  const int h = blockIdx.y, seq = blockIdx.z, t0 = blockIdx.x * TQ;
  const int tid = threadIdx.x, qi = tid >> 2, sub = tid & 3;
  const int pos0 = pos ? *pos : 0;
  const int nq = min(TQ, n_tok - t0);
  const int my_t = t0 + min(qi, nq - 1);       // out-of-range query threads shadow the last valid row
  const int my_pos = pos0 + my_t;
  const int last_key = pos0 + t0 + nq - 1;     // newest key any query of this tile may see

  for (int i = tid; i < TQ * (HS / 4); i += 128) {
    int r = i / (HS / 4), c4 = (i % (HS / 4)) * 4;
    int t = t0 + min(r, nq - 1);
    float4 v = *reinterpret_cast<const float4 *>(q + ((size_t)seq * n_tok + t) * ldq + h * HS + c4);
    Qs[r][c4] = v.x; Qs[r][c4 + 1] = v.y; Qs[r][c4 + 2] = v.z; Qs[r][c4 + 3] = v.w;
  }
  const float *kb = kc + (size_t)seq * kv_seq_stride * ldkv + h * HS;
  const float *vb = vc + (size_t)seq * kv_seq_stride * ldkv + h * HS;

  float m = -INFINITY, l = 0.f, o[DPT];
#pragma unroll
  for (int d = 0; d < DPT; d++) o[d] = 0.f;

  for (int j0 = 0; j0 <= last_key; j0 += TK) {
    __syncthreads();
    for (int i = tid; i < TK * (HS / 4); i += 128) {
      int r = i / (HS / 4), c4 = (i % (HS / 4)) * 4;
      int j = min(j0 + r, last_key);
      float4 kv = *reinterpret_cast<const float4 *>(kb + (size_t)j * ldkv + c4);
      float4 vv = *reinterpret_cast<const float4 *>(vb + (size_t)j * ldkv + c4);
      Ks[r][c4] = kv.x; Ks[r][c4 + 1] = kv.y; Ks[r][c4 + 2] = kv.z; Ks[r][c4 + 3] = kv.w;
      Vs[r][c4] = vv.x; Vs[r][c4 + 1] = vv.y; Vs[r][c4 + 2] = vv.z; Vs[r][c4 + 3] = vv.w;
    }
    __syncthreads();
    float s[TK / 4];
#pragma unroll
    for (int kk = 0; kk < TK / 4; kk++) s[kk] = 0.f;
    for (int d = 0; d < HS; d++) {
      float qv = Qs[qi][d];
#pragma unroll
      for (int kk = 0; kk < TK / 4; kk++) s[kk] += qv * Ks[sub + 4 * kk][d];
    }
    float tmax = -INFINITY;
#pragma unroll
    for (int kk = 0; kk < TK / 4; kk++) {
      int j = j0 + sub + 4 * kk;
      s[kk] = (j <= my_pos) ? s[kk] * scale : -INFINITY;
      tmax = fmaxf(tmax, s[kk]);
    }
    tmax = fmaxf(tmax, __shfl_xor_sync(0xffffffffu, tmax, 1));
    tmax = fmaxf(tmax, __shfl_xor_sync(0xffffffffu, tmax, 2));
    float mn = fmaxf(m, tmax);  // key j0 <= my_pos is visible in every processed tile? no: guard below
    float corr = (m == -INFINITY) ? 0.f : expf(m - mn);
    float psum = 0.f;
#pragma unroll
    for (int kk = 0; kk < TK / 4; kk++) {
      float p = (s[kk] == -INFINITY) ? 0.f : expf(s[kk] - mn);
      Ps[qi][sub + 4 * kk] = p;
      psum += p;
    }
    psum += __shfl_xor_sync(0xffffffffu, psum, 1);
    psum += __shfl_xor_sync(0xffffffffu, psum, 2);
    if (mn != -INFINITY) {
      l = l * corr + psum;
      m = mn;
    }
    __syncwarp();
#pragma unroll
    for (int d = 0; d < DPT; d++) o[d] *= corr;
    for (int k = 0; k < TK; k++) {
      float p = Ps[qi][k];
#pragma unroll
      for (int d = 0; d < DPT; d++) o[d] += p * Vs[k][sub + 4 * d];
    }
  }
  if (qi < nq) {
    float *op = out + ((size_t)seq * n_tok + t0 + qi) * ldo + h * HS;
    float inv = 1.f / l;
#pragma unroll
    for (int d = 0; d < DPT; d++) op[sub + 4 * d] = o[d] * inv;
  }
}

// ------------------------------------------------------------------------------------------------
// Prefill for head size 64 (every GPT-2 size and the char model), register-tiled: a CTA of 256 threads takes 64
// query rows against key tiles of 64, thread (ty, tx) of a 16 x 16 grid owns queries ty, ty+16, ty+32, ty+48 and
// keys tx, tx+16, tx+32, tx+48 of the tile for the scores, and the same queries with output dims 4tx..4tx+3 for
// the values. Q, K, V and the probabilities sit in shared memory in their natural row layout with rows padded to
// 68 floats; every inner step is 128-bit loads (the four keys of a lane are 16 rows apart, so a quarter-warp's
// eight addresses fall into different banks): 64 multiply-adds per eight loads, against one per load in the
// 32 x 32 kernel above. Online softmax per query row across tiles; the 16 lanes that share a row combine their
// maxima and sums with shuffles. Same mathematics as the chain it replaces (formatQ, fusedWeights with the causal
// mask, softmax, attentionValues: instructions.js:1101-1214, :593-666); masked keys contribute exactly zero.
constexpr int kAttn64Tile = 64, kAttn64Ld = 68;
constexpr size_t attn_prefill64_smem_bytes() { return (size_t)4 * kAttn64Tile * kAttn64Ld * sizeof(float); }

__global__ void __launch_bounds__(256)
attn_prefill64_kernel(const float *__restrict__ q, int ldq, const float *__restrict__ kc, const float *__restrict__ vc,
                      int ldkv, size_t kv_seq_stride, float *__restrict__ out, int ldo, int n_tok,
                      const int *__restrict__ pos, float scale) {
  constexpr int HS = 64, T = kAttn64Tile, LD = kAttn64Ld;
  extern __shared__ __align__(16) float attn_smem[];
  float *Qs = attn_smem, *Ks = Qs + T * LD, *Vs = Ks + T * LD, *Ps = Vs + T * LD;
  const int h = blockIdx.y, seq = blockIdx.z, t0 = blockIdx.x * T;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int pos0 = pos ? *pos : 0;
  const int nq = min(T, n_tok - t0);
  const int last_key = pos0 + t0 + nq - 1;  // newest key any query of this tile may see
  int my_pos[4];
#pragma unroll
  for (int i = 0; i < 4; i++) my_pos[i] = pos0 + t0 + min(ty + 16 * i, nq - 1);  // rows past the end shadow the last one

  for (int idx = tid; idx < T * (HS / 4); idx += 256) {
    const int r = idx >> 4, c4 = (idx & 15) * 4;
    const int t = t0 + min(r, nq - 1);
    *reinterpret_cast<float4 *>(Qs + r * LD + c4) =
        *reinterpret_cast<const float4 *>(q + ((size_t)seq * n_tok + t) * ldq + h * HS + c4);
  }
  const float *kb = kc + (size_t)seq * kv_seq_stride * ldkv + h * HS;
  const float *vb = vc + (size_t)seq * kv_seq_stride * ldkv + h * HS;

  float m[4], l[4], o[4][4];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    m[i] = -INFINITY;
    l[i] = 0.f;
#pragma unroll
    for (int d = 0; d < 4; d++) o[i][d] = 0.f;
  }

  for (int j0 = 0; j0 <= last_key; j0 += T) {
    __syncthreads();  // the previous tile's K, V and P are no longer read
    for (int idx = tid; idx < T * (HS / 4); idx += 256) {
      const int r = idx >> 4, c4 = (idx & 15) * 4;
      const int j = min(j0 + r, last_key);
      *reinterpret_cast<float4 *>(Ks + r * LD + c4) = *reinterpret_cast<const float4 *>(kb + (size_t)j * ldkv + c4);
      *reinterpret_cast<float4 *>(Vs + r * LD + c4) = *reinterpret_cast<const float4 *>(vb + (size_t)j * ldkv + c4);
    }
    __syncthreads();
    // ---- scores of 4 queries x 4 keys
    float s[4][4];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int k = 0; k < 4; k++) s[i][k] = 0.f;
#pragma unroll 4
    for (int d = 0; d < HS; d += 4) {
      float4 qv[4], kv[4];
#pragma unroll
      for (int i = 0; i < 4; i++) qv[i] = *reinterpret_cast<const float4 *>(Qs + (ty + 16 * i) * LD + d);
#pragma unroll
      for (int k = 0; k < 4; k++) kv[k] = *reinterpret_cast<const float4 *>(Ks + (tx + 16 * k) * LD + d);
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int k = 0; k < 4; k++) s[i][k] += dot4(qv[i], kv[k]);
    }
    // ---- online softmax per query row (the 16 lanes with this ty share the row)
#pragma unroll
    for (int i = 0; i < 4; i++) {
      float tmax = -INFINITY;
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const int j = j0 + tx + 16 * k;
        s[i][k] = (j <= my_pos[i]) ? s[i][k] * scale : -INFINITY;
        tmax = fmaxf(tmax, s[i][k]);
      }
#pragma unroll
      for (int off = 8; off > 0; off >>= 1) tmax = fmaxf(tmax, __shfl_xor_sync(0xffffffffu, tmax, off));
      const float mn = fmaxf(m[i], tmax);
      const float corr = (m[i] == -INFINITY) ? 0.f : expf(m[i] - mn);
      float psum = 0.f;
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const float p = (s[i][k] == -INFINITY) ? 0.f : expf(s[i][k] - mn);
        Ps[(ty + 16 * i) * LD + tx + 16 * k] = p;
        psum += p;
      }
#pragma unroll
      for (int off = 8; off > 0; off >>= 1) psum += __shfl_xor_sync(0xffffffffu, psum, off);
      if (mn != -INFINITY) {
        l[i] = l[i] * corr + psum;
        m[i] = mn;
      }
#pragma unroll
      for (int d = 0; d < 4; d++) o[i][d] *= corr;
    }
    __syncthreads();  // the probabilities of the tile are complete
    // ---- values: 4 queries x 4 output dims
#pragma unroll 4
    for (int k = 0; k < T; k += 4) {
      float4 pv[4], vv[4];
#pragma unroll
      for (int i = 0; i < 4; i++) pv[i] = *reinterpret_cast<const float4 *>(Ps + (ty + 16 * i) * LD + k);
#pragma unroll
      for (int kk = 0; kk < 4; kk++) vv[kk] = *reinterpret_cast<const float4 *>(Vs + (k + kk) * LD + 4 * tx);
#pragma unroll
      for (int i = 0; i < 4; i++) {
        o[i][0] += pv[i].x * vv[0].x + pv[i].y * vv[1].x + pv[i].z * vv[2].x + pv[i].w * vv[3].x;
        o[i][1] += pv[i].x * vv[0].y + pv[i].y * vv[1].y + pv[i].z * vv[2].y + pv[i].w * vv[3].y;
        o[i][2] += pv[i].x * vv[0].z + pv[i].y * vv[1].z + pv[i].z * vv[2].z + pv[i].w * vv[3].z;
        o[i][3] += pv[i].x * vv[0].w + pv[i].y * vv[1].w + pv[i].z * vv[2].w + pv[i].w * vv[3].w;
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int r = ty + 16 * i;
    if (r < nq) {
      const float inv = 1.f / l[i];
      *reinterpret_cast<float4 *>(out + ((size_t)seq * n_tok + t0 + r) * ldo + h * HS + 4 * tx) =
          make_float4(o[i][0] * inv, o[i][1] * inv, o[i][2] * inv, o[i][3] * inv);
    }
  }
}

}  // namespace wgpt

namespace wgpt {

// ------------------------------------------------------------------------------------------------
// Prefill for head size 64 on the tensor cores (warp-level mma.sync.m16n8k8, TF32 inputs, FP32 accumulation), used
// when the device computes products in TF32 or 3xTF32; the FP32 mode keeps attn_prefill64_kernel. A CTA of four
// warps takes 64 query rows (16 per warp) against key tiles of 64 held in shared memory; scores, online softmax and
// the probabilities never leave registers (the accumulator fragment of the score product is re-arranged into the
// A fragment of the value product with shuffles inside each quad of lanes). X3: every operand is split into
// hi = its top 19 bits and lo = x - hi, and each product is hi*hi + hi*lo + lo*hi, as in the GEMM kernels.
// Same mathematics as attn_prefill64_kernel (instructions.js:1101-1214, :593-666); masked keys contribute zero.
constexpr int kAttnMmaKLd = 68, kAttnMmaVLd = 72;  // row strides (floats) that keep the fragment loads conflict-free

__device__ __forceinline__ void mma_tf32_16x8x8(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t tf32_hi_bits(float x) { return __float_as_uint(x) & 0xFFFFE000u; }
__device__ __forceinline__ uint32_t tf32_lo_bits(float x) {
  return __float_as_uint(x - __uint_as_float(__float_as_uint(x) & 0xFFFFE000u));
}

template <bool X3>
__global__ void __launch_bounds__(128)
attn_prefill64_mma_kernel(const float *__restrict__ q, int ldq, const float *__restrict__ kc,
                          const float *__restrict__ vc, int ldkv, size_t kv_seq_stride, float *__restrict__ out,
                          int ldo, int n_tok, const int *__restrict__ pos, float scale) {
  constexpr int HS = 64, T = 64, KLD = kAttnMmaKLd, VLD = kAttnMmaVLd;
  __shared__ __align__(16) float Ks[T * KLD];
  __shared__ __align__(16) float Vs[T * VLD];
  const int h = blockIdx.y, seq = blockIdx.z, t0 = blockIdx.x * T;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int pos0 = pos ? *pos : 0;
  const int nq = min(T, n_tok - t0);
  const int last_key = pos0 + t0 + nq - 1;  // newest key any query of this tile may see
  const int r0 = 16 * warp + g, r1 = r0 + 8;  // this lane's two query rows inside the tile
  const int p0 = pos0 + t0 + min(r0, nq - 1), p1 = pos0 + t0 + min(r1, nq - 1);  // rows past the end shadow the last
  const int warp_last = pos0 + t0 + min(16 * warp + 15, nq - 1);

  // ---- Q fragments (A operand of the score product), staged through the K buffer
  for (int idx = tid; idx < T * (HS / 4); idx += 128) {
    const int r = idx >> 4, c4 = (idx & 15) * 4;
    const int tq = t0 + min(r, nq - 1);
    *reinterpret_cast<float4 *>(Ks + r * KLD + c4) =
        *reinterpret_cast<const float4 *>(q + ((size_t)seq * n_tok + tq) * ldq + h * HS + c4);
  }
  __syncthreads();
  uint32_t qh[8][4], ql[X3 ? 8 : 1][4];
#pragma unroll
  for (int ks = 0; ks < 8; ks++) {
    const float x0 = Ks[r0 * KLD + 8 * ks + t], x1 = Ks[r1 * KLD + 8 * ks + t];
    const float x2 = Ks[r0 * KLD + 8 * ks + t + 4], x3 = Ks[r1 * KLD + 8 * ks + t + 4];
    qh[ks][0] = tf32_hi_bits(x0); qh[ks][1] = tf32_hi_bits(x1); qh[ks][2] = tf32_hi_bits(x2); qh[ks][3] = tf32_hi_bits(x3);
    if (X3) {
      ql[ks][0] = tf32_lo_bits(x0); ql[ks][1] = tf32_lo_bits(x1); ql[ks][2] = tf32_lo_bits(x2); ql[ks][3] = tf32_lo_bits(x3);
    }
  }
  const float *kb = kc + (size_t)seq * kv_seq_stride * ldkv + h * HS;
  const float *vb = vc + (size_t)seq * kv_seq_stride * ldkv + h * HS;

  float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f;
  float o[8][4];
#pragma unroll
  for (int j = 0; j < 8; j++)
#pragma unroll
    for (int e = 0; e < 4; e++) o[j][e] = 0.f;

  for (int j0 = 0; j0 <= last_key; j0 += T) {
    __syncthreads();  // the previous tile (or the staged Q) is no longer read
    for (int idx = tid; idx < T * (HS / 4); idx += 128) {
      const int r = idx >> 4, c4 = (idx & 15) * 4;
      const int j = min(j0 + r, last_key);
      *reinterpret_cast<float4 *>(Ks + r * KLD + c4) = *reinterpret_cast<const float4 *>(kb + (size_t)j * ldkv + c4);
      *reinterpret_cast<float4 *>(Vs + r * VLD + c4) = *reinterpret_cast<const float4 *>(vb + (size_t)j * ldkv + c4);
    }
    __syncthreads();
    if (j0 > warp_last) continue;  // every key of the tile is masked for this warp's rows (same for the whole warp)

    // ---- scores: 16 rows x 64 keys as eight 16x8 accumulators
    float s[8][4];
#pragma unroll
    for (int j = 0; j < 8; j++) {
#pragma unroll
      for (int e = 0; e < 4; e++) s[j][e] = 0.f;
#pragma unroll
      for (int ks = 0; ks < 8; ks++) {
        const float k0 = Ks[(8 * j + g) * KLD + 8 * ks + t], k1 = Ks[(8 * j + g) * KLD + 8 * ks + t + 4];
        const uint32_t kh0 = tf32_hi_bits(k0), kh1 = tf32_hi_bits(k1);
        mma_tf32_16x8x8(s[j], qh[ks], kh0, kh1);
        if (X3) {
          mma_tf32_16x8x8(s[j], qh[ks], tf32_lo_bits(k0), tf32_lo_bits(k1));
          mma_tf32_16x8x8(s[j], ql[ks], kh0, kh1);
        }
      }
    }
    // ---- online softmax of rows r0 (elements 0, 1) and r1 (elements 2, 3); key of element e: j0 + 8j + 2t + (e & 1)
    float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll
    for (int j = 0; j < 8; j++) {
#pragma unroll
      for (int e = 0; e < 4; e++) {
        const int key = j0 + 8 * j + 2 * t + (e & 1);
        const int pq = e < 2 ? p0 : p1;
        s[j][e] = key <= pq ? s[j][e] * scale : -INFINITY;
      }
      mx0 = fmaxf(mx0, fmaxf(s[j][0], s[j][1]));
      mx1 = fmaxf(mx1, fmaxf(s[j][2], s[j][3]));
    }
    mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 1)); mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 2));
    mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 1)); mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 2));
    const float mn0 = fmaxf(m0, mx0), mn1 = fmaxf(m1, mx1);
    const float c0 = (m0 == -INFINITY) ? 0.f : expf(m0 - mn0), c1 = (m1 == -INFINITY) ? 0.f : expf(m1 - mn1);
    float ps0 = 0.f, ps1 = 0.f;
#pragma unroll
    for (int j = 0; j < 8; j++) {
      s[j][0] = (s[j][0] == -INFINITY) ? 0.f : expf(s[j][0] - mn0);
      s[j][1] = (s[j][1] == -INFINITY) ? 0.f : expf(s[j][1] - mn0);
      s[j][2] = (s[j][2] == -INFINITY) ? 0.f : expf(s[j][2] - mn1);
      s[j][3] = (s[j][3] == -INFINITY) ? 0.f : expf(s[j][3] - mn1);
      ps0 += s[j][0] + s[j][1];
      ps1 += s[j][2] + s[j][3];
    }
    if (mn0 != -INFINITY) { l0 = l0 * c0 + ps0; m0 = mn0; }  // l holds this lane's share of the row sum
    if (mn1 != -INFINITY) { l1 = l1 * c1 + ps1; m1 = mn1; }
#pragma unroll
    for (int j = 0; j < 8; j++) {
      o[j][0] *= c0; o[j][1] *= c0; o[j][2] *= c1; o[j][3] *= c1;
    }
    // ---- values: the probabilities of keys 8ks..8ks+7 become the A fragment of k-step ks
    const int src_lo = (lane & ~3) | (t >> 1), src_hi = src_lo + 2;
    const bool odd = (t & 1) != 0;
#pragma unroll
    for (int ks = 0; ks < 8; ks++) {
      // element (row, key 8ks + c) sits in the lane of the quad with 2*tig == c & ~1, as element c & 1 (row r0) / 2 + (c & 1) (row r1)
      const float e0a = __shfl_sync(0xffffffffu, s[ks][0], src_lo), e1a = __shfl_sync(0xffffffffu, s[ks][1], src_lo);
      const float e2a = __shfl_sync(0xffffffffu, s[ks][2], src_lo), e3a = __shfl_sync(0xffffffffu, s[ks][3], src_lo);
      const float e0b = __shfl_sync(0xffffffffu, s[ks][0], src_hi), e1b = __shfl_sync(0xffffffffu, s[ks][1], src_hi);
      const float e2b = __shfl_sync(0xffffffffu, s[ks][2], src_hi), e3b = __shfl_sync(0xffffffffu, s[ks][3], src_hi);
      const float a0 = odd ? e1a : e0a, a1 = odd ? e3a : e2a;  // keys 8ks + t of rows r0, r1
      const float a2 = odd ? e1b : e0b, a3 = odd ? e3b : e2b;  // keys 8ks + t + 4
      uint32_t ph[4] = {tf32_hi_bits(a0), tf32_hi_bits(a1), tf32_hi_bits(a2), tf32_hi_bits(a3)};
      uint32_t pl[4] = {0u, 0u, 0u, 0u};
      if (X3) { pl[0] = tf32_lo_bits(a0); pl[1] = tf32_lo_bits(a1); pl[2] = tf32_lo_bits(a2); pl[3] = tf32_lo_bits(a3); }
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const float v0 = Vs[(8 * ks + t) * VLD + 8 * j + g], v1 = Vs[(8 * ks + t + 4) * VLD + 8 * j + g];
        const uint32_t vh0 = tf32_hi_bits(v0), vh1 = tf32_hi_bits(v1);
        mma_tf32_16x8x8(o[j], ph, vh0, vh1);
        if (X3) {
          mma_tf32_16x8x8(o[j], ph, tf32_lo_bits(v0), tf32_lo_bits(v1));
          mma_tf32_16x8x8(o[j], pl, vh0, vh1);
        }
      }
    }
  }
  l0 += __shfl_xor_sync(0xffffffffu, l0, 1); l0 += __shfl_xor_sync(0xffffffffu, l0, 2);
  l1 += __shfl_xor_sync(0xffffffffu, l1, 1); l1 += __shfl_xor_sync(0xffffffffu, l1, 2);
  const float i0 = 1.f / l0, i1 = 1.f / l1;
#pragma unroll
  for (int j = 0; j < 8; j++) {
    if (r0 < nq)
      *reinterpret_cast<float2 *>(out + ((size_t)seq * n_tok + t0 + r0) * ldo + h * HS + 8 * j + 2 * t) =
          make_float2(o[j][0] * i0, o[j][1] * i0);
    if (r1 < nq)
      *reinterpret_cast<float2 *>(out + ((size_t)seq * n_tok + t0 + r1) * ldo + h * HS + 8 * j + 2 * t) =
          make_float2(o[j][2] * i1, o[j][3] * i1);
  }
}

// ------------------------------------------------------------------------------------------------
// The same for a model whose matrices are pairs of half-precision planes (pair.cuh): queries, keys, values and
// probabilities are split into pairs (scaled by powers of two whose bounds are known at load; probabilities by 2^15) and
// each product is h0 h0 + h0 h1 + h1 h0 through mma.sync.m16n8k16, half the instructions of the TF32 form at the same
// terms. K and V tiles are split once, while they are staged, instead of by every warp at every fragment; fragments come
// by ldmatrix; the score accumulators of two 8-key tiles are the A fragment of a 16-key value step as they are, so the
// probabilities need no shuffles. 16 WARPS query rows per CTA share a staged 64-key tile. KG > 1: KG groups of WARPS warps
// take the same rows and alternate key tiles (staged together), their results merged at the end - for grids that leave SMs
// idle, where the serial chain of a row's key tiles is what the kernel takes. Output as a pair.
//
// OWN: nothing is known of the operands (the per-operator attention, whose rows may be of any size). Every query, key and
// value row of the head gets its own power of two, found while it is staged; a key's returns with its scores and a value's
// goes into the probabilities, which are scaled by the largest weighted value a query has met so far (rescaled with the
// running maximum), so that a row is as accurate beside one 2^24 times its size as alone, and later rows leave no trace in
// earlier ones. Output as FP32 rows: their own exponents span all heads.
constexpr int kAttnPairLd = 72;  // halves per staged row: 144 bytes, so that the eight rows of an ldmatrix hit all banks

__device__ __forceinline__ void mma_f16_16x8x16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t saddr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(saddr));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t saddr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(saddr));
}
// Two values as a half pair: the first planes' word, and the second planes'.
__device__ __forceinline__ uint32_t pair_word(float x, float y, uint32_t &lo) {
  const __half2 a = __floats2half2_rn(x, y);
  const float2 f = __half22float2(a);
  const __half2 b = __floats2half2_rn(x - f.x, y - f.y);
  lo = *reinterpret_cast<const uint32_t *>(&b);
  return *reinterpret_cast<const uint32_t *>(&a);
}

constexpr size_t attn_pair_smem_bytes(int kg, bool own) { return (size_t)4 * kg * 64 * kAttnPairLd * 2 + (own ? (size_t)2 * kg * 64 * 4 : 0); }

// Largest of the four lanes that share a row of an accumulator fragment.
__device__ __forceinline__ float quad_max(float v) {
  v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 1));
  return fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 2));
}

template <int WARPS, int KG, bool OWN>
__global__ void __launch_bounds__(32 * WARPS * KG)
attn_prefill64_pair_kernel(const float *__restrict__ q, int ldq, const float *__restrict__ kc,
                           const float *__restrict__ vc, int ldkv, size_t kv_seq_stride, int n_tok,
                           const int *__restrict__ pos, float scale, float s_qk, float s_v,
                           __half *__restrict__ planes, size_t plane, float *__restrict__ out, int ldo, int H) {
  constexpr int HS = 64, TQ = 16 * WARPS, T = 64, LD = kAttnPairLd, NT = 32 * WARPS * KG;
  extern __shared__ __align__(16) __half attn_pair_smem[];
  __half *Ks = attn_pair_smem, *Vs = attn_pair_smem + 2 * KG * T * LD;  // [plane][KG tiles of T keys][LD]
  float *kd = reinterpret_cast<float *>(Vs + 2 * KG * T * LD), *vd = kd + KG * T;  // OWN: 1 / scale of every staged row
  // The query tiles with the most keys first: an SM takes its next CTA when one of its own ends, so the short ones fill up.
  const int order = (int)blockIdx.x;
  const int n_tiles = (n_tok + TQ - 1) / TQ, heads = (int)gridDim.x / n_tiles, hq = order % heads;
  const int h = hq % H, seq = hq / H;
  const int t0 = (n_tiles - 1 - order / heads) * TQ;
  const int tid = threadIdx.x, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int warp = (tid >> 5) % WARPS, kg = (tid >> 5) / WARPS;
  pdl_launch_dependents();
  pdl_wait();
  const int pos0 = pos ? __ldcg(pos) : 0;
  const int nq = min(TQ, n_tok - t0);
  const int last_key = pos0 + t0 + nq - 1;  // newest key any query of this tile may see
  const int r0 = 16 * warp + g, r1 = r0 + 8;
  const int p0 = pos0 + t0 + min(r0, nq - 1), p1 = pos0 + t0 + min(r1, nq - 1);  // rows past the end shadow the last
  const int warp_last = pos0 + t0 + min(16 * warp + 15, nq - 1);
  const bool warp_live = 16 * warp < nq;

  // ---- Q fragments: element (row, dim) pairs straight from global memory, once
  uint32_t qh[4][4], ql[4][4];
  float s_q0 = s_qk, s_q1 = s_qk;
  {
    const float *q0 = q + ((size_t)seq * n_tok + t0 + min(r0, nq - 1)) * ldq + h * HS + 2 * t;
    const float *q1 = q + ((size_t)seq * n_tok + t0 + min(r1, nq - 1)) * ldq + h * HS + 2 * t;
    float2 a[4], b[4], c[4], d[4];
    float top0 = 0.f, top1 = 0.f;
#pragma unroll
    for (int ks = 0; ks < 4; ks++) {
      a[ks] = __ldcg(reinterpret_cast<const float2 *>(q0 + 16 * ks));
      b[ks] = __ldcg(reinterpret_cast<const float2 *>(q1 + 16 * ks));
      c[ks] = __ldcg(reinterpret_cast<const float2 *>(q0 + 16 * ks + 8));
      d[ks] = __ldcg(reinterpret_cast<const float2 *>(q1 + 16 * ks + 8));
      top0 = fmaxf(top0, fmaxf(fmaxf(fabsf(a[ks].x), fabsf(a[ks].y)), fmaxf(fabsf(c[ks].x), fabsf(c[ks].y))));
      top1 = fmaxf(top1, fmaxf(fmaxf(fabsf(b[ks].x), fabsf(b[ks].y)), fmaxf(fabsf(d[ks].x), fabsf(d[ks].y))));
    }
    if (OWN) {
      s_q0 = pair_scale_for(quad_max(top0));
      s_q1 = pair_scale_for(quad_max(top1));
    }
#pragma unroll
    for (int ks = 0; ks < 4; ks++) {
      qh[ks][0] = pair_word(a[ks].x * s_q0, a[ks].y * s_q0, ql[ks][0]);
      qh[ks][1] = pair_word(b[ks].x * s_q1, b[ks].y * s_q1, ql[ks][1]);
      qh[ks][2] = pair_word(c[ks].x * s_q0, c[ks].y * s_q0, ql[ks][2]);
      qh[ks][3] = pair_word(d[ks].x * s_q1, d[ks].y * s_q1, ql[ks][3]);
    }
  }
  const float *kb = kc + (size_t)seq * kv_seq_stride * ldkv + h * HS;
  const float *vb = vc + (size_t)seq * kv_seq_stride * ldkv + h * HS;
  const float f0 = OWN ? scale / s_q0 : scale / (s_qk * s_qk), f1 = OWN ? scale / s_q1 : f0;  // OWN: times the key's

  float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f;
  float wt0 = 0.f, wt1 = 0.f, od0 = 1.f, od1 = 1.f;  // OWN: largest weighted value so far, 1 / scale of o
  float o[8][4];
#pragma unroll
  for (int j = 0; j < 8; j++)
#pragma unroll
    for (int e = 0; e < 4; e++) o[j][e] = 0.f;
  // ldmatrix row addresses of this lane: keys (lane & 7) + 8 (lane >> 4), dims 8 ((lane >> 3) & 1) for K (two 8-key tiles
  // x 16 dims); keys (lane & 15), dims 8 (lane >> 4) for V, transposed (16 keys x two 8-dim tiles)
  const uint32_t k_row = smem_addr(Ks) + 2u * (uint32_t)((kg * T + (lane & 7) + 8 * (lane >> 4)) * LD + 8 * ((lane >> 3) & 1));
  const uint32_t v_row = smem_addr(Vs) + 2u * (uint32_t)((kg * T + (lane & 15)) * LD + 8 * (lane >> 4));
  constexpr uint32_t kPlane = 2u * KG * T * LD;
  static_assert(KG * T * (HS / 4) == 8 * NT, "eight float4 of K and of V per thread");

  for (int jb = 0; jb <= last_key; jb += KG * T) {
    const int j0 = jb + kg * T;
    __syncthreads();  // the previous tile is no longer read
    {
      constexpr int PER = KG * T * (HS / 4) / NT;  // float4 of K (and of V) per thread: 8
      // sixteen lanes to a row; OWN: four, each with a quarter of it, so that a row's maximum is two exchanges away
      auto row_of = [&](int i) { return OWN ? (tid >> 2) + (NT / 4) * (i >> 2) : (tid + NT * i) >> 4; };
      auto col_of = [&](int i) { return OWN ? ((tid & 3) + 4 * (i & 3)) * 4 : ((tid + NT * i) & 15) * 4; };
      float4 kv[PER], vv[PER];
#pragma unroll
      for (int i = 0; i < PER; i++) {
        const size_t at = (size_t)min(jb + row_of(i), last_key) * ldkv + col_of(i);
        kv[i] = __ldcg(reinterpret_cast<const float4 *>(kb + at));
        vv[i] = __ldcg(reinterpret_cast<const float4 *>(vb + at));
      }
      float sk = s_qk, sv = s_v;
#pragma unroll
      for (int i = 0; i < PER; i++) {
        const int r = row_of(i), c4 = col_of(i);
        if (OWN && (i & 3) == 0) {
          float mk = 0.f, mv = 0.f;
#pragma unroll
          for (int u = i; u < i + 4; u++) {
            mk = fmaxf(mk, fmaxf(fmaxf(fabsf(kv[u].x), fabsf(kv[u].y)), fmaxf(fabsf(kv[u].z), fabsf(kv[u].w))));
            mv = fmaxf(mv, fmaxf(fmaxf(fabsf(vv[u].x), fabsf(vv[u].y)), fmaxf(fabsf(vv[u].z), fabsf(vv[u].w))));
          }
          sk = pair_scale_for(quad_max(mk));
          sv = pair_scale_for(quad_max(mv));
          if ((tid & 3) == 0) { kd[r] = 1.f / sk; vd[r] = 1.f / sv; }
        }
        uint2 a, b;
        pair_split4(scale4(kv[i], sk), a, b);
        *reinterpret_cast<uint2 *>(Ks + r * LD + c4) = a;
        *reinterpret_cast<uint2 *>(Ks + (KG * T + r) * LD + c4) = b;
        pair_split4(scale4(vv[i], sv), a, b);
        *reinterpret_cast<uint2 *>(Vs + r * LD + c4) = a;
        *reinterpret_cast<uint2 *>(Vs + (KG * T + r) * LD + c4) = b;
      }
    }
    __syncthreads();
    if (!warp_live || j0 > warp_last) continue;  // every key of the tile is masked for this warp's rows

    // ---- scores: 16 rows x 64 keys as eight 16x8 accumulators, two per ldmatrix
    float s[8][4];
#pragma unroll
    for (int j = 0; j < 8; j++)
#pragma unroll
      for (int e = 0; e < 4; e++) s[j][e] = 0.f;
#pragma unroll
    for (int jp = 0; jp < 4; jp++) {
#pragma unroll
      for (int ks = 0; ks < 4; ks++) {
        uint32_t kh[4], kl[4];
        ldmatrix_x4(kh, k_row + 2u * (uint32_t)(16 * jp * LD + 16 * ks));
        ldmatrix_x4(kl, k_row + kPlane + 2u * (uint32_t)(16 * jp * LD + 16 * ks));
        mma_f16_16x8x16(s[2 * jp], qh[ks], kh[0], kh[1]);
        mma_f16_16x8x16(s[2 * jp + 1], qh[ks], kh[2], kh[3]);
        mma_f16_16x8x16(s[2 * jp], qh[ks], kl[0], kl[1]);
        mma_f16_16x8x16(s[2 * jp + 1], qh[ks], kl[2], kl[3]);
        mma_f16_16x8x16(s[2 * jp], ql[ks], kh[0], kh[1]);
        mma_f16_16x8x16(s[2 * jp + 1], ql[ks], kh[2], kh[3]);
      }
    }
    // ---- online softmax of rows r0 (elements 0, 1) and r1 (elements 2, 3); key of element e: j0 + 8j + 2t + (e & 1)
    float mx0 = -INFINITY, mx1 = -INFINITY;
    const bool masked = j0 + T - 1 > pos0 + t0 + 16 * warp;  // same for the whole warp: some key is beyond some row
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const float2 kf = OWN ? *reinterpret_cast<const float2 *>(kd + kg * T + 8 * j + 2 * t) : make_float2(1.f, 1.f);
#pragma unroll
      for (int e = 0; e < 4; e++) {
        const float f = e < 2 ? f0 : f1;
        s[j][e] *= OWN ? f * (e & 1 ? kf.y : kf.x) : f;
        if (masked) {
          const int key = j0 + 8 * j + 2 * t + (e & 1);
          if (key > (e < 2 ? p0 : p1)) s[j][e] = -INFINITY;
        }
      }
      mx0 = fmaxf(mx0, fmaxf(s[j][0], s[j][1]));
      mx1 = fmaxf(mx1, fmaxf(s[j][2], s[j][3]));
    }
    mx0 = quad_max(mx0);
    mx1 = quad_max(mx1);
    float mn0 = fmaxf(m0, mx0), mn1 = fmaxf(m1, mx1);  // finite with KG == 1: every row sees key 0 of its first tile
    m0 = KG > 1 && mn0 == -INFINITY ? 0.f : m0;        // a row that has seen no key yet: everything below gives zero
    m1 = KG > 1 && mn1 == -INFINITY ? 0.f : m1;
    const float b0 = KG > 1 && mn0 == -INFINITY ? 0.f : mn0, b1 = KG > 1 && mn1 == -INFINITY ? 0.f : mn1;
    float c0 = expf(m0 - b0), c1 = expf(m1 - b1);
    float ps0 = 0.f, ps1 = 0.f;
#pragma unroll
    for (int j = 0; j < 8; j++) {
      s[j][0] = expf(s[j][0] - b0);
      s[j][1] = expf(s[j][1] - b0);
      s[j][2] = expf(s[j][2] - b1);
      s[j][3] = expf(s[j][3] - b1);
      ps0 += s[j][0] + s[j][1];
      ps1 += s[j][2] + s[j][3];
    }
    l0 = l0 * c0 + ps0; m0 = mn0;  // l holds this lane's share of the row sum
    l1 = l1 * c1 + ps1; m1 = mn1;
    float sp0 = kPairTop, sp1 = kPairTop;  // scale of the probabilities
    if (OWN) {
      float w0 = 0.f, w1 = 0.f;
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const float2 vf = *reinterpret_cast<const float2 *>(vd + kg * T + 8 * j + 2 * t);
        s[j][0] *= vf.x; s[j][1] *= vf.y; s[j][2] *= vf.x; s[j][3] *= vf.y;
        w0 = fmaxf(w0, fmaxf(s[j][0], s[j][1]));
        w1 = fmaxf(w1, fmaxf(s[j][2], s[j][3]));
      }
      wt0 = fmaxf(wt0 * c0, quad_max(w0));
      wt1 = fmaxf(wt1 * c1, quad_max(w1));
      sp0 = pair_scale_for(wt0);
      sp1 = pair_scale_for(wt1);
      c0 = c0 * sp0 * od0;  // wt0 never falls below its share of the old one: c0 sp0 od0 is at most 2
      c1 = c1 * sp1 * od1;
      od0 = 1.f / sp0;
      od1 = 1.f / sp1;
    }
#pragma unroll
    for (int j = 0; j < 8; j++) {
      o[j][0] *= c0; o[j][1] *= c0; o[j][2] *= c1; o[j][3] *= c1;
    }
    // ---- values
#pragma unroll
    for (int ks = 0; ks < 4; ks++) {
      uint32_t ph[4], pl[4];
      ph[0] = pair_word(s[2 * ks][0] * sp0, s[2 * ks][1] * sp0, pl[0]);
      ph[1] = pair_word(s[2 * ks][2] * sp1, s[2 * ks][3] * sp1, pl[1]);
      ph[2] = pair_word(s[2 * ks + 1][0] * sp0, s[2 * ks + 1][1] * sp0, pl[2]);
      ph[3] = pair_word(s[2 * ks + 1][2] * sp1, s[2 * ks + 1][3] * sp1, pl[3]);
#pragma unroll
      for (int jp = 0; jp < 4; jp++) {
        uint32_t vh[4], vl[4];
        ldmatrix_x4_trans(vh, v_row + 2u * (uint32_t)(16 * ks * LD + 16 * jp));
        ldmatrix_x4_trans(vl, v_row + kPlane + 2u * (uint32_t)(16 * ks * LD + 16 * jp));
        mma_f16_16x8x16(o[2 * jp], ph, vh[0], vh[1]);
        mma_f16_16x8x16(o[2 * jp + 1], ph, vh[2], vh[3]);
        mma_f16_16x8x16(o[2 * jp], ph, vl[0], vl[1]);
        mma_f16_16x8x16(o[2 * jp + 1], ph, vl[2], vl[3]);
        mma_f16_16x8x16(o[2 * jp], pl, vh[0], vh[1]);
        mma_f16_16x8x16(o[2 * jp + 1], pl, vh[2], vh[3]);
      }
    }
  }
  if (KG > 1) {  // merge the groups' results, in group order
    constexpr int REC = OWN ? 38 : 36;
    float *mg = reinterpret_cast<float *>(attn_pair_smem);  // [KG - 1][WARPS][REC][32]
    __syncthreads();
    if (kg > 0) {
      float *r = mg + (size_t)((kg - 1) * WARPS + warp) * REC * 32 + lane;
#pragma unroll
      for (int j = 0; j < 8; j++)
#pragma unroll
        for (int e = 0; e < 4; e++) r[(4 * j + e) * 32] = o[j][e];
      r[32 * 32] = m0; r[33 * 32] = m1; r[34 * 32] = l0; r[35 * 32] = l1;
      if (OWN) { r[36 * 32] = od0; r[37 * 32] = od1; }
    }
    __syncthreads();
    if (kg > 0) return;
#pragma unroll 1
    for (int k = 0; k < KG - 1; k++) {
      const float *r = mg + (size_t)(k * WARPS + warp) * REC * 32 + lane;
      const float n0 = r[32 * 32], n1 = r[33 * 32];
      const float x0 = fmaxf(m0, n0), x1 = fmaxf(m1, n1);  // finite: group 0 has seen key 0
      float a0 = expf(m0 - x0), a1 = expf(m1 - x1), d0 = expf(n0 - x0), d1 = expf(n1 - x1);
      l0 = l0 * a0 + r[34 * 32] * d0;
      l1 = l1 * a1 + r[35 * 32] * d1;
      m0 = x0; m1 = x1;
      if (OWN) {  // both in units of the larger one
        const float g0 = r[36 * 32], g1 = r[37 * 32], u0 = fmaxf(od0, g0), u1 = fmaxf(od1, g1);
        a0 *= od0 / u0; d0 *= g0 / u0; od0 = u0;
        a1 *= od1 / u1; d1 *= g1 / u1; od1 = u1;
      }
#pragma unroll
      for (int j = 0; j < 8; j++) {
        o[j][0] = o[j][0] * a0 + r[(4 * j) * 32] * d0; o[j][1] = o[j][1] * a0 + r[(4 * j + 1) * 32] * d0;
        o[j][2] = o[j][2] * a1 + r[(4 * j + 2) * 32] * d1; o[j][3] = o[j][3] * a1 + r[(4 * j + 3) * 32] * d1;
      }
    }
  }
  if (!warp_live) return;
  l0 += __shfl_xor_sync(0xffffffffu, l0, 1); l0 += __shfl_xor_sync(0xffffffffu, l0, 2);
  l1 += __shfl_xor_sync(0xffffffffu, l1, 1); l1 += __shfl_xor_sync(0xffffffffu, l1, 2);
  if (OWN) {
    const float i0 = 1.f / l0, i1 = 1.f / l1;
#pragma unroll
    for (int j = 0; j < 8; j++) {
      float *at = out + ((size_t)seq * n_tok + t0 + r0) * ldo + h * HS + 8 * j + 2 * t;
      if (r0 < nq) *reinterpret_cast<float2 *>(at) = make_float2(o[j][0] * i0 * od0, o[j][1] * i0 * od0);
      if (r1 < nq) *reinterpret_cast<float2 *>(at + (size_t)8 * ldo) = make_float2(o[j][2] * i1 * od1, o[j][3] * i1 * od1);
    }
    return;
  }
  // the values' own scale is also the output pair's
  const float i0 = 1.f / (l0 * kPairTop), i1 = 1.f / (l1 * kPairTop);
#pragma unroll
  for (int j = 0; j < 8; j++) {
    uint32_t lo;
    if (r0 < nq) {
      __half *at = planes + ((size_t)seq * n_tok + t0 + r0) * ldo + h * HS + 8 * j + 2 * t;
      *reinterpret_cast<uint32_t *>(at) = pair_word(o[j][0] * i0, o[j][1] * i0, lo);
      *reinterpret_cast<uint32_t *>(at + plane) = lo;
    }
    if (r1 < nq) {
      __half *at = planes + ((size_t)seq * n_tok + t0 + r1) * ldo + h * HS + 8 * j + 2 * t;
      *reinterpret_cast<uint32_t *>(at) = pair_word(o[j][2] * i1, o[j][3] * i1, lo);
      *reinterpret_cast<uint32_t *>(at + plane) = lo;
    }
  }
}

}  // namespace wgpt
