// fp32 SIMT tasks for the tiny model (widths that are not multiples of the tensor-core tile: D=64, head dim 16, V=65).
// Same task contract, layouts and epilogues as the bf16 path; every sum has a fixed order (a thread's own share of k upwards, then the
// shares in index order), so results are bitwise independent of the schedule.
//
// What bounds these tasks is latency: a step of the tiny model is some fifty dependent phases of 0.1 to 3 MFLOP each. So a phase is
// cut into enough tasks to spread over the blocks, a task asks for all its operands at once, and its 256 threads share one output
// tile by splitting k among themselves. One step of the char model (B=16, T=64, two layers): 1,060 us of kernel with 64 x 64 tiles
// walked 16 k at a time and one attention thread per query row.
#pragma once
#include "common.cuh"
#include "task_api.h"

namespace ofa {
namespace f32 {

// C tile of a task. NN / NT: 32 x 32, the operand panels (up to 256 k deep) in shared memory, four groups of 64 threads take every
// fourth k, a thread owns 4 x 4 outputs. TN (weight gradients: k runs over all tokens, outputs are few): 16 x 16, sixteen groups of 16
// threads read their rows straight from global memory, eight rows of both operands in flight per thread where both are 16-byte aligned, four
// otherwise and in remainders. The weight gradient of the head over 3,072 tokens: V = 300 27.6 us, V = 299, unaligned, 44.9 (40.9 and 55.7 with
// eight rows in one loop for both; V = 65 43.2 and 54.2).
constexpr int GT = 32, GT_TN = 16, GK = 256, GS = GT + 4;
constexpr int GEMM_SMEM = 2 * GK * GS * 4;
__host__ __device__ constexpr int gemm_tile(int layout) { return layout == GL_TN ? GT_TN : GT; }

__device__ __forceinline__ float4 zero4() { return make_float4(0.f, 0.f, 0.f, 0.f); }
__device__ __forceinline__ float4 ld4s(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void fma16(float (&acc)[4][4], const float4 a, const float4 b) {
  const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
}
// four consecutive elements of a row of length n; elements past n are zero. vec: rows are 16-byte aligned and n is a multiple of 4
__device__ __forceinline__ float4 row4(const float* row, int c, int n, bool vec) {
  if (vec) return c < n ? ld4s(row + c) : zero4();
  return make_float4(c < n ? row[c] : 0.f, c + 1 < n ? row[c + 1] : 0.f, c + 2 < n ? row[c + 2] : 0.f, c + 3 < n ? row[c + 3] : 0.f);
}
__device__ __forceinline__ bool aligned_rows(const void* p, int ld, int n) { return ((reinterpret_cast<uintptr_t>(p) & 15) | (ld & 3) | (n & 3)) == 0; }

// panel dst[k][GT] (stride GS) of an operand stored [rows][K]: lane = row, so the transposed stores of a warp hit 32 banks
__device__ __forceinline__ void panel_kmajor(float* dst, const float* X, int ld, int r0, int rows, int k0, int kc, int K) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool vec = aligned_rows(X, ld, K), in = r0 + lane < rows;
  const float* row = X + (size_t)(r0 + lane) * ld;
  auto put = [&](int k, const float4 v) { dst[k * GS + lane] = v.x; dst[(k + 1) * GS + lane] = v.y; dst[(k + 2) * GS + lane] = v.z; dst[(k + 3) * GS + lane] = v.w; };
  if (vec) {
#pragma unroll 4
    for (int k = warp * 4; k < kc; k += NTHR / 8) put(k, in ? row4(row, k0 + k, K, true) : zero4());
  } else {
#pragma unroll 1
    for (int k = warp * 4; k < kc; k += NTHR / 8) put(k, in ? row4(row, k0 + k, K, false) : zero4());
  }
}
// panel dst[k][GT] of an operand stored [K][cols]
__device__ __forceinline__ void panel_nmajor(float* dst, const float* X, int ld, int c0, int cols, int k0, int kc, int K) {
  const int c = (threadIdx.x & 7) * 4;
  const bool vec = aligned_rows(X, ld, cols);
  auto put = [&](int k, bool v4) { *reinterpret_cast<float4*>(dst + k * GS + c) = k0 + k < K ? row4(X + (size_t)(k0 + k) * ld, c0 + c, cols, v4) : zero4(); };
  if (vec) {
#pragma unroll 4
    for (int k = threadIdx.x >> 3; k < kc; k += NTHR / 8) put(k, true);
  } else {
#pragma unroll 1
    for (int k = threadIdx.x >> 3; k < kc; k += NTHR / 8) put(k, false);
  }
}
// Out of line, like the unaligned forms of the loads above in loops of their own: a block runs through most of the library in a step, so what a task's code
// occupies beyond what it executes often is fetched anew each time. The char model's step: 407 -> 376 us, a weight gradient of 64 x 256 13.1 -> 8.7 us.
__device__ __noinline__ void epilogue1(const GemmArgs& g, int epi, int m, int n, float v) {
  float* C = reinterpret_cast<float*>(g.C); float* aux = reinterpret_cast<float*>(g.aux);
  const size_t ci = (size_t)m * g.ldc + n, ai = (size_t)m * g.ldaux + n;
  switch (epi) {
    case GE_RES: v += aux[ai]; break;
    case GE_GELU: aux[ai] = v; v = gelu_fwd<false>(v); break;
    case GE_DGELU: v *= gelu_bwd<false>(aux[ai]); break;
    case GE_F32: if (g.accumulate) v += C[ci]; break;
    default: break;
  }
  C[ci] = v;
}

// one 32 x 32 tile of C; task -> (tm = task % tiles_m, tn = task / tiles_m)
template <bool B_KMAJOR>
__device__ __forceinline__ void gemm_task(const GemmArgs& g, int epi, int tiles_m, int task, unsigned char* smem) {
  float* sA = reinterpret_cast<float*>(smem);          // [GK][GS]
  float* sB = sA + GK * GS;
  const int tid = threadIdx.x, kg = tid >> 6, ty = (tid & 63) >> 3, tx = tid & 7;
  const int m0 = (task % tiles_m) * GT, n0 = (task / tiles_m) * GT;
  const float *A = reinterpret_cast<const float*>(g.A), *B = reinterpret_cast<const float*>(g.B);
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; i++) { acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f; }
  for (int k0 = 0; k0 < g.K; k0 += GK) {
    const int kc = (min(GK, g.K - k0) + 3) & ~3;       // whole groups of four: rows past K are zero in both panels
    panel_kmajor(sA, A, g.lda, m0, g.M, k0, kc, g.K);
    if (B_KMAJOR) panel_kmajor(sB, B, g.ldb, n0, g.N, k0, kc, g.K);
    else panel_nmajor(sB, B, g.ldb, n0, g.N, k0, kc, g.K);
    __syncthreads();
#pragma unroll 4
    for (int k = kg; k < kc; k += 4) fma16(acc, ld4s(sA + k * GS + ty * 4), ld4s(sB + k * GS + tx * 4));
    __syncthreads();
  }
  float* red = sA;                                     // [4][GT * GT]
#pragma unroll
  for (int i = 0; i < 4; i++) *reinterpret_cast<float4*>(red + kg * GT * GT + (ty * 4 + i) * GT + tx * 4) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
  __syncthreads();
#pragma unroll 1
  for (int q = 0; q < 4; q++) {                         // a warp's 32 outputs are one row of the tile
    const int o = tid + q * NTHR, m = m0 + o / GT, n = n0 + o % GT;
    const float v = (red[o] + red[GT * GT + o]) + (red[2 * GT * GT + o] + red[3 * GT * GT + o]);
    if (m < g.M && n < g.N) epilogue1(g, epi, m, n, v);
  }
  __syncthreads();
}
// one 16 x 16 tile of C = A[K,M]^T . B[K,N]
__device__ __forceinline__ void gemm_task_tn(const GemmArgs& g, int epi, int tiles_m, int task, unsigned char* smem) {
  float* red = reinterpret_cast<float*>(smem);         // [16][GT_TN * GT_TN]
  const int tid = threadIdx.x, kg = tid >> 4, ty = (tid & 15) >> 2, tx = tid & 3;
  const int m0 = (task % tiles_m) * GT_TN, n0 = (task / tiles_m) * GT_TN;
  const float *A = reinterpret_cast<const float*>(g.A), *B = reinterpret_cast<const float*>(g.B);
  const bool va = aligned_rows(A, g.lda, g.M), vb = aligned_rows(B, g.ldb, g.N);
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; i++) { acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f; }
  int k = kg;
  if (va && vb) {
#pragma unroll 1
    for (; k + 7 * 16 < g.K; k += 8 * 16) {
      float4 a[8], b[8];
#pragma unroll
      for (int u = 0; u < 8; u++) {
        a[u] = row4(A + (size_t)(k + u * 16) * g.lda, m0 + ty * 4, g.M, true);
        b[u] = row4(B + (size_t)(k + u * 16) * g.ldb, n0 + tx * 4, g.N, true);
      }
#pragma unroll
      for (int u = 0; u < 8; u++) fma16(acc, a[u], b[u]);
    }
  }
#pragma unroll 1
  for (; k + 3 * 16 < g.K; k += 4 * 16) {
    float4 a[4], b[4];
#pragma unroll
    for (int u = 0; u < 4; u++) { a[u] = row4(A + (size_t)(k + u * 16) * g.lda, m0 + ty * 4, g.M, va); b[u] = row4(B + (size_t)(k + u * 16) * g.ldb, n0 + tx * 4, g.N, vb); }
#pragma unroll
    for (int u = 0; u < 4; u++) fma16(acc, a[u], b[u]);
  }
#pragma unroll 1
  for (; k < g.K; k += 16) fma16(acc, row4(A + (size_t)k * g.lda, m0 + ty * 4, g.M, va), row4(B + (size_t)k * g.ldb, n0 + tx * 4, g.N, vb));
#pragma unroll
  for (int i = 0; i < 4; i++) *reinterpret_cast<float4*>(red + kg * 256 + (ty * 4 + i) * GT_TN + tx * 4) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
  __syncthreads();
  float v = 0.f;
#pragma unroll 4
  for (int q = 0; q < 16; q++) v += red[q * 256 + tid];
  const int m = m0 + tid / GT_TN, n = n0 + tid % GT_TN;
  if (m < g.M && n < g.N) epilogue1(g, epi, m, n, v);
  __syncthreads();
}
__device__ __noinline__ void gemm_run(const PhaseDesc& d, int task, unsigned char* smem) {
  switch (d.layout) {
    case GL_NN: gemm_task<false>(d.g, d.epi, d.tiles_m, task, smem); break;
    case GL_NT: gemm_task<true>(d.g, d.epi, d.tiles_m, task, smem); break;
    default:    gemm_task_tn(d.g, d.epi, d.tiles_m, task, smem); break;
  }
}

// ---------------------------------------------------------------------------------------------- attention (one task per (b, h))
// Four lanes share a row: lane l takes every fourth partner position, with the row's own vectors in registers; rows of scores have an odd
// length so that the rows of a warp fall into different banks (an even T is padded by a word; T = 151, the longest that fits a block, is odd).
__host__ __device__ constexpr int score_row(int T) { return T | 1; }
__host__ __device__ constexpr size_t attn_fwd_smem(int T, int DH) { return (size_t)(3 * T * DH + T * score_row(T)) * 4; }
__host__ __device__ constexpr size_t attn_bwd_smem(int T, int DH) { return (size_t)(5 * T * DH + 2 * T * score_row(T) + T) * 4; }

template <int DH> __device__ __forceinline__ void ld_row(const float* p, float (&f)[DH]) {
#pragma unroll
  for (int c = 0; c < DH; c += 4) { const float4 v = ld4s(p + c); f[c] = v.x; f[c + 1] = v.y; f[c + 2] = v.z; f[c + 3] = v.w; }
}
template <int DH> __device__ __forceinline__ float dot_row(const float (&a)[DH], const float* p) {
  float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
#pragma unroll
  for (int c = 0; c < DH; c += 4) { const float4 v = ld4s(p + c); s0 = fmaf(a[c], v.x, s0); s1 = fmaf(a[c + 1], v.y, s1); s2 = fmaf(a[c + 2], v.z, s2); s3 = fmaf(a[c + 3], v.w, s3); }
  return (s0 + s1) + (s2 + s3);
}
__device__ __forceinline__ float sum4(float v) { v += __shfl_xor_sync(0xffffffffu, v, 1); return v + __shfl_xor_sync(0xffffffffu, v, 2); }
// four consecutive floats of a row to global memory; vec: 16-byte aligned
__device__ __forceinline__ void st4row(float* p, const float4 v, bool vec) {
  if (vec) *reinterpret_cast<float4*>(p) = v;
  else { p[0] = v.x; p[1] = v.y; p[2] = v.z; p[3] = v.w; }
}
// rows [0, T) of one head's columns of a [.., ld] matrix into a [T][DH] array
template <int DH> __device__ __forceinline__ void load_heads(float* dst, const float* src, int ld, int T) {
  const bool vec = aligned_rows(src, ld, DH);
  for (int i = threadIdx.x; i < T * (DH / 4); i += NTHR) {
    const int r = i / (DH / 4), c = (i % (DH / 4)) * 4;
    *reinterpret_cast<float4*>(dst + r * DH + c) = row4(src + (size_t)r * ld, c, DH, vec);
  }
}

template <int DH>
__device__ __forceinline__ void attn_fwd_task(const float* qkv, float* o, float* lse, int b, int h, int T, int H, unsigned char* smem) {
  const int D = H * DH, ld = 3 * D, S = score_row(T);
  float* sq = reinterpret_cast<float*>(smem); float* sk = sq + T * DH; float* sv = sk + T * DH; float* sp = sv + T * DH;
  const float scale = rsqrtf((float)DH);
  const float* base = qkv + (size_t)b * T * ld + h * DH;
  load_heads<DH>(sq, base, ld, T); load_heads<DH>(sk, base + D, ld, T); load_heads<DH>(sv, base + 2 * D, ld, T);
  __syncthreads();
  const int l = threadIdx.x & 3;
  for (int r0 = 0; r0 < T; r0 += NTHR / 4) {
    const int i = r0 + (threadIdx.x >> 2), ir = min(i, T - 1);
    float q[DH], acc[DH];
    ld_row<DH>(sq + ir * DH, q);
    float m = -INFINITY;
    for (int j = l; j <= ir; j += 4) { const float s = dot_row<DH>(q, sk + j * DH) * scale; sp[ir * S + j] = s; m = fmaxf(m, s); }
    m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1)); m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
    float sum = 0.f;
#pragma unroll
    for (int c = 0; c < DH; c++) acc[c] = 0.f;
    for (int j = l; j <= ir; j += 4) {
      const float p = expf(sp[ir * S + j] - m);
      sum += p;
#pragma unroll
      for (int c = 0; c < DH; c += 4) { const float4 v = ld4s(sv + j * DH + c); acc[c] = fmaf(p, v.x, acc[c]); acc[c + 1] = fmaf(p, v.y, acc[c + 1]); acc[c + 2] = fmaf(p, v.z, acc[c + 2]); acc[c + 3] = fmaf(p, v.w, acc[c + 3]); }
    }
    sum = sum4(sum);
    const float inv = 1.f / sum;
#pragma unroll
    for (int c = 0; c < DH; c++) acc[c] = sum4(acc[c]) * inv;
    if (i < T) {
#pragma unroll
      for (int c = 0; c < DH; c += 4)
        if (c / 4 % 4 == l) st4row(o + (size_t)(b * T + i) * D + h * DH + c, make_float4(acc[c], acc[c + 1], acc[c + 2], acc[c + 3]), aligned_rows(o, D, DH));
      if (l == 0) lse[((size_t)b * H + h) * T + i] = m + logf(sum);
    }
  }
  __syncthreads();
}

// dq | dk | dv for one (b, h): recomputes P from lse, D = rowsum(dO * O), dS = P * (dP - D).
template <int DH>
__device__ __forceinline__ void attn_bwd_task(const float* qkv, const float* o, const float* dO, const float* lse, float* dqkv,
                                              int b, int h, int T, int H, unsigned char* smem) {
  const int D = H * DH, ld = 3 * D, S = score_row(T);
  float* sq = reinterpret_cast<float*>(smem); float* sk = sq + T * DH; float* sv = sk + T * DH; float* sdo = sv + T * DH; float* so = sdo + T * DH;
  float* sp = so + T * DH; float* sds = sp + T * S;
  const float scale = rsqrtf((float)DH);
  const float* base = qkv + (size_t)b * T * ld + h * DH;
  load_heads<DH>(sq, base, ld, T); load_heads<DH>(sk, base + D, ld, T); load_heads<DH>(sv, base + 2 * D, ld, T);
  load_heads<DH>(sdo, dO + (size_t)b * T * D + h * DH, D, T); load_heads<DH>(so, o + (size_t)b * T * D + h * DH, D, T);
  __syncthreads();
  const int l = threadIdx.x & 3;
  for (int r0 = 0; r0 < T; r0 += NTHR / 4) {
    const int i = r0 + (threadIdx.x >> 2);
    if (i >= T) continue;                              // whole groups of four lanes; no shuffles below
    float q[DH], d[DH];
    ld_row<DH>(sq + i * DH, q); ld_row<DH>(sdo + i * DH, d);
    const float Di = dot_row<DH>(d, so + i * DH), L = lse[((size_t)b * H + h) * T + i];
    for (int j = l; j <= i; j += 4) {
      const float p = expf(dot_row<DH>(q, sk + j * DH) * scale - L);
      sp[i * S + j] = p; sds[i * S + j] = p * (dot_row<DH>(d, sv + j * DH) - Di);
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < T * (DH / 4); e += NTHR) {
    const int r = e / (DH / 4), c = (e % (DH / 4)) * 4;
    float4 dq = zero4(), dk = zero4(), dv = zero4();
    auto add = [](float4& a, float w, const float4 x) { a.x = fmaf(w, x.x, a.x); a.y = fmaf(w, x.y, a.y); a.z = fmaf(w, x.z, a.z); a.w = fmaf(w, x.w, a.w); };
#pragma unroll 4
    for (int j = 0; j <= r; j++) add(dq, sds[r * S + j], ld4s(sk + j * DH + c));
#pragma unroll 4
    for (int i = r; i < T; i++) { add(dk, sds[i * S + r], ld4s(sq + i * DH + c)); add(dv, sp[i * S + r], ld4s(sdo + i * DH + c)); }
    float* row = dqkv + (size_t)(b * T + r) * ld + h * DH + c;
    const bool vec = aligned_rows(dqkv, ld, DH);
    st4row(row, make_float4(dq.x * scale, dq.y * scale, dq.z * scale, dq.w * scale), vec);
    st4row(row + D, make_float4(dk.x * scale, dk.y * scale, dk.z * scale, dk.w * scale), vec);
    st4row(row + 2 * D, dv, vec);
  }
  __syncthreads();
}

}  // namespace f32
}  // namespace ofa
