// Batch-1 KV-cache decode from the LIVE working-copy weights, as tasks of the serving job.
//
// Phase structure and every rounding point follow the reference's decode task set
// (llm/b200/megakernel/decode_wide.cuh:251-626): per layer QKV (LN1 prologue + 64-column GEMV slice, K/V row appended at
// `pos`), ATT+WO (one head's softmax attention + its slice of Wo), UP+DOWN (LN2 + 32 hidden units + their slice of Wdown);
// then HEAD (LN_f + 64 vocabulary rows per task, fp32 logits, chunk-local argmax / Gumbel-max) and SAMPLE (fixed-order
// final pick, prompt forcing / answer mode, position update, next embedding). The residual stream is kept in int64 fixed
// point (2^-30 units) and updated with integer atomics, so the result is bitwise independent of task order. LN output,
// attention output and GELU output are each rounded to the activation type T before the next product; q, K, V are stored
// as T; softmax uses expf; GELU uses tanhf; argmax ties go to the lower index and NaN never wins.
// Nothing synchronises the decoder with the trainer: it reads whatever the working copy holds.
//
// What is different from the reference is where the weights wait. A serving block knows its next task as soon as it has
// claimed the ticket, usually before the task's dependencies are complete. In that window it starts bulk copies (TMA,
// cp.async.bulk, completion counted on an mbarrier) of everything the task will read that does not depend on the current
// token - its weight slice, and for attention the K/V rows of earlier positions - into a 96 KB shared-memory buffer. When the
// dependencies resolve the task only runs its LayerNorm prologue and multiplies out of shared memory, so the 38 dependent
// phases of a token no longer each pay a DRAM round trip (measured before this change: 5 us of an 8.7 us QKV task was
// waiting for its second batch of weight loads).
//
// Unlike the reference, the code is generic over T in {bf16, float}, the width D and the head dim DH (the thread mappings
// are derived from the 16-byte vector width), so the tiny fp32 model runs through the same tasks.
#pragma once
#include "common.cuh"
#include "task_api.h"

namespace ofa {
namespace dec {

constexpr int HR = 64;                                // vocabulary rows per head task (one task's rows fill the weight buffer)
constexpr int HU = 32;                                // hidden units per UP+DOWN task
constexpr float FX_SCALE = 1073741824.0f;             // 2^30
constexpr float FX_INV = 1.0f / 1073741824.0f;
__device__ __forceinline__ unsigned long long fx(float v) { return (unsigned long long)llrintf(v * FX_SCALE); }
__device__ __forceinline__ float unfx(unsigned long long u) { return (float)(long long)u * FX_INV; }

__device__ __forceinline__ uint4 ldw16(const void* p) {   // streaming 16-byte load that never allocates in L1
  uint4 r;
  asm volatile("ld.global.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p) : "memory");
  return r;
}
template <class T> __device__ __forceinline__ void cvt16(uint4 u, float* f);      // 16 raw bytes -> Vec<T>::N floats
template <> __device__ __forceinline__ void cvt16<bf16>(uint4 u, float* f) { unpack8(u, f); }
template <> __device__ __forceinline__ void cvt16<float>(uint4 u, float* f) { f[0] = __uint_as_float(u.x); f[1] = __uint_as_float(u.y); f[2] = __uint_as_float(u.z); f[3] = __uint_as_float(u.w); }
template <class T> __device__ __forceinline__ float ldcg_f(const T* p);
template <> __device__ __forceinline__ float ldcg_f<bf16>(const bf16* p) { return __bfloat162float(__ldcg(p)); }
template <> __device__ __forceinline__ float ldcg_f<float>(const float* p) { return __ldcg(p); }

__device__ __forceinline__ bool better(float a, int ai, float b, int bi) {
  if (a != a) return false;
  if (b != b) return true;
  return a > b || (a == b && ai < bi);
}
__device__ __forceinline__ void block_argmax(float& v, int& idx, float* sv, int* si) {
  for (int o = 16; o; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, v, o);
    const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
    if (better(ov, oi, v, idx)) { v = ov; idx = oi; }
  }
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) { sv[w] = v; si[w] = idx; }
  __syncthreads();
  v = sv[0]; idx = si[0];
#pragma unroll
  for (int i = 1; i < 8; i++) if (better(sv[i], si[i], v, idx)) { v = sv[i]; idx = si[i]; }
  __syncthreads();
}
// counter-based Gumbel(0,1) noise keyed by (seed, step, vocabulary index)
static __device__ __noinline__ float gumbel(u64 seed, uint32_t step, uint32_t v) {
  const u64 r = splitmix64(splitmix64(seed ^ ((u64)step << 32)) + v);
  const float u = ((float)(uint32_t)(r >> 40) + 0.5f) * (1.0f / 16777216.0f);
  return -logf(-logf(u));
}

// stage stamps of one traced task instance (layer 0, task 0): slot base + i
__device__ __forceinline__ void trace(unsigned long long* tr, bool on, int slot) { if (on && tr && threadIdx.x == 0) tr[slot] = gtimer(); }

template <class T, int D, int DH> struct Geo {
  static constexpr int VN = Vec<T>::N;
  static constexpr int ES = (int)sizeof(T);
  static constexpr int CB = D < 256 ? D : 256;        // residual columns per attention/Wo task
  static constexpr int NCB = D / CB;
  static constexpr int WB = D * 64 * ES;              // weight buffer: one 64-column slice of a [D, *] matrix (98,304 B for GPT-S)
  static constexpr int WO_BYTES = DH * CB * ES;       // Wo slice of an attention task
  static constexpr int KV_ROWS = (WB - WO_BYTES) / 2 / (DH * ES);   // K (and V) rows of earlier positions that fit beside it
  static constexpr int LPK = DH / VN;                 // lanes per key row
  static constexpr int KPR = NTHR / LPK;              // keys per round
  static constexpr int RED = 1024;                    // floats of reduction scratch
  static_assert(D % CB == 0 && D % 64 == 0 && DH % VN == 0 && NTHR % LPK == 0 && HU * D * ES * 2 <= WB && HR * D * ES <= WB && KPR * DH <= 2048, "geometry");
};
// shared memory: weight buffer [WB] | floats xs[D] red[2048] res[64] scratch[32] hb[64] sc[T] lg[HR] | int meta[4]
// meta: 0 = position word the K/V prefetch saw (DS_POSKEY), 1 = launch step + 1 that word 3 belongs to, 2 = launch step + 1 whose final
// LayerNorm is in xs, 3 = position word of that step
template <class T, int D, int DH> __host__ __device__ constexpr size_t smem_bytes(int Tctx) {
  return (size_t)Geo<T, D, DH>::WB + (size_t)(D + 2048 + 64 + 32 + 64 + Tctx + HR + 4) * 4;
}
template <class T, int D, int DH> struct Smem {
  unsigned char* w; float *xs, *red, *res, *scratch, *hb, *sc, *lg; int* meta;
  __device__ __forceinline__ Smem(unsigned char* base, int Tctx) {
    w = base; xs = reinterpret_cast<float*>(base + Geo<T, D, DH>::WB); red = xs + D; res = red + 2048; scratch = res + 64; hb = scratch + 32;
    sc = hb + 64; lg = sc + Tctx; meta = reinterpret_cast<int*>(lg + HR);
  }
};

// once per serving block, before its first task
template <class T, int D, int DH>
__device__ __forceinline__ void block_init(unsigned char* smem, int Tctx) {
  Smem<T, D, DH> S(smem, Tctx);
  if (threadIdx.x < 4) S.meta[threadIdx.x] = 0;
}

__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}

// ---------------------------------------------------------------------------------------------- prefetch (runs while the task's dependencies are still pending)
// Starts the bulk copies of task (kind, layer, t) into the weight buffer; warp 0 only. Returns true (uniformly for the block)
// if the task has a fill to wait for. The LayerNorm's gamma comes along into `red`, which no task writes before its LayerNorm is done: read
// after the dependency wait it cost a DRAM round trip (the weights of a token are twice the L2, so it is never there), about 0.2 us per phase.
// `bar` is the block's fill barrier (count 1); each fill is one phase of it.
template <class T, int D, int DH>
__device__ __forceinline__ bool prefetch(const DecodeParams& P, const ModelDims& md, int kind, int layer, int t, int step, unsigned char* smem, uint32_t bar) {
  using G = Geo<T, D, DH>;
  if (kind == TK_DEC_SAMPLE) return false;
  if (threadIdx.x >= 32) return true;
  const int lane = threadIdx.x;
  const uint32_t dst = smem_u32(smem);
  Smem<T, D, DH> S(smem, md.T);
  fence_proxy_async();          // the previous task's ordinary accesses to the buffer come before these asynchronous writes
  switch (kind) {
    case TK_DEC_QKV: {
      constexpr int RBY = 64 * G::ES;
      if (lane == 0) mbar_expect_tx(bar, D * RBY + D * G::ES);
      __syncwarp();
      if (lane == 8) bulk_g2s(smem_u32(S.red), P.g1[layer], D * G::ES, bar);
      constexpr int BR = D < 256 ? D : 256;            // rows per TMA box
      if (lane < D / BR) tma_load_2d(dst + lane * BR * RBY, reinterpret_cast<const char*>(P.tm_qkv) + (size_t)layer * 128, bar, t * 64, lane * BR);
      break;
    }
    case TK_DEC_ATTWO: {
      const int head = t / G::NCB, cb = t % G::NCB;
      // rows of earlier positions: the position word may be older than the token this task belongs to (tickets are claimed
      // ahead), so the epoch it carries is kept and the task uses the copied rows only if it runs in the same context
      const int key = __ldcg(&P.st.scal[DS_POSKEY]);
      int np = key & 0xFFFF;
      np = np < G::KV_ROWS ? np : G::KV_ROWS;
      const uint32_t kvb = (uint32_t)np * DH * G::ES;
      if (lane == 0) { S.meta[0] = (key & ~0xFFFF) | np; mbar_expect_tx(bar, G::WO_BYTES + 2 * kvb); }
      __syncwarp();
      if (lane == 2) tma_load_2d(dst, reinterpret_cast<const char*>(P.tm_wo) + (size_t)layer * 128, bar, cb * G::CB, head * DH);
      if (np > 0 && lane < 2) {
        const T* kv = reinterpret_cast<const T*>(P.st.kv) + (((size_t)layer * 2 + lane) * md.H + head) * md.T * DH;
        bulk_g2s(dst + G::WO_BYTES + lane * G::KV_ROWS * DH * G::ES, kv, kvb, bar);
      }
      break;
    }
    case TK_DEC_UPDN: {
      constexpr int RBY = HU * G::ES;
      if (lane == 0) mbar_expect_tx(bar, 2 * D * RBY + D * G::ES);
      __syncwarp();
      if (lane == 8) bulk_g2s(smem_u32(S.red), P.g2[layer], D * G::ES, bar);
      constexpr int BR = D < 256 ? D : 256;
      if (lane >= 1 && lane <= D / BR) tma_load_2d(dst + (lane - 1) * BR * RBY, reinterpret_cast<const char*>(P.tm_up) + (size_t)layer * 128, bar, t * HU, (lane - 1) * BR);
      if (lane == 0) bulk_g2s(dst + D * RBY, reinterpret_cast<const T*>(P.wdn[layer]) + (size_t)t * HU * D, D * RBY, bar);
      break;
    }
    default: {  // TK_DEC_HEAD
      const int rows = min(HR, md.V - t * HR);
      const int gb = S.meta[2] != step + 1 ? D * G::ES : 0;      // the task makes the same test before its LayerNorm
      if (lane == 0) { mbar_expect_tx(bar, rows * D * G::ES + gb); if (gb) bulk_g2s(smem_u32(S.red), P.gf, gb, bar); bulk_g2s(dst, reinterpret_cast<const T*>(P.head) + (size_t)t * HR * D, rows * D * G::ES, bar); }
      break;
    }
  }
  return true;
}

// the block's fill has landed; out of line what comes after the first probe
static __device__ __noinline__ bool wait_fill_slow(uint32_t bar, uint32_t parity, DevStatus* status, int layer, int t) {
  const bool ok = mbar_wait_slow(bar, parity, status);
  if (!ok && !aborted(status)) raise_abort(status, ST_MBAR_FULL_TIMEOUT, -2, t, layer);
  return ok;
}
__device__ __forceinline__ bool wait_fill(uint32_t bar, uint32_t parity, DevStatus* status, int layer, int t) {
  return mbar_try(bar, parity) || wait_fill_slow(bar, parity, status, layer, t);
}

// xs[k] = round_T(LN(x)[k] * gamma[k]); x = fixed-point residual `src`, gamma in shared memory once the task's fill has landed. One block
// reduction of shifted sums. Ends with a block barrier; false (for all threads) if the fill never came.
template <class T, int D>
__device__ __forceinline__ bool prologue_ln(const unsigned long long* src, const T* gamma, float* xs, float* scratch, unsigned long long* copy_to,
                                            uint32_t bar, uint32_t parity, DevStatus* status, int layer, int t) {
  constexpr int NE = (D + NTHR - 1) / NTHR;
  const int tid = threadIdx.x;
  float x[NE];
  unsigned long long raw[NE];
  const unsigned long long raw0 = __ldcg(&src[0]);
#pragma unroll
  for (int i = 0; i < NE; i++) {                       // every load before the first store of copy_to, which the compiler cannot tell apart from them
    const int k = tid + i * NTHR;
    raw[i] = k < D ? __ldcg(&src[k]) : 0ull;
  }
  const float xref = unfx(raw0);
  float s1 = 0.f, s2 = 0.f;
#pragma unroll
  for (int i = 0; i < NE; i++) {
    const int k = tid + i * NTHR;
    if (k < D) {
      x[i] = unfx(raw[i]);
      const float d = x[i] - xref;
      s1 += d; s2 += d * d;
      if (copy_to) copy_to[k] = raw[i];
    }
  }
  for (int o = 16; o; o >>= 1) { s1 += __shfl_xor_sync(0xffffffffu, s1, o); s2 += __shfl_xor_sync(0xffffffffu, s2, o); }
  if ((tid & 31) == 0) { scratch[tid >> 5] = s1; scratch[8 + (tid >> 5)] = s2; }
  const bool ok = wait_fill(bar, parity, status, layer, t);
  __syncthreads();
  float t1 = 0.f, t2 = 0.f;
#pragma unroll
  for (int i = 0; i < 8; i++) { t1 += scratch[i]; t2 += scratch[8 + i]; }
  const float m1 = t1 * (1.0f / D);
  const float var = fmaxf(t2 * (1.0f / D) - m1 * m1, 0.f);
  const float mean = xref + m1, rstd = rsqrtf(var + 1e-5f);
#pragma unroll
  for (int i = 0; i < NE; i++) {
    const int k = tid + i * NTHR;
    if (k < D) xs[k] = round_to<T>((x[i] - mean) * rstd * to_f(gamma[k]));
  }
  return !__syncthreads_or(!ok);                       // uniform decision: nobody is left behind at a later barrier
}

// Sums a[0..N) over the lanes that differ in the bits O .. END / 2, handing each half of a pair half of the values as long as there are two:
// 4 + 2 + 1 shuffles for eight values over eight lanes instead of 24. scatter_index gives the first value a lane ends up with,
// scatter_left how many it holds (values that ran out early are held by several lanes).
template <int N, int O, int END = 32> __device__ __forceinline__ void reduce_scatter(float* a) {
  if constexpr (O < END) {
    if constexpr (N > 1) {
      const bool hi = (threadIdx.x & O) != 0;
#pragma unroll
      for (int i = 0; i < N / 2; i++) {
        const float send = hi ? a[i] : a[i + N / 2], keep = hi ? a[i + N / 2] : a[i];
        a[i] = keep + __shfl_xor_sync(0xffffffffu, send, O);
      }
      reduce_scatter<N / 2, 2 * O, END>(a);
    } else {
      a[0] += __shfl_xor_sync(0xffffffffu, a[0], O);
      reduce_scatter<1, 2 * O, END>(a);
    }
  }
}
template <int N, int O, int END = 32> __device__ __forceinline__ int scatter_index() {
  if constexpr (N > 1 && O < END) return ((threadIdx.x & O) ? N / 2 : 0) + scatter_index<N / 2, 2 * O, END>();
  else return 0;
}
template <int N, int O, int END = 32> __host__ __device__ constexpr int scatter_left() {
  if constexpr (N > 1 && O < END) return scatter_left<N / 2, 2 * O, END>();
  else return N;
}

// sum_k xs[k] * W[k][c] for a [D][NC] slice resident in shared memory (NC = 64 or 32); threads c < NC return column c. A thread reads
// 16 bytes of a row, so a warp moves 512 consecutive bytes per instruction (the slice costs 768 clocks of shared-memory bandwidth at
// 96 KB); the warp's row groups meet in shuffles, the eight warps in `red`, in index order. One 64-column slice: 1.4 us with four-byte
// reads and 24 rounds of four rows, 0.9 us now.
template <class T, int NC, int D>
__device__ __forceinline__ float gemv_smem(const T* W, const float* xs, float* red) {
  constexpr int VN = Vec<T>::N, LPR = NC / VN, RG = NTHR / LPR, LEFT = scatter_left<VN, LPR>();
  static_assert(D % RG == 0 && LPR <= 32, "gemv geometry");
  const int tid = threadIdx.x, w = tid >> 5, l = tid % LPR, rg = tid / LPR;
  float a[VN];
#pragma unroll
  for (int i = 0; i < VN; i++) a[i] = 0.f;
#pragma unroll 4
  for (int k = rg; k < D; k += RG) {
    float f[VN]; cvt16<T>(*reinterpret_cast<const uint4*>(W + (size_t)k * NC + l * VN), f);
    const float x = xs[k];
#pragma unroll
    for (int i = 0; i < VN; i++) a[i] = fmaf(x, f[i], a[i]);
  }
  reduce_scatter<VN, LPR>(a);
  const int c = l * VN + scatter_index<VN, LPR>();
#pragma unroll
  for (int i = 0; i < LEFT; i++) red[w * NC + c + i] = a[i];
  __syncthreads();
  float r = 0.f;
  if (tid < NC) {
#pragma unroll
    for (int g = 0; g < NTHR / 32; g++) r += red[g * NC + tid];
  }
  return r;
}
// part[kg][c] = sum over the kg-th share of x[0..NK) of x[k] * W[k][c], c < NC, W [NK][NC] in shared memory: every thread owns 16 bytes of
// a row. Returns the number of shares; the caller adds them in order after a barrier.
template <class T, int NC, int NK>
__device__ __forceinline__ void gemv_shares(const T* W, const float* x, float* part) {
  constexpr int VN = Vec<T>::N, CG = NC / VN, KG = NTHR / CG, KPT = NK / KG;
  static_assert(NK % KG == 0 && KG * NC <= 2048, "share geometry");
  const int tid = threadIdx.x, kg = tid / CG, c = (tid % CG) * VN;
  if (kg < KG) {
    float a[VN];
#pragma unroll
    for (int i = 0; i < VN; i++) a[i] = 0.f;
#pragma unroll                                         // whole: by fours a served token takes 182.2 instead of 181.4 us, on 24 SMs 340.3 instead of 339.7
    for (int q = 0; q < KPT; q++) {
      const int k = kg * KPT + q;
      float f[VN]; cvt16<T>(*reinterpret_cast<const uint4*>(W + (size_t)k * NC + c), f);
      const float xv = x[k];
#pragma unroll
      for (int i = 0; i < VN; i++) a[i] = fmaf(xv, f[i], a[i]);
    }
#pragma unroll
    for (int i = 0; i < VN; i += 4) *reinterpret_cast<float4*>(part + kg * NC + c + i) = make_float4(a[i], a[i + 1], a[i + 2], a[i + 3]);
  }
}
template <class T, int NC> __host__ __device__ constexpr int gemv_nshares() { return NTHR / (NC / Vec<T>::N); }

// ---------------------------------------------------------------------------------------------- tasks
// Every task: dependent prologue first, then wait (bounded) for its fill, then multiply out of shared memory.
#define OFA_DEC_WAIT_FILL()                                                                                        \
  {                                                                                                                 \
    const bool ok_ = wait_fill(bar, parity, status, layer, t);                                                      \
    if (__syncthreads_or(!ok_)) return;      /* uniform decision: nobody is left behind at a later barrier */       \
  }

// The position word (DS_POSKEY: context epoch, position) is written once per token, by SAMPLE: a block reads it in its first task of a
// step and keeps it, so that the later ones can ask for q and the newest K/V row without a round trip in front.
template <class SM> __device__ __forceinline__ int position_word(const SM& S, const DecodeState& st, int step) {
  return S.meta[1] == step + 1 ? S.meta[3] : __ldcg(&st.scal[DS_POSKEY]);
}
template <class SM> __device__ __forceinline__ void keep_position(const SM& S, int step, int key) {   // behind a block barrier that follows position_word
  if (threadIdx.x == 0) { S.meta[1] = step + 1; S.meta[3] = key; }
}

// QKV: task t = columns [64t, 64t+64) of [q|k|v]; ntasks = 3D/64.
template <class T, int D, int DH, bool PROF>
__device__ __forceinline__ void task_qkv(const DecodeParams& P, const ModelDims& md, int layer, int t, int step, unsigned char* smem, uint32_t bar, uint32_t parity, DevStatus* status) {
  Smem<T, D, DH> S(smem, md.T);
  const DecodeState& st = P.st;
  const bool tr = PROF && layer == 0 && t == 0;
  trace(P.trace, tr, 0);
  const int key = position_word(S, st, step);
  if (threadIdx.x == 0) S.meta[2] = 0;                 // xs no longer holds a final-LayerNorm row
  if (!prologue_ln<T, D>(st.xw, reinterpret_cast<const T*>(S.red), S.xs, S.scratch, t == 0 ? st.xr : nullptr, bar, parity, status, layer, t)) return;
  trace(P.trace, tr, 1);
  keep_position(S, step, key);
  trace(P.trace, tr, 2);
  const float r = gemv_smem<T, 64, D>(reinterpret_cast<const T*>(S.w), S.xs, S.red);
  trace(P.trace, tr, 3);
  if (threadIdx.x < 64) {
    const int col = t * 64 + threadIdx.x, which = col / D, within = col % D;
    const T o = from_f<T>(r);
    if (which == 0) reinterpret_cast<T*>(st.q)[within] = o;
    else {
      const int head = within / DH, i = within % DH, pos = key & 0xFFFF;
      reinterpret_cast<T*>(st.kv)[((((size_t)layer * 2 + (which - 1)) * md.H + head) * md.T + pos) * DH + i] = o;
    }
  }
  trace(P.trace, tr, 4);
}

// ATT+WO: task t -> head = t / NCB, column block cb = t % NCB; ntasks = H * NCB. K/V rows below min(prefetched, pos) come from
// shared memory, the first KPR rows above them, the current token's among them, from registers (asked for together with q), others
// from global memory.
// LPK lanes share a key; a group takes every KPR-th key, keeps a maximum of its own and weighs its keys against it, so the block meets
// once, when the eight warps' sums are brought to the largest maximum. With a maximum and a sum over the whole block first the task
// took 4.2 us on average over a 256-token answer (six block barriers, three round trips to L2 one after the other), now 3.2.
template <class T, int D, int DH, bool PROF>
__device__ __forceinline__ void task_attwo(const DecodeParams& P, const ModelDims& md, int layer, int t, int step, unsigned char* smem, uint32_t bar, uint32_t parity, DevStatus* status) {
  using G = Geo<T, D, DH>;
  constexpr int VN = G::VN, LPK = G::LPK, KPR = G::KPR, NW = NTHR / 32;
  static_assert((KPR & (KPR - 1)) == 0, "row ownership");
  Smem<T, D, DH> S(smem, md.T);
  float* ob = S.res;
  const DecodeState& st = P.st;
  const int tid = threadIdx.x, g = tid / LPK, l = tid % LPK, w = tid >> 5;
  const int head = t / G::NCB, cb = t % G::NCB;
  const bool tr = PROF && layer == 0 && t == 0;
  trace(P.trace, tr, 24);
  const int key = position_word(S, st, step), pos = key & 0xFFFF, n = pos + 1;
  const T* Kc = reinterpret_cast<const T*>(st.kv) + (((size_t)layer * 2 + 0) * md.H + head) * md.T * DH;
  const T* Vc = reinterpret_cast<const T*>(st.kv) + (((size_t)layer * 2 + 1) * md.H + head) * md.T * DH;
  const uint4 q4 = ldw16(reinterpret_cast<const T*>(st.q) + head * DH + l * VN);
  const int seen = S.meta[0];
  const int nres = ((seen ^ key) >> 16) == 0 ? min(seen & 0xFFFF, pos) : 0;   // rows valid in shared memory: same context epoch
  // this group's first row that is not: asked for now, beside q. A group has the rows j = g mod KPR wherever they come from, in rising
  // order, so that how far ahead a block prefetched does not change a bit
  const int jt = nres + ((g - nres) & (KPR - 1));
  uint4 kt = make_uint4(0u, 0u, 0u, 0u), vt = kt;
  if (jt < n) { kt = ldw16(Kc + (size_t)jt * DH + l * VN); vt = ldw16(Vc + (size_t)jt * DH + l * VN); }
  if (tid == 0) S.meta[2] = 0;
  OFA_DEC_WAIT_FILL();
  keep_position(S, step, key);
  trace(P.trace, tr, 25);
  const T* sK = reinterpret_cast<const T*>(S.w + G::WO_BYTES) + l * VN;
  const T* sV = sK + (size_t)G::KV_ROWS * DH;
  Kc += l * VN; Vc += l * VN;
  float qv[VN]; cvt16<T>(q4, qv);
#pragma unroll
  for (int i = 0; i < VN; i++) qv[i] *= rsqrtf((float)DH);
  constexpr int UK = 4;
  auto dot = [&](const uint4 k4) {                     // this lane's share of a score
    float f[VN]; cvt16<T>(k4, f);
    float d = 0.f;
#pragma unroll
    for (int i = 0; i < VN; i++) d = fmaf(qv[i], f[i], d);
    return d;
  };
  float m = -INFINITY;                                 // of the scores this lane ended up with
  const int us = scatter_index<UK, 1, LPK>();
  auto scores = [&](int j0, int end, const uint4 (&kw)[UK]) {      // rows j0, j0 + KPR, .. below `end`
    float d[UK];
#pragma unroll
    for (int u = 0; u < UK; u++) d[u] = dot(kw[u]);
    reduce_scatter<UK, 1, LPK>(d);
    const int j = j0 + KPR * us;
    if (j < end) { m = fmaxf(m, d[0]); S.sc[j] = d[0]; }
  };
  for (int j0 = g; j0 - g < nres; j0 += KPR * UK) {
    uint4 kw[UK];
#pragma unroll
    for (int u = 0; u < UK; u++) kw[u] = *reinterpret_cast<const uint4*>(sK + (size_t)min(j0 + KPR * u, nres - 1) * DH);
    scores(j0, nres, kw);
  }
  {
    float d = dot(kt);
#pragma unroll
    for (int o = 1; o < LPK; o <<= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
    if (jt < n) { m = fmaxf(m, d); if (l == 0) S.sc[jt] = d; }
  }
  for (int j0 = jt + KPR; __any_sync(0xffffffffu, j0 < n); j0 += KPR * UK) {
    uint4 kw[UK];
#pragma unroll
    for (int u = 0; u < UK; u++) kw[u] = ldw16(Kc + (size_t)min(j0 + KPR * u, pos) * DH);
    scores(j0, n, kw);
  }
#pragma unroll
  for (int o = 1; o < LPK; o <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));      // the group's maximum
  __syncwarp();                                        // its scores are read back by the same warp
  trace(P.trace, tr, 26);
  float acc[VN], sum = 0.f;
  const float mg = m == -INFINITY ? 0.f : m;           // no key, or only scores of -inf: every weight is 0
#pragma unroll
  for (int i = 0; i < VN; i++) acc[i] = 0.f;
  auto weigh = [&](int j, int end, const uint4 v4) {
    if (j < end) {
      const float p = expf(S.sc[j] - mg);
      sum += p;
      float f[VN]; cvt16<T>(v4, f);
#pragma unroll
      for (int i = 0; i < VN; i++) acc[i] = fmaf(p, f[i], acc[i]);
    }
  };
  for (int j0 = g; j0 - g < nres; j0 += KPR * UK) {
    uint4 vb[UK];
#pragma unroll
    for (int u = 0; u < UK; u++) vb[u] = *reinterpret_cast<const uint4*>(sV + (size_t)min(j0 + KPR * u, nres - 1) * DH);
#pragma unroll
    for (int u = 0; u < UK; u++) weigh(j0 + KPR * u, nres, vb[u]);
  }
  weigh(jt, n, vt);
  for (int j0 = jt + KPR; j0 < n; j0 += KPR * UK) {
    uint4 vb[UK];
#pragma unroll
    for (int u = 0; u < UK; u++) vb[u] = ldw16(Vc + (size_t)min(j0 + KPR * u, pos) * DH);
#pragma unroll
    for (int u = 0; u < UK; u++) weigh(j0 + KPR * u, n, vb[u]);
  }
  float mw = m;                                        // the warp's groups, brought to the warp's maximum
#pragma unroll
  for (int o = LPK; o < 32; o <<= 1) mw = fmaxf(mw, __shfl_xor_sync(0xffffffffu, mw, o));
  const float fg = m == -INFINITY ? 0.f : expf(m - mw);
  sum *= fg;
#pragma unroll
  for (int o = LPK; o < 32; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
#pragma unroll
  for (int i = 0; i < VN; i++) acc[i] *= fg;
  reduce_scatter<VN, LPK>(acc);
  constexpr int LEFT = scatter_left<VN, LPK>();
  const int ci = l * VN + scatter_index<VN, LPK>();
#pragma unroll
  for (int i = 0; i < LEFT; i++) S.red[w * DH + ci + i] = acc[i];
  if ((tid & 31) == 0) { S.scratch[w] = mw; S.scratch[NW + w] = sum; }
  __syncthreads();
  trace(P.trace, tr, 27);
  if (tid < DH) {
    static_assert(NW == 8 && DH <= NTHR, "one exponential a lane");
    float M = S.scratch[0];
#pragma unroll
    for (int i = 1; i < NW; i++) M = fmaxf(M, S.scratch[i]);
    const float mine = S.scratch[tid & 7], fl = mine == -INFINITY ? 0.f : expf(mine - M);      // lane i: the factor of warp i % 8
    float o = 0.f, sm = 0.f;
#pragma unroll
    for (int i = 0; i < NW; i++) {
      const float fw = __shfl_sync(DH >= 32 ? 0xffffffffu : (1u << (DH & 31)) - 1u, fl, i);
      o += fw * S.red[i * DH + tid]; sm += fw * S.scratch[NW + i];
    }
    ob[tid] = round_to<T>(o / sm);
  }
  __syncthreads();
  gemv_shares<T, G::CB, DH>(reinterpret_cast<const T*>(S.w), ob, S.red);      // o[DH] . Wo slice
  __syncthreads();
  trace(P.trace, tr, 28);
  if (tid < G::CB) {
    float r = 0.f;
#pragma unroll
    for (int i = 0; i < gemv_nshares<T, G::CB>(); i++) r += S.red[i * G::CB + tid];
    const unsigned long long u = fx(r);
    atomicAdd(&st.xr[cb * G::CB + tid], u);
    atomicAdd(&st.xw[cb * G::CB + tid], u);
  }
  trace(P.trace, tr, 29);
}

// UP+DOWN: task t = hidden units [32t, 32t+32); ntasks = FF/32.
template <class T, int D, int DH, bool PROF>
__device__ __forceinline__ void task_updn(const DecodeParams& P, const ModelDims& md, int layer, int t, unsigned char* smem, uint32_t bar, uint32_t parity, DevStatus* status) {
  using G = Geo<T, D, DH>;
  Smem<T, D, DH> S(smem, md.T);
  const DecodeState& st = P.st;
  const bool tr = PROF && layer == 0 && t == 0;
  trace(P.trace, tr, 8);
  if (threadIdx.x == 0) S.meta[2] = 0;
  if (!prologue_ln<T, D>(st.xr, reinterpret_cast<const T*>(S.red), S.xs, S.scratch, nullptr, bar, parity, status, layer, t)) return;
  trace(P.trace, tr, 9);
  trace(P.trace, tr, 10);
  const float h = gemv_smem<T, HU, D>(reinterpret_cast<const T*>(S.w), S.xs, S.red);
  if (threadIdx.x < HU) S.hb[threadIdx.x] = round_to<T>(gelu_fwd<false>(h));
  __syncthreads();
  trace(P.trace, tr, 11);
  // the shares go through shared memory so that a warp's atomics cover consecutive columns (16 bytes a thread would touch four times the sectors)
  gemv_shares<T, D, HU>(reinterpret_cast<const T*>(S.w + (size_t)D * HU * G::ES), S.hb, S.red);      // Wdown rows [HU][D]
  __syncthreads();
  trace(P.trace, tr, 13);
  for (int c = threadIdx.x; c < D; c += NTHR) {
    float r = 0.f;
#pragma unroll
    for (int i = 0; i < gemv_nshares<T, D>(); i++) r += S.red[i * D + c];
    atomicAdd(&st.xw[c], fx(r));
  }
  trace(P.trace, tr, 12);
}

// HEAD: task t = vocabulary rows [64t, 64t+64); ntasks = ceil(V/64). Warp w owns rows 8w..8w+7; a lane keeps its share of the LayerNorm
// row in registers for all of them (read from shared memory for each row, it was two thirds of the task's shared-memory traffic).
template <class T, int D, int DH>
__device__ __forceinline__ void task_head(const DecodeParams& P, const ModelDims& md, int t, int step, unsigned char* smem, uint32_t bar, uint32_t parity, DevStatus* status) {
  using G = Geo<T, D, DH>;
  constexpr int VN = G::VN, VPR = D / VN, RPW = HR / 8;
  Smem<T, D, DH> S(smem, md.T);
  const DecodeState& st = P.st;
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31, layer = -1;
  // the final LayerNorm is the same for every head task of a token: a block that runs several of them in a row keeps it
  if (S.meta[2] != step + 1) {
    if (!prologue_ln<T, D>(st.xw, reinterpret_cast<const T*>(S.red), S.xs, S.scratch, nullptr, bar, parity, status, layer, t)) return;
    if (tid == 0) S.meta[2] = step + 1;
  } else OFA_DEC_WAIT_FILL();
  const T* Wh = reinterpret_cast<const T*>(S.w) + (size_t)w * RPW * D;
  float s[RPW];                                        // rows past the vocabulary hold whatever the buffer held: they are not read below
#pragma unroll
  for (int rr = 0; rr < RPW; rr++) s[rr] = 0.f;
#pragma unroll                                         // as a rolled loop 181.7 instead of 181.1 us a token, on 24 SMs, where a block runs 16 of these, 340.0 instead of 336.2
  for (int i = 0; i < (VPR + 31) / 32; i++) {
    const int vi = lane + 32 * i;
    if (VPR % 32 != 0 && vi >= VPR) break;
    float x[VN];
#pragma unroll
    for (int k = 0; k < VN; k += 4) {
      const float4 v = *reinterpret_cast<const float4*>(S.xs + vi * VN + k);
      x[k] = v.x; x[k + 1] = v.y; x[k + 2] = v.z; x[k + 3] = v.w;
    }
#pragma unroll
    for (int rr = 0; rr < RPW; rr++) {
      float f[VN]; cvt16<T>(*reinterpret_cast<const uint4*>(Wh + (size_t)rr * D + vi * VN), f);
#pragma unroll
      for (int k = 0; k < VN; k++) s[rr] = fmaf(x[k], f[k], s[rr]);
    }
  }
  reduce_scatter<RPW, 1>(s);
  if (lane < RPW) S.lg[w * RPW + scatter_index<RPW, 1>()] = s[0];
  __syncthreads();
  if (w == 0) {                                        // one warp, two rows a lane: no further block barriers
    const float temp = P.temperature, invT = temp > 0.f ? 1.f / temp : 1.f;
    const uint32_t dstep = temp > 0.f ? (uint32_t)__ldcg(&st.scal[DS_STEP]) : 0u;
    const int nchunk = (md.V + HR - 1) / HR;
    float b0 = -INFINITY, b1 = -INFINITY; int i0 = t * HR + lane, i1 = i0;
#pragma unroll
    for (int q = 0; q < HR / 32; q++) {
      const int gi = t * HR + q * 32 + lane;
      if (gi < md.V) {
        const float lv = S.lg[q * 32 + lane];
        st.logits[gi] = lv;
        if (gi < md.valid_vocab) {
          if (better(lv, gi, b0, i0)) { b0 = lv; i0 = gi; }
          if (temp > 0.f) { const float nv = lv * invT + gumbel(P.seed, dstep, gi); if (better(nv, gi, b1, i1)) { b1 = nv; i1 = gi; } }
        }
      }
    }
    auto pick = [](float& v, int& idx) {
#pragma unroll
      for (int o = 16; o; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, v, o);
        const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
        if (better(ov, oi, v, idx)) { v = ov; idx = oi; }
      }
    };
    pick(b0, i0);
    if (temp > 0.f) pick(b1, i1); else { b1 = b0; i1 = i0; }
    if (lane == 0) { st.cand_v[t] = b0; st.cand_i[t] = i0; st.cand_v[nchunk + t] = b1; st.cand_i[nchunk + t] = i1; }
  }
}
#undef OFA_DEC_WAIT_FILL

// xw := fixed point (wte[tok] + wpe[pos])
template <class T, int D>
__device__ __forceinline__ void write_embed(const DecodeParams& P, int tok, int pos) {
  constexpr int NE = (D + NTHR - 1) / NTHR;
  float a[NE], b[NE];
#pragma unroll
  for (int i = 0; i < NE; i++) {                       // all loads before the first store
    const int k = threadIdx.x + i * NTHR;
    a[i] = k < D ? ldcg_f<T>(reinterpret_cast<const T*>(P.wte) + (size_t)tok * D + k) : 0.f;
    b[i] = k < D ? ldcg_f<T>(reinterpret_cast<const T*>(P.wpe) + (size_t)pos * D + k) : 0.f;
  }
#pragma unroll
  for (int i = 0; i < NE; i++) { const int k = threadIdx.x + i * NTHR; if (k < D) P.st.xw[k] = fx(a[i] + b[i]); }
}

// SAMPLE: one task. Final pick over the chunk candidates, prompt forcing / answer mode, pos/step update, next embedding.
template <class T, int D, int DH>
__device__ __forceinline__ void task_sample(const DecodeParams& P, const ModelDims& md, Live* live, unsigned char* smem) {
  const DecodeState& st = P.st;
  float* sv = reinterpret_cast<float*>(smem); int* si = reinterpret_cast<int*>(sv + 8); int* sn = si + 8;
  const int tid = threadIdx.x, mode = P.temperature > 0.f ? 1 : 0;
  const int nchunk = (md.V + HR - 1) / HR;
  int step = 0, pos = 0, astep = 0, epoch = 0;
  if (tid == 0) { step = __ldcg(&st.scal[DS_STEP]); pos = __ldcg(&st.scal[DS_POS]); astep = __ldcg(&st.scal[DS_ASTEP]); epoch = __ldcg(&st.scal[DS_EPOCH]); }   // on their way beside the candidates
  float bv = -INFINITY; int bi = 0x7fffffff;
  constexpr int UC = 4;
  for (int c0 = tid; c0 < nchunk; c0 += UC * NTHR) {
    float v[UC]; int i[UC];
#pragma unroll
    for (int u = 0; u < UC; u++) {
      const int c = c0 + u * NTHR;
      v[u] = c < nchunk ? __ldcg(&st.cand_v[mode * nchunk + c]) : -INFINITY;
      i[u] = c < nchunk ? __ldcg(&st.cand_i[mode * nchunk + c]) : 0x7fffffff;
    }
#pragma unroll
    for (int u = 0; u < UC; u++) if (better(v[u], i[u], bv, bi)) { bv = v[u]; bi = i[u]; }
  }
  block_argmax(bv, bi, sv, si);
  if (tid == 0) {
    int next = bi;
    if (P.answer_len > 0) {                            // answer mode: the prompt is fed again before every answer
      const bool forcing = astep + 1 < P.nforced;
      if (forcing) next = P.forced[astep + 1];
      if (st.out_tokens) st.out_tokens[step % st.out_cap] = forcing ? (astep == 0 ? OUT_RESTART : OUT_FORCED) : bi;
      pos += 1; astep += 1;
      if (astep >= P.nforced - 1 + P.answer_len) { next = P.forced[0]; pos = 0; astep = 0; }
      st.scal[DS_ASTEP] = astep;
    } else {
      if (step + 1 < P.nforced) next = P.forced[step + 1];
      if (st.out_tokens) st.out_tokens[step % st.out_cap] = bi;
      pos += 1;
    }
    st.scal[DS_CTXFULL] = (pos >= md.T);
    if (pos >= md.T && P.auto_reset) pos = 0;
    if (pos == 0) { epoch = (epoch + 1) & 0x7FFF; st.scal[DS_EPOCH] = epoch; }      // a new context starts
    st.scal[DS_POSKEY] = (epoch << 16) | pos;
    st.scal[DS_TOKEN] = next; st.scal[DS_POS] = pos; st.scal[DS_STEP] = step + 1;
    if (live) live->dec_steps = (unsigned)(step + 1);
    sn[0] = next; sn[1] = pos;
  }
  __syncthreads();
  write_embed<T, D>(P, sn[0], sn[1]);
}

}  // namespace dec
}  // namespace ofa
