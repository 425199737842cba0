// bf16 tensor-core GEMM task for sm_100a: TMA -> swizzled shared memory -> tcgen05.mma -> TMEM -> epilogue.
//
// Task contract (replaces the reference's `tg::tile<LAYOUT,EPI>` = gemm::sm100::tile_tc,
// llm/b200/gemm_tcgen05/gemm_sm100.cuh:174-289, with the layouts/epilogues of llm/gemm/gemm.cuh:18-50):
//   one task = a STRIP of `nsub` consecutive 128 x BN tiles of C that share their 128 rows; all 256 threads call
//   gemm_tc_task() together. BN is 128 by default; 256 is an opt-in per GEMM. Differences in design from the reference tile:
//     * two tile widths. With every SM busy a 64-deep K step of a 128x128 tile takes 0.66 us per block (~14 TB/s of operand
//       reads GPU-wide); a 128x256 tile moves 48 KB instead of 64 KB per 128x256x64 of work but fits only two stages per
//       block, and measured slower on all model shapes except lm_head dW: the loop is bound by bytes in flight;
//     * the mbarriers and the 256 TMEM columns of a block live for the whole kernel; phase parities are derived from running
//       counters kept in `GemmPipe` (one set of barriers and counters per tile width, because the widths use different
//       pipeline depths), so nothing is re-initialised or invalidated between tiles or tasks;
//     * inside a strip the TMA producer (warp 0) and the MMA issuer (warp 1) run ahead of the epilogue; with BN = 128 the
//       accumulator is double-buffered in TMEM (2 x 128 columns) and drained by warps 4..7 while the next tile's MMAs are in
//       flight; with BN = 256 one accumulator fills the block's TMEM and the SM's other resident block provides the overlap;
//     * the epilogue never touches the pipeline buffers: each epilogue warp transposes 32x32 fp32 blocks through its own
//       4 KB staging area (XOR-swizzled, conflict-free) and then moves whole 64/128-byte row segments to global memory;
//       epilogues that read `aux` fetch their row segments before waiting for the accumulator;
//     * every wait is bounded and aborts the grid cleanly on expiry.
//   K order is fixed (k ascending, one accumulator) => results are deterministic and independent of the schedule and of BN.
//
// Operand staging (SWIZZLE_128B everywhere; one pipeline stage = 64 values of K: 16 KB of A + BN x 128 B of B):
//   K-major operand  X[rows][K]  (A of NN/NT, B of NT): TMA boxes {64 k, 128 rows} -> 128 rows x 128 B each; UMMA descriptor
//     SBO = 1024 B (8 rows), a step of 16 in K advances the start address by 32 B.
//   MN-major operand X[K][cols]  (B of NN/TN, A of TN): TMA boxes {64 cols, 64 k}, 8 KB apart -> per box 64 k-rows x
//     128 B; UMMA descriptor LBO = 8192 B (between 64-wide column groups), SBO = 1024 B (8 k-rows), a step of 16 in K
//     advances the start address by 2048 B.
#pragma once
#include "common.cuh"
#include "task_api.h"

namespace ofa {
namespace gemm_tc {

constexpr int BM = 128, BK = 64;
constexpr int A_BYTES = BM * BK * 2;                 // 16 KB
constexpr int PIPE_BYTES = 96 * 1024;                // 3 stages x 32 KB (BN 128) or 2 stages x 48 KB (BN 256)
constexpr int EPI_WARPS = 4;                         // warps 4..7
constexpr int STAGING_BYTES = EPI_WARPS * 32 * 32 * 4;   // 16 KB
constexpr int BAR_OFFSET = PIPE_BYTES + STAGING_BYTES;   // control area: barriers, TMEM slot, scheduler words
constexpr int BAR_BYTES = CTRL_BYTES;
constexpr int SMEM_BYTES = BAR_OFFSET + BAR_BYTES;   // 115,712 B: two blocks per SM use the whole 228 KB (1 KB per block is reserved by the system)
constexpr int TMEM_COLS = 256;

template <int BN> struct Cfg {
  static constexpr int W = BN == 128 ? 0 : 1;                    // which barrier set / counter set
  static constexpr int STAGES = BN == 128 ? 3 : 2;
  static constexpr int B_BYTES = BN * BK * 2;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int NBUF = BN == 128 ? 2 : 1;                  // accumulators in TMEM
  static constexpr int BAR0 = BN == 128 ? 0 : 176;                // byte offset of this width's barriers in the control area
  static_assert(STAGES * STAGE_BYTES <= PIPE_BYTES, "pipeline does not fit");
};
// control area (1 KB at smem + BAR_OFFSET = the last 1,024 bytes of dynamic shared memory):
//   [  0, 80) BN128: full[3] empty[3] accf[2] acce[2]     [ 80, 84) TMEM base slot     [ 96,104) serving fill barrier   [104,112) training bulk-copy barrier
//   [112,128) and [160,176) streamed cross-entropy stage barriers [4]
//   [176,224) BN256: full[2] empty[2] accf[1] acce[1]      [224,248) AdamW stage barriers [3]      [248,256), [1008,1024) time tables (CTRL_T_*)
//   [256,448) and [448,640) two slots for phase descriptors: the one being worked on and the next phase's, fetched ahead
//   [640,832) the block's scheduling state and pipeline counters (BlockState)      [832,1008) attention barriers
template <int BN> __device__ __forceinline__ uint32_t bar_full(uint32_t base, int s) { return base + BAR_OFFSET + Cfg<BN>::BAR0 + 8u * s; }
template <int BN> __device__ __forceinline__ uint32_t bar_empty(uint32_t base, int s) { return base + BAR_OFFSET + Cfg<BN>::BAR0 + 8u * (Cfg<BN>::STAGES + s); }
template <int BN> __device__ __forceinline__ uint32_t bar_accf(uint32_t base, int b) { return base + BAR_OFFSET + Cfg<BN>::BAR0 + 8u * (2 * Cfg<BN>::STAGES + b); }
template <int BN> __device__ __forceinline__ uint32_t bar_acce(uint32_t base, int b) { return base + BAR_OFFSET + Cfg<BN>::BAR0 + 8u * (2 * Cfg<BN>::STAGES + Cfg<BN>::NBUF + b); }
constexpr int TMEM_SLOT_OFFSET = BAR_OFFSET + 80;

// Running counters, one set per tile width; in shared memory, read at the start of a task and advanced by thread 0 behind its closing barrier.
struct GemmPipe {
  uint32_t stage_count[2];   // pipeline stages produced/consumed since block start
  uint32_t tile_count[2];    // accumulator tiles since block start
  uint32_t tmem_base;
};

template <int BN> __device__ __forceinline__ void init_bars(uint32_t base) {
  for (int s = 0; s < Cfg<BN>::STAGES; s++) { mbar_init(bar_full<BN>(base, s), 1); mbar_init(bar_empty<BN>(base, s), 1); }
  for (int b = 0; b < Cfg<BN>::NBUF; b++) { mbar_init(bar_accf<BN>(base, b), 1); mbar_init(bar_acce<BN>(base, b), EPI_WARPS); }
}
// Once per block, before its first GEMM task. All 256 threads. Returns false (and aborts) if shared memory is misaligned.
__device__ __forceinline__ bool block_init(GemmPipe& gp, unsigned char* smem, DevStatus* st) {
  const uint32_t base = smem_u32(smem);
  const bool ok = (base & 1023u) == 0;
  if (!ok) { if (threadIdx.x == 0) raise_abort(st, ST_SMEM_MISALIGNED, -1, -1, (int)base); }
  if (threadIdx.x == 0) { init_bars<128>(base); init_bars<256>(base); mbar_fence_init(); }
  if (threadIdx.x < 32) tmem_alloc(base + TMEM_SLOT_OFFSET, TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (threadIdx.x == 0) { gp.stage_count[0] = gp.stage_count[1] = 0; gp.tile_count[0] = gp.tile_count[1] = 0; gp.tmem_base = *reinterpret_cast<volatile uint32_t*>(smem + TMEM_SLOT_OFFSET); }
  __syncthreads();
  return ok;
}
// Once per block before it exits. All 256 threads. TMA copies still in flight when a task gives up are waited for
// (bounded) by the producer inside that task; here an aborting block only adds a short fixed delay before freeing TMEM.
__device__ __forceinline__ void block_exit(GemmPipe& gp, unsigned char* smem, DevStatus* st) {
  (void)smem;
  if (aborted(st)) __nanosleep(20000);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (threadIdx.x < 32) tmem_dealloc(gp.tmem_base, TMEM_COLS);
}

// Asks for the B operand of a task whose B is a weight matrix (PhaseDesc::i1) to be brought to L2, while the block waits for the tasks
// that produce A. With few tokens every weight tile comes from HBM and the three-stage pipeline sees its latency on every third
// k-step. One of the tasks that share a strip of B does it; at most 64 boxes (1 MB of K-major, 0.5 MB of MN-major tiles).
__device__ __forceinline__ void l2_prefetch_box(const void* tmap, int c0, int c1) {
  asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global.tile [%0, {%1, %2}];" ::"l"(tmap), "r"(c0), "r"(c1) : "memory");
}
__device__ __forceinline__ void prefetch_weights(const PhaseDesc& d, int task) {
  const GemmArgs& g = d.g;
  if (task % d.tiles_m != 0) return;
  const int n0 = (task / d.tiles_m) * g.nsub * g.bn, n1 = min(g.N, n0 + g.nsub * g.bn);
  const bool kmajor = d.layout == GL_NT;
  int left = 64;
  for (int n = n0; n < n1 && left > 0; n += kmajor ? 128 : 64)
    for (int k = 0; k < g.K && left > 0; k += BK, left--) { if (kmajor) l2_prefetch_box(g.tmB, k, n); else l2_prefetch_box(g.tmB, n, k); }
}

// ---------------------------------------------------------------------------------------------- epilogue math
// The epilogues that meet their second operand in fp32 before the one rounding (and the fp32 result): eight consecutive
// columns of one row, after the fp32 transpose. Everything else is stored from the bf16-staged pass of the task itself.
template <int EPI>
__device__ __forceinline__ void epi_store8(const GemmArgs& g, size_t row, int col, const float* acc, uint4 auxv) {
  static_assert(EPI == GE_F32 || EPI == GE_RES || EPI == GE_DGELU, "bf16 results without a second fp32 operand take the staged pass");
  if constexpr (EPI == GE_F32) {
    float* dst = reinterpret_cast<float*>(g.C) + row * g.ldc + col;
    float4 v0 = make_float4(acc[0], acc[1], acc[2], acc[3]), v1 = make_float4(acc[4], acc[5], acc[6], acc[7]);
    if (g.accumulate) {
      const float4 o0 = *reinterpret_cast<const float4*>(dst), o1 = *reinterpret_cast<const float4*>(dst + 4);
      v0.x += o0.x; v0.y += o0.y; v0.z += o0.z; v0.w += o0.w; v1.x += o1.x; v1.y += o1.y; v1.z += o1.z; v1.w += o1.w;
    }
    *reinterpret_cast<float4*>(dst) = v0; *reinterpret_cast<float4*>(dst + 4) = v1;
  } else {
    float v[8], a8[8];
    unpack8(auxv, a8);
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = EPI == GE_RES ? acc[i] + a8[i] : acc[i] * gelu_bwd<true>(a8[i]);
    *reinterpret_cast<uint4*>(reinterpret_cast<bf16*>(g.C) + row * g.ldc + col) = pack8(v);
  }
}

// ---------------------------------------------------------------------------------------------- the task
// task index -> (tile_m, first tile_n): consecutive tasks walk down M first so that neighbouring blocks share the B strip.
template <int LAYOUT, int EPI, int BN>
__device__ __forceinline__ void gemm_tc_task(const GemmArgs& g, int tiles_m, int task, unsigned char* smem, GemmPipe& gp,
                                             DevStatus* st, int phase_id, EarlyTicket& et, int nfast) {
  using CF = Cfg<BN>;
  constexpr bool A_MN = (LAYOUT == GL_TN), B_MN = (LAYOUT != GL_NT);
  constexpr bool HAS_AUX_IN = (EPI == GE_RES || EPI == GE_DGELU || EPI == GE_DR);
  constexpr bool BF16_STAGED = (EPI == GE_STORE || EPI == GE_GELU || EPI == GE_LSE || EPI == GE_DR);   // epilogues whose stored value is the rounded accumulator
  constexpr uint32_t IDESC = umma_idesc(A_MN, B_MN, BM, BN);
  constexpr int STAGES = CF::STAGES, W = CF::W;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t base = smem_u32(smem);
  const uint32_t stage0 = gp.stage_count[W], tile0 = gp.tile_count[W], tmem = gp.tmem_base;
  const int KT = g.K / BK;
  const int tiles_n = g.N / BN;
  // nfast: consecutive tasks walk along N first, so the tasks that stream the same rows of a large A run side by side and the
  // second and third reader find them in L2 (the LM head's weight gradient); otherwise down M first, sharing the B strip
  const int nstrips = (tiles_n + g.nsub - 1) / g.nsub;
  const int tm = nfast ? task / nstrips : task % tiles_m, strip = nfast ? task % nstrips : task / tiles_m;
  const int tn0 = strip * g.nsub;
  const int nt = min(g.nsub, tiles_n - tn0);
  const int m0 = tm * BM;

  if (warp == 0) {
    if (lane == 0) {                                                           // ---- TMA producer
      fence_proxy_async();     // operands were written with ordinary stores by earlier phases (possibly other SMs)
      uint32_t sc = stage0;
      bool ok = true;
      for (int t = 0; t < nt && ok; t++) {
        const int n0 = (tn0 + t) * BN;
        for (int kt = 0; kt < KT; kt++, sc++) {
          const int s = sc % STAGES; const uint32_t use = sc / STAGES;
          const uint32_t full = bar_full<BN>(base, s);
          if (!mbar_wait(bar_empty<BN>(base, s), (use & 1) ^ 1, st)) { if (!aborted(st)) raise_abort(st, ST_MBAR_EMPTY_TIMEOUT, phase_id, task, kt); ok = false; break; }
          mbar_expect_tx(full, CF::STAGE_BYTES);
          const uint32_t sA = base + s * CF::STAGE_BYTES, sB = sA + A_BYTES;
          const int k0 = kt * BK;
          if (!A_MN) tma_load_2d(sA, g.tmA, full, k0, m0);
          else { tma_load_2d(sA, g.tmA, full, m0, k0); tma_load_2d(sA + 8192, g.tmA, full, m0 + 64, k0); }
          if (!B_MN) {
#pragma unroll
            for (int h = 0; h < BN / 128; h++) tma_load_2d(sB + h * 16384, g.tmB, full, k0, n0 + h * 128);
          } else {
#pragma unroll
            for (int h = 0; h < BN / 64; h++) tma_load_2d(sB + h * 8192, g.tmB, full, n0 + h * 64, k0);
          }
        }
      }
      if (ok) take_early_ticket(et);     // every copy of the task is on its way: this thread has nothing left to do but the closing barrier
      if (aborted(st)) {       // giving up: wait (bounded) until the copies this task issued into our shared memory have landed
        const uint32_t issued = sc - stage0;
        for (uint32_t i = 0; i < issued && i < (uint32_t)STAGES; i++) {
          const uint32_t c = sc - 1 - i; const int s = c % STAGES; const uint32_t use = c / STAGES;
          for (int spin = 0; spin < 100000; spin++) if (mbar_try(bar_full<BN>(base, s), use & 1)) break;
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {                                                           // ---- MMA issuer
      uint32_t sc = stage0, tc = tile0;
      bool ok = true;
      for (int t = 0; t < nt && ok; t++, tc++) {
        const int b = tc % CF::NBUF; const uint32_t use = tc / CF::NBUF;
        if (!mbar_wait(bar_acce<BN>(base, b), (use & 1) ^ 1, st)) { if (!aborted(st)) raise_abort(st, ST_MBAR_ACC_TIMEOUT, phase_id, task, 100 + t); ok = false; break; }
        tc_fence_after();
        const uint32_t d_tmem = tmem + (uint32_t)(b * BN);
        for (int kt = 0; kt < KT; kt++, sc++) {
          const int s = sc % STAGES; const uint32_t suse = sc / STAGES;
          if (!mbar_wait(bar_full<BN>(base, s), suse & 1, st)) { if (!aborted(st)) raise_abort(st, ST_MBAR_FULL_TIMEOUT, phase_id, task, kt); ok = false; break; }
          tc_fence_after();
          const uint32_t sA = base + s * CF::STAGE_BYTES, sB = sA + A_BYTES;
#pragma unroll
          for (int kk = 0; kk < BK / 16; kk++) {
            const u64 da = A_MN ? umma_smem_desc(sA + kk * 2048, 8192, 1024) : umma_smem_desc(sA + kk * 32, 16, 1024);
            const u64 db = B_MN ? umma_smem_desc(sB + kk * 2048, 8192, 1024) : umma_smem_desc(sB + kk * 32, 16, 1024);
            umma_bf16(d_tmem, da, db, IDESC, (kt > 0 || kk > 0) ? 1u : 0u);
          }
          umma_commit(bar_empty<BN>(base, s));       // stage s reusable once these MMAs retire
        }
        if (ok) umma_commit(bar_accf<BN>(base, b));  // accumulator b complete
      }
    }
  } else if (warp >= 4) {                                                      // ---- epilogue warps
    const int e = warp - 4;                      // TMEM lane quadrant == warp % 4
    float* stg = reinterpret_cast<float*>(smem + PIPE_BYTES + e * 4096);
    uint32_t tc = tile0;
    bool ok = true;
    const int cg = lane & 3;
    // An epilogue's code runs once per tile and has left the instruction caches by the block's next task of the kind (a step runs through
    // hundreds of KB of task code), so straight-line code pays a fetch from L2 for every line of it: the passes over the columns are loops.
    // One-tile tasks of K = 768, 128 columns unrolled -> loops: GELU' 25 -> 14 us, softmax partials 19 -> 11, row term 15 -> 11.5. `aux` is
    // fetched a pass at a time; fetching it one pass ahead as well spilled, and with next to no L1 a spill goes to L2 (residual 9 -> 14 us).
    for (int t = 0; t < nt && ok; t++, tc++) {
      const int b = tc % CF::NBUF; const uint32_t use = tc / CF::NBUF;
      const int n0 = (tn0 + t) * BN;
#pragma unroll 1
      for (int half = 0; half < BN / 128; half++) {          // 128 columns at a time
        const uint32_t tacc = tmem + ((uint32_t)(e * 32) << 16) + (uint32_t)(b * BN + half * 128);
        const int nh = n0 + half * 128;
        // Epilogues that read `aux` (residual, pre-activation) fetch this thread's row segments of the first pass BEFORE waiting for the
        // accumulator, so the loads travel while the MMAs run.
        constexpr int NAUX = EPI == GE_DR ? 8 : 4;             // row segments of 8 columns per pass (64 columns for the staged pass, 32 otherwise)
        uint4 auxr[HAS_AUX_IN ? NAUX : 1];
        const bf16* auxp = nullptr;
        if constexpr (EPI == GE_DR) auxp = reinterpret_cast<const bf16*>(g.aux) + (size_t)(m0 + e * 32 + (lane >> 3)) * g.ldaux + nh + (lane & 7) * 8;   // row = it*4 + lane/8
        else if constexpr (HAS_AUX_IN) auxp = reinterpret_cast<const bf16*>(g.aux) + (size_t)(m0 + e * 32 + (lane >> 2)) * g.ldaux + nh + cg * 8;       // row = it*8 + lane/4
        auto fetch_aux = [&](uint4 (&dst)[HAS_AUX_IN ? NAUX : 1], int col) {
          if constexpr (HAS_AUX_IN) {
#pragma unroll
            for (int it = 0; it < NAUX; it++) dst[it] = *reinterpret_cast<const uint4*>(auxp + (size_t)(it * (32 / NAUX)) * g.ldaux + col);
          }
        };
        fetch_aux(auxr, 0);
        if (half == 0) {
          if (!mbar_wait(bar_accf<BN>(base, b), use & 1, st)) { if (lane == 0 && !aborted(st)) raise_abort(st, ST_MBAR_ACC_TIMEOUT, phase_id, task, t); ok = false; }
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          tc_fence_after();
        }
        if constexpr (BF16_STAGED) {
          // The stored value is the bf16 rounding of the accumulator itself, so the accumulator is rounded BEFORE the transpose:
          // the thread that owns row `lane` packs 64 columns into eight 16-byte chunks of a 32 x 128 B tile (chunk j at
          // position j ^ (lane & 7)), and the warp reads it back as 4 rows x 128 B per instruction - whole lines for the
          // stores, half the shared-memory traffic of an fp32 transpose (the pipeline's own traffic nearly saturates it).
          unsigned char* sb = reinterpret_cast<unsigned char*>(stg);
          const int sub = lane >> 3, ch = lane & 7;
          float lm = -INFINITY, ls = 0.f;                  // GE_LSE: maximum (log2 domain) and sum of 2^(x - max) of this thread's row so far
#pragma unroll 1
          for (int cp = 0; cp < 2; cp++) {                 // 64 columns at a time
            if (EPI == GE_DR && cp == 1) fetch_aux(auxr, 64);
#pragma unroll(EPI == GE_LSE ? 1 : 2)
            for (int hc = 0; hc < 2; hc++) {
              uint32_t r[32], pk[16];
              tmem_ld32(tacc + (uint32_t)(cp * 64 + hc * 32), r);
              if (half == BN / 128 - 1 && cp == 1 && hc == 1) {    // all TMEM reads of this accumulator are done: hand it back early
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_acce<BN>(base, b));
              }
#pragma unroll
              for (int q = 0; q < 16; q++) pk[q] = pack2f(__uint_as_float(r[2 * q]), __uint_as_float(r[2 * q + 1]));
#pragma unroll
              for (int q = 0; q < 4; q++)
                *reinterpret_cast<uint4*>(sb + lane * 128 + (((hc * 4 + q) ^ (lane & 7)) << 4)) = make_uint4(pk[4 * q], pk[4 * q + 1], pk[4 * q + 2], pk[4 * q + 3]);
              if constexpr (EPI == GE_LSE) {               // over the STORED values, which are what cross-entropy will read
                float gm[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY}, s4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int q = 0; q < 16; q++) gm[q & 3] = fmaxf(gm[q & 3], fmaxf(__uint_as_float(pk[q] << 16), __uint_as_float(pk[q] & 0xffff0000u)));
                const float cm = fmaxf(fmaxf(gm[0], gm[1]), fmaxf(gm[2], gm[3])) * 1.4426950408889634f;
                if (cm > lm) { ls *= ex2_approx(lm - cm); lm = cm; }
#pragma unroll
                for (int q = 0; q < 16; q++)
                  s4[q & 3] += ex2_approx(fmaf(__uint_as_float(pk[q] << 16), 1.4426950408889634f, -lm)) + ex2_approx(fmaf(__uint_as_float(pk[q] & 0xffff0000u), 1.4426950408889634f, -lm));
                ls += (s4[0] + s4[1]) + (s4[2] + s4[3]);
              }
            }
            __syncwarp();
            const size_t row0 = (size_t)(m0 + e * 32 + sub);
            const int col = nh + cp * 64 + ch * 8;
            if constexpr (EPI == GE_GELU) {
#pragma unroll 2
              for (int it = 0; it < 8; it++) {
                const int rr = it * 4 + sub;
                const uint4 out = *reinterpret_cast<const uint4*>(sb + rr * 128 + ((ch ^ (rr & 7)) << 4));
                *reinterpret_cast<uint4*>(reinterpret_cast<bf16*>(g.aux) + (row0 + it * 4) * g.ldaux + col) = out;   // bf16-rounded pre-activation is what backward sees
                float pv[8]; unpack8(out, pv);
#pragma unroll
                for (int i = 0; i < 8; i++) pv[i] = gelu_fwd<true>(pv[i]);
                *reinterpret_cast<uint4*>(reinterpret_cast<bf16*>(g.C) + (row0 + it * 4) * g.ldc + col) = pack8(pv);
              }
            } else {
              // all eight reads first: a global store between two shared-memory reads keeps the compiler from moving the second
              // read up (it cannot rule out aliasing), and the pass would pay eight shared-memory latencies in a row
              uint4 ov[8];
#pragma unroll
              for (int it = 0; it < 8; it++) { const int rr = it * 4 + sub; ov[it] = *reinterpret_cast<const uint4*>(sb + rr * 128 + ((ch ^ (rr & 7)) << 4)); }
#pragma unroll
              for (int it = 0; it < 8; it++) *reinterpret_cast<uint4*>(reinterpret_cast<bf16*>(g.C) + (row0 + it * 4) * g.ldc + col) = ov[it];
              if constexpr (EPI == GE_DR) {                // one pass = the 64 columns of one head; a row's share sits in 8 lanes
                // the 128 rows of a tile belong to one sequence (the context length is a multiple of 128): one division per tile
                const int bseq = m0 / g.dr_T, t0 = m0 - bseq * g.dr_T + e * 32 + sub;
                float* drow = g.dr + ((size_t)bseq * g.dr_H + nh / 64 + cp) * g.dr_T + t0;
#pragma unroll
                for (int it = 0; it < 8; it++) {
                  float c8[8], o8[8]; unpack8(ov[it], c8); unpack8(auxr[it], o8);
                  float v = 0.f;
#pragma unroll
                  for (int i = 0; i < 8; i++) v = fmaf(c8[i], o8[i], v);
                  v += __shfl_xor_sync(0xffffffffu, v, 1); v += __shfl_xor_sync(0xffffffffu, v, 2); v += __shfl_xor_sync(0xffffffffu, v, 4);
                  if (ch == 0) drow[it * 4] = v;
                }
              }
            }
            __syncwarp();
          }
          if constexpr (EPI == GE_LSE) reinterpret_cast<float2*>(g.dr)[(size_t)(m0 + e * 32 + lane) * (g.N / 128) + nh / 128] = make_float2(lm, ls);
        } else {
#pragma unroll 1
          for (int c = 0; c < 4; c++) {
            if (c > 0) fetch_aux(auxr, c * 32);
            uint32_t r[32];
            tmem_ld32(tacc + (uint32_t)(c * 32), r);
            if (half == BN / 128 - 1 && c == 3) {    // all TMEM reads of this accumulator are done: hand it back early
              tc_fence_before();
              __syncwarp();
              if (lane == 0) mbar_arrive(bar_acce<BN>(base, b));
            }
            // thread = row `lane` of the 32x32 block; 16-byte chunk j goes to position j ^ (lane & 7)
#pragma unroll
            for (int j = 0; j < 8; j++)
              *reinterpret_cast<float4*>(stg + lane * 32 + ((j ^ (lane & 7)) << 2)) =
                  make_float4(__uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1]), __uint_as_float(r[4 * j + 2]), __uint_as_float(r[4 * j + 3]));
            __syncwarp();
            // 8 rows per instruction: lane -> (row = it*8 + lane/4, 8 consecutive columns (lane%4)*8..)
            float4 av[8];                            // all reads before the first global store (see the bf16-staged pass)
#pragma unroll
            for (int it = 0; it < 4; it++) {
              const int rr = it * 8 + (lane >> 2);
              av[2 * it] = *reinterpret_cast<const float4*>(stg + rr * 32 + (((2 * cg) ^ (rr & 7)) << 2));
              av[2 * it + 1] = *reinterpret_cast<const float4*>(stg + rr * 32 + (((2 * cg + 1) ^ (rr & 7)) << 2));
            }
#pragma unroll
            for (int it = 0; it < 4; it++) {
              const float4 a0 = av[2 * it], a1 = av[2 * it + 1];
              const float acc[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
              epi_store8<EPI>(g, (size_t)(m0 + e * 32 + it * 8 + (lane >> 2)), nh + c * 32 + cg * 8, acc, auxr[HAS_AUX_IN ? it : 0]);
            }
            __syncwarp();
          }
        }
      }
    }
  }
  __syncthreads();
  if (tid == 0) { gp.stage_count[W] = stage0 + (uint32_t)(nt * KT); gp.tile_count[W] = tile0 + (uint32_t)nt; }
}

template <int LAYOUT, int EPI>
__device__ __forceinline__ void dispatch_bn(const PhaseDesc& d, int task, unsigned char* smem, GemmPipe& gp, DevStatus* st, int phase_id, EarlyTicket& et) {
  if (d.g.bn == 256) gemm_tc_task<LAYOUT, EPI, 256>(d.g, d.tiles_m, task, smem, gp, st, phase_id, et, d.i0);
  else gemm_tc_task<LAYOUT, EPI, 128>(d.g, d.tiles_m, task, smem, gp, st, phase_id, et, d.i0);
}
// run-time dispatch over the (layout, epilogue) pairs the training graph uses
__device__ __forceinline__ void run(const PhaseDesc& d, int task, unsigned char* smem, GemmPipe& gp, DevStatus* st, int phase_id, EarlyTicket& et) {
  switch (d.layout * 8 + d.epi) {
    case GL_NN * 8 + GE_STORE: dispatch_bn<GL_NN, GE_STORE>(d, task, smem, gp, st, phase_id, et); break;
    case GL_NN * 8 + GE_RES:   dispatch_bn<GL_NN, GE_RES>(d, task, smem, gp, st, phase_id, et); break;
    case GL_NN * 8 + GE_GELU:  dispatch_bn<GL_NN, GE_GELU>(d, task, smem, gp, st, phase_id, et); break;
    case GL_NN * 8 + GE_F32:   dispatch_bn<GL_NN, GE_F32>(d, task, smem, gp, st, phase_id, et); break;      // split-K partial products
    case GL_NT * 8 + GE_STORE: dispatch_bn<GL_NT, GE_STORE>(d, task, smem, gp, st, phase_id, et); break;
    case GL_NT * 8 + GE_DGELU: dispatch_bn<GL_NT, GE_DGELU>(d, task, smem, gp, st, phase_id, et); break;
    case GL_NT * 8 + GE_DR:    gemm_tc_task<GL_NT, GE_DR, 128>(d.g, d.tiles_m, task, smem, gp, st, phase_id, et, d.i0); break;
    case GL_NT * 8 + GE_LSE:   gemm_tc_task<GL_NT, GE_LSE, 128>(d.g, d.tiles_m, task, smem, gp, st, phase_id, et, d.i0); break;
    case GL_TN * 8 + GE_F32:   dispatch_bn<GL_TN, GE_F32>(d, task, smem, gp, st, phase_id, et); break;
    case GL_TN * 8 + GE_STORE: dispatch_bn<GL_TN, GE_STORE>(d, task, smem, gp, st, phase_id, et); break;
    default: if (threadIdx.x == 0) raise_abort(st, ST_BAD_DESC, phase_id, task, d.layout * 8 + d.epi); __syncthreads(); break;
  }
}

}  // namespace gemm_tc
}  // namespace ofa
