// The persistent kernel: one launch, blocks that never exit until their job is finished, on-GPU ticket queues with
// dependency counters, and a static split of the SMs between the training job, the serving (decode) job and a reserved
// idle partition.
//
// Scheduling model (same contract as the reference's job_loop / ofa_kernel, llm/b200/megakernel/ofa.cu:220-326):
//   thread 0 of a block takes the next ticket g of its job with one fetch-add; g -> (step, phase, task) through the prefix
//   table; warp 0 then waits until every dependency (phase p, step delta d) satisfies done[p] >= ntasks[p]*(step+1+d); the
//   whole block runs the task; thread 32 then bumps done[phase], training and the last phase of a serving step after a
//   device-scope fence, other serving phases with a releasing increment. Phases are topologically ordered and
//   cross-step dependencies point backwards, so every dependency is a lower ticket and the lowest unfinished ticket is
//   always runnable: no deadlock as long as every claimed ticket is eventually run, which holds because a block holds at
//   most one ticket.
// What differs from the reference: the phase lookup walks on from the block's last phase; every wait is bounded (%globaltimer deadline and a
// grid-wide abort word) so that a wedged task makes the kernel RETURN with a status instead of hanging the GPU; the
// per-block tensor-core state (mbarriers, TMEM) is created once per block, not per task; external (host / other-rank)
// events enter the graph as ordinary 1-task phases (TK_EXT_WAIT / TK_EXT_SIGNAL).
#pragma once
#include "common.cuh"
#include "task_api.h"
#include "tickets.h"
#include "elementwise.cuh"
#include "gemm_tc.cuh"
#include "attn_common.cuh"
#include "attn_tc.cuh"
#include "simt_f32.cuh"
#include "decode.cuh"
#include <type_traits>

namespace ofa {

template <class T> struct IsBf16 { static constexpr bool value = std::is_same<T, bf16>::value; };

// What a block keeps between tasks. It sits in the control area, not in registers: next to task functions that use all 128 of them it was
// spilled (408 bytes of it), and behind the device-scope fence that ends a task, which empties L1, every reload went to L2 - five of them in a
// row for each task. An empty task 2.51 -> 1.27 us, a phase of one empty task per block 4.69 -> 2.12.
struct BlockState {
  int4 sel[2];                       // hand-off from thread 0 to the block: {what to do, step, phase, task}; two in turn, so that the thread that signals may still read the last one
  int4 stop[2];                      // copies of the second 16 bytes of DevStatus (y = abort word) and, serving, of the finished word, asked for with each task's end
  int4 cur;                          // thread 0: current phase, its tickets [y, z) within a step; all threads: w = outcome of the dependency wait
  int2 pos;                          // thread 0: current step and its first ticket
  int2 ready;                        // thread 0: (step, phase) last seen ready, unless the phase has row-block dependencies, which are per task: {-1, -1}
  int rbw[2];                        // thread 32: counter of the row block that the task writes, -1: none
  EarlyTicket early;
  attn_tc::AttnPipe ap; gemm_tc::GemmPipe gp;
  uint32_t bulk_uses, adam_tiles, ce_chunks;       // uses of the bulk-copy barrier (control area byte 104), tiles staged by AdamW (CTRL_ADAM_BAR), chunks staged by the streamed cross-entropy (112, 120, 160, 168)
};
constexpr int CTRL_DESC = 256, CTRL_STATE = CTRL_DESC + 2 * (int)sizeof(PhaseDesc);
constexpr int CTRL_ADAM_BAR = 224, CTRL_T_END = 248, CTRL_T_BUSY = 1008, CTRL_T_START = 1016;      // the time tables' words
static_assert(offsetof(DevStatus, abort) == 20 && sizeof(DevStatus) <= 32, "copied as its second 16 bytes");
static_assert(sizeof(PhaseDesc) == 192 && sizeof(SchedRec) == 48, "control area map");
static_assert(CTRL_STATE + sizeof(BlockState) <= attn_tc::BAR0, "scheduling state does not fit the control area");
static_assert(attn_tc::BAR0 + 8 * attn_tc::NBAR <= CTRL_T_BUSY && CTRL_T_START + 8 <= CTRL_BYTES, "attention barriers reach into the time tables' words");
static_assert(CTRL_ADAM_BAR + 8 * ew::ADAM_STAGES <= CTRL_T_END && CTRL_T_END + 8 <= CTRL_DESC, "AdamW barriers reach into the time tables' words");

// ---------------------------------------------------------------------------------------------- one training task
// The tasks are inlined here: as functions they saved the registers they use in local memory, which next to no L1 sends to L2, and took their
// arguments from there (small model of 384 tokens 1,525 -> 1,471 us for two steps, one layer of 4,096 540 -> 520, attention forward 25.2 -> 24.6,
// GELU' product 35.2 -> 33.3). LayerNorm forward is the exception, 6.4 us as a function and 7.2 inlined, where it spills.
template <class T, int D, int DH>
__device__ __forceinline__ void run_train_task(const Ctx& C, const PhaseDesc& d, int ph, int local, int step, unsigned char* smem, BlockState& B) {
  const ModelDims& md = C.md;
  gemm_tc::GemmPipe& gp = B.gp; attn_tc::AttnPipe& ap = B.ap; EarlyTicket& et = B.early;
  switch (d.kind) {
    case TK_DATA:
      ew::data_task(local, step + C.step_base, C.data, C.ntok, C.starts, C.nstarts, C.seed, C.tok_in, C.tok_tgt, md.T, md.B);
      break;
    case TK_EMBED:
      ew::embed_fwd_task<T, D>(local, (T*)d.p[0], (const T*)d.p[1], (const T*)d.p[2], (const int*)d.p[3], md.N, md.T);
      break;
    case TK_LN_FWD:
      ew::ln_fwd_task<T, D>(local, (T*)d.p[0], (float*)d.p[1], (float*)d.p[2], (const T*)d.p[3], (const T*)d.p[4], md.N);
      break;
    case TK_GEMM:
      if constexpr (IsBf16<T>::value) gemm_tc::run(d, local, smem, gp, C.status, ph, et);
      else f32::gemm_run(d, local, smem);
      break;
    case TK_ATT_FWD: {
      if constexpr (IsBf16<T>::value) {
        const int BH = md.B * md.H, QT = md.T / attn::QTILE;
        const int qt = QT - 1 - local / BH, bh = local % BH;      // heavy (late) query tiles first
        attn_tc::fwd_task((const attn_tc::Maps*)d.p[6], (bf16*)d.p[1], (float*)d.p[2], bh / md.H, bh % md.H, qt, md.T, md.H, smem, ap, gp.tmem_base, C.status, ph, local, et);
      } else {
        f32::attn_fwd_task<DH>((const float*)d.p[0], (float*)d.p[1], (float*)d.p[2], local / md.H, local % md.H, md.T, md.H, smem);
      }
      break;
    }
    case TK_ATT_PREP: {
      if constexpr (IsBf16<T>::value) {
        const int BH = md.B * md.H;
        const int rt = local / BH, bh = local % BH;
        attn::bwd_prep_task((const bf16*)d.p[0], (const bf16*)d.p[1], (float*)d.p[2], bh / md.H, bh % md.H, rt, md.T, md.H);
      }
      break;
    }
    case TK_ATT_BWD: {
      if constexpr (IsBf16<T>::value) {
        const int BH = md.B * md.H, QT = md.T / attn::QTILE;
        if (local < BH * QT) {                                     // dK/dV: early key tiles see the most queries -> first
          const int kt = local / BH, bh = local % BH;
          attn_tc::bwd_dkdv_task((const attn_tc::Maps*)d.p[6], (const float*)d.p[2], (const float*)d.p[3], (bf16*)d.p[4], bh / md.H, bh % md.H, kt, md.T, md.H, smem, ap, gp.tmem_base, C.status, ph, local, et);
        } else {                                                   // dQ: late query tiles see the most keys -> first
          const int l2 = local - BH * QT, qt = QT - 1 - l2 / BH, bh = l2 % BH;
          attn_tc::bwd_dq_task((const attn_tc::Maps*)d.p[6], (const float*)d.p[2], (const float*)d.p[3], (bf16*)d.p[4], bh / md.H, bh % md.H, qt, md.T, md.H, smem, ap, gp.tmem_base, C.status, ph, local, et);
        }
      } else {
        f32::attn_bwd_task<DH>((const float*)d.p[0], (const float*)d.p[5], (const float*)d.p[1], (const float*)d.p[2], (float*)d.p[4],
                               local / md.H, local % md.H, md.T, md.H, smem);
      }
      break;
    }
    case TK_CE:
      if constexpr (IsBf16<T>::value) {
        if (d.p[3] && md.V % 8 == 0) {                 // the LM-head GEMM left softmax partials: one streamed pass over the logits
          ew::ce_task_stream(local, (bf16*)d.p[0], (const int*)d.p[1], (float*)d.p[2], (const float2*)d.p[3], d.i2, md.N, md.V, 1.0f / (float)md.N, smem,
                             smem_u32(smem + C.smem_bytes - CTRL_BYTES + 112), smem_u32(smem + C.smem_bytes - CTRL_BYTES + 160), B.ce_chunks, C.status);
          break;
        }
        if ((size_t)md.V * 2 <= (size_t)d.i0 && md.V % 8 == 0) {
          ew::ce_task_bulk(local, (bf16*)d.p[0], (const int*)d.p[1], (float*)d.p[2], md.N, md.V, 1.0f / (float)md.N, smem,
                           smem_u32(smem + C.smem_bytes - CTRL_BYTES + 104), B.bulk_uses, C.status);
          break;
        }
      }
      if constexpr (!IsBf16<T>::value) {
        if (md.V <= ew::CE_WARP_MAX_V) { ew::ce_task_warp(local, (float*)d.p[0], (const int*)d.p[1], (float*)d.p[2], md.N, md.V, 1.0f / (float)md.N); break; }
      }
      ew::ce_task<T>(local, (T*)d.p[0], (const int*)d.p[1], (float*)d.p[2], md.N, md.V, 1.0f / (float)md.N, smem, d.i0);
      break;
    case TK_CE_MEAN: {
      const float lv = ew::ce_mean_task((float*)d.p[0], (const float*)d.p[1], md.N, smem);
      if (threadIdx.x == 0) { C.loss_hist[step] = lv; if (C.live) C.live->loss = lv; }
      break;
    }
    case TK_LN_BWD:
      ew::ln_bwd_task<T, D>(local, (T*)d.p[0], (float*)d.p[1], (const T*)d.p[2], (const T*)d.p[3], (const float*)d.p[4],
                            (const float*)d.p[5], (const T*)d.p[6], (const T*)d.p[7], md.N, smem);
      break;
    case TK_LN_DG:
      if (d.i1) ew::ln_dgamma_reduce_task<bf16>(local, (bf16*)d.p[0], (const float*)d.p[1], (md.N + ew::ROWS_PER_TASK - 1) / ew::ROWS_PER_TASK, D, d.i0, smem);
      else ew::ln_dgamma_reduce_task<float>(local, (float*)d.p[0], (const float*)d.p[1], (md.N + ew::ROWS_PER_TASK - 1) / ew::ROWS_PER_TASK, D, d.i0, smem);
      break;
    case TK_EMB_WTE:
      if (d.i1) ew::embed_bwd_wte_task<T, D, bf16>(local, (bf16*)d.p[0], (const T*)d.p[1], (const int*)d.p[2], md.N, md.V, d.tiles_m, d.i0, smem);
      else ew::embed_bwd_wte_task<T, D, float>(local, (float*)d.p[0], (const T*)d.p[1], (const int*)d.p[2], md.N, md.V, d.tiles_m, d.i0, smem);
      break;
    case TK_EMB_WPE:
      if (d.i1) ew::embed_bwd_wpe_task<T, bf16>(local, (bf16*)d.p[0], (const T*)d.p[1], md.N, md.T, D);
      else ew::embed_bwd_wpe_task<T, float>(local, (float*)d.p[0], (const T*)d.p[1], md.N, md.T, D);
      break;
    case TK_ADAMW: {
      const ew::AdamHP hp = ew::adam_hp(C.hp, step + C.step_base);
      if constexpr (IsBf16<T>::value) {               // inputs staged by the copy engine (the fp32 preset's blocks have no room for the stages)
        const uint32_t bar0 = smem_u32(smem + C.smem_bytes - CTRL_BYTES + CTRL_ADAM_BAR);
        if (d.i2 == 0) {
          if (d.i1) ew::adamw_task_bulk<T, bf16>(local, (float*)d.p[0], (const bf16*)d.p[1], (float*)d.p[2], (float*)d.p[3], (T*)d.p[4], d.n, hp, (const int2*)d.p[5], d.i0, d.tiles_m, smem, bar0, B.adam_tiles, C.status);
          else ew::adamw_task_bulk<T, float>(local, (float*)d.p[0], (const float*)d.p[1], (float*)d.p[2], (float*)d.p[3], (T*)d.p[4], d.n, hp, (const int2*)d.p[5], d.i0, d.tiles_m, smem, bar0, B.adam_tiles, C.status);
          break;
        }
      }
      if (d.i1) ew::adamw_task<T, bf16>(local, (float*)d.p[0], (const bf16*)d.p[1], (float*)d.p[2], (float*)d.p[3], (T*)d.p[4], d.n, hp, (const int2*)d.p[5], d.i0, d.tiles_m);
      else ew::adamw_task<T, float>(local, (float*)d.p[0], (const float*)d.p[1], (float*)d.p[2], (float*)d.p[3], (T*)d.p[4], d.n, hp, (const int2*)d.p[5], d.i0, d.tiles_m);
      break;
    }
    case TK_SUMCAST:
      ew::sumcast_task<T>(local, (T*)d.p[0], &d.p[1], d.i0, d.n);
      break;
    case TK_EXT_SIGNAL:
      // flag values count steps since the context was created, so a stale value from an earlier launch is always too small
      if (threadIdx.x == 0) { __threadfence_system(); *reinterpret_cast<volatile int*>(d.p[0]) = C.step_base + step + 1; __threadfence_system(); }
      break;
    case TK_EXT_WAIT:
      if (threadIdx.x == 0) {
        const volatile int* flag = reinterpret_cast<const volatile int*>(d.p[0]);
        const u64 t0 = gtimer();
        while (*flag < C.step_base + step + 1) {
          if (aborted(C.status)) break;
          if (gtimer() - t0 > C.dep_timeout_ns) { raise_abort(C.status, ST_EXTERNAL_TIMEOUT, ph, local, step); break; }
          __nanosleep(200);
        }
        __threadfence_system();
      }
      break;
    default: break;   // TK_BARRIER
  }
}

template <class T, int D, int DH, bool PROF>
__device__ __forceinline__ void run_decode_task(const Ctx& C, const PhaseDesc& d, int local, int step, unsigned char* smem, uint32_t bar, uint32_t parity) {
  switch (d.kind) {
    case TK_DEC_QKV: dec::task_qkv<T, D, DH, PROF>(C.dp, C.md, d.i0, local, step, smem, bar, parity, C.status); break;
    case TK_DEC_ATTWO: dec::task_attwo<T, D, DH, PROF>(C.dp, C.md, d.i0, local, step, smem, bar, parity, C.status); break;
    case TK_DEC_UPDN: dec::task_updn<T, D, DH, PROF>(C.dp, C.md, d.i0, local, smem, bar, parity, C.status); break;
    case TK_DEC_HEAD: dec::task_head<T, D, DH>(C.dp, C.md, local, step, smem, bar, parity, C.status); break;
    case TK_DEC_SAMPLE: dec::task_sample<T, D, DH>(C.dp, C.md, C.live, smem); break;
    default: break;
  }
}

// ---------------------------------------------------------------------------------------------- scheduler
// row block a task writes (x) and the row blocks it reads from its row-block-grain producers (first, number). Out of line: once per task, divisions
static __device__ __noinline__ int3 rb_of_task(int rb_map, int BH, int H, int QT, int local) {
  const int kind = rb_map & 0xFF, a = rb_map >> 8;
  int prod = 0;
  if (kind == RB_MOD) prod = local % a;
  else if (kind == RB_DIV) prod = local / a;
  else if (kind != RB_NONE) {
    const bool dq = kind == RB_ATT_BWD && local >= BH * QT;
    if (dq) local -= BH * QT;
    const int t = local / BH, b = (local - t * BH) / H;
    if (kind == RB_ATT_FWD) { const int qt = QT - 1 - t; return make_int3(b * QT + qt, b * QT, qt + 1); }
    if (!dq) return make_int3(b * QT + t, b * QT + t, QT - t);
    prod = b * QT + QT - 1 - t;
  }
  return make_int3(prod, prod, 1);
}
// after every 64 polls: true when the block must leave (abort, or the deadline has passed)
static __device__ __noinline__ bool wait_over(DevStatus* st, u64 t0, u64 limit, int ph, int local, int step) {
  if (aborted(st)) return true;
  if (gtimer() - t0 <= limit) return false;
  raise_abort(st, ST_DEP_TIMEOUT, ph, local, step);
  return true;
}
// Dependency wait (bounded) of warp 0, whose lanes share the counters: up to four dependencies of the phase's record, the row blocks of one
// that has them over eight lanes each; more than four (AdamW, the end of a step) over all lanes. cnt, w, nt = the record's number of
// dependencies and, for lane l, its dependency l % 4; h = {.., step, phase, task}, rb = {first, number} of the row blocks that the task
// reads. Returns 0 when every dependency is satisfied, -2 when the block must leave (job finished elsewhere, abort, or deadline).
// Acquire loads: relaxed ones and a fence behind the last cost 310 clocks more per wait.
template <int JOB>
__device__ __forceinline__ int wait_deps(const Ctx& C, const Job& J, const int cnt, const int w, const int nt, const int4 h, const int2 rb) {
  const int lane = threadIdx.x & 31, k = lane & 3;
  const bool grain = (w & DEP_RB) != 0;
  const int* ctr = J.done + (w & DEP_WORD) + (grain ? (rb.x + (lane >> 2)) * RB_STRIDE : 0);
  const int left = k >= cnt ? 0 : grain ? rb.y - (lane >> 2) : lane < 4 ? 1 : 0;
  const int need = nt * (h.y + 1 - ((w & DEP_PREV) ? 1 : 0));
  const int off = cnt < 0 ? __ldg(J.dep_off + h.z) : 0, n = cnt < 0 ? __ldg(J.dep_cnt + h.z) : 0;
  const u64 t0 = gtimer();
  for (unsigned spins = 1;; spins++) {
    bool ready = true;
    const int* p = ctr;
#pragma unroll 1
    for (int q = left; q > 0; q -= 8, p += 8 * RB_STRIDE) ready = ld_acquire(p) >= need && ready;
#pragma unroll 1
    for (int i = lane; i < n; i += 32) {
      const Dep e = J.deps[off + i];
      ready = ld_acquire(J.done + e.phase * DONE_STRIDE) >= __ldg(J.ntasks + e.phase) * (h.y + 1 + e.delta) && ready;
    }
    if (__all_sync(0xffffffffu, ready)) return 0;
    if (JOB == 1 && C.use_train && (spins & 7u) == 0 && __any_sync(0xffffffffu, ld_relaxed(C.finished) != 0)) return -2;
    // a dependency may legitimately sit behind an external wait that is about to give up: the bound here is half as long again, so
    // that the status names the external flag that was never raised and not one of the tasks queued behind it
    if ((spins & 63u) == 0) {
      const bool over = lane == 0 && wait_over(C.status, t0, C.dep_timeout_ns + (C.dep_timeout_ns >> 1), h.z, h.w, h.y);
      if (__any_sync(0xffffffffu, over)) return -2;
    }
    // No pause for 512 polls, 80 to 180 us, which is longer than nearly every wait: best of four with limits of 32 / 128 / 512 / 2,048, char step 359.5 / 356.3 /
    // 354.7 / 355.1 us, two steps of 384 tokens (3 layers) 1,489 / 1,488 / 1,485 / 1,486, a layer as a list of phases 525.5 / 524.7 / 524.6 / 524.5. Nothing is
    // slower for it: a step of 4 x 1,024 tokens 6,087 / 6,127 / 6,119, beside a serving job 7,285 / 7,282 / 7,285 (2,352 / 2,352 / 2,358 tokens/s), a served
    // token 182.4 with 32 and 512, and a copy by other SMs while all blocks wait for an external flag takes 0.186 ms each time.
    // A counter seen complete is read again with the others: a step takes the same either way, a served token is 3 % slower if each lane remembers.
    if (spins > 512u) __nanosleep(JOB == 1 ? 20 : 80);
  }
}
static __device__ __noinline__ void end_of_step(unsigned long long* done, Live* live, int step, unsigned long long* t_end, int* finished) {
  const u64 t1 = gtimer();
  *done = t1;
  if (live) live->steps = (unsigned)(step + 1);
  if (t_end) { *t_end = t1; __threadfence(); atomicExch(finished, 1); }
}
// test hook (Job::perm, 0 in production): tickets of a phase are handed out in a permuted task order, which
// must not change any result - the reference's shuffled-order check (llm/gemm/test_gemm.cu:20-49)
static __device__ __noinline__ int permuted(int local, int mul, int n) { return mul == 0 ? local : (int)(((long long)local * mul + (mul >> 1)) % (long long)n); }

__device__ __forceinline__ void sched_cp16(uint32_t dst, const void* src) { asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory"); }
__device__ __forceinline__ void sched_cp_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// threadIdx.x read anew: what is derived from it is not worth a register over a whole task
__device__ __forceinline__ int thread_index() { int t; asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t)); return t; }

template <class T, int D, int DH, int JOB, bool PROF>
__device__ __forceinline__ void job_loop(const Ctx& C, const Job& J, unsigned char* smem) {
  constexpr bool TRAIN = JOB == 0, RB = TRAIN && IsBf16<T>::value;        // RB: phases may count completions per row block
  unsigned char* ctrl = smem + (IsBf16<T>::value ? gemm_tc::SMEM_BYTES : C.smem_bytes) - CTRL_BYTES;   // the last bytes of dynamic shared memory are the block's control area (map in gemm_tc.cuh)
  BlockState& B = *reinterpret_cast<BlockState*>(ctrl + CTRL_STATE);
  u64 &t_busy = *reinterpret_cast<u64*>(ctrl + CTRL_T_BUSY), &t_start = *reinterpret_cast<u64*>(ctrl + CTRL_T_START), &t_end = *reinterpret_cast<u64*>(ctrl + CTRL_T_END);   // profiling only: thread 0, serving the end of a task by thread 64
  const int* pre = TRAIN ? C.train_pre : C.dec_pre;   // first tickets of the phases inside the kernel parameter, when they fit
  const bool ptab = (TRAIN ? C.train_pre_n : C.dec_pre_n) > 0;
  int tid = thread_index();
  constexpr bool use_tc = IsBf16<T>::value && TRAIN;
  const uint32_t fill_bar = smem_u32(ctrl + 96);     // serving blocks: counts the bytes of the weight prefetch of the task they hold a ticket for
  if (tid == 0) {
    B.cur = make_int4(-1, 0, 0, 0); B.pos = make_int2(0, 0); B.ready = make_int2(-1, -1);
    B.early.counter = (use_tc && (C.sched_flags & 4) == 0) ? J.ticket : nullptr;       // (flag 4: tickets only at the end of a task, for A/B measurements)
    B.early.taken = 0;
    B.stop[0] = B.stop[1] = make_int4(0, 0, 0, 0); t_busy = 0; t_end = 0; B.bulk_uses = 0; B.adam_tiles = 0; B.ce_chunks = 0;
  }
  if constexpr (use_tc) {
    if (tid == 0) {
      mbar_init(smem_u32(ctrl + 104), 1);
      for (int q = 0; q < ew::ADAM_STAGES; q++) mbar_init(smem_u32(ctrl + CTRL_ADAM_BAR + 8 * q), 1);
      for (int q = 0; q < 2; q++) { mbar_init(smem_u32(ctrl + 112 + 8 * q), 1); mbar_init(smem_u32(ctrl + 160 + 8 * q), 1); }   // streamed cross-entropy: four stages
    }
    attn_tc::block_init(B.ap, smem); gemm_tc::block_init(B.gp, smem, C.status);
  }
  if constexpr (!TRAIN) {
    if (tid == 0) { mbar_init(fill_bar, 1); mbar_fence_init(); }
    dec::block_init<T, D, DH>(smem, C.md.T);
    __syncthreads();
  }
  uint32_t fills = 0;                                // serving: fills of the weight buffer so far
  int slot = 0;                                      // which of the two descriptor slots holds the phase being worked on
  int cached_ph = -1, ahead_ph = -1;                 // phases held by that slot and by the other one (fetched ahead)
  const unsigned total = (unsigned)J.nsteps * (unsigned)J.tasks_per_step;
  auto add_time = [&](int what, u64 dt) { if (C.blk_wait) C.blk_wait[(size_t)what * gridDim.x + blockIdx.x] += dt; };     // 0 dependency wait, 1 claim, 2 hand-off, 3 signalling
  unsigned next_g = 0; bool have_next = false;       // thread 0, from the end of a task to the next claim: the ticket taken
  for (int turn = 0;; turn ^= 1) {
    if (tid == 0) {                                  // ---- claim
      u64 tl0 = 0;
      if (TRAIN && PROF) { tl0 = gtimer(); if (t_end) add_time(3, tl0 - t_end); }
      int4 cur = B.cur; int2 pos = B.pos; const int2 rdy = B.ready;      // on their way beside the ticket
      int4 h = make_int4(-2, 0, 0, 0);
      const unsigned g = have_next ? next_g : atomicAdd(J.ticket, 1u);
      if (g < total) {
        int step = pos.x; unsigned first = (unsigned)pos.y;
        const int r = (int)place_ticket(g, (unsigned)J.tasks_per_step, step, first);
        if (step != pos.x) {                             // a new step
          pos = make_int2(step, (int)first);
          cur.x = -1; cur.z = 0;
          B.pos = pos;
        }
        // A block's tickets grow, so within a step it only moves forward through the phases: keep the current phase's tickets and walk on.
        if (r >= cur.z) {
          int ph = cur.x, hi = cur.z, lo;
#pragma unroll 1
          do { lo = hi; ph++; hi = ptab ? pre[ph + 1] : __ldg(J.prefix + ph + 1); } while (r >= hi);
          cur.x = ph; cur.y = lo; cur.z = hi;
          B.cur = cur;
        }
        int local = r - cur.y;
        if (C.sched_flags & 1) local = permuted(local, J.perm[cur.x], cur.z - cur.y);
        // a phase whose dependencies are all phase-level stays ready once it has been seen ready; row-block dependencies are per task
        h = make_int4((pos.x == rdy.x && cur.x == rdy.y) ? 0 : 1, pos.x, cur.x, local);      // 1: the dependencies have to be waited for
      }
      B.sel[turn] = h;
      if (TRAIN && PROF) { const u64 t = gtimer(); t_start = t; add_time(1, t - tl0); }
    } else if (tid < 16) {
      sched_cp_wait();                               // the descriptor requested at the end of the last task: visible to all after the barrier below
    }
    __syncthreads();
    const int4 h = B.sel[turn];
    const int res = h.x;
    // the abort and finished words are looked at inside every wait loop; here in a copy that was asked for at the end of the last task
    if (res < 0 || B.stop[0].y != 0 || (!TRAIN && C.use_train && B.stop[1].x != 0)) break;
    // The descriptor is read from shared memory: every dependency check ends with a device-scope acquire, after which L1 no
    // longer holds it, and the chain of dependent global loads that decoding it would take was a measurable part of the
    // per-task overhead. Two slots: the next phase's descriptor is requested at the end of a task (below), so a block that
    // moves on by one phase - the common case when phases have about as many tasks as there are blocks - finds it here.
    bool settle = TRAIN && res == 1, fetched = false;   // a second barrier is due before the task starts
    {
      const int ph = h.z;
      if (ph != cached_ph) {
        if (ph == ahead_ph) { slot ^= 1; ahead_ph = cached_ph; cached_ph = ph; }      // already there: no second barrier (-0.9 % per step)
        else {
          const int q = tid - 64;
          if (q >= 0 && q < (int)(sizeof(PhaseDesc) / 4)) reinterpret_cast<uint32_t*>(ctrl + CTRL_DESC + sizeof(PhaseDesc) * slot)[q] = __ldg(reinterpret_cast<const uint32_t*>(J.ph + ph) + q);
          cached_ph = ph;
          settle = fetched = true;
        }
      }
    }
    const PhaseDesc& d = *reinterpret_cast<const PhaseDesc*>(ctrl + CTRL_DESC + sizeof(PhaseDesc) * slot);
    const SchedRec& rec = fetched ? J.ph[h.z].rec : d.rec;      // a descriptor that was not fetched ahead is on its way: what the waiting warp needs of it comes beside it
    auto wait_ready = [&]() {                        // warp 0: the dependencies of the task at hand
      const int k = 2 * (tid & 3), cnt = rec.ndeps, w = rec.dep[k], nt = rec.dep[k + 1];
      bool any_rb = false;
      int3 q = make_int3(0, 0, 0);
      if (RB) { any_rb = rec.any_rb != 0; if (any_rb) q = rb_of_task(rec.rb_map, C.md.B * C.md.H, C.md.H, C.md.T >> 7, h.w); }
      const int r2 = wait_deps<JOB>(C, J, cnt, w, nt, h, make_int2(q.y, q.z));
      if (tid == 0) { B.ready = r2 == 0 && !any_rb ? make_int2(h.y, h.z) : make_int2(-1, -1); B.cur.w = r2; }
    };
    // where the task's completion is counted besides its phase's counter: worked out now, so that signalling does not wait for it
    if (RB && tid == 32) {
      const int o = rec.rb_off;
      B.rbw[turn] = o < 0 ? -1 : (o + rb_of_task(rec.rb_map, C.md.B * C.md.H, C.md.H, C.md.T >> 7, h.w).x) * RB_STRIDE;
    }
    // Warp 0 waits for the dependencies while other threads fetch the descriptor: behind the wait, a descriptor that was not
    // fetched ahead cost its round trip on the critical path of every phase change.
    if (settle) {
      if (TRAIN && tid < 32 && res == 1) {
        const u64 w0 = PROF ? gtimer() : 0;
        wait_ready();
        if (PROF && tid == 0) {
          const u64 w = gtimer() - w0;
          add_time(0, w);
          if (C.phase_busy && w > 200) atomicAdd(C.phase_busy + J.nph + h.z, w);
          t_start = gtimer();
        }
      }
      // meanwhile the weights of the task, which no task of this step writes, start on their way to L2
      if constexpr (use_tc) if (tid == 32 && res == 1) {
        const PhaseDesc& dd = fetched ? J.ph[h.z] : d;
        if (dd.kind == TK_GEMM && dd.i1) gemm_tc::prefetch_weights(dd, h.w);
      }
      __syncthreads();
      if (TRAIN && res == 1 && B.cur.w < 0) break;
    }
    bool filled = false;
    if constexpr (!TRAIN) {                          // ---- serving: start the weight prefetch, THEN wait for the dependencies
      filled = dec::prefetch<T, D, DH>(C.dp, C.md, d.kind, d.i0, h.w, h.y, smem, fill_bar);
      if (tid < 32 && res == 1) wait_ready();
      __syncthreads();
      if (res == 1 && B.cur.w < 0) {                             // leaving with copies in flight: give them a bounded chance to land
        if (filled) mbar_wait(fill_bar, fills & 1u, C.status);
        __syncthreads();
        break;
      }
    }
    if (PROF && tid == 0) {
      const u64 t0 = gtimer();
      if (TRAIN) add_time(2, t0 - t_start);
      t_start = t0;
      if (!TRAIN && C.dp.trace && h.w == 0 && (h.z == 0 || h.z == 2)) C.dp.trace[16 + h.z] = t0;
    }
    // tensor-core tasks let their copy producer (this block's thread 0) take the next ticket as soon as its last copy is issued
    if constexpr (TRAIN) run_train_task<T, D, DH>(C, d, h.z, h.w, h.y, smem, B);
    else { run_decode_task<T, D, DH, PROF>(C, d, h.w, h.y, smem, fill_bar, fills & 1u); if (filled) fills++; }
    __syncthreads();
    tid = thread_index();
    {                                                // ask for the next phase's descriptor now
      const int nxt = cached_ph + 1 < J.nph ? cached_ph + 1 : 0;
      if (nxt != ahead_ph) {
        if (tid >= 1 && tid <= (int)(sizeof(PhaseDesc) / 16))
          sched_cp16(smem_u32(ctrl + CTRL_DESC + sizeof(PhaseDesc) * (slot ^ 1)) + 16 * (tid - 1), reinterpret_cast<const char*>(J.ph + nxt) + 16 * (tid - 1));
        ahead_ph = nxt;
      }
      if (tid == 14) sched_cp16(smem_u32(&B.stop[0]), reinterpret_cast<const char*>(C.status) + 16);
      if (!TRAIN && tid == 15) sched_cp16(smem_u32(&B.stop[1]), C.finished);
    }
    auto task_over = [&](u64 t1) {                   // the time tables' part of it
      const u64 t0 = t_start;
      const int4 e = B.sel[turn]; const int ph = e.z;
      t_busy += t1 - t0;
      if constexpr (TRAIN) {
        t_end = t1;
        if (C.phase_busy) {
          atomicAdd(C.phase_busy + ph, t1 - t0);
          if (e.y == C.prof_step) { atomicMin(C.phase_first + ph, t0); atomicMax(C.phase_last + ph, t1); }
        }
      } else {
        if (C.dp.trace && e.w == 0 && (ph == 0 || ph == 2)) C.dp.trace[17 + ph] = t1;
        if (C.dec_phase_busy) atomicAdd(C.dec_phase_busy + ph, t1 - t0);
      }
    };
    // Two threads share the end of a task. Thread 0 takes the next ticket at once (a fetch-add whose value it needs only at the
    // top of the loop: the task is finished, so holding the next ticket cannot delay anything this block still has to do, every
    // dependency being a lower ticket). Thread 32 publishes the completion: ONE device-scope fence - the block barrier above
    // ordered every thread's writes of this task before it - and relaxed increments of the completion counters. The fence waits
    // for the SM's outstanding stores (about a microsecond after a GEMM epilogue); on its own thread it runs beside the ticket's
    // round trip and the next claim instead of in front of them.
    if (tid == 0) {
      const u64 t1 = TRAIN && PROF ? gtimer() : 0;     // before the ticket: behind it the task would seem to last until it is there
      unsigned early = 0;
      if constexpr (use_tc) { early = B.early.taken; B.early.taken = 0; }
      if (early != 0) next_g = early - 1u; else next_g = atomicAdd(J.ticket, 1u);
      have_next = true;
      if (TRAIN && PROF) task_over(t1);
    } else if (!TRAIN && PROF && tid == 64) {          // thread 0 asks for the ticket meanwhile: in front of it the timer cost 0.13 us a phase (24 SMs, 361.3 -> 355.2 us a token)
      task_over(gtimer());
    } else if (tid == 32) {
      const int4 e = B.sel[turn]; const int ph = e.z, step = e.y;      // read again: nothing stays in registers over a task
      const int rbw = RB ? B.rbw[turn] : -1;
      // one counter (serving): a releasing increment, 0.7 % per decoded token faster than fence and increment; with two, two of them are slower than one fence
      const bool last = ph == J.last_phase;
      if (TRAIN || last) fence_acq_rel();
      if (rbw >= 0) red_relaxed_add(J.done_rb + rbw, 1);      // completions per row block first: their waiters are the ones on the critical chain
      if (!last) { if (TRAIN) red_relaxed_add(J.done + ph * DONE_STRIDE, 1); else red_release_add(J.done + ph * DONE_STRIDE, 1); }
      else {                                           // the step's last phase needs the old value
        const int old = atomicAdd(J.done + ph * DONE_STRIDE, 1);
        if (TRAIN && old == __ldg(J.ntasks + ph) * (step + 1) - 1) {     // last task of the step
          end_of_step(C.step_done + step, C.live, step, step == J.nsteps - 1 ? C.t_end : nullptr, C.finished);
        }
      }
    }
  }
  sched_cp_wait();
  if constexpr (use_tc) gemm_tc::block_exit(B.gp, smem, C.status);
  if (PROF && tid == 0 && C.blk_busy) C.blk_busy[blockIdx.x * 2 + JOB] = t_busy;
}

// A block of an idle partition must not leave before the whole grid has been placed: the hardware refills the slot of an
// exited block first, so early exits would steal the second block of the working SMs (measured: the 24-SM serving partition
// ran with one block per SM). Idle blocks therefore wait (bounded) until every block of the grid has reported in.
__device__ __forceinline__ void idle_block(const Ctx& C) {
  if (threadIdx.x == 0 && C.arrived) {
    const u64 t0 = gtimer();
    while (ld_relaxed(C.arrived) < (int)gridDim.x && gtimer() - t0 < 20000000ull) __nanosleep(500);
  }
}

// For the first launch that uses TMA descriptors the host has just written. Out of line: later launches, which have nothing to fence, run past
// a call (a served token takes the same with the loop inlined, 180.9 / 180.6 us, on 24 SMs 336.0 / 336.3).
__device__ __noinline__ void fence_maps(const unsigned char* maps, int n) { for (int q = threadIdx.x; q < n; q += NTHR) tmap_fence(maps + 128 * (size_t)q); }

// One kernel for launches that train, one for those that serve (bf16), one for both, each with and without time tables, because what a launch does not
// run lies between what it does: a served token takes 182.4 us from the form that only serves and 182.9 from the one that does both, a step of 384
// tokens 3,332 and 3,345, a char step 364 and 366. The char model alone serves faster from the form that does both (launch_kernel). Code that is not met
// again before the instruction caches have lost it is slow to run, 6 clocks a warp instruction in a loop of 48 KB or more, 2 in one of 16 KB, but it is not
// what a block waits for most: of the warps that are not held at a block barrier, 9 % wait for an instruction in small training steps and 4 % while
// serving, 33 and 37 % for a load (profiles/scheduler_parts_and_stalls.md). So only what a sound run never executes is out of line, and loops are as timed.
template <class T, int D, int DH, bool TRAIN, bool SERVE, bool PROF>
__global__ void __launch_bounds__(NTHR, 2) ofa_kernel(const __grid_constant__ Ctx C) {
  extern __shared__ __align__(1024) unsigned char dsm[];
  const unsigned hw = smid();
  const int rank = C.smid_rank ? C.smid_rank[hw] : (int)hw;
  const int isms = SERVE && C.use_decode ? C.infer_sms : 0;
  if (C.nmaps > 0) fence_maps(C.maps, C.nmaps);      // barriers come before the first use of any
  if (threadIdx.x == 0 && C.arrived) atomicAdd(C.arrived, 1);
  const int role = rank < isms ? 1 : rank < isms + C.reserved_sms ? 2 : (TRAIN && C.use_train && rank < isms + C.reserved_sms + C.train_sms) ? 3 : 4;
  if (threadIdx.x == 0 && C.blk_info) C.blk_info[blockIdx.x] = (int)hw | (role << 16);
  if constexpr (IsBf16<T>::value && TRAIN) {
    // Blocks that never allocate TMEM give up their allocation permit at once. Measured on B200: while a resident block of a
    // kernel that contains tcgen05.alloc still holds the permit, the hardware does not place a second block of that kernel on
    // the SM; the serving partition ran with one block per SM (24 instead of 48 blocks) until this line was added.
    if (role != 3 && threadIdx.x < 32) asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if constexpr (SERVE) if (role == 1) { job_loop<T, D, DH, 1, PROF>(C, C.dec, dsm); return; }
  if constexpr (TRAIN) if (role == 3) { job_loop<T, D, DH, 0, PROF>(C, C.train, dsm); return; }
  idle_block(C);
}

// one resident block per slot records its %smid so the host can build a dense rank table
__global__ void __launch_bounds__(NTHR, 2) smid_probe_kernel(unsigned* seen) {
  extern __shared__ __align__(1024) unsigned char dsm[];
  if (threadIdx.x == 0) {
    const unsigned id = smid();
    atomicOr(&seen[id >> 5], 1u << (id & 31));
    const u64 t0 = gtimer();
    while (gtimer() - t0 < 2000000ull) {}      // 2 ms: keeps the block resident so that every SM receives its share
    dsm[0] = 0;
  }
}

// first embedding of a decode context: xw := fx(wte[token] + wpe[pos])
template <class T, int D>
__global__ void decode_init_embed_kernel(DecodeParams P) { dec::write_embed<T, D>(P, P.st.scal[DS_TOKEN], P.st.scal[DS_POS]); }

}  // namespace ofa
