// One persistent kernel: causal varlen GQA FlashAttention -> O_proj GEMM -> AllReduce.
//
// Work identity is a 128-row tile.  A CTA repeatedly asks the in-kernel scheduler for a
// task (protocol of the reference's FusedFaOprojAr kernel,
// src/mega_attention/kernels/sm90/fused_fa_oproj_ar.py:148-398):
//   FA task    (row_tile, q head[s])  : S = Q K^T and O += P V as tcgen05 MMAs with fp32
//                                       accumulators in TMEM, online softmax by one thread
//                                       per row, result to O_scratch (bf16) by TMA store
//   O_proj task                       : one rank: up to two row tiles x 256 columns, C =
//                                       O_scratch tiles @ W_o columns, a TMEM accumulator
//                                       per row tile, W stages shared.  Several ranks:
//                                       (row_tile, n super-group), C[128, <=512] in two
//                                       passes of 256 columns into the two accumulators
//   AR task    (owned slot)           : multimem.ld_reduce / multimem.st over the NVLS
//                                       multicast view of the symmetric output (or plain
//                                       peer loads / stores with two ranks)
//
// Warp roles (12 warps, 384 threads):
//   warp 0 (lane 0)  TMA producer: Q tiles, the K/V ring, O_proj stages
//   warp 1           MMA issuer of both attention tiles and of every O_proj task; allocates
//                    and frees TMEM
//   warp 2 (lane 0)  scheduler: claims tasks, fills one of two descriptor slots, publishes
//                    completions (runs one task ahead of the workers)
//   warp 3 (lane 0)  stores the attention output tiles
//   warps 4-7, 8-11  two compute warpgroups: online softmax (one thread per row), both
//                    epilogues, AllReduce slots
// An FA task is two q heads of one row tile whenever the rank has two: the two compute
// warpgroups alternate, so the tensor pipe runs one tile's MMAs under the other tile's
// softmax.  With an even number of q heads per kv head the two heads share a kv head and
// every K/V stage of the ring; otherwise (MHA included) each head gets K/V stages of its
// own in the same ring (K of both heads, then V of both heads, per key block), and the
// head an odd count leaves over runs alone.
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "kparams.h"
#include "launch.cuh"
#include "ptx.cuh"

namespace ma {

namespace {

constexpr uint32_t kTile = 32768;          // 128 x 128 bf16
constexpr uint32_t kPanel = 16384;         // 128 rows x 64 bf16 (one 128-byte-swizzle panel)
constexpr uint32_t kSmQ = 0;               // two Q tiles
constexpr uint32_t kSmKV = 2 * kTile;      // ring of five K/V tiles
constexpr int kKvSlots = 5;
constexpr uint32_t kSmOpStaging = 4 * (16384 + 32768);   // O_proj output staging, 2 x 16 KB
// O_proj stages, by what the launch's tasks are.  (Three of the large ones for every task of one
// rank: K_local 4096, hidden 8192, 1024 and 2048 tokens took 170 and 177 us for 144 and 154.)
constexpr uint32_t kOpStage = 16384 + 32768;   // one row tile: A 128x64 + W 64x256 (4 stages)
constexpr uint32_t kOpStage2 = 2 * 16384 + 32768;   // two row tiles: A 256x64 + W 64x256 (3 stages)
constexpr uint32_t kWPanel = 8192;         // 64 k-rows x 64 n bf16
constexpr uint32_t kTmemS = 0;             // S0 at 0, S1 at 128 (P aliases the first 64 cols)
constexpr uint32_t kTmemO = 256;           // O0 at 256, O1 at 384
constexpr uint32_t kIdescQK = make_idesc_bf16(128, 128, 0, 0);
constexpr uint32_t kIdescPV = make_idesc_bf16(128, 128, 0, 1);
constexpr float kRescaleThreshold = 8.0f;  // in log2 units

struct Bars {
  uint64_t task_full[2];    // scheduler -> roles: descriptor k is valid        (count 1)
  uint64_t task_empty[2];   // roles -> scheduler: task in slot k is finished   (count 11)
  uint64_t loads_done[2];   // producer: every load of the task in slot k is issued (count 1)
  uint64_t q_full[2];       // TMA: Q tile i landed
  uint64_t q_empty[2];      // MMA: last Q K^T of tile i done + epilogue: staging released (count 2)
  uint64_t kv_full[kKvSlots];
  uint64_t kv_empty[kKvSlots];   // MMA: the last product that reads the slot completed (count 1)
  uint64_t s_full[2];       // MMA: S_i ready
  uint64_t p_part[2];       // softmax warps: key columns 0-95 of P_i written (count 4)
  uint64_t p_full[2];       // softmax warps: P_i written (count 4, one arrival per warp)
  uint64_t o_staged[2];     // epilogue warps: O_i staged in shared memory (count 4)
  uint64_t o_done[2];       // MMA: last P V of the task for tile i completed
  uint64_t o_free[2];       // epilogue warps: O_i read out (count 4)
  uint64_t op_full[4];
  uint64_t op_empty[4];
  uint64_t acc_full[2];     // MMA: O_proj accumulator half h complete
  uint64_t acc_free[2];     // epilogue warps: half h read out (count 8)
  uint64_t drain;           // abort path only: the issuer's outstanding MMAs have retired
};

struct Env {
  const KParams* p;
  volatile int* abort_flag;
};

__device__ __noinline__ void report(const Env& e, uint32_t code, uint32_t site, uint32_t aux) {
  if (atomicCAS(e.p->status, 0u, code) == 0u) {
    e.p->status[1] = site;
    e.p->status[2] = blockIdx.x;
    e.p->status[3] = aux;
  }
  __threadfence();
  *e.abort_flag = 1;
}

// Bounded mbarrier wait.  Returns false once the wait limit passed or the CTA aborted.  The
// first look is a test_wait: on a phase that is complete it takes 45 cycles, a try_wait 120,
// and these waits stand on the pipelines' chains.  What follows is short on purpose (a loop
// of 32 quick tries before it cost the attention stage 3 %), and inline: as a call it made
// every value that is live across a wait go through memory.
constexpr uint32_t kWaitSleepNs = 20000;
__device__ __forceinline__ bool wait_bar(const Env& e, uint32_t bar, uint32_t parity,
                                         uint32_t site) {
  if (mbar_test_wait(bar, parity)) return true;
  if (mbar_try_wait_for(bar, parity, kWaitSleepNs)) return true;
  const uint64_t t0 = globaltimer_ns();
#pragma unroll 1
  while (!mbar_try_wait_for(bar, parity, kWaitSleepNs)) {
    if (*e.abort_flag) return false;
    if (globaltimer_ns() - t0 > e.p->wait_limit_ns) {
      report(e, ST_TIMEOUT_MBAR, site, parity);
      return false;
    }
  }
  return true;
}

// A compute warp's look at the next task.  An abort does not end it, the scheduler's end does (all of
// whose waits have limits): the four warps of a warpgroup look one by one, their epilogues have
// barriers that wait for all of them without a limit, and a task that is posted after the abort has to
// be found by all of them or by none.
__device__ __noinline__ bool wait_task_or_end(uint32_t bar, uint32_t parity, const volatile int* posted_all) {
  while (!mbar_try_wait_for(bar, parity, kWaitSleepNs)) {
    if (*posted_all) {
      __threadfence_block();               // (the flag was set behind the last post)
      return mbar_test_wait(bar, parity);
    }
  }
  return true;
}

// ---------------------------------------------------------------- scheduler (thread 0)
// One rank, or partial sums only: what a task leaves is read by nobody in this launch.
__device__ __forceinline__ bool without_ar(const KParams& p) { return p.tp == 1 || (p.flags & 16u); }

// Attention task ids come from the counter, the first of every CTA too: a task belongs to a CTA
// only once that CTA runs.  (Ids by CTA number save that atomic, but then a CTA that gets its
// SM late - another stream's kernel holds it - keeps its task from all the others, which wait
// for it up to the wait limit.)
// An id stands for one head, two heads of a kv group (pair), or two heads that share no kv
// head and the last head of an odd count alone (sep), of one position of the claim order.
__device__ __forceinline__ int fa_tasks_per_tile(const KParams& p) {
  return (p.pair || p.sep) ? (p.H + 1) >> 1 : p.H;
}

// Pop from the published O_proj ready queue.  The reference pops with a CAS on the consume
// index (fused_fa_oproj_ar.py:168-189); with one CTA per SM all polling, a CAS admits one
// winner per L2 round trip and the queue drains at ~2 tasks/us.  Here a CTA takes a ticket
// with one atomicAdd (every attempt succeeds) after seeing head < tail.  A ticket that lost
// the race to a not-yet-published entry stays pending in this CTA (at most one) and is
// served as soon as the publish index passes it; meanwhile the CTA keeps taking other work.
// The queue holds row-tile groups in the order they became ready; each stands for its
// `per_group` tasks, so ticket t is task t % per_group of entry t / per_group.  An entry is the
// group's number plus one, written with release behind its reservation and zero before: who holds a
// ticket waits for the entry itself.  (With a publish count that the publishers advanced in their
// turn, a row tile's last head and its first O_proj task were two trips to L2 and two fences
// further apart, 2 us.)
// `head` and `tail` are the consume and reserve counts as the caller read them.
__device__ __forceinline__ bool try_pop_oproj(const KParams& p, int total_op, int per_group,
                                              uint32_t head, uint32_t tail, int* pending, int* arg) {
  if (*pending < 0) {
    if (head >= tail) return false;
    const uint32_t t = atom_add_relaxed_gpu(p.ctrl + C_OP_CONSUME, 1u);
    if (static_cast<int>(t) >= total_op) return false;    // past the end: nothing there
    *pending = static_cast<int>(t);
  }
  const uint32_t entry = ld_acquire_gpu(p.oproj_queue + *pending / per_group);
  if (entry == 0u) return false;
  *arg = static_cast<int>(entry - 1u) * per_group + *pending % per_group;
  *pending = -1;
  return true;
}

// Claim one ready AllReduce slot of this (owner) rank.
//
// The reference has the last of the tp arriving ranks set a bit in the owner's ready
// bitset, found by its atomic add returning tp-1, and owners claim by clearing the lowest
// set bit (fused_fa_oproj_ar.py:192-239, 294-317).  On NVSwitch that costs every O_proj
// task a blocking remote round trip (tens of microseconds once the links carry the
// AllReduce itself) and makes all polling CTAs fight for one bit.  Here arrivals are
// fire-and-forget adds on the owner's ready counts and the owner finds ready slots by
// reading the counts: they are packed as one byte per slot (tp <= 8 arrivals; bit 7 marks
// a slot as claimed), so sixteen slots come with one 16-byte load and a scan of all the
// slots a rank owns is a handful of loads - cheap enough that every CTA looks at every
// slot each time it asks for work, and no ready slot waits to be discovered.  A CTA starts
// its scan at a place of its own so that CTAs polling at the same moment do not all go for
// the same slot; the claim is an atomic OR of the slot's flag, won by whoever sees the
// flag clear in the value that comes back.  The reference's ready bitset has no role here
// (the plan descriptor still has the field so that the workspace keeps the reference's
// buffer list; it may be 0).
__device__ __noinline__ int try_claim_ar(const KParams& p, int local_owned, uint32_t poll_no) {
  if (local_owned <= 0) return -1;
  const uint32_t tp = static_cast<uint32_t>(p.tp);
  const uint32_t n_words = (static_cast<uint32_t>(local_owned) + 3u) >> 2;   // 4 slots per word
  const uint32_t n_vec = (n_words + 3u) >> 2;                                // 16 slots per load
  const uint32_t cap_words = static_cast<uint32_t>(p.max_owner_slots);       // buffer length
  const uint32_t start = (blockIdx.x * 5u + poll_no) % n_vec;
  for (uint32_t v0 = 0; v0 < n_vec; v0 += 8) {
    uint4 w[8];
    uint32_t vi[8];
#pragma unroll
    for (uint32_t u = 0; u < 8; ++u) {
      uint32_t v = start + v0 + u;
      if (v >= n_vec) v -= n_vec;
      vi[u] = v;
      w[u] = make_uint4(0u, 0u, 0u, 0u);
      if (v0 + u < n_vec) {
        // (gpu-scope loads: a hint only - the atomic below is the synchronising access)
        const uint32_t* src = p.ready_count + v * 4;
        if (v * 4 + 4 <= cap_words) {
          w[u] = ld_relaxed_gpu_b128(src);
        } else {                     // last, partial vector of a short buffer
          if (v * 4 + 0 < cap_words) w[u].x = ld_relaxed_gpu(src + 0);
          if (v * 4 + 1 < cap_words) w[u].y = ld_relaxed_gpu(src + 1);
          if (v * 4 + 2 < cap_words) w[u].z = ld_relaxed_gpu(src + 2);
        }
      }
    }
#pragma unroll
    for (uint32_t u = 0; u < 8; ++u) {
      const uint32_t ws[4] = {w[u].x, w[u].y, w[u].z, w[u].w};
#pragma unroll
      for (uint32_t k = 0; k < 4; ++k) {
        // bytes equal to tp (a claimed slot reads tp | 0x80, an unfinished one < tp)
        const uint32_t x = ws[k] ^ (tp * 0x01010101u);
        uint32_t hit = (x - 0x01010101u) & ~x & 0x80808080u;
        while (hit) {
          const uint32_t b = (__ffs(hit) - 1) >> 3;            // byte number 0..3
          hit &= ~(0xFFu << (b * 8));
          if (((ws[k] >> (b * 8)) & 0xFFu) != tp) continue;      // borrow artefact
          const uint32_t idx = (vi[u] * 4 + k) * 4 + b;
          if (idx >= static_cast<uint32_t>(local_owned)) continue;
          const uint32_t old = atom_or_relaxed_sys(p.ready_count + vi[u] * 4 + k, 0x80u << (b * 8));
          if (((old >> (b * 8)) & 0xFFu) == tp) {
            fence_acq_rel_sys();      // the tp arrivals (release) happen before what follows
            return static_cast<int>(idx * tp + p.rank);
          }
        }
      }
    }
  }
  return -1;
}

// What limits a claim is the number of trips to L2 that wait for one another, 600-700 cycles
// each: the words that decide it are read together.  (One after the other, with the tile's
// descriptor behind them, a claim took 6500 cycles - most of what lies between two attention
// tasks, and several times in the chain of a small launch.  In-kernel cycles of a whole launch:
// three short prompts 77400 -> 71700, six ragged prompts of 13400 tokens 371200 -> 363600, 12
// short turns on cached prompts 199300 -> 193100, a wide layer 2191000 -> 2193000.)
__device__ __noinline__ void schedule_pick(const Env& e, int role, int num_fa, int n_fa_tasks, int total_op,
                                           int per_group, int local_owned, uint32_t poll_no, bool busy,
                                           bool* fa_left, int* pending, int* mode, int* arg) {
  const KParams& p = *e.p;
  *mode = MODE_IDLE;
  *arg = -1;
  const uint32_t status = ld_relaxed_gpu(p.status);
  const uint32_t fa_next = ld_relaxed_gpu(p.ctrl + C_FA_COUNTER), fa_d = ld_relaxed_gpu(p.ctrl + C_FA_DONE);
  const uint32_t op_next = ld_relaxed_gpu(p.ctrl + C_OP_CONSUME), op_d = ld_relaxed_gpu(p.ctrl + C_OP_DONE);
  const uint32_t ar_next = ld_relaxed_gpu(p.ctrl + C_AR_CURSOR), ar_d = ld_relaxed_gpu(p.ctrl + C_AR_DONE);
  const uint32_t tail = ld_relaxed_gpu(p.ctrl + C_OP_RESERVE);
  if (status != 0u) {       // some CTA (or rank) gave up: leave
    *e.abort_flag = 1;
    *mode = MODE_DONE;
    return;
  }
  if (p.flags & 8u) {
    // AllReduce-only launch: every owned slot is taken as ready (the caller made sure all
    // ranks' partials are in place); slots are handed out by a counter
    if (static_cast<int>(ar_d) >= local_owned) { *mode = MODE_DONE; return; }
    if (static_cast<int>(ar_next) < local_owned) {
      const int idx = static_cast<int>(atom_add_relaxed_gpu(p.ctrl + C_AR_CURSOR, 1u));
      if (idx < local_owned) { *mode = MODE_AR; *arg = idx * p.tp + p.rank; }
    }
    return;
  }
  if (p.flags & 32u) {
    // O_proj-only launch (single rank): O_scratch is taken as complete, slots are handed
    // out in order by the consume counter
    *mode = MODE_DONE;
    if (static_cast<int>(op_next) < total_op) {
      const int t = static_cast<int>(atom_add_relaxed_gpu(p.ctrl + C_OP_CONSUME, 1u));
      if (t < total_op) { *mode = MODE_OPROJ; *arg = t; }
    }
    return;
  }
  const bool fa_only = (p.flags & 1u) != 0;
  // With an AllReduce to come everybody stays until all of it is done: slots become ready by other
  // ranks' work.  (Each count is final once it is at its target; what they stand for is read by
  // nobody before the exit protocol's fence.)  Without one a CTA leaves once every task is handed
  // out and it holds no ticket: what is left is running, and the last CTA out ends the launch.  (To
  // wait for the counts instead was a poll or two, 2 us, at the end of every launch.)
  const bool done = without_ar(p)
                        ? static_cast<int>(fa_next) >= n_fa_tasks && *pending < 0 &&
                              (fa_only || static_cast<int>(op_next) >= total_op)
                        : static_cast<int>(fa_d) >= num_fa &&
                              (fa_only || (static_cast<int>(op_d) >= total_op && static_cast<int>(ar_d) >= local_owned));
  if (done) { *mode = MODE_DONE; return; }
  // probe order by role: 0: FA,OPROJ,AR  1: OPROJ,AR,FA  2: AR,FA,OPROJ (the reference's
  // three orders).  With the "drain first" launch flag downstream work goes first so that
  // AllReduce traffic starts early and keeps flowing: roles 0/1 become 3: OPROJ,FA,AR and
  // role 2 becomes 4: AR,OPROJ,FA.
  for (int i = 0; i < 3; ++i) {
    int m;
    if (role == 3) m = (i == 0) ? MODE_OPROJ : (i == 1) ? MODE_FA : MODE_AR;
    else if (role == 4) m = MODE_AR - i;
    else {
      const int src = (role == 0) ? (MODE_FA + i) : (role == 1) ? (MODE_OPROJ + i) : (MODE_AR + i);
      m = (src > MODE_AR) ? src - 3 : src;
    }
    bool ok = false;
    if (m == MODE_FA) {
      if (*fa_left && static_cast<int>(fa_next) < n_fa_tasks) {
        *arg = static_cast<int>(atom_add_relaxed_gpu(p.ctrl + C_FA_COUNTER, 1u));
        ok = *arg < n_fa_tasks;
      }
      if (!ok) *fa_left = false;
    } else if (fa_only) ok = false;
    else if (m == MODE_OPROJ) ok = try_pop_oproj(p, total_op, per_group, op_next, tail, pending, arg);
    else if (!without_ar(p) && !(busy && static_cast<int>(op_next) >= total_op)) {
      // (once every O_proj task has been handed out only reductions are left and CTAs go
      // idle: a CTA that still has a task running leaves ready slots to them instead of
      // queueing one behind its own)
      const int q = try_claim_ar(p, local_owned, poll_no);
      if (q >= 0) { *arg = q; ok = true; }
    }
    if (ok) { *mode = m; return; }
  }
}

// Publish the O_proj tasks of one row-tile group (the caller has acquired what made it ready).
__device__ __forceinline__ void publish_oproj(const KParams& p, int group, int per_group) {
  const uint32_t n = static_cast<uint32_t>(per_group);
  const uint32_t start = atom_add_relaxed_gpu(p.ctrl + C_OP_RESERVE, n);
  st_release_gpu(p.oproj_queue + start / n, static_cast<uint32_t>(group) + 1u);
}

__device__ __forceinline__ void finish_ar_slot(const KParams& p, int slot) {
  const int owner_idx = slot / p.tp;
  const uint64_t bit = 1ull << (owner_idx & 63);
  const uint64_t old = atom_or_acqrel_gpu_u64(
      reinterpret_cast<uint64_t*>(p.ar_done_bits) + (owner_idx >> 6), bit);
  if ((old & bit) == 0) atom_add_release_gpu(p.ctrl + C_AR_DONE, 1u);
}

// After an O_proj task: tell the slot's owner rank that this rank's partial is in place.
__device__ __noinline__ void publish_ar_ready(const KParams& p, int slot) {
  // (the partial is the result, or partial sums only (measurement aid): nothing to account)
  if (without_ar(p)) return;
  const int owner_rank = slot % p.tp;
  const int owner_idx = slot / p.tp;
  red_add_release_sys(reinterpret_cast<uint32_t*>(p.peer_rc[owner_rank]) + (owner_idx >> 2),
                      1u << ((owner_idx & 3) * 8));      // one byte per slot
  atom_add_release_gpu(p.ctrl + C_OP_DONE, 1u);
}

// ---------------------------------------------------------------- rank barrier
// Cross-rank barrier at kernel exit: two signal slots (phase) counted up to tp and back
// down to 0 (sign), selected by a rank-local counter, so it is reusable without any reset
// (fused_fa_oproj_ar.py:99-143).  Run by one CTA (the last one to finish).
__device__ __noinline__ void rank_barrier(const Env& e) {
  const KParams& p = *e.p;
  __syncthreads();
  if (!*e.abort_flag) {
    const uint32_t st = ld_relaxed_gpu(p.sync_ctrl + S_NVL_COUNTER);
    const int phase = st & 1u;
    const int down = (st >> 1) & 1u;
    if (static_cast<int>(threadIdx.x) < p.tp) {
      int* peer = reinterpret_cast<int*>(p.peer_nvl[threadIdx.x]) + phase;
      atom_add_release_sys_s32(peer, down ? -1 : 1);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      atom_add_relaxed_gpu(p.sync_ctrl + S_NVL_COUNTER, 1u);
      const int target = down ? 0 : p.tp;
      const uint64_t t0 = globaltimer_ns();
      uint32_t it = 0;
      while (ld_acquire_sys_s32(p.nvl_signal + phase) != target) {
        if ((++it & 63u) == 0 && globaltimer_ns() - t0 > p.wait_limit_ns) {
          report(e, ST_TIMEOUT_NVL, phase, target);
          break;
        }
      }
    }
  }
  __syncthreads();
}

// ---------------------------------------------------------------- FA: MMA helpers
constexpr uint64_t kDescK = smem_desc_template(16, 1024);          // K-major, 128-B swizzle
constexpr uint64_t kDescVmn = smem_desc_template(kPanel, 1024);    // V tile [kv][d], MN-major
constexpr uint64_t kDescWmn = smem_desc_template(kWPanel, 1024);   // W slab [k][n], MN-major

// S = Q K^T over d = 128: 8 k-steps; both tiles are two 64-wide swizzled panels.
__device__ __forceinline__ void issue_qk(uint32_t tmem_s, uint32_t sm_q, uint32_t sm_k) {
  const uint32_t q16 = sm_q >> 4, k16 = sm_k >> 4;
#pragma unroll
  for (int kk = 0; kk < 8; ++kk) {
    const uint32_t off16 = ((kk >> 2) * kPanel + (kk & 3) * 32) >> 4;
    mma_ss(tmem_s, smem_desc_at(kDescK, q16 + off16), smem_desc_at(kDescK, k16 + off16),
           kIdescQK, kk > 0);
  }
}
// O (+)= P V over the 16-key steps [k0, k1): P is bf16 in TMEM (8 columns per 16 kv), V tile
// is [kv][d] in two d panels.
template <int k0, int k1>
__device__ __forceinline__ void issue_pv(uint32_t tmem_o, uint32_t tmem_p, uint32_t sm_v,
                                         bool acc) {
  const uint32_t v16 = sm_v >> 4;
#pragma unroll
  for (int kk = k0; kk < k1; ++kk)
    mma_ts(tmem_o, tmem_p + kk * 8, smem_desc_at(kDescVmn, v16 + kk * 128), kIdescPV,
           (acc || kk > 0) ? 1u : 0u);
}

// Convert N fp32 values (columns col0..col0+N-1 of this thread's row, N and col0 multiples of 8) to
// bf16 and put them into a [128 rows][64 columns] staging panel laid out as TMA expects
// for a 128-byte-swizzled box: 16-byte chunk c of row r lives at chunk c ^ (r & 7).
template <int N>
__device__ __forceinline__ void stage_row(uint32_t panel, int row, int col0,
                                          const uint32_t (&v)[N], float scale) {
  const uint32_t rbase = panel + static_cast<uint32_t>(row) * 128u;
  const uint32_t sw = static_cast<uint32_t>(row & 7);
#pragma unroll
  for (int q = 0; q < N / 8; ++q) {
    const uint32_t c = static_cast<uint32_t>((col0 >> 3) + q);
    st_shared_v4(rbase + ((c ^ sw) << 4),
                 pack_bf16x2(__uint_as_float(v[8 * q + 0]) * scale, __uint_as_float(v[8 * q + 1]) * scale),
                 pack_bf16x2(__uint_as_float(v[8 * q + 2]) * scale, __uint_as_float(v[8 * q + 3]) * scale),
                 pack_bf16x2(__uint_as_float(v[8 * q + 4]) * scale, __uint_as_float(v[8 * q + 5]) * scale),
                 pack_bf16x2(__uint_as_float(v[8 * q + 6]) * scale, __uint_as_float(v[8 * q + 7]) * scale));
  }
}

// A whole panel row already in bf16.
__device__ __forceinline__ void stage_panel_row(uint32_t panel, int row, const uint32_t (&pk)[32]) {
  const uint32_t rbase = panel + static_cast<uint32_t>(row) * 128u;
  const uint32_t sw = static_cast<uint32_t>(row & 7);
#pragma unroll
  for (uint32_t c = 0; c < 8; ++c)
    st_shared_v4(rbase + ((c ^ sw) << 4), pk[4 * c], pk[4 * c + 1], pk[4 * c + 2], pk[4 * c + 3]);
}

// ---------------------------------------------------------------- AllReduce of one slot
// One AllReduce slot: 128 rows x (vnt x 128) bf16 columns, reduced in the switch and
// written back to every rank.  `nthr` threads cooperate; each keeps U 16-byte reductions in
// flight before its first store (NVLink round trips are microseconds).
template <int U>
__device__ __forceinline__ void ar_batch(const KParams& p, int ft, int base_out, int c0, int nthr) {
  auto chunk_addr = [&](int c) -> unsigned long long {
    const int o_t = c >> 11, m = (c >> 4) & 127, nc = c & 15;
    const size_t elem =
        ((static_cast<size_t>(ft * 128 + m) * p.num_out + base_out + o_t) * 128) + nc * 8;
    return p.csym_mc + elem * 2;
  };
  uint4 v[U];
#pragma unroll
  for (int u = 0; u < U; ++u) v[u] = multimem_ld_reduce_bf16x8(chunk_addr(c0 + u * nthr));
#pragma unroll
  for (int u = 0; u < U; ++u) multimem_st_b128(chunk_addr(c0 + u * nthr), v[u]);
}

// The same batch with plain peer loads and stores, two ranks only: the owner reads its own
// and the peer's partial, adds in fp32, rounds once and writes both copies.  With two GPUs
// the multicast path is several times slower than the NVLink copy rate; this one is not.
template <int U>
__device__ __forceinline__ void ar_batch_p2p(const KParams& p, int ft, int base_out, int c0, int nthr) {
  auto chunk_off = [&](int c) -> unsigned long long {
    const int o_t = c >> 11, m = (c >> 4) & 127, nc = c & 15;
    const size_t elem =
        ((static_cast<size_t>(ft * 128 + m) * p.num_out + base_out + o_t) * 128) + nc * 8;
    return elem * 2;
  };
  const unsigned long long mine = p.peer_csym[p.rank], peer = p.peer_csym[p.rank ^ 1];
  uint4 a[U], b[U];
#pragma unroll
  for (int u = 0; u < U; ++u) b[u] = ld_relaxed_sys_b128(peer + chunk_off(c0 + u * nthr));
#pragma unroll
  for (int u = 0; u < U; ++u)      // this GPU's own partial: gpu scope is enough
    a[u] = ld_relaxed_gpu_b128(reinterpret_cast<const void*>(mine + chunk_off(c0 + u * nthr)));
#pragma unroll
  for (int u = 0; u < U; ++u) {
    uint4 r;
    r.x = add_bf16x2_via_f32(a[u].x, b[u].x); r.y = add_bf16x2_via_f32(a[u].y, b[u].y);
    r.z = add_bf16x2_via_f32(a[u].z, b[u].z); r.w = add_bf16x2_via_f32(a[u].w, b[u].w);
    const unsigned long long off = chunk_off(c0 + u * nthr);
    st_relaxed_sys_b128(peer + off, r);
    st_relaxed_sys_b128(mine + off, r);
  }
}

// One AllReduce slot: 128 rows x (vnt x 128) bf16 columns, reduced in the switch and
// written back to every rank.  `nthr` (256) threads cooperate; each keeps 16 16-byte
// reductions in flight before its first store (NVLink round trips are microseconds).  A
// slot is vnt x 2048 chunks: whole batches of nthr x 16, then one of nthr x 8 if vnt is odd.
__device__ __forceinline__ void ar_slot(const KParams& p, int ft, int base_out, int vnt, int t,
                                        int nthr) {
  const int total = vnt * 2048;
  int c0 = t;
  if (p.flags & 64u) {      // MA_FLAG_AR_P2P (host side admits it at tp == 2 only)
    for (; c0 + nthr * 7 < total; c0 += nthr * 8) ar_batch_p2p<8>(p, ft, base_out, c0, nthr);
    return;
  }
  for (; c0 + nthr * 15 < total; c0 += nthr * 16) ar_batch<16>(p, ft, base_out, c0, nthr);
  if (c0 + nthr * 7 < total) ar_batch<8>(p, ft, base_out, c0, nthr);
}

}  // namespace

// O_proj task of a single rank: nrt row tiles x nnt column tiles in one pass.  A task's time per
// 64 k, from what a further round of tasks adds to the stage alone (K_local 2048): 0.35 us for
// 1 x 1, 0.42 for 1 x 2, 0.75 for 2 x 2 - so 2 x 2 does the same work in nine tenths of the time of
// 1 x 2, and a 1 x 1 task costs almost what a 1 x 2 one does.  (The tensor pipe needs 0.14, 0.28
// and 0.56; what holds the small shapes up is not established.)
// O_proj-only launches: every task is ready at the start, so 2 x 2 from half a wave of such tasks
// and 1 x 1 only below a quarter.  The stage in us as 1 x 1 / 1 x 2 / 2 x 2 at K_local 2048: 0.2 waves
// 30 / 32 / 42, 0.4 42 / 34 / 44, 0.65 53 / 45 / 44, 0.9 64 / 46 / 44, 1.3 86 / 59 / 67, 1.7 99 / 73 /
// 68, 2.05 121 / 87 / 90, 2.8 155 / 106 / 92, 3.5 179 / 119 / 117.
// Behind attention, with few tasks what counts is how soon the last row tile's product is done:
// one column tile per task up to 1.25 waves, two up to 2.25.  Whole launches, us, as 1 x 1 / 1 x 2 /
// 2 x 2: 0.1 waves (520 tokens, hidden 1024) 44 / 46 / 51, 0.9 waves (four prompts of 1024, hidden
// 2048, K_local 2048) 90 / 93 / 103, 1.3 waves (3072 tokens, hidden 4096, K_local 512, 1024, 2048,
// 4096) 70 / 70 / 62, 78 / 70 / 72, 107 / 87 / 101, 178 / 138 / 162.  As 1 x 2 / 2 x 2, hidden 4096 and
// the same K_local: 1.95 waves 78 / 67, 85 / 82, 110 / 117, 197 / 190; 2.05 81 / 68, 88 / 84, 113 / 119,
// 218 / 209; 2.3 86 / 70, 92 / 85, 122 / 124, 225 / 228; 2.8 101 / 76, 106 / 95, 147 / 137, 283 / 267.
// (K_local 512 would take 2 x 2 from one wave on, a longer product has the longer last task.)
// These figures compare the shapes under an issuer that was converged per stage and with W in two
// loads; since then every shape is faster (2 x 2 alone at 0.9 waves 44 -> 42 us, 2.6 91 -> 86, 3.5 117
// -> 110; 0.9 waves as a whole launch 90 -> 86), and the lines were not moved.
__device__ __forceinline__ void op_task_shape(const KParams& p, int n_tiles, int ctas, int* nrt,
                                              int* nnt) {
  const int t22 = (n_tiles + 1) / 2 * ((p.num_out + 1) / 2);
  *nrt = 4 * t22 >= p.op_two_from * ctas ? 2 : 1;
  *nnt = 4 * t22 >= p.op_cols2_from * ctas ? 2 : 1;
}

template <bool kSeparate> struct Layout { static constexpr bool value = kSeparate; };   // of K/V stages

// Task descriptor words written by the scheduler (shared memory, two slots).
enum : int { T_MODE = 0, T_FT = 1,
             TF_HEAD0 = 2, TF_NT = 3, TF_KVH = 4, TF_QROW0 = 5, TF_VALID = 6, TF_KSTART = 7,
             TF_KLEN = 8, TF_OFFSET = 9, TF_NBLK = 10, TF_MB = 11,
             TF_PARTS = 12,     // parts its keys are split into (1: none); TF_PART: which of them
             TF_PART = 13, TF_SLOT = 14,
             TF_FIN0 = 15, TF_FIN1 = 16,   // head 0 / 1 of the task is finished when the task is
             TO_BASE = 2, TO_VNT = 3, TO_SLOT = 5, TO_NRT = 6, TO_TWO = 8,
             T_WORDS = 17 };

// End of a head's attention over a part of its keys.  The part's O (not divided), reference maximum
// and row sum go to memory in fp32; whichever part of the head is there last adds them all up and
// stages the head's output - nobody waits for anybody.  Its own O it has in TMEM, but it adds in the
// parts' order, so that the result does not depend on who was last.
// What it costs is trips to L2: 4.5 us to put a part of 64 KB there and look, 2.5 us for each part
// that is read.  A thread's row of it lies strided ([column / 4][row] of float4: a warp's accesses are
// 512 bytes in a row).  More than 32 columns of one part in flight would take the registers that the
// attention loop lives on (two parts': the kernel's spills 240 -> 1000 bytes, every task slower).
__device__ __noinline__ void finish_part(const KParams& p, int* d, int wg, int row, uint32_t t_o,
                                         uint32_t stg, uint32_t bar_o_free, float m, float l) {
  const int n = d[TF_PARTS], own = d[TF_PART], head = d[TF_HEAD0] + wg, first = d[TF_SLOT];
  const size_t pitch = static_cast<size_t>(p.H) * kPartFloats;      // from one part to the next
  float* base = p.part_o + static_cast<size_t>(first) * pitch + static_cast<size_t>(head) * kPartFloats;
  float* mine = base + own * pitch;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    uint32_t o[32];
    tmem_ld32(t_o + c * 32, o);
    tc_wait_ld();
#pragma unroll
    for (int q = 0; q < 8; ++q)
      __stcg(reinterpret_cast<uint4*>(mine) + (c * 8 + q) * 128 + row,
             make_uint4(o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]));
  }
  __stcg(mine + kPartMax + row, m);
  __stcg(mine + kPartSum + row, l);
  named_bar_sync(1 + wg, 128);
  if (row == 0) {
    uint32_t* count = p.part_count + first * p.H + head;
    fence_acq_rel_gpu();                        // (the warpgroup's stores: ordered by the barrier)
    const bool last = atom_add_relaxed_gpu(count, 1u) == static_cast<uint32_t>(n - 1);
    fence_acq_rel_gpu();
    if (last) *count = 0u;                      // (the next launch's parts count from zero)
    d[TF_FIN0 + wg] = last ? 1 : 0;
  }
  named_bar_sync(1 + wg, 128);
  if (d[TF_FIN0 + wg] != 0) {
    float top = -INFINITY, sum = 0.f;
#pragma unroll 4
    for (int i = 0; i < n; ++i) top = fmaxf(top, __ldcg(base + i * pitch + kPartMax + row));
    auto weight = [&](float mi) { return mi == -INFINITY ? 0.f : ex2((mi - top) * p.scale_log2); };
#pragma unroll 4
    for (int i = 0; i < n; ++i)
      sum += weight(__ldcg(base + i * pitch + kPartMax + row)) * __ldcg(base + i * pitch + kPartSum + row);
    const float inv = (row < d[TF_VALID] && sum > 0.f) ? (1.f / sum) : 0.f;
    const float w_own = weight(m);
#pragma unroll 1
    for (int c = 0; c < 4; ++c) {
      float acc[32];
#pragma unroll
      for (int q = 0; q < 32; ++q) acc[q] = 0.f;
      auto add_own = [&]() {
        uint32_t o[32];
        tmem_ld32(t_o + c * 32, o);
        tc_wait_ld();
#pragma unroll
        for (int q = 0; q < 32; ++q) acc[q] += w_own * __uint_as_float(o[q]);
      };
#pragma unroll 1
      for (int j = 0; j < n - 1; ++j) {
        const float* part = base + (j + (j >= own ? 1 : 0)) * pitch;
        const float4* src = reinterpret_cast<const float4*>(part) + c * 8 * 128 + row;
        float4 x[8];
        const float mi = __ldcg(part + kPartMax + row);
#pragma unroll
        for (int q = 0; q < 8; ++q) x[q] = __ldcg(src + q * 128);
        if (j == own) add_own();
        const float w = weight(mi);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          acc[4 * q] += w * x[q].x; acc[4 * q + 1] += w * x[q].y;
          acc[4 * q + 2] += w * x[q].z; acc[4 * q + 3] += w * x[q].w;
        }
      }
      if (own == n - 1) add_own();
      uint32_t bits[32];
#pragma unroll
      for (int q = 0; q < 32; ++q) bits[q] = __float_as_uint(acc[q]);
      stage_row(stg + (c >> 1) * kPanel, row, (c & 1) * 32, bits, inv);
    }
  }
  tc_fence_before();
  __syncwarp();
  if ((row & 31) == 0) mbar_arrive(bar_o_free);
}

__device__ __forceinline__ bool is_tile_mode(int m) { return m == MODE_FA || m == MODE_OPROJ; }

__global__ void __launch_bounds__(kThreads, 1)
fused_prefill_kernel(const __grid_constant__ CUtensorMap tmQ,
                     const __grid_constant__ CUtensorMap tmK,
                     const __grid_constant__ CUtensorMap tmV,
                     const __grid_constant__ CUtensorMap tmO,
                     const __grid_constant__ CUtensorMap tmW,
                     const __grid_constant__ CUtensorMap tmC,
                     const __grid_constant__ CUtensorMap tmW2,
                     const __grid_constant__ KParams p) {
  extern __shared__ uint8_t dyn_smem[];
  // The abort flag, read in every wait loop, gets a 128-byte line of its own: where the
  // compiler put it next to the barrier block by default depended on the block's size, and one
  // such placement cost the attention stage 2.5 % (0.1597 vs 0.1560 ms).
  __shared__ __align__(128) Bars bars;
  __shared__ uint32_t s_tmem;
  __shared__ __align__(128) int s_abort_line[32];
  __shared__ __align__(128) int s_desc[2][T_WORDS];
  int& s_abort = s_abort_line[0];
  int& s_posted_all = s_abort_line[1];       // the scheduler has left: no task will follow

  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane = tid & 31;
  const uint32_t smem0 = (smem_u32(dyn_smem) + 1023u) & ~1023u;
  Env env{&p, &s_abort};

  if (tid == 0) {
    s_abort = s_posted_all = 0;
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&bars.task_full[i]), 1);
      mbar_init(smem_u32(&bars.task_empty[i]), 11);
      mbar_init(smem_u32(&bars.loads_done[i]), 1);
      mbar_init(smem_u32(&bars.q_full[i]), 1);
      mbar_init(smem_u32(&bars.q_empty[i]), 2);
      mbar_init(smem_u32(&bars.s_full[i]), 1);
      mbar_init(smem_u32(&bars.p_part[i]), 4);
      mbar_init(smem_u32(&bars.p_full[i]), 4);
      mbar_init(smem_u32(&bars.o_staged[i]), 4);
      mbar_init(smem_u32(&bars.o_done[i]), 1);
      mbar_init(smem_u32(&bars.o_free[i]), 4);
      mbar_init(smem_u32(&bars.acc_full[i]), 1);
      mbar_init(smem_u32(&bars.acc_free[i]), 8);
    }
    for (int i = 0; i < kKvSlots; ++i) {
      mbar_init(smem_u32(&bars.kv_full[i]), 1);
      mbar_init(smem_u32(&bars.kv_empty[i]), 1);
    }
    for (int i = 0; i < 4; ++i) {
      mbar_init(smem_u32(&bars.op_full[i]), 1);
      mbar_init(smem_u32(&bars.op_empty[i]), 1);
    }
    mbar_init(smem_u32(&bars.drain), 1);
    fence_mbar_init();
    fence_proxy_async_smem();
    tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV);
    tma_prefetch_desc(&tmO); tma_prefetch_desc(&tmW); tma_prefetch_desc(&tmC);
    tma_prefetch_desc(&tmW2);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&s_tmem), 512);
    tmem_relinquish();
  }
  wait_for_previous();        // (what is above touches nothing of the kernels before this one)
  // The scheduler's first trip to L2: whether an earlier launch gave up, the counts, and its first
  // attention task, which is there for the taking (nothing else can be ready).
  const bool has_fa = !(p.flags & (8u | 32u));
  const int* tasks = (p.flags & 4u) ? nullptr : p.tasks;
  uint32_t status0 = 0, first_fa = 0;
  int num_fa = 0, total_op = 0, n_tiles = 0, local_owned = 0, n_pos = 0;
  if (tid == 64) {
    status0 = ld_relaxed_gpu(p.status);
    num_fa = p.actv[0]; total_op = p.actv[1]; n_tiles = p.actv[2]; local_owned = p.actv[5];
    if (tasks) n_pos = tasks[0];
    if (has_fa) first_fa = atom_add_relaxed_gpu(p.ctrl + C_FA_COUNTER, 1u);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = s_tmem;

  // Every role walks the two descriptor slots in turn.  A role arrives on task_empty[k]
  // when its part of the task in slot k is finished; the scheduler publishes the task's
  // completion and refills the slot once all eleven arrivals are in (producer, MMA issuer,
  // attention store, eight compute warps), so the scheduler runs
  // one task ahead of the workers.  Attention tiles and O_proj tiles overlay the same
  // shared memory and TMEM: a role that goes from one kind to the other first waits for
  // the previous task to finish completely (same-kind neighbours overlap freely).
  int slot_k = 0;
  uint32_t tf_par = 0, arrived = 0;        // a bit per slot: phase to wait for, arrivals made (mod 2)
  int prev_mode = MODE_IDLE, prev_k = 0;

#define MA_TASK_FULL                                                                       \
  wait_bar(env, smem_u32(&bars.task_full[slot_k]), (tf_par >> slot_k) & 1u, 0x100 + warp)
#define MA_NEXT_TASK_IF(full, desc_ptr, mode_var)                                          \
  if (!(full)) break;                                                                      \
  tf_par ^= 1u << slot_k;                                                                  \
  const int* desc_ptr = s_desc[slot_k];                                                    \
  const int mode_var = desc_ptr[T_MODE];                                                   \
  if (mode_var == MODE_DONE) break;
#define MA_NEXT_TASK(desc_ptr, mode_var) MA_NEXT_TASK_IF(MA_TASK_FULL, desc_ptr, mode_var)
// A whole warp takes the task or leaves together: its lanes may see an abort at different
// times, and what follows has instructions that wait for all of them.
#define MA_NEXT_TASK_WARP(desc_ptr, mode_var) \
  MA_NEXT_TASK_IF(__all_sync(0xffffffffu, MA_TASK_FULL), desc_ptr, mode_var)
// A compute warpgroup finds the task with all of its warps or with none (wait_task_or_end).
#define MA_TASK_FULL_OR_END                                                                \
  (mbar_test_wait(smem_u32(&bars.task_full[slot_k]), (tf_par >> slot_k) & 1u) ||          \
   wait_task_or_end(smem_u32(&bars.task_full[slot_k]), (tf_par >> slot_k) & 1u, &s_posted_all))
#define MA_NEXT_TASK_WARPGROUP(desc_ptr, mode_var) \
  MA_NEXT_TASK_IF(__all_sync(0xffffffffu, MA_TASK_FULL_OR_END), desc_ptr, mode_var)
#define MA_DRAIN_IF_SWITCH(mode_var)                                                       \
  if (is_tile_mode(mode_var) && is_tile_mode(prev_mode) && mode_var != prev_mode)          \
    wait_bar(env, smem_u32(&bars.task_empty[prev_k]), ((arrived >> prev_k) & 1u) ^ 1u, 0x110 + warp);
#define MA_TASK_DONE(mode_var)                                                             \
  mbar_arrive(smem_u32(&bars.task_empty[slot_k]));                                         \
  arrived ^= 1u << slot_k;                                                                     \
  prev_mode = mode_var; prev_k = slot_k; slot_k ^= 1;

  if (warp < 4) {
    reg_dec<88>();
    if (warp == 2 && lane == 0) {
      // ==================================================================== scheduler
      // O_proj tasks.  With several ranks a task is an AllReduce slot: one row tile, up to
      // `sg` column tiles in two passes (TO_NRT = 0).  One rank is free to choose: nrt row
      // tiles x nnt column tiles (<= 2 x 2) in one pass, the row tiles sharing every W stage.
      int nrt = 0, nnt = p.sg, per_group = p.nsg;
      // the table of attention tasks, in claim order (none: the claim order's arrays)
      if (n_pos == 0) { tasks = nullptr; n_pos = num_fa / p.H; }
      const int n_fa_tasks = n_pos * fa_tasks_per_tile(p);
      bool fa_left = has_fa;
      if (p.tp == 1 && !(p.flags & 16u)) {      // (without AllReduce: slots, as with several)
        op_task_shape(p, n_tiles, static_cast<int>(gridDim.x), &nrt, &nnt);
        per_group = (p.num_out + nnt - 1) / nnt;
        // (plus what the host's count of slots is off by: such a launch must not end well)
        total_op = (n_tiles + nrt - 1) / nrt * per_group + (total_op - n_tiles * p.nsg);
      }
      const int grp = max(nrt, 1);              // row tiles whose attention a task group needs
#ifdef MA_AUDIT
      if (p.audit && blockIdx.x == 0) { p.status[6] = nrt; p.status[7] = nnt; }   // for tests
#endif
      int role;
      {
        const int wsum = p.w_fa + p.w_oproj + p.w_ar;
        const int r = static_cast<int>(blockIdx.x) % wsum;
        role = (r < p.w_fa) ? 0 : (r < p.w_fa + p.w_oproj) ? 1 : 2;
        if (p.flags & 2u) role = (role == 2) ? 4 : 3;
      }
      int k = 0;
      bool occupied[2] = {false, false};
      uint32_t te_par[2] = {0, 0}, ld_par[2] = {0, 0};
      bool ld_pending[2] = {false, false}, ld_skip[2] = {false, false};
      int pending_ticket = -1;
      uint32_t poll_no = 0;
      bool first = true;
      int occ_mode[2] = {0, 0}, occ_a[2] = {0, 0};
#ifdef MA_AUDIT
      int occ_h[2] = {0, 0};
#endif
      auto publish = [&](int kk) {
        if (s_abort) return;
#ifdef MA_AUDIT
        if (p.audit) {      // exactly-once audit (audit build only): one count per finished unit
          if (occ_mode[kk] == MODE_FA) {
            for (int i = 0; i < 2; ++i)
              if (s_desc[kk][TF_FIN0 + i]) atomicAdd(p.audit + occ_a[kk] * p.H + occ_h[kk] + i, 1u);
          } else if (occ_mode[kk] == MODE_OPROJ && nrt == 0) {
            atomicAdd(p.audit + p.audit_op_base + occ_a[kk], 1u);
          } else if (occ_mode[kk] == MODE_OPROJ) {     // a slot counts with its first column tile
            const int r0 = occ_a[kk] / per_group * nrt, o0 = occ_a[kk] % per_group * nnt;
            for (int r = r0; r < min(r0 + nrt, n_tiles); ++r)
              for (int o = o0; o < min(o0 + nnt, p.num_out); ++o)
                if (o % p.sg == 0) atomicAdd(p.audit + p.audit_op_base + r * p.nsg + o / p.sg, 1u);
          } else if (occ_mode[kk] == MODE_AR) {
            atomicAdd(p.audit + p.audit_ar_base + occ_a[kk] / p.tp, 1u);
          }
        }
#endif
        if (occ_mode[kk] == MODE_FA) {
          // heads that are finished (one of which another part is still running counts with that)
          const int heads = s_desc[kk][TF_FIN0] + s_desc[kk][TF_FIN1];
          if (heads == 0) return;
          if (!(p.flags & 1u)) {
            fence_acq_rel_gpu();
            const int g = occ_a[kk] / grp;
            const uint32_t old = atom_add_relaxed_gpu(p.head_ready + g, static_cast<uint32_t>(heads));
            if (static_cast<int>(old) + heads == p.H * min(grp, n_tiles - g * grp)) {
              fence_acq_rel_gpu();
              publish_oproj(p, g, per_group);
            }
          }
          // (Without an AllReduce nobody reads the count.  Left out there, the attention loop's code
          // comes out with more spills: MHA, six ragged prompts 252 -> 254 us, three short ones 29.8 -> 29.5.)
          if (without_ar(p)) red_add_relaxed_gpu(p.ctrl + C_FA_DONE, static_cast<uint32_t>(heads));
          else atom_add_release_gpu(p.ctrl + C_FA_DONE, static_cast<uint32_t>(heads));
        } else if (occ_mode[kk] == MODE_OPROJ) {
          publish_ar_ready(p, occ_a[kk]);
        } else if (occ_mode[kk] == MODE_AR) {
          fence_acq_rel_sys();
          finish_ar_slot(p, occ_a[kk]);
        }
      };
      while (true) {
        if (occupied[k]) {
          // (who gives up here posts nothing more: the slot may still be looked at)
          if (!wait_bar(env, smem_u32(&bars.task_empty[k]), te_par[k], 0x120 + k)) break;
          te_par[k] ^= 1u;
          occupied[k] = false;
          publish(k);
        }
        // A long attention task must not sit claimed behind another one: take the next
        // task only once the producer has issued the running task's last load (a few
        // blocks before its end), which keeps the claim order close to greedy.
        if (ld_pending[k ^ 1]) {
          wait_bar(env, smem_u32(&bars.loads_done[k ^ 1]), ld_par[k ^ 1], 0x128 + k);
          ld_par[k ^ 1] ^= 1u;
          ld_pending[k ^ 1] = false;
        } else if (ld_skip[k ^ 1]) {
          ld_par[k ^ 1] ^= 1u;        // that task's loads_done phase is never waited for
          ld_skip[k ^ 1] = false;
        }
        int mode, arg;
        int* d = s_desc[k];
        do {
          mode = MODE_IDLE;
          arg = -1;
          if (fa_left && (first || role == 0)) {
            // An attention task where that is what the CTA asks for first: one atomic, and whether
            // somebody gave up comes with it.  (The first was taken before the set-up's barrier.  A launch after
            // one that gave up does nothing until the state has been cleared.)
            const uint32_t status = first ? status0 : ld_relaxed_gpu(p.status);
            if (status == 0u) {
              arg = static_cast<int>(first ? first_fa : atom_add_relaxed_gpu(p.ctrl + C_FA_COUNTER, 1u));
              if (arg < n_fa_tasks) mode = MODE_FA; else fa_left = false;
            }
            first = false;
          }
          uint64_t idle_t0 = 0;
          while (mode == MODE_IDLE) {
            schedule_pick(env, role, num_fa, n_fa_tasks, total_op, per_group, local_owned, poll_no++,
                          occupied[k ^ 1], &fa_left, &pending_ticket, &mode, &arg);
            if (mode != MODE_IDLE) break;
            // nothing to do and not finished: bounded like every other wait (a rank that
            // never shows up, or counts that can never be reached, must not hang the GPU)
            if ((poll_no & 15u) == 0) {
              const uint64_t now = globaltimer_ns();
              if (idle_t0 == 0) idle_t0 = now;
              else if (now - idle_t0 > p.wait_limit_ns) {
                report(env, ST_TIMEOUT_IDLE, poll_no, static_cast<uint32_t>(pending_ticket));
                mode = MODE_DONE;
                break;
              }
            }
            const int o = k ^ 1;
            if (occupied[o] && mbar_try_wait(smem_u32(&bars.task_empty[o]), te_par[o])) {
              te_par[o] ^= 1u;
              occupied[o] = false;
              publish(o);
            } else {
              __nanosleep(100);
            }
          }
          if (mode == MODE_FA) {
            const int per_tile = fa_tasks_per_tile(p);
            const int pos = arg / per_tile, head0 = (arg % per_tile) * ((p.pair || p.sep) ? 2 : 1);
            const int nt = p.pair ? 2 : (p.sep ? min(2, p.H - head0) : 1);
            int ft, b, mb, q0, q_len, k0, k_len;
            uint32_t split = 1u;           // parts | which << 8 | first slot of the row tile's << 16
            if (tasks) {          // one trip to L2; by the arrays below it is three
              const int4* r = reinterpret_cast<const int4*>(tasks + 4 + pos * kTaskWords);
              const int4 r0 = r[0], r1 = r[1];
              ft = r0.x; b = r0.y; mb = r0.z; q0 = r0.w;
              q_len = r1.x; k0 = r1.y; k_len = r1.z; split = static_cast<uint32_t>(r1.w);
            } else {
              ft = (p.fa_order && !(p.flags & 4u)) ? p.fa_order[pos] : pos;
              b = p.fa_b[ft]; mb = p.fa_mb[ft];
              q0 = p.cu_q[b]; q_len = p.cu_q[b + 1] - q0;
              k0 = p.cu_k[b]; k_len = p.cu_k[b + 1] - k0;
            }
            // contiguous KV: rows [k0, k0 + k_len) of K/V; paged KV: k0 is the sequence's row
            // in the page table and the length comes from cache_seqlens
            if (p.page_table) { k0 = b * p.pps; k_len = p.cache_seqlens[b]; }
            int offset = k_len - q_len;
            int nblk = (k_len + 127) >> 7;
            const int nb2 = ((mb + 1) * 128 + offset + 127) >> 7;
            if (nb2 < nblk) nblk = nb2;
            // A part of the keys: its blocks are counted from its first one, for which the start moves
            // up and the lengths shrink.  (The host split by its own lengths; with fewer blocks than
            // parts, or nowhere to put parts, the last of them are empty.)
            const int parts = max(1, min(static_cast<int>(split & 255u), p.part_o ? nblk : 1));
            const int part = static_cast<int>(split >> 8 & 255u);
            if (part >= parts) { mode = MODE_IDLE; continue; }
            if (parts > 1) {
              const int lo = nblk * part / parts;
              nblk = nblk * (part + 1) / parts - lo;
              k0 += p.page_table ? lo : lo * 128;
              offset -= lo * 128;
              k_len -= lo * 128;
            }
            d[T_FT] = ft; d[TF_HEAD0] = head0; d[TF_NT] = nt; d[TF_KVH] = head0 / p.q_per_kv;
            d[TF_QROW0] = q0 + mb * 128; d[TF_VALID] = min(128, q_len - mb * 128);
            d[TF_KSTART] = k0; d[TF_KLEN] = k_len; d[TF_OFFSET] = offset; d[TF_NBLK] = nblk;
            d[TF_MB] = mb;
            d[TF_PARTS] = parts; d[TF_PART] = part; d[TF_SLOT] = static_cast<int>(split >> 16);
            d[TF_FIN0] = 1; d[TF_FIN1] = nt - 1;
            occ_a[k] = ft;
#ifdef MA_AUDIT
            occ_h[k] = head0;
#endif
          }
        } while (mode == MODE_IDLE);
        if (mode == MODE_OPROJ || mode == MODE_AR) {
          const bool own = mode == MODE_OPROJ && nrt > 0;     // a shape of this rank's choice
          const int ft = own ? arg / per_group * nrt : arg / p.nsg;
          const int width = own ? nnt : p.sg;
          const int base_out = (own ? arg % per_group : arg % p.nsg) * width;
          const int rows = own ? min(nrt, n_tiles - ft) : 1;
          d[T_FT] = ft; d[TO_BASE] = base_out; d[TO_VNT] = min(width, p.num_out - base_out);
          d[TO_NRT] = own ? rows : 0; d[TO_SLOT] = arg; d[TO_TWO] = nrt == 2;
          occ_a[k] = arg;
        }
        d[T_MODE] = mode;
        occ_mode[k] = mode;
        mbar_arrive(smem_u32(&bars.task_full[k]));
        if (mode == MODE_DONE) {
          // (without an AllReduce a CTA is done when nothing is left to claim, with a task running)
          if (occupied[k ^ 1]) {
            wait_bar(env, smem_u32(&bars.task_empty[k ^ 1]), te_par[k ^ 1], 0x122 + k);
            publish(k ^ 1);
          }
          break;
        }
        occupied[k] = true;
        // claim-ahead is only held back behind long attention tasks; short tasks (O_proj,
        // AllReduce, a few key blocks) want their successor posted before they end
        ld_pending[k] = (mode == MODE_FA && d[TF_NBLK] > 6);
        ld_skip[k] = !ld_pending[k];
        k ^= 1;
      }
      __threadfence_block();
      *const_cast<volatile int*>(&s_posted_all) = 1;
    } else if (warp == 0 && lane == 0) {
      // ==================================================================== TMA producer
      uint32_t kv_slot = 0, kv_ph = 0, op_st = 0, op_ph = 0, q_uses = 0;
      while (true) {
        MA_NEXT_TASK(d, mode)
        MA_DRAIN_IF_SWITCH(mode)
        if (mode == MODE_FA) {
          const int nt = d[TF_NT], nblk = d[TF_NBLK];
          // a wait that gave up (abort) ends the task's loads: nothing is written into a
          // buffer that was not waited for
          bool ok = true;
          for (int i = 0; i < nt && ok; ++i) {
            ok = wait_bar(env, smem_u32(&bars.q_empty[i]), ((q_uses >> i) & 1u) ^ 1u, 0x18 + i);
            if (!ok) break;
            q_uses ^= 1u << i;
            const uint32_t bar = smem_u32(&bars.q_full[i]);
            mbar_expect_tx(bar, kTile);
            tma_load_4d(smem0 + kSmQ + i * kTile, &tmQ, bar, 0, d[TF_QROW0], 0, d[TF_HEAD0] + i);
          }
          // shared stages: one K and one V tile per key block; separate stages (p.sep): the
          // K tiles of the task's heads, then their V tiles
          const int nld = p.sep ? nt : 1;
          const int kvh0 = p.sep ? d[TF_HEAD0] / p.q_per_kv : d[TF_KVH];
          const int kvh1 = p.sep ? (d[TF_HEAD0] + 1) / p.q_per_kv : kvh0;
          const int k_base = d[TF_KSTART];
          for (int jj = 0; jj < nblk && ok; ++jj) {
            const int blk = nblk - 1 - jj;
            // key block -> first row of its 128-row tile (paged: one page is one block)
            const int kv_row = p.page_table ? p.page_table[k_base + blk] * 128 : k_base + blk * 128;
            for (int ld = 0; ld < 2 * nld; ++ld) {
              const int which = ld >= nld, i = which ? ld - nld : ld;
              if (!(ok = wait_bar(env, smem_u32(&bars.kv_empty[kv_slot]), kv_ph ^ 1u, 0x10 + kv_slot)))
                break;
              const uint32_t bar = smem_u32(&bars.kv_full[kv_slot]);
              mbar_expect_tx(bar, kTile);
              tma_load_4d(smem0 + kSmKV + kv_slot * kTile, which ? &tmV : &tmK, bar, 0, kv_row, 0,
                          i ? kvh1 : kvh0);
              if (++kv_slot == kKvSlots) { kv_slot = 0; kv_ph ^= 1u; }
            }
          }
        } else if (mode == MODE_OPROJ) {
          const int ft = d[T_FT], base_out = d[TO_BASE], vnt = d[TO_VNT], nrt = d[TO_NRT];
          const int nkc = p.K_local >> 6;
          const int rows = max(nrt, 1), passes = nrt ? 1 : (vnt + 1) >> 1;
          const bool two = d[TO_TWO] != 0;      // (the launch's, also for a last row tile alone)
          const uint32_t stage = two ? kOpStage2 : kOpStage, w_off = two ? 2 * kPanel : kPanel;
          const uint32_t stages = two ? 3 : 4;
          fence_proxy_async_global();   // O_scratch was written by other CTAs' TMA stores
          bool ok = true;
          for (int h = 0; h < passes && ok; ++h) {
            const int nw = min(2, vnt - 2 * h);            // column tiles of this pass
            for (int kc = 0; kc < nkc; ++kc) {
              ok = wait_bar(env, smem_u32(&bars.op_empty[op_st]), op_ph ^ 1u, 0x90 + op_st);
              if (!ok) break;
              const uint32_t bar = smem_u32(&bars.op_full[op_st]);
              const uint32_t dst = smem0 + op_st * stage;
              // A chunks of 128 x 64, and a W slab of 64 k x 128 or 256 columns in one load (2 or 4
              // panels; panels past the padded width are filled with zeros).  256 columns as two
              // loads: launches of slots 1 to 8 % slower (K_local 4096, hidden 1024, 2048 tokens
              // 123 us for 112).
              mbar_expect_tx(bar, rows * kPanel + nw * 2 * kWPanel);
              for (int r = 0; r < rows; ++r)
                tma_load_2d(dst + r * kPanel, &tmO, bar, kc * 64, (ft + r) * 128);
              tma_load_3d(dst + w_off, nw == 2 ? &tmW2 : &tmW, bar, 0, kc * 64, (base_out + 2 * h) * 2);
              if (++op_st == stages) { op_st = 0; op_ph ^= 1u; }
            }
          }
        }
        mbar_arrive(smem_u32(&bars.loads_done[slot_k]));
        MA_TASK_DONE(mode)
      }
    } else if (warp == 1) {
      // ============================================= MMA issuer of both attention tiles and of
      // every O_proj task.  A task is one elected lane's from start to end (see elect_one).
      uint32_t kv_slot = 0, kv_ph = 0, op_st = 0, op_ph = 0;
      uint32_t q_par = 0, p_par = 0, o_uses = 0, acc_uses = 0;     // a bit per tile / accumulator
      while (true) {
        MA_NEXT_TASK_WARP(d, mode)
        MA_DRAIN_IF_SWITCH(mode)
        if (mode == MODE_FA) {
          // A tile's chain softmax -> P V -> next Q K^T is what bounds the loop: the V tile
          // and the next K tile are looked at before P is waited for, and P V starts on the
          // first three quarters of P.  The tiles take turns, which keeps them half a period
          // apart: one tile's MMAs run under the other's softmax.
          const int nblk = d[TF_NBLK], nt = d[TF_NT];
          // The task's first operands are nearly always there: one look at all their barriers, a
          // lane each.  The lane that issues has seen one of them at most, and a vote orders no
          // memory: the __syncwarp hands it what the other lanes acquired.
          const uint32_t bar0 = smem_u32(lane == 0 ? &bars.q_full[0] : lane == 1 && nt == 2 ? &bars.q_full[1]
                                                                     : &bars.kv_full[kv_slot]);
          const uint32_t par0 = lane == 0 ? q_par & 1u : lane == 1 && nt == 2 ? q_par >> 1 : kv_ph;
          const bool there = __all_sync(0xffffffffu, mbar_test_wait(bar0, par0));
          __syncwarp();
          // Shared K/V stages: one slot per operand and key block.  Separate stages (p.sep):
          // nt slots, the i-th for tile i.  Two instances of the loop: a test of the layout in it
          // costs the shared one 2 %.  One elected lane runs the whole task, what every lane keeps
          // is advanced after it, and the parities are bits (arrays indexed by the tile lived in
          // local memory).  With a converged warp that waited and elected per batch the issuer
          // itself was late where the K tiles are: MHA, six ragged prompts of 13400 tokens,
          // attention stage 147 -> 137 us; shared stages the same time.
          auto run = [&](auto layout) {
            constexpr bool sep = decltype(layout)::value;
            const uint32_t per = sep ? nt : 1;
            uint32_t slot = kv_slot, ph = kv_ph;
            struct SlotAt { uint32_t slot, ph; };
            auto take = [&]() {                       // the next `per` slots of the ring
              const SlotAt r{slot, ph};
              slot += per;
              if (slot >= static_cast<uint32_t>(kKvSlots)) { slot -= kKvSlots; ph ^= 1u; }
              return r;
            };
            auto at = [&](SlotAt r, int i) {          // tile i's slot among them
              if (sep && i) {
                if (++r.slot == static_cast<uint32_t>(kKvSlots)) { r.slot = 0; r.ph ^= 1u; }
              }
              return r;
            };
            auto wait_kv = [&](SlotAt r, uint32_t site) {
              wait_bar(env, smem_u32(&bars.kv_full[0]) + r.slot * 8, r.ph, site + r.slot);
            };
            auto kv_at = [&](SlotAt r) { return smem0 + kSmKV + r.slot * kTile; };
            auto free_kv = [&](SlotAt r) { tc_commit(smem_u32(&bars.kv_empty[0]) + r.slot * 8); };
            SlotAt k = take();
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              if (i < nt) {
                if (!there) wait_bar(env, smem_u32(&bars.q_full[i]), (q_par >> i) & 1u, 0x20 + i);
                if (sep ? i == 1 || !there : i == 0 && !there) wait_kv(at(k, i), 0x30);
                tc_fence_after();
                issue_qk(tmem + kTmemS + i * 128, smem0 + kSmQ + i * kTile, kv_at(at(k, i)));
                tc_commit(smem_u32(&bars.s_full[i]));
                if (sep || i == nt - 1) free_kv(at(k, i));
                if (nblk == 1) tc_commit(smem_u32(&bars.q_empty[i]));
              }
            }
            uint32_t par = p_par;
            for (int jj = 0; jj < nblk; ++jj) {
              const bool has_next = (jj + 1 < nblk);
              const SlotAt v = take();
              if (has_next) k = take();
              if (!sep) {
                wait_kv(v, 0x40);
                if (has_next) wait_kv(k, 0x50);
              }
#pragma unroll
              for (int i = 0; i < 2; ++i) {
                if (i < nt) {
                  const uint32_t t_s = tmem + kTmemS + i * 128, t_o = tmem + kTmemO + i * 128;
                  const bool last_use = sep || i == nt - 1;
                  if (sep) wait_kv(at(v, i), 0x40);
                  // (the previous task's epilogue must have read O out)
                  if (jj == 0) wait_bar(env, smem_u32(&bars.o_free[i]), ((o_uses >> i) & 1u) ^ 1u, 0x68 + i);
                  wait_bar(env, smem_u32(&bars.p_part[i]), (par >> i) & 1u, 0x58 + i);
                  tc_fence_after();
                  issue_pv<0, 6>(t_o, t_s, kv_at(at(v, i)), jj > 0);
                  wait_bar(env, smem_u32(&bars.p_full[i]), (par >> i) & 1u, 0x60 + i);
                  tc_fence_after();
                  issue_pv<6, 8>(t_o, t_s, kv_at(at(v, i)), true);
                  if (has_next) {
                    if (sep) {
                      // The ring holds 1.25 key blocks here: the next K tile comes late, and P V must
                      // not wait for it (looked at before P, the stage lost up to 12 % on MHA).
                      free_kv(at(v, i));
                      wait_kv(at(k, i), 0x50);
                      tc_fence_after();
                    }
                    issue_qk(t_s, smem0 + kSmQ + i * kTile, kv_at(at(k, i)));
                    tc_commit(smem_u32(&bars.s_full[i]));
                    if (last_use) {
                      if (!sep) free_kv(at(v, i));
                      free_kv(at(k, i));
                    }
                    if (jj + 2 == nblk) tc_commit(smem_u32(&bars.q_empty[i]));
                  } else {
                    tc_commit(smem_u32(&bars.o_done[i]));
                    if (last_use) free_kv(at(v, i));
                  }
                }
              }
              par ^= 3u;
            }
          };
          if (elect_one()) {
            if (p.sep) run(Layout<true>{}); else run(Layout<false>{});
          }
          __syncwarp();
          const uint32_t used = static_cast<uint32_t>(2 * nblk) * (p.sep ? nt : 1) + kv_slot;
          kv_ph ^= (used / kKvSlots) & 1u;
          kv_slot = used % kKvSlots;
          const uint32_t tiles = nt == 2 ? 3u : 1u;
          q_par ^= tiles;
          o_uses ^= tiles;
          if (nblk & 1) p_par ^= tiles;
        } else if (mode == MODE_OPROJ) {
          const int vnt = d[TO_VNT], nrt = d[TO_NRT];
          const int nkc = p.K_local >> 6;
          const int rows = max(nrt, 1), passes = nrt ? 1 : (vnt + 1) >> 1;
          const bool two = d[TO_TWO] != 0;      // (the launch's, also for a last row tile alone)
          const uint32_t stage = two ? kOpStage2 : kOpStage, w_off = two ? 2 * kPanel : kPanel;
          const uint32_t stages = two ? 3 : 4;
          // One lane runs the whole task, waits included, and what every lane keeps is advanced after
          // it.  (A converged warp that waits and elects per stage, as for attention, takes 50 ns
          // longer for each: K_local 4096, hidden 1024, 2048 tokens in slots 128 us for 123.)
          if (elect_one()) {
            uint32_t st = op_st, ph = op_ph;
            for (int h = 0; h < passes; ++h) {
              const uint32_t idesc = make_idesc_bf16(128, min(2, vnt - 2 * h) * 128, 0, 1);
              for (int kc = 0; kc < nkc; ++kc) {
                wait_bar(env, smem_u32(&bars.op_full[st]), ph, 0xA0 + st);
                const uint32_t a16 = (smem0 + st * stage) >> 4;
                const uint32_t w16 = a16 + (w_off >> 4);
                // accumulator h + r: row tile r's (the passes of a slot have one row tile)
                for (int r = 0; r < rows; ++r) {
                  if (kc == 0)
                    wait_bar(env, smem_u32(&bars.acc_free[h + r]), ((acc_uses >> (h + r)) & 1u) ^ 1u,
                             0xA8 + h + r);
                  tc_fence_after();
                  const uint32_t a16r = a16 + r * (kPanel >> 4);
#pragma unroll
                  for (int kk = 0; kk < 4; ++kk)
                    mma_ss(tmem + (h + r) * 256, smem_desc_at(kDescK, a16r + kk * 2),
                           smem_desc_at(kDescWmn, w16 + kk * 128), idesc,
                           (kc > 0 || kk > 0) ? 1u : 0u);
                  if (r + 1 == rows) tc_commit(smem_u32(&bars.op_empty[st]));
                  if (kc + 1 == nkc) tc_commit(smem_u32(&bars.acc_full[h + r]));
                }
                if (++st == stages) { st = 0; ph ^= 1u; }
              }
            }
          }
          __syncwarp();
          const uint32_t end = op_st + static_cast<uint32_t>(passes * nkc);
          op_ph ^= (end / stages) & 1u;
          op_st = end % stages;
          acc_uses ^= (rows == 2 || passes == 2) ? 3u : 1u;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&bars.task_empty[slot_k]));
        arrived ^= 1u << slot_k;
        prev_mode = mode; prev_k = slot_k; slot_k ^= 1;
      }
    } else if (warp == 3 && lane == 0) {
      // ==================================== attention output stores: O_scratch[ft, :, head, :]
      // (a warp of their own, so that no softmax warp waits for a store to complete)
      uint32_t st_par = 0;
      while (true) {
        MA_NEXT_TASK(d, mode)
        if (mode == MODE_FA) {
          const int ft = d[T_FT], head0 = d[TF_HEAD0], nt = d[TF_NT];
          for (int i = 0; i < nt; ++i) {
            if (!wait_bar(env, smem_u32(&bars.o_staged[i]), (st_par >> i) & 1u, 0x88 + i)) break;
            st_par ^= 1u << i;
            if (d[TF_FIN0 + i]) {       // (else a part of the keys, and not the last)
              const uint32_t stg = smem0 + kSmQ + i * kTile;
              tma_store_2d(&tmO, stg, (head0 + i) * 128, ft * 128);
              tma_store_2d(&tmO, stg + kPanel, (head0 + i) * 128 + 64, ft * 128);
              tma_store_commit();
              tma_store_wait_read();
            }
            mbar_arrive(smem_u32(&bars.q_empty[i]));     // the producer may refill this Q buffer
          }
          tma_store_wait_all();
          fence_proxy_async_all();     // O_scratch is read back by TMA loads of other CTAs (the
                                       // scheduler's fence covers them)
        }
        MA_TASK_DONE(mode)
      }
    }
    __syncwarp();
  } else {
    // ====================================================================== compute warps
    reg_inc<208>();
    const int wg = (warp - 4) >> 2;                            // compute warpgroup 0 / 1
    const int row = (warp & 3) * 32 + lane;                    // TMEM lane == tile row
    const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
    uint32_t s_par = 0, o_par = 0, acc_par = 0;
    while (true) {
      MA_NEXT_TASK_WARPGROUP(d, mode)
      if (mode == MODE_FA && wg < d[TF_NT]) {
        // -------------------------------------------- softmax + epilogue of tile `wg`
        const int valid_m = d[TF_VALID];
        const int k_len = d[TF_KLEN], offset = d[TF_OFFSET], nblk = d[TF_NBLK], mb = d[TF_MB];
        const uint32_t t_s = tmem + kTmemS + wg * 128 + lane_base;
        const uint32_t t_o = tmem + kTmemO + wg * 128 + lane_base;
        const uint32_t bar_s = smem_u32(&bars.s_full[wg]);
        const uint32_t bar_pp = smem_u32(&bars.p_part[wg]), bar_p = smem_u32(&bars.p_full[wg]);
        const float sl2 = p.scale_log2;
        // last kv position this row may see (bottom-right causal, clipped to k_len)
        const int lim_abs = min(mb * 128 + row + offset, k_len - 1);
        float m_ref = -INFINITY;      // max the exponent is taken against (raw score units)
        float l_run = 0.f;            // running row sum of exp2
        for (int jj = 0; jj < nblk; ++jj) {
          const int j = nblk - 1 - jj;
          wait_bar(env, bar_s, s_par, 0x70 + wg);
          s_par ^= 1u;
          tc_fence_after();
          // Four chunks of 32 scores.  The last is read for the maximum and read again for its
          // exponentials: held all along it takes the registers that the rest of the kernel
          // needs (spilled, the attention stage lost 3 %).
          uint32_t s[3][32], last[32];
#pragma unroll
          for (int c = 0; c < 3; ++c) tmem_ld32(t_s + c * 32, s[c]);
          tmem_ld32(t_s + 96, last);
          tc_wait_ld();
          const bool need_mask = ((j + 1) * 128 - 1 > mb * 128 + offset) || ((j + 1) * 128 > k_len);
          const int lim = lim_abs - j * 128;      // columns > lim are masked
          auto mask = [&](uint32_t (&x)[32], int c) {
#pragma unroll
            for (int kx = 0; kx < 32; ++kx)
              if (c * 32 + kx > lim) x[kx] = 0xff800000u;   // -inf
          };
          if (need_mask) {
            mask(s[0], 0);
            mask(s[1], 1);
            mask(s[2], 2);
            mask(last, 3);
          }
          float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
          for (int kx = 0; kx < 32; kx += 2) {
#pragma unroll
            for (int c = 0; c < 3; ++c)
              mx[c] = fmax3(mx[c], __uint_as_float(s[c][kx]), __uint_as_float(s[c][kx + 1]));
            mx[3] = fmax3(mx[3], __uint_as_float(last[kx]), __uint_as_float(last[kx + 1]));
          }
          const float m_blk = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
          // lazy rescale: move the reference max only when it would grow by > 2^8
          const bool grow = (m_blk > -INFINITY) &&
                            ((m_ref == -INFINITY) || ((m_blk - m_ref) * sl2 > kRescaleThreshold));
          if (__any_sync(0xffffffffu, grow)) {
            float o_scale = 1.f;
            if (grow) {
              o_scale = (m_ref == -INFINITY) ? 0.f : ex2((m_ref - m_blk) * sl2);
              m_ref = m_blk;
              l_run *= o_scale;
            }
            if (jj > 0) {
              // the P V MMA of the previous block completed before this block's S was
              // committed (in-order tensor pipe), so O is quiescent here
#pragma unroll 1
              for (int c = 0; c < 8; ++c) {
                uint32_t o[16];
                tmem_ld16(t_o + c * 16, o);
                tc_wait_ld();
#pragma unroll
                for (int kx = 0; kx < 16; ++kx)
                  o[kx] = __float_as_uint(__uint_as_float(o[kx]) * o_scale);
                tmem_st16(t_o + c * 16, o);
              }
            }
          }
          // Scale-and-subtract and the row sums work on packed pairs (fma / add on two
          // floats per instruction).  P goes out chunk by chunk over the S columns already
          // in registers; three quarters of it are handed to the issuer while the last
          // quarter's exponentials run.
          const float neg_m = (m_ref == -INFINITY) ? 0.f : -m_ref * sl2;
          const uint64_t sl2x2 = pack_f32x2(sl2, sl2), negm2 = pack_f32x2(neg_m, neg_m);
          uint64_t sum2[2] = {pack_f32x2(0.f, 0.f), pack_f32x2(0.f, 0.f)};
          auto exps = [&](const uint32_t (&x)[32], uint32_t (&pk)[16]) {
#pragma unroll
            for (int kx = 0; kx < 16; ++kx) {
              const uint64_t a2 = fma_f32x2(
                  pack_f32x2(__uint_as_float(x[2 * kx]), __uint_as_float(x[2 * kx + 1])), sl2x2,
                  negm2);
              float a0, a1;
              unpack_f32x2(a2, a0, a1);
              const float e0 = ex2(a0), e1 = ex2(a1);
              sum2[kx & 1] = add_f32x2(sum2[kx & 1], pack_f32x2(e0, e1));
              pk[kx] = pack_bf16x2(e0, e1);
            }
          };
          {
            uint32_t pk[16];
            exps(s[0], pk);
            tmem_st16(t_s, pk);
          }
          uint32_t x3[32];
          tmem_ld32(t_s + 96, x3);                // (P takes columns 0-63 only)
#pragma unroll
          for (int c = 1; c < 3; ++c) {
            uint32_t pk[16];
            exps(s[c], pk);
            tmem_st16(t_s + c * 16, pk);
          }
          {
            uint32_t pk[16];
            tc_wait_ld();
            if (need_mask) mask(x3, 3);
            exps(x3, pk);
            tc_wait_st();                         // (stores 0-2 were issued a quarter ago)
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_pp);
            tmem_st16(t_s + 48, pk);
          }
          tc_wait_st();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar_p);   // 4 arrivals, not 128 serialised ones
          float s0, s1, s2, s3;
          unpack_f32x2(sum2[0], s0, s1);
          unpack_f32x2(sum2[1], s2, s3);
          l_run += (s0 + s1) + (s2 + s3);
        }
        // epilogue: O / l -> bf16 -> O_scratch[ft, row, head, :]; tail rows are zeros
        wait_bar(env, smem_u32(&bars.o_done[wg]), o_par, 0x80 + wg);
        o_par ^= 1u;
        tc_fence_after();
        const uint32_t stg = smem0 + kSmQ + wg * kTile;
        if (d[TF_PARTS] > 1) {
          finish_part(p, s_desc[slot_k], wg, row, t_o, stg, smem_u32(&bars.o_free[wg]), m_ref, l_run);
        } else {
          const float inv = (row < valid_m && l_run > 0.f) ? (1.f / l_run) : 0.f;
          // O / l -> bf16 -> this tile's Q buffer (free: every Q K^T of the task is done),
          // then two TMA stores of 128 rows x 64 columns into O_scratch[ft, :, head, :].
#pragma unroll
          for (int hh = 0; hh < 2; ++hh) {
            uint32_t o[2][32];
            tmem_ld32(t_o + hh * 64, o[0]);
            tmem_ld32(t_o + hh * 64 + 32, o[1]);
            tc_wait_ld();
            if (hh == 1) {            // all of O is in registers: the next task may overwrite it
              tc_fence_before();
              __syncwarp();
              if (lane == 0) mbar_arrive(smem_u32(&bars.o_free[wg]));
            }
            stage_row(stg + hh * kPanel, row, 0, o[0], inv);
            stage_row(stg + hh * kPanel, row, 32, o[1], inv);
          }
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&bars.o_staged[wg]));   // warp 3 stores the tile
      } else if (mode == MODE_OPROJ) {
        const int ft0 = d[T_FT], base_out = d[TO_BASE], vnt = d[TO_VNT], nrt = d[TO_NRT];
        const bool leader = ((warp & 3) == 0 && lane == 0);
        const uint32_t stg = smem0 + kSmOpStaging + wg * kPanel;   // [128 rows][64 cols] bf16
        bool direct = false;
        // rows of the task's row tiles, looked up while the product runs (by the scheduler they were
        // two trips to L2 of every claim)
        auto rows_of = [&](int ft) {
          const int b = p.fa_b[ft];
          return min(128, p.cu_q[b + 1] - p.cu_q[b] - p.fa_mb[ft] * 128);
        };
        const int rows0 = rows_of(ft0), rows1 = nrt == 2 ? rows_of(ft0 + 1) : 0;
        // Accumulator h holds row tile h of the task, or columns 2h and 2h + 1 of a slot; this
        // warpgroup's 128 columns of it go out as two panels of 64, by way of bf16 words in
        // registers.
        auto wait_acc = [&](int h) {
          wait_bar(env, smem_u32(&bars.acc_full[h]), (acc_par >> h) & 1u, 0xB0 + h);
          acc_par ^= 1u << h;
          tc_fence_after();
        };
        auto free_acc = [&](int h) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&bars.acc_free[h]));
        };
        auto load_panel = [&](int h, int hh, uint32_t (&pk)[32]) {
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            uint32_t r[32];
            tmem_ld32(tmem + lane_base + h * 256 + wg * 128 + hh * 64 + c * 32, r);
            tc_wait_ld();
#pragma unroll
            for (int kx = 0; kx < 16; ++kx)
              pk[c * 16 + kx] =
                  pack_bf16x2(__uint_as_float(r[2 * kx]), __uint_as_float(r[2 * kx + 1]));
          }
        };
        auto emit_panel = [&](int h, int hh, const uint32_t (&pk)[32]) {
          const int ft = nrt ? ft0 + h : ft0;
          const int out_n = base_out + (nrt ? 0 : 2 * h) + wg;
          const int valid_m = (nrt && h) ? rows1 : rows0;
          if (valid_m == 128) {
            // full row tile: stage 64 columns, one TMA store (clipped at `hidden`)
            if (leader) tma_store_wait_read();
            named_bar_sync(1 + wg, 128);
            stage_panel_row(stg, row, pk);
            fence_proxy_async_smem();
            named_bar_sync(1 + wg, 128);
            if (leader) {
              tma_store_2d(&tmC, stg, out_n * 128 + hh * 64, ft * 128);
              tma_store_commit();
            }
            return;
          }
          // last tile of a sequence: rows past valid_m must stay untouched
          direct = true;
          if (row >= valid_m) return;
          const int col0 = out_n * 128 + hh * 64;
          uint16_t* dst = p.csym + static_cast<size_t>(ft * 128 + row) * p.num_out * 128 + col0;
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            if (col0 + c * 8 + 8 <= p.hidden) {
              reinterpret_cast<uint4*>(dst)[c] =
                  make_uint4(pk[4 * c], pk[4 * c + 1], pk[4 * c + 2], pk[4 * c + 3]);
            } else {
#pragma unroll
              for (int kx = 0; kx < 8; ++kx)
                if (col0 + c * 8 + kx < p.hidden)
                  dst[c * 8 + kx] = static_cast<uint16_t>(pk[4 * c + (kx >> 1)] >> ((kx & 1) * 16));
            }
          }
        };
        // Both panels leave TMEM before the first is written out, so that the accumulator is
        // soon free for the next task's MMAs.  (All of the second accumulator as well, before
        // the first is written, takes more registers than there are: spilled, 129 us for 105.)
        const int halves = nrt ? nrt : (vnt + 1) >> 1;
#pragma unroll 1
        for (int h = 0; h < halves; ++h) {
          const bool mine = (nrt ? 0 : 2 * h) + wg < vnt;
          uint32_t pa[32], pb[32];
          wait_acc(h);
          if (mine) {
            load_panel(h, 0, pa);
            load_panel(h, 1, pb);
          }
          free_acc(h);
          if (mine) {
            emit_panel(h, 0, pa);
            emit_panel(h, 1, pb);
          }
        }
        // Ordering towards other CTAs / ranks: the leader waits for its TMA stores, rows
        // written directly get a gpu-scope fence; the one system-scope fence per task is
        // the scheduler's, after it has seen every warp arrive.  (A system fence by each of
        // the 256 threads costs tens of microseconds per task while NVLink is busy.)
        // Without an AllReduce nobody looks before the launch has ended: the leader waits only until
        // its staging has been read.
        if (without_ar(p)) {
          if (leader) tma_store_wait_read();
        } else {
          if (leader) {
            tma_store_wait_all();
            fence_proxy_async_all();
          }
          if (direct) __threadfence();
        }
      } else if (mode == MODE_AR) {
        ar_slot(p, d[T_FT], d[TO_BASE], d[TO_VNT], tid - 128, 256);
        if (lane == 0) __threadfence_system();   // one per warp; the scheduler fences again
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&bars.task_empty[slot_k]));
      arrived ^= 1u << slot_k;
      prev_mode = mode; prev_k = slot_k; slot_k ^= 1;
    }
  }
#undef MA_TASK_FULL
#undef MA_NEXT_TASK_IF
#undef MA_NEXT_TASK
#undef MA_NEXT_TASK_WARP
#undef MA_NEXT_TASK_WARPGROUP
#undef MA_TASK_FULL_OR_END
#undef MA_DRAIN_IF_SWITCH
#undef MA_TASK_DONE

  // ------------------------------------------------------------------ exit protocol
  // The reference ends with grid barrier -> every CTA clears the per-launch control state
  // -> grid barrier -> cross-rank barrier (fused_fa_oproj_ar.py:1154-1177).  Here each CTA
  // only counts itself out; the last one to do so (every other CTA has stopped touching
  // the control words by then) clears the state at full capacity, resets the counter and,
  // with tp > 1, runs the cross-rank barrier that also opens the next launch.  No CTA
  // waits for another one.
  __syncthreads();
  if (!s_abort) {
    __shared__ int s_last;
    if (tid == 0) {
      fence_acq_rel_gpu();
      s_last = (atom_add_relaxed_gpu(p.sync_ctrl + S_GS_QUIESCE, 1u) == gridDim.x - 1) ? 1 : 0;
      if (s_last) fence_acq_rel_gpu();
    }
    __syncthreads();
    if (s_last) {
      for (int i = tid; i < p.max_row_tiles; i += kThreads) {
        p.head_ready[i] = 0u;
        p.oproj_queue[i] = 0u;      // (an entry per row-tile group at most)
      }
      for (int i = tid; i < p.max_owner_slots; i += kThreads) p.ready_count[i] = 0u;
      for (int i = tid; i < p.max_owner_words; i += kThreads) p.ar_done_bits[i] = 0ull;
      if (tid < 8) p.ctrl[tid] = 0u;
      if (tid == 8) p.sync_ctrl[S_GS_QUIESCE] = 0u;
      if (p.tp > 1) __threadfence_system();
      if (p.tp > 1 && !(p.flags & (1u | 16u))) rank_barrier(env);
    }
  }

  if (s_abort) {
    // A wait ran out (here or in another CTA) and the roles left their loops wherever they
    // were: MMAs, TMA loads and TMA stores of this CTA may still be in flight, and none of
    // them may outlive the CTA's shared memory and TMEM.  Each issuer waits (bounded) for
    // its own MMAs, the store leaders for their bulk stores, and everybody gives loads
    // already issued 100 us to land (nothing issues new ones any more).
    if (warp == 1) {
      const uint32_t bar = smem_u32(&bars.drain);
      __syncwarp();
      if (elect_one()) tc_commit(bar);      // (the lane that issued the MMAs)
      __syncwarp();
      for (int it = 0; it < (1 << 20); ++it)
        if (mbar_try_wait(bar, 0)) break;
    }
    if ((warp == 3 || warp == 4 || warp == 8) && lane == 0) tma_store_wait_all();
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 100000ull) {}
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, 512);
}

// ---------------------------------------------------------------------- host launcher
cudaError_t launch_fused_prefill(const CUtensorMap* maps, const KParams& kp, int num_ctas,
                                 cudaStream_t stream) {
  static bool attr_set[64] = {};
  int dev = 0;
  cudaError_t err = cudaGetDevice(&dev);
  if (err != cudaSuccess) return err;
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    err = cudaFuncSetAttribute(fused_prefill_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               kSmemDynamic);
    if (err != cudaSuccess) return err;
    attr_set[dev] = true;
  }
  return launch_behind(fused_prefill_kernel, num_ctas, kThreads, kSmemDynamic, stream, maps[0], maps[1], maps[2],
                       maps[3], maps[4], maps[5], maps[6], kp);
}

cudaError_t fused_prefill_attributes(cudaFuncAttributes* out) {
  return cudaFuncGetAttributes(out, fused_prefill_kernel);
}

}  // namespace ma
