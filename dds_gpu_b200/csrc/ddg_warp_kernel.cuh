// The warp kernel: one search per warp (ddg_warp.cuh), warps fed from the job queue.
//
// A block is up to WARP_MAX searchers on an SM of its own. A searcher takes a job, runs it to
// its end and takes the next; searchers share nothing but the queue, so there is no
// barrier in the loop and the SM's schedulers always have the other warps to issue from.
// Searcher w of block b owns the TT slice, the stack area and the save slot of lane
// b * warps + w.
//
// What bounds it: instruction fetch and issue. A node takes about 434 warp instructions (a
// lane of batch_kernel took ~3,030 thread instructions on one thread of a warp that was
// 35 % full), and 16 warps on an SM issue as much as 32 (1.8 a cycle), since warps that
// stand at different places of the code share few fetches. Measured against batch_kernel
// (block phases, 512 lanes to an SM): random 13-card deals with every SM full 1.18 against
// 0.70 G nodes/s; one job alone on an SM about 1 M against 0.15 M nodes/s; 240 quick
// 13-card deals 109 against 1,405 ms; 65,536 six-card endings 158 against 376 ms; 1,200
// nine-card endings 135 against 1,117 ms; the 20 leads of a five-card ending asked one by
// one 3.2 against 19.2 ms. batch_kernel stays for helping and for its own options.
#pragma once
#include "ddg_kernel.cuh"
#include "ddg_warp.cuh"

#ifndef DDG_TT_SIG

namespace ddg {

enum { WARP_MAX = 32 };

// A searcher between two slices of a resumable solve, in its lane's save slot. (The frames
// below the top go to the lane's stack area.)
struct WarpSave {
  uint16_t m[16], all[4], now[4];
  u32 trick;
  u32 code[4];
  int8_t trump, leader, nplayed, left, need, sp;
  WarpJob job;
};
static_assert(sizeof(WarpSave) <= sizeof(LaneSave), "a searcher's state fits its lane's save slot");

struct WarpBlock {
  BatchArgs args;
  u64 idle_since;  // stream: global time since which no searcher had work (0 = busy)
  int polling;     // stream: a searcher of the block is looking at the ring
  int busy;        // stream: searchers with a job
  int idle_exit;   // stream: waiting searchers end (1: nothing will come, 2: stopped by the host)
  unsigned polls;  // stream: looks at the ring
  int running;     // searchers that did not end idle
  unsigned long long nodes, jobs_done, total[WCNT_COUNT];
  WarpMem warp[1];  // as many as the block has warps
};
inline size_t warp_smem(int warps) { return sizeof(WarpBlock) + sizeof(WarpMem) * (size_t)(warps - 1); }

struct WarpEnv {
  WarpBlock* sh;
  TTBucket* tt;
  u64 t_end;
  long long lane;
  int wid;

  __device__ __forceinline__ TTBucket* table() { return tt; }
  __device__ __forceinline__ u32 mask() const { return (1u << sh->args.tt_log2) - 1; }
  __device__ __forceinline__ long long out_row(const WarpJob& j) const {
    return sh->args.ring ? (j.deal & sh->args.ring_mask) : j.deal;
  }
  __device__ __forceinline__ long long entry(const WarpJob& j) const { return out_row(j) * 20 + j.strain * 4 + j.decl; }
  // Ring slots are rewritten while the kernel runs: their values come from L2.
  __device__ __forceinline__ int seed(const WarpJob& j) const {
    const BatchArgs& a = sh->args;
    if (a.mode == MODE_STEP) return (int)__ldcg(reinterpret_cast<const signed char*>(a.seeds) + entry(j));
    return a.first_target ? a.first_target : 7;
  }
  __device__ __forceinline__ int root_hint(const WarpJob& j) const {
    const BatchArgs& a = sh->args;
    return a.hint20 ? (int)__ldcg(reinterpret_cast<const signed char*>(a.hint20) + entry(j)) : -1;
  }
  __device__ __forceinline__ void root_best(const WarpJob& j, int card) {
    if (sh->args.best20 && (threadIdx.x & 31) == 0) sh->args.best20[entry(j)] = (int8_t)card;
  }
  __device__ __forceinline__ void answer(const WarpJob& j, int ns) {
    if ((threadIdx.x & 31) == 0) sh->args.out20[entry(j)] = (uint8_t)((j.decl & 1) == 0 ? ns : 13 - ns);
  }
  __device__ __forceinline__ void job_done(WarpJob& j) {
    const BatchArgs& a = sh->args;
    if ((threadIdx.x & 31) == 0) {
      if (a.job_nodes) a.job_nodes[j.job] = j.nodes - j.start_nodes;
      if (a.job_end_ns) a.job_end_ns[j.job] = global_ns();
      j.jobs_done++;
      if (a.ring) {
        stream_deal_done(a, j.deal);
        atomicSub(&sh->busy, 1);
      }
    }
    __syncwarp();
  }

  // The stream's next job, in thread 0: 1 taken, 0 nothing will come, -1 stopped. One
  // searcher of a block looks at the ring at a time; the others wait longer the more of
  // the block's searchers are busy, so that deals spread over the SMs.
  __device__ __noinline__ int stream_next(unsigned long long& job) {
    const BatchArgs& a = sh->args;
    volatile int* vbusy = &sh->busy;
    volatile int* vexit = &sh->idle_exit;
    volatile u64* vsince = &sh->idle_since;
    DevEnv q;
    q.a = &a;
    for (;;) {
      if (*vexit) return *vexit == 1 ? 0 : -1;
      if (atomicCAS(&sh->polling, 0, 1) == 0) {
        int got = -2;
        const bool closing = *reinterpret_cast<const volatile int*>(a.closing) != 0;
        // The host's flag costs a read over the bus: looked at in every 256th look, here
        // only (a read by every waiting searcher held up the whole kernel: 400 deals took
        // 1.76 s).
        if ((sh->polls++ & 255u) == 255u && stop_requested(a, 0)) {
          *vexit = 2;
          got = -1;
        } else if (closing && !q.stream_more()) {
          *vexit = 1;  // nothing more will come for any searcher
          got = 0;
        } else if (q.stream_take(job)) {
          atomicAdd(&sh->busy, 1);
          *vsince = 0;
          got = 1;
        } else if (*vbusy == 0) {
          const u64 now = global_ns();
          if (!*vsince) *vsince = now;
          else if (now - *vsince > a.idle_ns) *vexit = 1;
        } else {
          *vsince = 0;
        }
        __threadfence_block();
        atomicExch(&sh->polling, 0);
        if (got != -2) return got;
      }
      __nanosleep(1000u + 500u * (unsigned)*vbusy);
    }
  }

  __device__ __forceinline__ bool take(WarpState& w, const WarpIds& id, WarpMem& sm) {
    const BatchArgs& a = sh->args;
    WarpJob& j = sm.job;
    __syncwarp();
    int got = 1;
    unsigned long long job = 0;
    if (id.t == 0) {
      if (a.ring) {
        got = stream_next(job);
      } else if ((t_end && global_ns() > t_end) || ((j.jobs_done & 15u) == 15u && stop_requested(a, 0))) {
        got = -1;  // (the host's flag costs a read over the bus: looked at for every 16th job)
      } else {
        // The first job of the launch is dealt round-robin over the blocks, so that a small
        // batch spreads over every SM; later ones come from the shared counter.
        const long long rr = (long long)wid * gridDim.x + blockIdx.x;
        if (j.job < 0 && rr < a.rr_jobs) job = (unsigned long long)rr;
        else job = atomicAdd(a.next_job, 1ull) + (unsigned long long)a.rr_jobs;
        if ((long long)job >= a.n_jobs) got = 0;
      }
      if (got != 1) {
        j.stage = got == 0 ? ST_IDLE : ST_TAKE;
      } else {
        j.job = (long long)job;
        j.deal = j.job / a.jpd;
        const int sub = (int)(j.job - j.deal * a.jpd);
        j.strain = (int8_t)(a.jpd == 5 ? sub : sub >> 2);
        j.decl = (int8_t)(a.jpd == 5 ? 0 : sub & 3);
        j.last_decl = (int8_t)(a.jpd == 5 ? 3 : sub & 3);
        if (a.one_job) {
          j.strain = (int8_t)a.one_strain;
          j.decl = (int8_t)(a.one_decl >= 0 ? a.one_decl : 0);
          j.last_decl = (int8_t)(a.one_decl >= 0 ? a.one_decl : 3);
        }
        j.mode = (int8_t)a.mode;
        j.start_nodes = j.nodes;
        if (a.job_start_ns) a.job_start_ns[j.job] = global_ns();
      }
    }
    got = __shfl_sync(0xFFFFFFFFu, got, 0);
    if (got != 1) return false;
    __syncwarp();
    const long long row = a.ring ? (j.deal & a.ring_mask) : j.deal;
    const unsigned short* h = reinterpret_cast<const unsigned short*>((a.ring ? a.ring : a.hands) + row * 4);
    w.m = (a.ring ? __ldcg(h + 4 * id.p + id.s) : h[4 * id.p + id.s]) & 0x1FFFu;
    w.all = w.now = w_shfl(w.m, id.s) | w_shfl(w.m, 4 + id.s) | w_shfl(w.m, 8 + id.s) | w_shfl(w.m, 12 + id.s);
    w.code = w_build_code(w, id);
    const int cards = (int)w_add(id.t < 4 ? (u32)w_popc(w.m) : 0u);
    w.trump = strain_trump(j.strain);
    // A new TT generation; at the wrap all tags are cleared, by the whole warp.
    w.gen++;
    if (w.gen >= (1u << GEN_BITS)) {
      const u32 n = (mask() + 1) * 4;
      for (u32 k = id.t; k < n; k += 32) reinterpret_cast<uint4*>(tt[k >> 2].tag)[k & 3] = make_uint4(0, 0, 0, 0);
      w.gen = 1;
    }
    if (id.t == 0) j.cards = (int8_t)(cards > 13 ? 13 : cards);
    __syncwarp();
    return true;
  }

  __device__ __forceinline__ bool stop(WarpState& w, const WarpIds& id, WarpMem& sm) {
    const bool look = (w.nodes & 1023u) == 1023u;  // the host's flag costs a read over the bus
    if (!look && !t_end) return false;
    int end = 0;
    if (id.t == 0) {
      if (look) end = stop_requested(sh->args, t_end);
      else end = global_ns() > t_end;
    }
    end = __shfl_sync(0xFFFFFFFFu, end, 0);
    if (end || (w.nodes & 0xFFFFu) == 0xFFFFu) w_flush(w, id, sm);
    if (end && id.t == 0) sm.job.stage = ST_ENTER;
    return end != 0;
  }
};

__global__ void __launch_bounds__(WARP_MAX * 32, 1) warp_kernel(BatchArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  WarpBlock& sh = *reinterpret_cast<WarpBlock*>(smem_raw);
  const int wid = threadIdx.x >> 5, t = threadIdx.x & 31, warps = blockDim.x >> 5;
  const long long lane = (long long)blockIdx.x * warps + wid;
  const u64 t_end = a.slice_ns ? global_ns() + a.slice_ns : 0;
  if (threadIdx.x == 0) {
    sh.args = a;
    sh.idle_since = 0;
    sh.polling = sh.busy = sh.idle_exit = sh.running = 0;
    sh.polls = 0;
    sh.nodes = sh.jobs_done = 0;
    for (int k = 0; k < WCNT_COUNT; k++) sh.total[k] = 0;
  }
  __syncthreads();
  const WarpIds id = {t, t & 3, (t >> 2) & 3};
  WarpMem& sm = sh.warp[wid];
  WarpState w;
  memset(&w, 0, sizeof(w));
  w.gen = a.lane_gen[lane];
  WarpFrame* stack = reinterpret_cast<WarpFrame*>(a.stacks) + lane * STACK_DEPTH;
  WarpSave* sv = a.save ? reinterpret_cast<WarpSave*>(a.save + lane) : nullptr;
  if (a.resume) {
    w.m = sv->m[t & 15];
    w.all = sv->all[id.s];
    w.now = sv->now[id.s];
    w.trick = sv->trick;
    w.trump = sv->trump;
    w.leader = sv->leader;
    w.nplayed = sv->nplayed;
    w.left = sv->left;
    w.need = sv->need;
    w.code = sv->code[id.s];
    w.sp = sv->sp;
    for (int k = t; k < w.sp * 4; k += 32) reinterpret_cast<uint4*>(sm.fr)[k] = reinterpret_cast<const uint4*>(stack)[k];
    if (t == 0) {
      sm.job = sv->job;
      sm.job.start_nodes = 0ull - (sm.job.nodes - sm.job.start_nodes);
    }
  } else if (t == 0) {
    memset(&sm.job, 0, sizeof(sm.job));
    sm.job.job = -1;
    sm.job.stage = ST_TAKE;
  }
  __syncwarp();
  if (t == 0) {
    sm.job.nodes = 0;
    sm.job.jobs_done = 0;
    for (int k = 0; k < WCNT_COUNT; k++) sm.job.total[k] = 0;
  }
  __syncwarp();
  WarpEnv env;
  env.sh = &sh;
  env.tt = a.tt + (lane << a.tt_log2);
  env.t_end = t_end;
  env.lane = lane;
  env.wid = wid;
  if (sm.job.stage != ST_IDLE) w_run(w, id, sm, env);
  __syncwarp();
  // The generation, the totals and, for a resumable solve, the search as it stands.
  if (t == 0) {
    a.lane_gen[lane] = w.gen;
    if (sm.job.stage != ST_IDLE) atomicAdd(&sh.running, 1);
    atomicAdd(&sh.nodes, (unsigned long long)sm.job.nodes);
    atomicAdd(&sh.jobs_done, (unsigned long long)sm.job.jobs_done);
    for (int k = 0; k < WCNT_COUNT; k++) atomicAdd(&sh.total[k], (unsigned long long)sm.job.total[k]);
  }
  if (sv) {
    if (t < 16) sv->m[t] = (uint16_t)w.m;
    if (t < 4) {
      sv->all[t] = (uint16_t)w.all;
      sv->now[t] = (uint16_t)w.now;
      sv->code[t] = w.code;
    }
    for (int k = t; k < w.sp * 4; k += 32) reinterpret_cast<uint4*>(stack)[k] = reinterpret_cast<const uint4*>(sm.fr)[k];
    if (t == 0) {
      sv->trick = w.trick;
      sv->trump = (int8_t)w.trump;
      sv->leader = (int8_t)w.leader;
      sv->nplayed = (int8_t)w.nplayed;
      sv->left = (int8_t)w.left;
      sv->need = (int8_t)w.need;
      sv->sp = (int8_t)w.sp;
      sv->job = sm.job;
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    atomicAdd(a.counters + CNT_NODES, sh.nodes);
    atomicAdd(a.counters + CNT_PROBES, sh.total[WCNT_PROBES]);
    atomicAdd(a.counters + CNT_HITS, sh.total[WCNT_HITS]);
    atomicAdd(a.counters + CNT_STORES, sh.total[WCNT_STORES]);
    atomicAdd(a.counters + CNT_TT_BYTES, sh.total[WCNT_BYTES] + 64 * sh.total[WCNT_PROBES] + 16 * sh.total[WCNT_READS]);
    atomicAdd(a.counters + CNT_ENTRY_READS, sh.total[WCNT_READS]);
    atomicAdd(a.counters + CNT_BOUNDS, sh.total[WCNT_BOUNDS]);
    atomicAdd(a.counters + CNT_JOBS_DONE, sh.jobs_done);
    if (!sh.running) atomicAdd(a.counters + CNT_BLOCKS_DONE, 1ull);
  }
}

}  // namespace ddg

#endif  // DDG_TT_SIG
