// The warp kernel: one search per warp (ddg_warp.cuh), warps fed from the job queue.
//
// A block is up to WARP_MAX searchers on an SM of its own. A searcher takes a job, runs it to
// its end and takes the next; searchers share nothing but the queue, so there is no
// barrier in the loop and the SM's schedulers always have the other warps to issue from.
// Searcher w of block b owns the TT slice, stack area and save slot number b * warps + w.
//
// What bounds it: on a full SM the integer pipe (85 % of its cycles busy) and instruction fetch
// (2.6 of 11.2 stall cycles an issue; 2.76 instructions a cycle); alone on an SM one warp's chain of instructions, 1,500 cycles a node, of which the
// table's memory is a twentieth. Measured against batch_kernel (block phases, 512 lanes to
// an SM): random 13-card deals with every SM full 2.36 against 0.70 G nodes/s; one job
// alone on an SM 1.3 M against 0.15 M nodes/s; 240 quick 13-card deals 75 against 1,381 ms;
// 65,536 six-card endings 122 against 371 ms; 1,200 nine-card endings (a job per lead) 95
// against 1,074 ms; the 20 leads of a five-card ending asked one by one 2.8 against 23 ms.
// batch_kernel stays for helping and for its own options.
#pragma once
#include "ddg_kernel.cuh"
#include "ddg_shape.hpp"
#include "ddg_warp.cuh"

#ifndef DDG_TT_SIG

namespace ddg {

// A launch of at most WARP_FEW searchers an SM takes a build with 104 registers a thread instead
// of 64. Measured on hard 13-card deals, nodes/s of the GPU with n searches on each of 148 SMs,
// this build against the other: n = 1: 200 against 193 M, 4: 784 / 748, 8: 1,375 / 1,348, 12: 1,817
// / 1,772, 16: 2,045 / 2,004. From 17 on the other's further searches are worth more than 16 of
// these with the rest waiting (2,050 M): 17: 2,073, 20: 2,172, 24: 2,263, 32: 2,384.
enum { WARP_FEW = 16 };

// A searcher between two slices of a resumable solve (the solver's save area). (The frames
// below the top go to the lane's stack area.)
struct WarpSave {
  uint16_t m[16], all[4], now[4];
  u32 code[4];
  u32 st, trick;
  int trump;
  u64 hash[14];
  WarpJob job;
};

struct WarpBlock {
  BatchArgs args;
  u64 idle_since;  // stream: global time since which no searcher had work (0 = busy)
  int polling;     // stream: a searcher of the block is looking at the ring
  int busy;        // stream: searchers with a job
  int idle_exit;   // stream: waiting searchers end (1: nothing will come, 2: stopped by the host)
  unsigned polls;  // stream: looks at the ring
  int halt;        // stopped by the host
  unsigned turn;   // of the clock, in which the host's flag was last read
  int running;     // searchers that did not end idle
  unsigned long long nodes, jobs_done, total[WCNT_COUNT];
  WarpMem warp[1];  // as many as the block has warps
};
inline size_t warp_smem(int warps) { return sizeof(WarpBlock) + sizeof(WarpMem) * (size_t)(warps - 1); }

// Is the slice over, or the solve stopped by the host? In one thread, asked at the first trick
// start after 256 nodes and before a job is taken. The host's flag is a read over the bus, and the
// GPU does about 1.15 M of those a second however many SMs ask (one read by every searcher each
// 1,024 nodes held the whole GPU at 1.18 G nodes/s). So a block reads it once in 2^FLAG_SHIFT
// clock cycles, about four milliseconds: the first question after that does, and the others see
// what it found. Counted in questions instead, one in 64, it held sets of small endings at 74 M
// jobs/s; read each millisecond, a search alone on an SM was 0.1 % slower (29.82 against 29.77 ms).
enum { FLAG_SHIFT = 23 };
__device__ __forceinline__ u32 flag_turn() { return (u32)(clock64() >> FLAG_SHIFT); }
__device__ __forceinline__ int warp_ask(WarpBlock* sh, u64 t_end) {
  const BatchArgs& a = sh->args;
  volatile int* halt = &sh->halt;
  const u32 turn = flag_turn();
  if (turn != *reinterpret_cast<volatile u32*>(&sh->turn) && atomicExch(&sh->turn, turn) != turn && a.stop && *a.stop) *halt = 1;
  return *halt | (int)(t_end && global_ns() > t_end);
}

// One look at the stream's ring, in one thread: 1 a job taken, 0 nothing will come, -1 stopped
// by the host, -2 nothing now. One searcher of a block looks at a time.
__device__ __forceinline__ int warp_stream_look(WarpBlock* sh, unsigned long long& job) {
  const BatchArgs& a = sh->args;
  volatile int* vexit = &sh->idle_exit;
  volatile u64* vsince = &sh->idle_since;
  int got = -2;
  if (*vexit) return *vexit == 1 ? 0 : -1;
  if (atomicCAS(&sh->polling, 0, 1) != 0) return got;
  DevEnv q;
  q.a = &a;
  const bool closing = *reinterpret_cast<const volatile int*>(a.closing) != 0;
  // The host's flag costs a read over the bus: looked at in every 256th look, here only (a
  // read by every waiting searcher held up the whole kernel: 400 deals took 1.76 s).
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
  } else if (*reinterpret_cast<volatile int*>(&sh->busy) == 0) {
    const u64 now = global_ns();
    if (!*vsince) *vsince = now;
    else if (now - *vsince > a.idle_ns) *vexit = 1;
  } else {
    *vsince = 0;
  }
  __threadfence_block();
  atomicExch(&sh->polling, 0);
  return got;
}

// The next job of a batch, in one thread: 1 taken, 0 none left, -1 stopped.
__device__ __forceinline__ int warp_next_job(WarpBlock* sh, const WarpJob& j, int wid, u64 t_end, unsigned long long& job) {
  const BatchArgs& a = sh->args;
  // A searcher that has not searched in this launch takes a job all the same: a slice that is over
  // before the kernel has started up still gets on, by 256 nodes a searcher or a job.
  if (warp_ask(sh, t_end) && j.nodes) return -1;
  // The first job of the launch is dealt round-robin over the blocks, so that a small batch
  // spreads over every SM; later ones come from the shared counter.
  const long long rr = (long long)wid * gridDim.x + blockIdx.x;
  if (j.job < 0 && rr < a.rr_jobs) job = (unsigned long long)rr;
  else job = atomicAdd(a.next_job, 1ull) + (unsigned long long)a.rr_jobs;
  return (long long)job < a.n_jobs;
}

// The job's record.
__device__ __forceinline__ void warp_set_job(const BatchArgs& a, WarpJob& j, unsigned long long job, int t) {
  const unsigned long long deal = a.jpd == 5 ? job / 5 : job / 20;
  const int sub = (int)(job - deal * a.jpd);
  const bool all = a.jpd == 5;
  j.job = (long long)job;
  j.deal = (long long)deal;
  j.strain = (int8_t)(a.one_job ? a.one_strain : all ? sub : sub >> 2);
  j.decl = (int8_t)(a.one_job ? (a.one_decl >= 0 ? a.one_decl : 0) : all ? 0 : sub & 3);
  j.last_decl = (int8_t)(a.one_job ? (a.one_decl >= 0 ? a.one_decl : 3) : all ? 3 : sub & 3);
  j.mode = (int8_t)a.mode;
  j.start_nodes = j.nodes;
  if (a.job_start_ns && t == 0) a.job_start_ns[job] = global_ns();
}

// A job's end, in one thread.
template <bool STREAM>
__device__ __forceinline__ void warp_job_done(WarpBlock* sh, WarpJob* j) {
  const BatchArgs& a = sh->args;
  if (a.job_nodes) a.job_nodes[j->job] = j->nodes - j->start_nodes;
  if (a.job_end_ns) a.job_end_ns[j->job] = global_ns();
  j->jobs_done++;
  if (STREAM) {
    stream_deal_done(a, j->deal);
    atomicSub(&sh->busy, 1);
  }
}

// STREAM: the jobs come from a stream's ring. (A kernel of its own, so that other launches carry
// nothing of the waiting for deals.)
template <bool STREAM>
struct WarpEnv {
  WarpBlock* sh;
  TTBucket* tt;
  u64 t_end;
  int wid;

  __device__ __forceinline__ TTBucket* table() { return tt; }
  __device__ __forceinline__ u32 mask() const { return (1u << sh->args.tt_log2) - 1; }
  __device__ __forceinline__ long long out_row(const WarpJob& j) const {
    return STREAM ? (j.deal & sh->args.ring_mask) : j.deal;
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
    if ((threadIdx.x & 31) == 0) warp_job_done<STREAM>(sh, &j);
    __syncwarp();
  }

  __device__ __forceinline__ bool take(WarpState& w, const WarpIds& id, WarpMem& sm) {
    const BatchArgs& a = sh->args;
    WarpJob& j = sm.job;
    __syncwarp();
    unsigned long long job = 0;
    int got = -2;
    if (STREAM) {
      for (;;) {
        if (id.t == 0) got = warp_stream_look(sh, job);
        got = (int)w_uni((u32)got);
        if (got != -2) break;
        // the busier the block, the longer the wait: deals spread over the SMs
        __nanosleep(1000u + 500u * (unsigned)*reinterpret_cast<volatile int*>(&sh->busy));
      }
    } else {
      if (id.t == 0) got = warp_next_job(sh, j, wid, t_end, job);
      got = (int)w_uni((u32)got);
    }
    if (id.t == 0) j.stage = got == 0 ? ST_IDLE : ST_TAKE;
    if (got != 1) return false;
    // By all threads, which write the same values: no branch takes the warp apart here.
    warp_set_job(a, j, (unsigned long long)w_uni((u32)(job >> 32)) << 32 | w_uni((u32)job), id.t);
    __syncwarp();
    const long long row = STREAM ? (j.deal & a.ring_mask) : j.deal;
    const unsigned short* h = reinterpret_cast<const unsigned short*>((STREAM ? a.ring : a.hands) + row * 4);
    w.m = (STREAM ? __ldcg(h + 4 * id.p + id.s) : h[4 * id.p + id.s]) & 0x1FFFu;
    w.all = w.now = w_shfl(w.m, id.s) | w_shfl(w.m, 4 + id.s) | w_shfl(w.m, 8 + id.s) | w_shfl(w.m, 12 + id.s);
    w.code = w_build_code(w, id);
    const int cards = (int)w_add(id.t < 4 ? (u32)w_popc(w.m) : 0u);
    w.trump = strain_trump(j.strain);
    // A new TT generation; at the wrap all tags are cleared, by the whole warp.
    w.gen++;
    if (w_any(w.gen >= (1u << GEN_BITS))) {
      const u32 n = (mask() + 1) * 4;
      for (u32 k = id.t; k < n; k += 32) reinterpret_cast<uint4*>(tt[k >> 2].tag)[k & 3] = make_uint4(0, 0, 0, 0);
      w.gen = 1;
    }
    if (id.t == 0) j.cards = (int8_t)(cards > 13 ? 13 : cards);
    __syncwarp();
    return true;
  }

  __device__ __forceinline__ bool stop(WarpState& w, const WarpIds& id, WarpMem& sm) {
    int end = 0;
    if (id.t == 0) end = warp_ask(sh, t_end);
    const bool over = w_any(end != 0);
    if (over && id.t == 0) sm.job.stage = ST_ENTER;
    return over;
  }
};

template <int WARPS, bool STREAM>
__global__ void __launch_bounds__(WARPS * 32, 1) warp_kernel(BatchArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  WarpBlock& sh = *reinterpret_cast<WarpBlock*>(smem_raw);
  const int wid = (int)w_uni(threadIdx.x >> 5), t = threadIdx.x & 31, warps = blockDim.x >> 5;
  const long long lane = (long long)blockIdx.x * warps + wid;
  const u64 t_end = a.slice_ns ? global_ns() + a.slice_ns : 0;
  if (threadIdx.x == 0) {
    sh.args = a;
    sh.idle_since = 0;
    sh.polling = sh.busy = sh.idle_exit = sh.running = 0;
    sh.polls = 0;
    sh.turn = flag_turn();
    sh.halt = 0;
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
  WarpSave* sv = a.save ? reinterpret_cast<WarpSave*>(a.save) + lane : nullptr;
  if (a.resume) {
    w.m = sv->m[t & 15];
    w.all = sv->all[id.s];
    w.now = sv->now[id.s];
    w.code = sv->code[id.s];
    w.st = sv->st;
    w.trick = sv->trick;
    w.trump = sv->trump;
    if (t < 14) sm.hash[t] = sv->hash[t];
    const int words = (int)(w.st & SW_OFF) / (16 << 8);
    for (int k = t; k < words; k += 32) reinterpret_cast<uint4*>(sm.fr)[k] = reinterpret_cast<const uint4*>(stack)[k];
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
  WarpEnv<STREAM> env;
  env.sh = &sh;
  env.tt = a.tt + (lane << a.tt_log2);
  env.t_end = t_end;
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
    if (t < 14) sv->hash[t] = sm.hash[t];
    if (t < 4) {
      sv->all[t] = (uint16_t)w.all;
      sv->now[t] = (uint16_t)w.now;
      sv->code[t] = w.code;
    }
    const int words = (int)(w.st & SW_OFF) / (16 << 8);
    for (int k = t; k < words; k += 32) reinterpret_cast<uint4*>(stack)[k] = reinterpret_cast<const uint4*>(sm.fr)[k];
    if (t == 0) {
      sv->st = w.st;
      sv->trick = w.trick;
      sv->trump = w.trump;
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
