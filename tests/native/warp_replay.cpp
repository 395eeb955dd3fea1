// Test infrastructure: the warp search (dds_gpu_b200/csrc/ddg_warp.cuh) on emulated warps
// (warp_emu.hpp), so that the CPU test suite compares its tables and its node counts, job
// for job, with the oracle's fixtures. Never part of the product path.
#include <string.h>

#include <atomic>
#include <thread>

#include "warp_emu.hpp"
#include "ddg_warp.cuh"

using namespace ddg;

namespace {
struct Batch {
  const u64* hands;
  long long n_jobs;
  int jpd, mode, tt_log2, stop_every;
  const int8_t* seeds;
  const int8_t* hints;
  int* out20;
  int8_t* best20;
  uint64_t* job_nodes;
  std::atomic<long long> next{0};
};

struct Searcher {  // one emulated warp
  Batch* b;
  std::vector<TTBucket> tt;
  WarpMem sm;
  WarpState lane[32];
  u32 gen = 0;
  long long taken = 0;
  u64 asked = 0;
  bool resume = false;
};

struct Env {
  Searcher* x;
  TTBucket* table() { return x->tt.data(); }
  u32 mask() { return (1u << x->b->tt_log2) - 1; }
  bool take(WarpState& w, const WarpIds& id, WarpMem& sm) {
    w_sync();
    if (id.t == 0) x->taken = x->b->next++;
    w_sync();
    if (x->taken >= x->b->n_jobs) {
      if (id.t == 0) sm.job.stage = ST_IDLE;
      return false;
    }
    if (id.t == 0) {
      WarpJob& j = sm.job;
      j.job = x->taken;
      j.deal = j.job / x->b->jpd;
      const int sub = (int)(j.job % x->b->jpd);
      j.strain = (int8_t)(x->b->jpd == 5 ? sub : sub / 4);
      j.decl = (int8_t)(x->b->jpd == 5 ? 0 : sub % 4);
      j.last_decl = (int8_t)(x->b->jpd == 5 ? 3 : sub % 4);
      j.mode = (int8_t)x->b->mode;
      j.cards = (int8_t)popc(x->b->hands[j.deal * 4]);
      j.start_nodes = j.nodes;
      x->gen = tt_next_gen(x->tt.data(), mask(), x->gen);
    }
    w_sync();
    w.gen = x->gen;
    w.trump = strain_trump(sm.job.strain);
    w.m = (u32)(x->b->hands[sm.job.deal * 4 + id.p] >> (16 * id.s)) & 0x1FFF;
    w.all = w.now = w_shfl(w.m, id.s) | w_shfl(w.m, 4 + id.s) | w_shfl(w.m, 8 + id.s) | w_shfl(w.m, 12 + id.s);
    w.code = w_build_code(w, id);
    return true;
  }
  // Every stop_every-th question ends the run; the caller resumes it.
  bool stop(WarpState& w, const WarpIds& id, WarpMem& sm) {
    w_sync();
    if (id.t == 0) x->asked++;
    w_sync();
    const bool end = x->b->stop_every && x->asked % x->b->stop_every == 0;
    if (end && id.t == 0) sm.job.stage = ST_ENTER;
    w_sync();
    return end;
  }
  int seed(const WarpJob& j) { return x->b->mode == MODE_STEP ? x->b->seeds[j.deal * 20 + j.strain * 4 + j.decl] : 7; }
  int root_hint(const WarpJob& j) { return x->b->hints ? x->b->hints[j.deal * 20 + j.strain * 4 + j.decl] : -1; }
  void answer(const WarpJob& j, int ns) {
    x->b->out20[j.deal * 20 + j.strain * 4 + j.decl] = (j.decl & 1) == 0 ? ns : 13 - ns;
  }
  void root_best(const WarpJob& j, int card) {
    if (x->b->best20) x->b->best20[j.deal * 20 + j.strain * 4 + j.decl] = (int8_t)card;
  }
  void job_done(const WarpJob& j) { x->b->job_nodes[j.job] = j.nodes - j.start_nodes; }
};

void fiber(void* arg, int t) {
  Searcher* x = (Searcher*)arg;
  const WarpIds id = {t, t & 3, (t >> 2) & 3};
  Env env = {x};
  w_run(x->lane[t], id, x->sm, env);
  w_sync();
}
}  // namespace

extern "C" {
// n deals; stats[0..5] = nodes, probes, hits, stores, entry reads, TT bytes. `stop_every`:
// every so many stop questions (256 nodes or a few more each) the warp's registers are kept, it ends and
// is started again. `backwards`: the fibers run ahead of one another in the other order.
int warp_replay(const uint64_t* hands, long long n, int tt_log2, int jpd, int mode, const int8_t* seeds,
                const int8_t* hints, int threads, int stop_every, int backwards, int* out20, int8_t* best20,
                uint64_t* job_nodes, uint64_t* stats) {
  if (tt_log2 < TT_MIN_LOG2 || tt_log2 > 16 || (jpd != 5 && jpd != 20) || threads < 1) return -1;
  Batch b;
  b.hands = hands;
  b.n_jobs = n * jpd;
  b.jpd = jpd;
  b.mode = mode;
  b.tt_log2 = tt_log2;
  b.stop_every = stop_every;
  b.seeds = seeds;
  b.hints = hints;
  b.out20 = out20;
  b.best20 = best20;
  b.job_nodes = job_nodes;
  std::atomic<uint64_t> sum[6];
  for (auto& s : sum) s = 0;
  std::vector<std::thread> pool;
  for (int k = 0; k < threads; k++)
    pool.emplace_back([&] {
      Searcher* x = new Searcher();
      x->b = &b;
      x->tt.resize((size_t)1 << tt_log2);
      memset(x->tt.data(), 0, x->tt.size() * sizeof(TTBucket));
      memset(&x->sm, 0, sizeof(x->sm));
      memset(x->lane, 0, sizeof(x->lane));
      x->sm.job.stage = ST_TAKE;
      WarpEmu* e = new WarpEmu();
      e->backwards = backwards != 0;
      do {
        e->run(fiber, x);
      } while (x->sm.job.stage != ST_IDLE);
      sum[0] += x->sm.job.nodes;
      for (int c = 0; c < 5; c++) sum[1 + c] += x->sm.job.total[c];
      delete e;
      delete x;
    });
  for (auto& t : pool) t.join();
  for (int c = 0; c < 6; c++) stats[c] = sum[c];
  return 0;
}
}
