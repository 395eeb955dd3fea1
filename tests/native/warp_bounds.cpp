// Test infrastructure: warp_replay.cpp's searchers in a build with -DDDG_BOUNDS_CHECK, reporting
// the failed checks and whether anything was written behind the frames. Never part of the
// product path.
#include "warp_replay.cpp"

extern "C" {
// n deals (binary search, five jobs each); report[0] = failed checks, report[1] = searchers whose
// memory behind the frames was written: the hashes of the 12th and 13th trick, which no ending of
// fewer cards uses. Answers in out20 (left alone where a searcher ended).
int warp_bounds(const uint64_t* hands, long long n, int tt_log2, int* out20, uint64_t* job_nodes, uint64_t* report) {
  std::vector<int8_t> best((size_t)n * 20);
  report[0] = report[1] = 0;
  for (long long d = 0; d < n; d++) {  // a searcher a deal: one that ends drops no other deal
    Batch b;
    b.hands = hands + d * 4;
    b.n_jobs = b.jpd = 5;
    b.mode = MODE_BISECT;
    b.tt_log2 = tt_log2;
    b.stop_every = 0;
    b.seeds = b.hints = nullptr;
    b.out20 = out20 + d * 20;
    b.best20 = best.data() + d * 20;
    b.job_nodes = job_nodes + d * 5;
    Searcher* x = new Searcher();
    x->b = &b;
    x->tt.resize((size_t)1 << tt_log2);
    memset(x->tt.data(), 0, x->tt.size() * sizeof(TTBucket));
    memset(&x->sm, 0, sizeof(x->sm));
    memset(x->lane, 0, sizeof(x->lane));
    x->sm.job.stage = ST_TAKE;
    WarpEmu* e = new WarpEmu();
    e->run(fiber, x);
    report[0] += x->sm.job.total[WCNT_BOUNDS];
    report[1] += (x->sm.hash[12] | x->sm.hash[13]) != 0;
    delete e;
    delete x;
  }
  return 0;
}
}
