// Launch shapes of the warp kernel (host code; the CPU tests call it).
#pragma once
#include <algorithm>

namespace ddg {

// Searchers to an SM at most.
enum { WARP_MAX = 32 };

// Tables of a pool of `lanes` lanes: those that a launch can use.
inline long long warp_tables(int sms, long long lanes) { return std::min<long long>(lanes, (long long)sms * WARP_MAX); }

struct WarpShape {
  int grid, warps;  // blocks, one to an SM; searchers to a block
};

// The blocks and searchers of a launch on at most `sms` SMs, each searcher with one of `lanes`
// tables. A batch with fewer jobs than lanes takes fewer searchers, spread over the SMs; a
// stream's jobs are yet to come, so it takes all.
inline WarpShape warp_shape(int sms, int lanes, long long n_jobs, bool stream) {
  const long long want = stream || n_jobs > lanes ? lanes : n_jobs;
  WarpShape s;
  s.grid = (int)std::min<long long>(sms, want);
  const long long warps = std::min<long long>(WARP_MAX, stream ? want / s.grid : (want + s.grid - 1) / s.grid);
  s.warps = (int)std::min<long long>(warps, lanes / s.grid);
  return s;
}

// SMs a stream's kernel may take on a GPU of `sms`, by a pool whose lanes make `blocks` blocks. It
// stays there for as long as the stream is open, so a pool that leaves SMs free (a guided
// stream's must, for the guide's kernels) leaves up to two free as a stream as well.
inline int stream_sms(int sms, int blocks) { return std::max(1, std::max(sms - 2, std::min(sms, blocks))); }

// Deals a stream takes in at once: two jobs a search that can be under way, one running and one
// waiting.
inline long long stream_deals(long long searches, int jobs_per_deal) {
  return std::max<long long>(1, searches * 2 / jobs_per_deal);
}

}  // namespace ddg
