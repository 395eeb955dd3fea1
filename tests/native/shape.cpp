// Test infrastructure: the warp kernel's launch shapes (dds_gpu_b200/csrc/ddg_shape.hpp) for the
// CPU test suite. Never part of the product path.
#include "ddg_shape.hpp"

extern "C" {
void shape_of(int sms, int lanes, long long n_jobs, int stream, int* grid, int* warps) {
  const ddg::WarpShape s = ddg::warp_shape(sms, lanes, n_jobs, stream != 0);
  *grid = s.grid;
  *warps = s.warps;
}
long long shape_tables(int sms, long long lanes) { return ddg::warp_tables(sms, lanes); }
int shape_stream_sms(int sms, int blocks) { return ddg::stream_sms(sms, blocks); }
long long shape_stream_deals(long long searches, int jpd) { return ddg::stream_deals(searches, jpd); }
}
