// Test infrastructure: the guide kernels' row arithmetic (dds_gpu_b200/csrc/ddg_guide_rows.cuh)
// for the CPU test suite. Never part of the product path.
#include "ddg_guide_rows.cuh"

extern "C" {
int64_t rows_tiles(int64_t rows) { return guide_nn::tiles_of(rows); }
int rows_block_tiles(int tiles, int block, int grid) { return guide_nn::block_tiles(tiles, block, grid); }
int64_t rows_first(int t, int block, int grid) { return guide_nn::first_row(t, block, grid); }
}
