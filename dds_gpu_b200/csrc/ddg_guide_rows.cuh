// Which rows (examples) a block of the guide's kernels works on. Tiles of TILE_M rows are dealt
// round-robin over the blocks of a launch; a set of 107,374,183 deals has more than 2^31 rows,
// so a row is a 64-bit number. Host code as well: the CPU tests walk a launch's tiles.
#pragma once
#include "ddg_bits.cuh"

namespace guide_nn {

enum : int { TILE_M = 128 };

// Tiles of `rows` rows, those of block `block` of `grid`, and its t-th one's first row.
DDG_HD int64_t tiles_of(int64_t rows) { return (rows + TILE_M - 1) / TILE_M; }
DDG_HD int block_tiles(int tiles, int block, int grid) { return block < tiles ? (tiles - 1 - block) / grid + 1 : 0; }
DDG_HD int64_t first_row(int t, int block, int grid) { return ((int64_t)t * grid + block) * TILE_M; }

}  // namespace guide_nn
