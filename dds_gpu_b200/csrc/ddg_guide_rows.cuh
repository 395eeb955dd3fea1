// Bookkeeping of the guide's kernels that host code can run (the CPU tests do).
//
// Which rows (examples) a block works on: tiles of TILE_M rows are dealt
// round-robin over the blocks of a launch; a set of 107,374,183 deals has more than 2^31 rows,
// so a row is a 64-bit number.
#pragma once
#include "ddg_bits.cuh"

namespace guide_nn {

enum : int { TILE_M = 128 };

// Tiles of `rows` rows, those of block `block` of `grid`, and its t-th one's first row.
DDG_HD int64_t tiles_of(int64_t rows) { return (rows + TILE_M - 1) / TILE_M; }
DDG_HD int block_tiles(int tiles, int block, int grid) { return block < tiles ? (tiles - 1 - block) / grid + 1 : 0; }
DDG_HD int64_t first_row(int t, int block, int grid) { return ((int64_t)t * grid + block) * TILE_M; }

// Parity of a thread's (n + 1)-th wait on a barrier, whose phases it waits for in turn, and of
// waiting once more for the phase of the last of its n waits. (A wait for a parity returns at
// once unless the phase under way has that parity, so the next wait's parity would not do.)
DDG_HD uint32_t wait_parity(uint32_t n) { return n & 1; }
DDG_HD uint32_t again_parity(uint32_t n) { return (n - 1) & 1; }

}  // namespace guide_nn
