"""The rows of a guide launch: its blocks' tiles cover every example once, also where a set has
more examples than 31 bits count (107,374,183 deals and up)."""
import ctypes
import os
import re
import subprocess

import pytest

from conftest import NATIVE, ROOT

CSRC = os.path.join(ROOT, "dds_gpu_b200", "csrc")


@pytest.fixture(scope="module")
def rows_lib():
    out = os.path.join(NATIVE, "_build", "libguide_rows.so")
    os.makedirs(os.path.dirname(out), exist_ok=True)
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-Wno-unknown-pragmas", "-I" + CSRC, "-o", out + ".tmp",
                    os.path.join(NATIVE, "guide_rows.cpp")], check=True)
    os.replace(out + ".tmp", out)
    lib = ctypes.CDLL(out)
    lib.rows_tiles.restype = lib.rows_first.restype = ctypes.c_int64
    lib.rows_tiles.argtypes = [ctypes.c_int64]
    return lib


@pytest.mark.parametrize("deals,grid", [(1, 1), (6, 1), (7, 2), (1000, 148), (107374182, 148), (107374183, 148),
                                        (150000000, 148), (400000000, 132)])
def test_tiles_cover_the_examples(rows_lib, deals, grid):
    rows = deals * 20
    tiles = rows_lib.rows_tiles(rows)
    grid = min(grid, tiles)
    count = [rows_lib.rows_block_tiles(tiles, b, grid) for b in range(grid)]
    assert sum(count) == tiles == -(-rows // 128)
    for b in range(grid):
        assert rows_lib.rows_first(0, b, grid) == 128 * b
        for t in {0, 1, count[b] // 2, count[b] - 1}:  # every grid-th tile, to the last one
            assert rows_lib.rows_first(t, b, grid) == 128 * (b + t * grid)
        assert 0 <= rows_lib.rows_first(count[b] - 1, b, grid) < rows <= rows_lib.rows_first(count[b], b, grid) + 128 * (grid - 1)
    last = max(rows_lib.rows_first(count[b] - 1, b, grid) for b in range(grid))
    assert last < rows <= last + 128


def test_kernel_takes_its_rows_from_there():
    """mlp_rows holds no row in 32 bits: its first rows come from first_row, as int64_t."""
    src = open(os.path.join(CSRC, "ddg_guide.cuh")).read()
    assert not re.search(r"\bint m0\b|\* TILE_M, sA|tile \* TILE_M", src)
    assert len(re.findall(r"\bfirst_row\(", src)) == 4


def test_the_last_wait_is_for_the_products_in_flight():
    """A wait for a parity returns while the phase under way has the other one, so a wait after
    one that gave up on a product needs a phase that nothing has completed: a barrier of its
    own, which a last commit arrives on when all products issued are done."""
    src = open(os.path.join(CSRC, "ddg_guide.cuh")).read()
    end = src[src.index("if (!ok && tid == 0) {"):]
    end = end[:end.index("tcgen05.dealloc")]
    assert end.index("commit(last);") < end.index("mbar_wait(last, 0);")
    assert len(re.findall(r"\blast\b[,;)]", src)) == 2  # used nowhere else
    assert "mbar_wait(done" not in end
    barriers = int(re.search(r"b < (\d+); b\+\+\) asm volatile\(\"mbarrier.init", src).group(1))
    assert "done = bars + 64, last = bars + 72" in src and barriers == 72 // 8 + 1
    assert "sm + SM_BAR + 80)" in src and "MLP_SMEM = SM_BAR + 11 * 8" in src  # then tensor memory's address
