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


@pytest.mark.parametrize("done_before", [0, 1, 2, 5, 12])
def test_the_last_wait_is_for_the_product_that_did_not_finish(rows_lib, done_before):
    """A wait for parity p returns while the phase under way has the other parity. After
    `done_before` products one does not complete in time: its wait gives up, and so must the
    wait that is made before the kernel frees what the product uses, until it completes."""
    class Barrier:
        phase = 0

        def ready(self, parity):
            return self.phase & 1 != parity

    bar, waits = Barrier(), 0
    for _ in range(done_before):
        assert not bar.ready(rows_lib.rows_wait_parity(waits))
        bar.phase += 1
        assert bar.ready(rows_lib.rows_wait_parity(waits))
        waits += 1
    assert not bar.ready(rows_lib.rows_wait_parity(waits))  # gives up
    waits += 1
    assert not bar.ready(rows_lib.rows_again_parity(waits))
    bar.phase += 1
    assert bar.ready(rows_lib.rows_again_parity(waits))
    src = open(os.path.join(CSRC, "ddg_guide.cuh")).read()
    assert re.findall(r"mbar_wait\(done, (\w+)", src) == ["wait_parity", "again_parity"]
