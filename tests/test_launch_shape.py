"""What a call reports of its launch is the launch that ran, for the warp kernel (a search to a
warp) and the lane-per-thread ones (a search to a thread)."""
import ctypes
import os
import subprocess
import time

import numpy as np
import pytest

from conftest import NATIVE, ROOT, load_golden


@pytest.fixture(scope="module")
def shape_lib():
    out = os.path.join(NATIVE, "_build", "libshape.so")
    os.makedirs(os.path.dirname(out), exist_ok=True)
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-I" + os.path.join(ROOT, "dds_gpu_b200", "csrc"), "-o",
                    out + ".tmp", os.path.join(NATIVE, "shape.cpp")], check=True)
    os.replace(out + ".tmp", out)
    lib = ctypes.CDLL(out)
    lib.shape_tables.restype = ctypes.c_longlong
    lib.shape_tables.argtypes = [ctypes.c_int, ctypes.c_longlong]
    lib.shape_stream_deals.restype = ctypes.c_longlong
    lib.shape_stream_deals.argtypes = [ctypes.c_longlong, ctypes.c_int]
    return lib


def shape(lib, sms, lanes, jobs, stream=0):
    grid, warps = ctypes.c_int(), ctypes.c_int()
    lib.shape_of(sms, lanes, ctypes.c_longlong(jobs), stream, ctypes.byref(grid), ctypes.byref(warps))
    return grid.value, warps.value


@pytest.mark.parametrize("lanes", [512, 2560, 4096, 4736, 75776])
@pytest.mark.parametrize("sms", [1, 146, 148])
def test_every_searcher_has_a_table_and_every_sm_its_share(shape_lib, lanes, sms):
    for jobs in (1, 2, sms - 1, sms, sms + 1, 16 * sms, 16 * sms + 1, 32 * sms, 10 ** 6):
        if jobs < 1:
            continue
        grid, warps = shape(shape_lib, sms, lanes, jobs)
        assert 1 <= grid <= sms and 1 <= warps <= 32 and grid * warps <= lanes
        assert grid == min(sms, jobs)
        assert warps == min(32, lanes // grid, -(-jobs // grid))  # enough for the jobs, where they fit
    grid, warps = shape(shape_lib, sms, lanes, 0, 1)
    assert grid == sms and warps == min(32, lanes // sms)


@pytest.mark.parametrize("blocks,want", [(1, 146), (32, 146), (146, 146), (147, 147), (148, 148), (500, 148)])
def test_a_stream_leaves_what_its_pool_leaves_up_to_two(shape_lib, blocks, want):
    assert shape_lib.shape_stream_sms(148, blocks) == want


def test_admission_is_two_jobs_a_search(shape_lib):
    assert shape_lib.shape_stream_deals(4736, 5) == 1894 and shape_lib.shape_stream_deals(4736, 20) == 473
    assert shape_lib.shape_stream_deals(4096, 5) == 1638 and shape_lib.shape_stream_deals(3, 20) == 1


def test_tables_are_those_a_launch_can_use(shape_lib):
    for lanes, want in ((512, 512), (600, 600), (4735, 4735), (4736, 4736), (4737, 4736), (75776, 4736), (1 << 34, 4736)):
        assert shape_lib.shape_tables(148, lanes) == want
        # with fewer tables a launch of any size is the same as with all that were asked for
        for jobs in (1, 147, 149, 2000, 4700, 10 ** 6):
            assert shape(shape_lib, 148, want, jobs) == shape(shape_lib, 148, min(lanes, 10 ** 6), jobs)
        for sms in (146, 148):
            assert shape(shape_lib, sms, want, 0, 1) == shape(shape_lib, sms, min(lanes, 10 ** 6), 0, 1)


# ---- on the GPU ------------------------------------------------------------------------------


def sm_count():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


def solve(solver, hands):
    import torch
    d_h = torch.from_numpy(np.ascontiguousarray(hands).view(np.int64)).cuda()
    d_o = torch.empty(len(hands) * 20, dtype=torch.uint8, device="cuda")
    return solver.solve_device(d_h.data_ptr(), len(hands), d_o.data_ptr())


@pytest.mark.gpu
@pytest.mark.parametrize("deals", [1, 31, 600, 4096])
def test_batch(ddg, deals):
    hands = load_golden("k6_4096.npz")["hands"][:deals]
    s = ddg.Solver()
    try:
        st = solve(s, hands)
    finally:
        s.close()
    sms, jobs = sm_count(), deals * 5
    warps = min(32, -(-jobs // min(sms, jobs)))
    assert (st["grid"], st["block"], st["lanes"]) == (min(sms, jobs), 32 * warps, min(sms, jobs) * warps)


@pytest.mark.gpu
def test_lane_per_thread(ddg):
    s = ddg.Solver(lanes=1024, free_below=96)
    try:
        st = solve(s, load_golden("k4_120.npz")["hands"])
    finally:
        s.close()
    assert (st["grid"], st["block"], st["lanes"]) == (2, 512, 1024)


@pytest.mark.gpu
@pytest.mark.parametrize("kw", [{}, {"lanes": 1024, "free_below": 96}])
def test_stream(ddg, kw):
    g = load_golden("k4_120.npz")
    s = ddg.Solver(**kw)
    try:
        st = ddg.Stream(s, ring_slots=64, idle_timeout_s=5)
        assert st.submit(g["hands"][:20]) == 20
        seen, t0 = 0, time.time()
        while seen < 20 and time.time() - t0 < 60:
            idx, tab = st.poll()
            assert (tab == g["tricks"][idx.astype(int)]).all()
            seen += len(idx)
        stats = st.close()
    finally:
        s.close()
    want = (2, 512, 1024) if kw else (sm_count(), 1024, 32 * sm_count())
    assert seen == 20 and (stats["grid"], stats["block"], stats["lanes"]) == want


@pytest.mark.gpu
@pytest.mark.parametrize("kw,searches", [({}, 148 * 32), ({"jobs_per_deal": 20}, 148 * 32), ({"lanes": 146 * 512}, 146 * 32),
                                         ({"lanes": 512}, 146 * 3), ({"lanes": 1024, "free_below": 96}, 1024)])
def test_stream_capacity(ddg, kw, searches):
    """Two jobs for every search that can be under way, whatever the pool's size."""
    if sm_count() != 148:
        pytest.skip("figures for 148 SMs")
    s = ddg.Solver(**kw)
    try:
        st = ddg.Stream(s, ring_slots=65536, idle_timeout_s=1)
        assert st.capacity == searches * 2 // s.jobs_per_deal
        stats = st.close()
        assert stats["lanes"] == searches
    finally:
        s.close()


@pytest.mark.gpu
def test_other_kernels_run_beside_a_stream(ddg):
    """A stream of (SMs - 2) * 512 lanes, busy for minutes, leaves SMs on which another solver's
    call ends."""
    hard = load_golden("k13_24.npz")["hands"]
    g = load_golden("k5_120.npz")
    s, other = ddg.Solver(lanes=(sm_count() - 2) * 512), ddg.Solver(lanes=512)
    try:
        assert (other.solve(g["hands"]) == g["tricks"]).all()  # kernels loaded, buffers there
        st = ddg.Stream(s, ring_slots=64, idle_timeout_s=5)
        assert st.submit(hard) == 24
        t0 = time.time()
        assert (other.solve(g["hands"]) == g["tricks"]).all()
        assert st.in_flight > 0 and time.time() - t0 < 20
        stats = st.close(drain=False)
        assert stats["grid"] == sm_count() - 2
    finally:
        s.close()
        other.close()


@pytest.mark.gpu
def test_pool(ddg):
    """The warp kernel's pool has a table a searcher; the other kernels' pools are whole blocks."""
    most = 32 * sm_count()
    tt = 320 << 10
    for kw, lanes in (({}, most), ({"lanes": 4 * most}, most), ({"lanes": most}, most), ({"lanes": 700}, 700),
                      ({"lanes": 700, "free_below": 96}, 512), ({"lanes": 4 * most, "free_below": 96}, 4 * most // 512 * 512)):
        s = ddg.Solver(**kw)
        try:
            assert s.lanes == lanes and lanes * tt <= s.nbytes < lanes * (tt + 8192)
            g = load_golden("k5_120.npz")
            assert (s.solve(g["hands"]) == g["tricks"]).all()
        finally:
            s.close()
    for kw in ({"lanes": 511}, {"lanes": 511, "free_below": 96}, {"lanes": 10 ** 7}):  # less than a block; 3.3 TB
        with pytest.raises(ddg.DDGError):
            ddg.Solver(**kw)


@pytest.mark.gpu
def test_tuned_pool_with_helping(ddg):
    """A setting tuned on the warp kernel, run with helping: on every lane of the other kernel."""
    import torch
    from dds_gpu_b200 import autotune
    g = load_golden("k6_120.npz")
    d_h = torch.from_numpy(g["hands"].view(np.int64)).cuda()
    made = []

    class Recorded(ddg.Solver):
        def __init__(self, **kw):
            super().__init__(**kw)
            made.append(self.lanes)

    solver, autotune.Solver = autotune.Solver, Recorded
    try:
        cfg = {"block": 512, "min_blocks": 1, "schedule": 0, "tt_log2": 10, "lanes": 32 * sm_count()}
        for help in (False, True):
            rep = autotune.run_batch(cfg, d_h, 120, 60.0, torch, tables=True, help=help)
            assert (rep["tables"] == g["tricks"]).all()
    finally:
        autotune.Solver = solver
    assert made == [32 * sm_count(), 512 * sm_count()]


@pytest.mark.gpu
@pytest.mark.parametrize("kw", [{}, {"free_below": 96}])
def test_guided_stream(ddg, kw):
    """The guide's kernels get the two SMs that a stream leaves, beside the warp kernel and beside
    the lane-per-thread one (any of whose options asks for it)."""
    from dds_gpu_b200 import guide as ddg_guide
    params = ddg_guide.load_weights()
    if params is None:
        pytest.skip("no guide weights file")
    g = load_golden("k7_120.npz")
    guide, s = ddg.Guide(max_rows=4096, params=params), ddg.Solver(lanes=(sm_count() - 2) * 512, **kw)
    try:
        st = ddg.Stream(s, ring_slots=64, idle_timeout_s=2, guide=guide)
        got, sent, seen, t0 = np.full_like(g["tricks"], 255), 0, 0, time.time()
        while seen < 120 and time.time() - t0 < 60:
            if sent < 120:
                sent += st.submit(g["hands"][sent:])
            idx, tab = st.poll()
            got[idx.astype(int)] = tab
            seen += len(idx)
        stats = st.close()
    finally:
        s.close()
        guide.close()
    assert seen == 120 and (got == g["tricks"]).all()
    assert stats["grid"] == sm_count() - 2 and stats["block"] == (512 if kw else 1024)
