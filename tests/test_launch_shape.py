"""What a call reports of its launch is the launch that ran, for the warp kernel (a search to a
warp) and the lane-per-thread ones (a search to a thread)."""
import time

import numpy as np
import pytest

from conftest import load_golden

pytestmark = pytest.mark.gpu


def sm_count():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


def solve(solver, hands):
    import torch
    d_h = torch.from_numpy(np.ascontiguousarray(hands).view(np.int64)).cuda()
    d_o = torch.empty(len(hands) * 20, dtype=torch.uint8, device="cuda")
    return solver.solve_device(d_h.data_ptr(), len(hands), d_o.data_ptr())


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


def test_lane_per_thread(ddg):
    s = ddg.Solver(lanes=1024, free_below=96)
    try:
        st = solve(s, load_golden("k4_120.npz")["hands"])
    finally:
        s.close()
    assert (st["grid"], st["block"], st["lanes"]) == (2, 512, 1024)


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
