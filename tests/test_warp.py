"""One warp per search (ddg_warp.cuh, the default kernel): on the CPU its code runs on
emulated warps (tests/native/warp_emu.hpp: 32 fibers that meet at every collective) and
must give the reference's tables and, job for job, its node counts, and the counters of the
host replay of the lane-per-thread stage machine; on the GPU the same through the C ABI for
pools from one block to the whole GPU, resumable slices and streams dropped in mid-search."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import NATIVE, ROOT, load_golden

P = ctypes.c_void_p
CSRC = os.path.join(ROOT, "dds_gpu_b200", "csrc")
LIGHT_13 = [1, 3, 15, 17, 22]  # full deals of k13_24 whose largest job is < 600k nodes


@pytest.fixture(scope="module")
def warp_lib():
    srcs = [os.path.join(NATIVE, f) for f in ("warp_replay.cpp", "warp_emu.hpp")]
    srcs += [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cuh")]
    out = os.path.join(NATIVE, "_build", "libwarp_replay.so")
    if not os.path.exists(out) or any(os.path.getmtime(s) > os.path.getmtime(out) for s in srcs):
        os.makedirs(os.path.dirname(out), exist_ok=True)
        subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-fPIC", "-shared", "-Wno-unknown-pragmas",
                        "-I" + CSRC, "-o", out + ".tmp", srcs[0]], check=True)
        os.replace(out + ".tmp", out)
    return ctypes.CDLL(out)


def ptr(a):
    return None if a is None else a.ctypes.data_as(P)


def replay(lib, hands, tt=10, jpd=5, seeds=None, hints=None, stop_every=0, backwards=0):
    n = hands.shape[0]
    h = np.ascontiguousarray(hands, dtype=np.uint64)
    out, best = np.full(n * 20, -1, np.int32), np.full(n * 20, -1, np.int8)
    nodes, stats = np.zeros(n * jpd, np.uint64), np.zeros(6, np.uint64)
    sd = None if seeds is None else np.ascontiguousarray(seeds, dtype=np.int8).reshape(-1)
    hd = None if hints is None else np.ascontiguousarray(hints, dtype=np.int8).reshape(-1)
    rc = lib.warp_replay(ptr(h), ctypes.c_longlong(n), tt, jpd, 0 if seeds is None else 1, ptr(sd), ptr(hd), 8,
                         stop_every, backwards, ptr(out), ptr(best), ptr(nodes), ptr(stats))
    assert rc == 0
    return out.reshape(n, 5, 4), nodes, stats, best.reshape(n, 5, 4)


@pytest.mark.parametrize("name,jpd,backwards", [("k1_120.npz", 5, 0), ("k2_120.npz", 20, 1), ("k4_120.npz", 5, 1),
                                                ("k5_120.npz", 20, 0), ("k7_120.npz", 5, 0), ("k9_120.npz", 20, 1)])
def test_endings(warp_lib, name, jpd, backwards):
    g = load_golden(name)
    n = 24 if name.startswith("k9") else 120
    t, nodes, _, _ = replay(warp_lib, g["hands"][:n], jpd=jpd, backwards=backwards)
    assert (t == g["tricks"][:n]).all()
    assert (nodes == g[f"nodes_jpd{jpd}"][:n * jpd]).all()


@pytest.mark.parametrize("tt", [9, 12])
def test_tt_sizes(warp_lib, tt):
    g = load_golden(f"k7_200_tt{tt}.npz")
    t, nodes, _, _ = replay(warp_lib, g["hands"][:80], tt=tt)
    assert (t == g["tricks"][:80]).all() and (nodes == g["nodes_jpd5"][:400]).all()


def test_seeded_and_full_deal(warp_lib):
    g = load_golden("k8_200_seeded.npz")
    t, nodes, _, _ = replay(warp_lib, g["hands"][:60], seeds=g["seeds"][:60])
    assert (t == g["tricks"][:60]).all() and (nodes == g["nodes_jpd5"][:300]).all()
    g = load_golden("k13_24.npz")
    t, nodes, _, _ = replay(warp_lib, g["hands"][LIGHT_13[:2]])
    want = g["nodes_jpd5"].reshape(-1, 5)[LIGHT_13[:2]].reshape(-1)
    assert (t == g["tricks"][LIGHT_13[:2]]).all() and (nodes == want).all()


def test_uneven_deals(warp_lib):
    """Long suits facing voids (many candidates, many discards)."""
    g = load_golden("mixed_300.npz")
    per_deal = g["nodes_jpd5"].astype(np.int64).reshape(-1, 5)
    sel = np.where(per_deal.max(axis=1) < 3000)[0][:100]
    t, nodes, _, _ = replay(warp_lib, g["hands"][sel])
    assert (t == g["tricks"][sel]).all() and (nodes == per_deal[sel].reshape(-1)).all()


@pytest.mark.parametrize("stop_every", [1, 7])
def test_stopped_and_resumed(warp_lib, stop_every):
    g = load_golden("k6_120.npz")
    t, nodes, _, _ = replay(warp_lib, g["hands"][:60], stop_every=stop_every)
    assert (t == g["tricks"][:60]).all() and (nodes == g["nodes_jpd5"][:300]).all()


def test_counters_and_hints_match_the_stage_machine(warp_lib, replay_lib):
    """Probes, hits, stores and TT bytes, and the nodes of searches with root leads given,
    as the host replay of the lane-per-thread stage machine counts them."""
    g = load_golden("k6_120.npz")
    n = 60
    h = np.ascontiguousarray(g["hands"][:n])
    rng = np.random.default_rng(3)
    hints = rng.integers(-1, 64, (n, 20)).astype(np.int8)
    seeds = rng.integers(0, 7, (n, 20)).astype(np.int8)
    out, nodes, stats = np.zeros(n * 20, np.int32), np.zeros(n * 5, np.uint64), np.zeros(13, np.uint64)
    rc = replay_lib.replay_solve_hinted(ptr(h), ctypes.c_longlong(n), 10, 5, 1, ptr(seeds), ptr(hints), 8, ptr(out),
                                        ptr(nodes), ptr(stats))
    assert rc == 0
    t, wn, ws, best = replay(warp_lib, h, seeds=seeds, hints=hints)
    assert (t.reshape(-1) == out).all() and (wn == nodes).all()
    assert ws[0] == nodes.sum()
    assert list(ws[1:4]) == list(stats[1:4])  # probes, hits, stores
    # the replay counts all TT bytes together, the warp those of probes by their events
    assert int(ws[5]) + 64 * int(ws[1]) + 16 * int(ws[4]) == int(stats[4])
    # a best lead is one of the leader's cards
    for d in range(n):
        for e in range(20):
            b = int(best[d, e // 4, e % 4])
            assert b == -1 or int(h[d, (e % 4 + 1) & 3]) >> b & 1


# ---- on the GPU ------------------------------------------------------------------------------


def device_solve(solver, hands, jpd=5):
    import torch
    n = hands.shape[0]
    d_h = torch.from_numpy(np.ascontiguousarray(hands).view(np.int64)).cuda()
    d_o = torch.empty(n * 20, dtype=torch.uint8, device="cuda")
    d_n = torch.zeros(n * jpd, dtype=torch.int64, device="cuda")
    st = solver.solve_device(d_h.data_ptr(), n, d_o.data_ptr(), d_job_nodes=d_n.data_ptr())
    return d_o.cpu().numpy().reshape(n, 5, 4), d_n.cpu().numpy().view(np.uint64), st


@pytest.mark.gpu
@pytest.mark.parametrize("lanes", [512, 2048, 2560, 0])
def test_pool_sizes(ddg, lanes):
    """From three searchers to an SM to the most one holds, on both sides of the 16 up to which
    a launch takes the build with more registers; jobs fewer and more than them, and more than
    63 to a searcher of the smallest pool (its TT generation wraps)."""
    s = ddg.Solver(lanes=lanes)
    try:
        for name, sel in (("k6_4096.npz", slice(0, 4096)), ("k6_4096.npz", slice(0, 4096)), ("k9_120.npz", slice(0, 1)),
                          ("k3_120.npz", slice(0, 120)), ("k5_120.npz", slice(0, 31))):
            g = load_golden(name)
            t, nodes, st = device_solve(s, g["hands"][sel])
            assert (t == g["tricks"][sel]).all()
            assert (nodes == g["nodes_jpd5"].reshape(-1, 5)[sel].reshape(-1)).all()
            assert st["nodes"] == int(nodes.sum()) and st["jobs_done"] == len(nodes)
            assert st["phase_warps"] == [0] * 5 and st["free_rounds"] == 0  # no other kernel ran
    finally:
        s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("lanes", [512, 0])
def test_slices(ddg, lanes):
    import torch
    g = load_golden("k9_120.npz")
    n = g["hands"].shape[0]
    s = ddg.Solver(lanes=lanes)
    try:
        d_h = torch.from_numpy(g["hands"].view(np.int64)).cuda()
        d_o = torch.empty(n * 20, dtype=torch.uint8, device="cuda")
        s.begin(d_h.data_ptr(), n, d_o.data_ptr())
        nodes = jobs = slices = 0
        finished = False
        while not finished:
            finished, st = s.resume(0.001)
            nodes, jobs, slices = nodes + st["nodes"], jobs + st["jobs_done"], slices + 1
            assert slices < 10000
        assert slices > 3
        assert (d_o.cpu().numpy().reshape(n, 5, 4) == g["tricks"]).all()
        assert nodes == int(g["nodes_jpd5"].astype(np.int64).sum()) and jobs == n * 5
    finally:
        s.close()


@pytest.mark.gpu
def test_time_limit_and_dropped_stream(ddg):
    """Searches cut off leave 255; the solver works normally afterwards."""
    hard = load_golden("k13_24.npz")["hands"]
    g = load_golden("k6_120.npz")
    s = ddg.Solver(time_limit_s=0.05)
    try:
        t = s.solve(hard)
        assert (t == 255).any()
        st = ddg.Stream(s, ring_slots=64, idle_timeout_s=5)
        assert st.submit(hard[:12]) == 12
        st.close(drain=False)
    finally:
        s.close()
    s = ddg.Solver()
    try:
        st = ddg.Stream(s, ring_slots=256, idle_timeout_s=0.2)
        assert st.submit(g["hands"]) == 120
        got = np.full((120, 5, 4), 255, np.uint8)
        import time
        t0 = time.time()
        seen = 0
        while seen < 120 and time.time() - t0 < 60:
            idx, tab = st.poll()
            got[idx.astype(int)] = tab
            seen += len(idx)
        time.sleep(1.0)  # the kernel ends by its idle timeout and is launched again
        assert st.submit(g["hands"][:3]) == 3
        t0 = time.time()
        while seen < 123 and time.time() - t0 < 60:
            idx, tab = st.poll()
            seen += len(idx)
            for i, x in zip(idx, tab):
                assert (x == g["tricks"][int(i) - 120]).all()
        st.close()
        assert seen == 123 and (got == g["tricks"]).all()
    finally:
        s.close()
