"""The warp search stays inside its memory (warp_replay.cpp: ddg_warp.cuh on emulated warps,
compiled with the compiler's array bounds checks): also for deals that the device-memory calls
take unchecked, whose hands need not have 13 cards at most."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import NATIVE, ROOT, load_golden

P = ctypes.c_void_p
CSRC = os.path.join(ROOT, "dds_gpu_b200", "csrc")
SANITIZE = ["-fsanitize=bounds", "-fno-sanitize-recover=bounds", "-static-libubsan"]


def build(name, defines, src="warp_replay.cpp"):
    out = os.path.join(NATIVE, "_build", name)
    os.makedirs(os.path.dirname(out), exist_ok=True)
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-fPIC", "-shared", "-Wno-unknown-pragmas", "-I" + CSRC]
                   + defines + ["-o", out + ".tmp", os.path.join(NATIVE, src)], check=True)
    os.replace(out + ".tmp", out)
    return out


@pytest.fixture(scope="module")
def sanitized():
    return build("libwarp_replay_ubsan.so", SANITIZE)


def run(lib_path, hands, jpd=5):
    """The replay in a process of its own, since a failed check ends it: tricks and nodes, or None."""
    code = """
import ctypes, sys, numpy as np
lib, h, jpd = ctypes.CDLL(sys.argv[1]), np.load(sys.argv[2]), int(sys.argv[3])
n = h.shape[0]
p = lambda a: a.ctypes.data_as(ctypes.c_void_p)
out, best = np.full(n * 20, -1, np.int32), np.full(n * 20, -1, np.int8)
nodes, stats = np.zeros(n * jpd, np.uint64), np.zeros(6, np.uint64)
assert lib.warp_replay(p(h), ctypes.c_longlong(n), 10, jpd, 0, None, None, 2, 0, 0, p(out), p(best), p(nodes), p(stats)) == 0
np.savez(sys.argv[2], out=out, nodes=nodes)
"""
    path = os.path.join(NATIVE, "_build", f"bounds_{os.getpid()}.npy")
    np.save(path, np.ascontiguousarray(hands, dtype=np.uint64))
    try:
        r = subprocess.run([sys.executable, "-c", code, lib_path, path, str(jpd)], capture_output=True, text=True, timeout=300)
        if r.returncode != 0:
            return None, r.stderr
        with np.load(path + ".npz") as z:
            return (z["out"], z["nodes"]), ""
    finally:
        for f in (path, path + ".npz"):
            if os.path.exists(f):
                os.remove(f)


def test_within_bounds_on_the_fixtures(sanitized):
    g = load_golden("k5_120.npz")
    got, err = run(sanitized, g["hands"][:40])
    assert got is not None, err
    assert (got[0].reshape(-1, 5, 4) == g["tricks"][:40]).all() and (got[1] == g["nodes_jpd5"][:200]).all()


def unchecked_deal(seat, north, top, void):
    """All 52 cards: `seat` holds every other rank from `top` down of the suits but `void` (each a
    candidate of its own), North `north` cards, which sets the tricks, the others the rest."""
    own = [16 * s + r for s in range(4) if s != void for r in range(top, -1, -2)]
    rest = [16 * s + r for s in [void] + [x for x in range(4) if x != void] for r in range(13)]
    rest = [c for c in rest if c not in own]
    hands = np.zeros(4, np.uint64)
    hands[seat] = sum(1 << c for c in own)
    cards = rest[::len(rest) // north][:north]
    hands[0] = sum(1 << c for c in cards)
    rest = [c for c in rest if c not in cards]
    for k, other in enumerate(x for x in (1, 2, 3) if x != seat):
        hands[other] = sum(1 << c for c in rest[k::2])
    return hands


@pytest.mark.parametrize("seat,north,top,void", [(1, 2, 11, 0), (2, 2, 12, 2), (3, 3, 11, 3), (1, 3, 12, 1)])
def test_hands_of_more_than_thirteen_cards(sanitized, seat, north, top, void):
    """A discard from 18 or 21 candidates, where a hand of 13 has at most 13: what the search
    finds is of no use, but it ends and touches nothing else."""
    got, err = run(sanitized, unchecked_deal(seat, north, top, void)[None])
    assert got is not None, err
    assert (got[0] >= 0).all() and (got[0] <= 13).all()


# ---- the bounds-checked build ----------------------------------------------------------------


def checked(lib_path, hands):
    lib = ctypes.CDLL(lib_path)
    h = np.ascontiguousarray(hands, dtype=np.uint64).reshape(-1, 4)
    out, nodes = np.full(h.shape[0] * 20, -1, np.int32), np.zeros(h.shape[0] * 5, np.uint64)
    report = np.zeros(2, np.uint64)
    p = [a.ctypes.data_as(P) for a in (h, out, nodes, report)]
    assert lib.warp_bounds(p[0], ctypes.c_longlong(h.shape[0]), 10, *p[1:]) == 0
    return out.reshape(-1, 5, 4), nodes, int(report[0]), int(report[1])


def test_checks_change_nothing():
    lib = build("libwarp_bounds.so", ["-DDDG_BOUNDS_CHECK"], "warp_bounds.cpp")
    for name, n in (("k5_120.npz", 60), ("k8_120.npz", 8)):
        g = load_golden(name)
        t, nodes, faults, written = checked(lib, g["hands"][:n])
        assert faults == 0 and written == 0
        assert (t == g["tricks"][:n]).all() and (nodes == g["nodes_jpd5"][:n * 5]).all()
    # more candidates than a hand of 13 has: counted, and the searcher ends
    t, _, faults, _ = checked(lib, unchecked_deal(1, 3, 12, 1))
    assert faults > 0 and (t == -1).any()


def test_planted_small_stack_is_caught_before_the_access():
    """A K-card ending writes 4 (K - 1) frames (its last trick is decided at the lead): a stack
    of 12 holds those of four cards and not those of five."""
    lib = build("libwarp_bounds12.so", ["-DDDG_BOUNDS_CHECK", "-DDDG_STACK_DEPTH=12"], "warp_bounds.cpp")
    g = load_golden("k4_120.npz")
    t, nodes, faults, written = checked(lib, g["hands"][:40])
    assert faults == 0 and written == 0 and (t == g["tricks"][:40]).all() and (nodes == g["nodes_jpd5"][:200]).all()
    g = load_golden("k5_120.npz")
    t, _, faults, written = checked(lib, g["hands"][:40])
    assert written == 0  # nothing behind the twelfth frame
    assert faults > 0 and (t == -1).any() and ((t == -1) | (t == g["tricks"][:40])).all()


@pytest.mark.gpu
@pytest.mark.parametrize("name,kw", [("k6_4096.npz", {}), ("k9_120.npz", {"jobs_per_deal": 20}), ("mixed_300.npz", {})])
def test_checked_lane_per_thread_kernel(ddg, name, kw):
    """The checked library's other kernel (any of its options asks for it) on the large fixtures."""
    import torch
    lib = ddg.load_library(ddg.CHECK_LIB_PATH)
    g = load_golden(name)
    sel = np.arange(len(g["hands"]))
    if name.startswith("mixed"):
        sel = np.where(g["nodes_jpd5"].astype(np.int64).reshape(-1, 5).max(axis=1) < 3_000_000)[0]
    hands = np.ascontiguousarray(g["hands"][sel])
    s = ddg.Solver(free_below=96, library=lib, **kw)  # 96: its default, said aloud
    try:
        d_h = torch.from_numpy(hands.view(np.int64)).cuda()
        d_o = torch.empty(len(sel) * 20, dtype=torch.uint8, device="cuda")
        st = s.solve_device(d_h.data_ptr(), len(sel), d_o.data_ptr())  # raises if a check failed
        assert (d_o.cpu().numpy().reshape(-1, 5, 4) == g["tricks"][sel]).all()
        assert sum(st["phase_warps"]) + st["free_rounds"] > 0 and sum(st["enter_exit"]) > 0  # that kernel ran
    finally:
        s.close()
