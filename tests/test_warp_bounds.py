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


def build(name, defines):
    out = os.path.join(NATIVE, "_build", name)
    os.makedirs(os.path.dirname(out), exist_ok=True)
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-fPIC", "-shared", "-Wno-unknown-pragmas", "-I" + CSRC]
                   + defines + ["-o", out + ".tmp", os.path.join(NATIVE, "warp_replay.cpp")], check=True)
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
