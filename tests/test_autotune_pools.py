"""The autotuner measures a pool once: lane counts that make the same pool (the warp kernel's, at
most 32 lanes an SM) are one candidate, and the larger TT is tried on the pool that won."""
import types

from dds_gpu_b200 import autotune


class FakeSolver:
    made = []
    most = 4736  # of the warp kernel: 32 lanes an SM

    def __init__(self, tt_log2, lanes, block, min_blocks, jobs_per_deal, schedule):
        warp = (block, min_blocks, schedule) == (512, 1, 0)
        lanes = lanes or 75776
        self.lanes = min(lanes, self.most) if warp else lanes // block * block
        self.key = (block, min_blocks, schedule, self.lanes, tt_log2)
        self.rate = 2000.0 if warp else 600.0 + self.lanes / 1000

    def begin(self, *a):
        pass

    def resume(self, seconds):
        FakeSolver.made.append(self.key)
        return False, {"kernel_ms": 1000.0 * seconds, "nodes": self.rate * seconds, "jobs_done": 7, "lanes": 1}

    def close(self):
        pass


def test_each_pool_once(monkeypatch):
    monkeypatch.setattr(autotune, "Solver", FakeSolver)
    FakeSolver.made = []
    buffer = types.SimpleNamespace(data_ptr=lambda: 0, device="cpu")
    torch = types.SimpleNamespace(empty=lambda *a, **k: buffer, uint8=None)
    best, results = autotune.tune(buffer, 10, 2.0, torch, log=lambda s: None)
    measured = FakeSolver.made[::2]  # a warm-up slice, then the scored one
    assert len(measured) == len(set(measured)) == len(results)
    assert sum(k[:3] == (512, 1, 0) for k in measured) == 2  # its pool, at 2^10 and at the largest TT
    assert len([k for k in measured if k[:3] == (256, 2, 0)]) == len(autotune.LANES)  # four pools there
    assert (best["block"], best["lanes"], best["tt_log2"]) == (512, 4736, max(autotune.TT_LOG2))
