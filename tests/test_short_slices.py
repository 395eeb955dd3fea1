"""A resumable solve ends whatever the length of its slices: in each, a searcher without a job
takes one, also when the slice was over before the kernel had started up."""
import numpy as np
import pytest

from conftest import load_golden

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seconds", [1e-9, 1e-6, 5e-6])
@pytest.mark.parametrize("kw", [{"lanes": 512}, {}, {"lanes": 512, "free_below": 96}])
def test_any_slice_gets_on(ddg, kw, seconds):
    import torch
    g = load_golden("k5_120.npz")
    n = len(g["hands"])
    s = ddg.Solver(**kw)
    try:
        d_h = torch.from_numpy(g["hands"].view(np.int64)).cuda()
        d_o = torch.empty(n * 20, dtype=torch.uint8, device="cuda")
        s.begin(d_h.data_ptr(), n, d_o.data_ptr())
        finished, slices, jobs = False, 0, 0
        while not finished and slices < 3000:  # 600 jobs of at most 1,245 nodes
            finished, st = s.resume(seconds)
            slices, jobs = slices + 1, jobs + st["jobs_done"]
        assert finished and jobs == n * 5
        assert (d_o.cpu().numpy().reshape(n, 5, 4) == g["tricks"]).all()
    finally:
        s.close()
