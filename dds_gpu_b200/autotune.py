"""Autotuner and the uneven-hardness batch in one persistent, graph-launched solve.

    python -m dds_gpu_b200.autotune [--jobs 200000] [--window 3] [--limit 300] [--out FILE]

Workload: (deal, strain) jobs over deals from ddg_make_deals_mixed (K uniform in 5..13
cards per seat, 30 % skewed with a 7-10 card suit facing a void), seed 7.

The tuner sweeps the launch shape (512 threads x 1 block or 256 x 2 per SM), solver lanes
and the kernel's stage schedule (block phases or per-warp queues) at one TT size; each
candidate runs a short resumable slice of the same set and is scored by the search nodes
it covers per second. The TT size (2^9..2^12 buckets per lane) is then the largest that
fits beside the chosen lanes (tune() says why node rates do not rank TT sizes). Lane counts
that make the same pool (of the warp kernel, which 512 x 1 with block phases runs: at most 32
an SM) are one candidate. The chosen setting then solves the whole set as one CUDA-graph launch of the persistent kernel
(optionally with helping: idle lanes split the last hard jobs in shared TTs; --help-lanes),
with per-job completion times for the tail.
"""
import argparse
import itertools
import json
import time

import numpy as np

from . import DDGError, Solver, make_deals_mixed

LANES = (16384, 32768, 49152, 0)  # 0 = every resident lane (148 SMs x 512)
SHAPES = ((512, 1), (256, 2))     # threads per block, resident blocks per SM
TT_LOG2 = (9, 10, 11, 12)
SCHEDULES = (0, 1)
SEED = 7


def measure(cfg, d_hands, n, window_s, torch, seen=()):
    """Search nodes and finished jobs per second, and the pool's lanes (None for the rates of a
    pool whose lanes are among `seen`), in one slice of `window_s` after a 1 s
    warm-up slice. Nodes per second scores a setting: a short slice's finished jobs
    favour settings that turn over the smallest jobs quickly, while the batch's end is set
    by how fast the search work as a whole goes."""
    s = Solver(tt_log2=cfg["tt_log2"], lanes=cfg["lanes"], block=cfg["block"], min_blocks=cfg["min_blocks"],
               jobs_per_deal=5, schedule=cfg["schedule"])
    try:
        if s.lanes in seen:
            return None, None, s.lanes
        d_out = torch.empty(n * 20, dtype=torch.uint8, device=d_hands.device)
        s.begin(d_hands.data_ptr(), n, d_out.data_ptr())
        _, warm = s.resume(1.0)
        _, st = s.resume(window_s)
        if st["kernel_ms"] == 0:  # a small set was solved in the warm-up slice: score that one
            st = warm
        sec = st["kernel_ms"] * 1e-3
        return st["nodes"] / sec, st["jobs_done"] / sec, s.lanes
    finally:
        s.close()


def tune(d_hands, n, window_s, torch, log=print):
    """Launch shape, lanes and stage schedule by node rate at one TT size (a job then costs
    the same nodes in every candidate, so nodes per second compares them fairly); then the
    TT size: the largest of TT_LOG2 that fits beside the chosen lanes. Node rates of other
    TT sizes are not comparable (a larger table answers more positions, so the same job
    takes fewer nodes: 1.5-2.5x fewer for hard 13-card jobs at 2^12 than at 2^10, at about
    the same node rate), so they are measured and reported, not used to rank."""
    results, seen = [], {}
    base_tt = 10 if 10 in TT_LOG2 else TT_LOG2[0]
    for (block, minb), lanes, sch in itertools.product(SHAPES, LANES, SCHEDULES):
        cfg = {"block": block, "min_blocks": minb, "lanes": lanes, "tt_log2": base_tt, "schedule": sch}
        pools = seen.setdefault((block, minb, sch), set())
        try:
            rate, jobs_rate, used = measure(cfg, d_hands, n, window_s, torch, pools)
        except DDGError as e:  # e.g. the TTs do not fit
            log(f"  {cfg}: {e}")
            continue
        if rate is None:
            log(f"  {cfg}: the pool of {used} lanes again")
            continue
        pools.add(used)
        cfg["lanes"] = used
        cfg["jobs_per_s"] = jobs_rate
        results.append((rate, cfg))
        log(f"  block {block}x{minb} lanes {used:6d} TT 2^{base_tt} schedule {sch}: {rate / 1e6:7.1f} M nodes/s, "
            f"{jobs_rate:9.1f} jobs/s")
    results.sort(key=lambda r: -r[0])
    best = dict(results[0][1])
    for tt in sorted(TT_LOG2, reverse=True):
        cfg = dict(best, tt_log2=tt)
        try:
            rate, jobs_rate, used = measure(cfg, d_hands, n, window_s, torch)
        except DDGError as e:
            log(f"  TT 2^{tt}: {e}")
            continue
        if used < best["lanes"]:  # the larger tables do not fit beside the chosen lanes
            log(f"  TT 2^{tt}: only {used} lanes fit")
            continue
        cfg["jobs_per_s"] = jobs_rate
        results.append((rate, cfg))
        log(f"  TT 2^{tt} at the chosen shape: {rate / 1e6:7.1f} M nodes/s")
        best = cfg
        break
    return best, results


def run_batch(cfg, d_hands, n, limit_s, torch, tables=False, help=False):
    """The whole set as one graph-launched persistent solve; completion-time tail (and the
    tables, (n, 5, 4) uint8 with 255 = unsolved, under "tables" when asked)."""
    help = help and cfg["schedule"] != 1
    # Helping runs on the lane-per-thread kernel: a pool tuned for the warp kernel (a search to a
    # warp, at most 32 on an SM) would fill few of its blocks, so it takes every lane instead.
    by_warp = (cfg["block"], cfg["min_blocks"], cfg["schedule"]) == (512, 1, 0)
    s = Solver(tt_log2=cfg["tt_log2"], lanes=0 if help and by_warp else cfg["lanes"], block=cfg["block"],
               min_blocks=cfg["min_blocks"], jobs_per_deal=5, schedule=cfg["schedule"], help=1 if help else 0,
               time_limit_s=limit_s)
    try:
        d_out = torch.empty(n * 20, dtype=torch.uint8, device=d_hands.device)
        d_end = torch.zeros(n * 5, dtype=torch.int64, device=d_hands.device)
        s.set_job_times(d_end.data_ptr())
        st = s.solve_graph(d_hands.data_ptr(), n, d_out.data_ptr())
        ends = d_end.cpu().numpy().astype(np.float64)
        out = d_out.cpu().numpy()
    finally:
        s.close()
    done = ends[ends > 0]
    t0 = done.min() if len(done) else 0.0
    rel = np.sort(done - t0) / 1e6  # ms after the first job finished
    q = (lambda p: float(rel[min(len(rel) - 1, int(p * len(rel)))])) if len(rel) else (lambda p: None)
    unsolved = int((out == 255).sum())
    deals_done = int(((out.reshape(n, 20) != 255).all(axis=1)).sum())
    rep = {"kernel_ms": st["kernel_ms"], "jobs": n * 5, "jobs_done": int(st["jobs_done"]),
           "deals_complete": deals_done, "deals_per_s": deals_done / (st["kernel_ms"] * 1e-3),
           "nodes": int(st["nodes"]), "helping_tasks": int(st["tasks"]), "unsolved_results": unsolved,
           "completion_ms": {"p50": q(0.5), "p90": q(0.9), "p99": q(0.99), "last": q(1.0)},
           "tail_ms_last_1pct": (q(1.0) - q(0.99)) if len(rel) else None,
           "time_limit_s": limit_s}
    if tables:
        rep["tables"] = out.reshape(n, 5, 4)
    return rep


def main():
    import torch
    p = argparse.ArgumentParser()
    p.add_argument("--jobs", type=int, default=200000, help="(deal, strain) jobs: deals = jobs / 5")
    p.add_argument("--window", type=float, default=3.0, help="tuning slice per candidate, seconds")
    p.add_argument("--limit", type=float, default=300.0, help="time limit of the full batch, seconds")
    p.add_argument("--help-lanes", action="store_true", help="idle lanes help with the last hard jobs")
    p.add_argument("--out", default="")
    a = p.parse_args()
    n = a.jobs // 5
    hands = make_deals_mixed(SEED, 0, n, 5, 13, 0.3)
    d_hands = torch.from_numpy(hands.view(np.int64)).cuda()
    t0 = time.time()
    best, results = tune(d_hands, n, a.window, torch)
    print(f"autotuner ({time.time() - t0:.0f} s): block {best['block']}x{best['min_blocks']}, lanes {best['lanes']}, "
          f"TT 2^{best['tt_log2']}, schedule {best['schedule']}", flush=True)
    rep = run_batch(best, d_hands, n, a.limit, torch, help=a.help_lanes)
    rep.update({"workload": f"{n} deals from ddg_make_deals_mixed(seed {SEED}, K 5..13, 30% skewed), "
                            f"{a.jobs} (deal, strain) jobs, one CUDA-graph launch, "
                            f"helping {'on' if a.help_lanes else 'off'}",
                "autotuner_choice": best,
                "autotuner_table": [{"nodes_per_s": r, **c} for r, c in results]})
    print(json.dumps(rep), flush=True)
    if a.out:
        with open(a.out, "w") as f:
            json.dump(rep, f, indent=1)


if __name__ == "__main__":
    main()
