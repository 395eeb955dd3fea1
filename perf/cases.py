"""Cases that time the solver's public calls: what a user has it do, from one lead of an
ending to a set of 65,536 deals, a stream, and the learned guide's inference and training.

Deals are seeded (``make_deals``, ``make_deals_mixed``). A uniformly random 13-card deal
takes a lane from a second to hours, so the 13-card cases use the quick ones of the
benchmark stream (seed 2), each under a random relabelling of its suits and a rotation of
its seats: the game's symmetries, under which these deals stay quick (none of a deal's 96
versions has a strain of more than 96,000 search nodes).
"""
import numpy as np
import torch

import dds_gpu_b200 as ddg
from dds_gpu_b200.guide import load_weights

# Deals of the benchmark stream, of its first 2,000, whose hardest strain stays quick.
QUICK_13 = (53, 116, 119, 163, 314, 373, 402, 603, 613, 645, 791, 797, 883, 910, 979, 982, 1084, 1095, 1193,
            1216, 1242, 1254, 1315, 1488, 1494, 1505, 1601, 1632, 1754, 1784, 1852, 1874)
# Mean search nodes of a random deal with K cards a hand (five strains, four leads each),
# and of a quick 13-card deal; a node costs at least 33 bytes of transposition table.
NODES = {3: 90, 4: 330, 5: 1100, 6: 3400, 7: 7100, 8: 16800, 9: 39300, 13: 180000}
NODE_BYTES = 33
DEAL_BYTES = 32 + 20  # hands in, table out

# The guide's layers, for its arithmetic.
G_IN, G_HID, G_OUT, G_TRICKS = 217, 256, 66, 14


def listed():
    return [
        # Every lead of a small ending, asked one at a time (dd_ns_tricks): an analysis tool's questions.
        {"name": "leads_k5", "do": "leads", "k": 5, "stepping": False},
        # The strains of a seven-card ending in turn, four declarers each (dd_solve_strain).
        {"name": "strains_k7", "do": "strains", "k": 7},
        # The table of a few endings from host memory: a teaching or play program's call.
        {"name": "tables_k7_9", "do": "tables", "n": 9, "k": 7},
        # The 4,096 six-card endings of the parity set, host to host.
        {"name": "set_k6_4096", "do": "tables", "n": 4096, "k": 6},
        # A large set of endings resident on the GPU, with each job's node count.
        {"name": "set_k6_65536", "do": "device", "n": 65536, "k": 6, "jpd": 5},
        # Nine-card endings, one job per lead.
        {"name": "set_k9_1200", "do": "device", "n": 1200, "k": 9, "jpd": 20},
        # Full deals as one resumable solve, inputs and tables through pinned host memory.
        {"name": "full_240", "do": "slices", "n": 240},
        # A handful of full deals steered by the learned guide: its seeds and leads, then the solve.
        {"name": "full_guided_11", "do": "guided", "n": 11},
        # Uneven deals (K = 5..9, 30 % skewed) as a replayed graph with a larger table.
        {"name": "uneven_graph_6001", "do": "graph", "n": 6001, "k": 9, "tt": 11, "lanes": 32768},
        # A stream's continuous batching: endings and full deals arriving in bursts.
        {"name": "stream_400", "do": "stream", "n": 400, "k": 8},
        # The guide's inference over a benchmark set.
        {"name": "guide_predict_20000", "do": "predict", "n": 20000, "rows": 8192},
        # One training step of the guide (its default batch), with the gradients.
        {"name": "guide_step_4096", "do": "step", "rows": 4096},
    ]


def _log(rng, lo, hi):
    return int(round(np.exp(rng.uniform(np.log(lo), np.log(hi)))))


def draw(rng):
    do = rng.choice(("leads", "strains", "tables", "tables", "device", "device", "slices", "guided", "graph", "stream",
                     "predict", "step"))
    if do == "leads":
        return {"do": do, "k": rng.randint(4, 7), "stepping": rng.random() < 0.5}
    if do == "strains":
        return {"do": do, "k": rng.randint(4, 8)}
    if do == "tables":
        k = rng.randint(4, 8)
        return {"do": do, "n": _log(rng, 1, {4: 20000, 5: 12000, 6: 8000, 7: 4000, 8: 2000}[k]), "k": k}
    if do == "device":
        k = rng.randint(5, 9)
        return {"do": do, "n": _log(rng, 30, {5: 60000, 6: 60000, 7: 20000, 8: 8000, 9: 1200}[k]), "k": k,
                "jpd": rng.choice((5, 20))}
    if do == "slices":
        return {"do": do, "n": _log(rng, 16, 240)}
    if do == "guided":
        return {"do": do, "n": _log(rng, 3, 150)}
    if do == "graph":
        return {"do": do, "n": _log(rng, 200, 6000), "k": rng.randint(7, 9), "tt": rng.choice((9, 10, 11)),
                "lanes": rng.choice((16384, 32768, 49152))}
    if do == "stream":
        return {"do": do, "n": _log(rng, 50, 400), "k": rng.randint(6, 8)}
    if do == "predict":
        return {"do": do, "n": _log(rng, 20, 20000), "rows": rng.choice((1024, 4096, 8192))}
    return {"do": "step", "rows": _log(rng, 100, 4096)}


def _seed(seed):
    return 1 + (int(seed) * 2654435761) % (1 << 40)


def _full(seed, n):
    """n quick 13-card deals, each under its own symmetry of the game."""
    rng = np.random.default_rng(_seed(seed))
    pool = np.concatenate([ddg.make_deals(2, i, 1, 13) for i in QUICK_13])
    old = pool[rng.integers(0, len(pool), n)]
    perm = np.argsort(rng.random((n, 4)), axis=1)
    new = np.zeros_like(old)
    for s in range(4):
        part = (old >> np.uint64(16 * s)) & np.uint64(0x1FFF)
        new |= part << (np.uint64(16) * perm[:, s].astype(np.uint64))[:, None]
    seat = (np.arange(4)[None, :] + rng.integers(0, 4, n)[:, None]) % 4
    return np.ascontiguousarray(np.take_along_axis(new, seat, axis=1))


def _device(hands):
    return torch.from_numpy(hands.view(np.int64)).cuda()


def prepare(case, seed):
    do, c = case["do"], dict(case)
    if do in ("leads", "strains"):
        rng = np.random.default_rng(_seed(seed))
        return {"case": c, "solver": ddg.Solver(), "hands": ddg.make_deals(_seed(seed), 0, 1, case["k"])[0],
                "guess": int(rng.integers(case["k"] + 1))}
    if do == "tables":
        return {"case": c, "solver": ddg.Solver(), "hands": ddg.make_deals(_seed(seed), 0, case["n"], case["k"])}
    if do == "device":
        n = case["n"]
        return {"case": c, "solver": ddg.Solver(jobs_per_deal=case["jpd"]),
                "hands": _device(ddg.make_deals(_seed(seed), 0, n, case["k"])),
                "out": torch.empty((n, 5, 4), dtype=torch.uint8, device="cuda"),
                "nodes": torch.empty((n, case["jpd"]), dtype=torch.int64, device="cuda")}
    if do == "slices":
        n = case["n"]
        return {"case": c, "solver": ddg.Solver(), "host": torch.from_numpy(_full(seed, n).view(np.int64)).pin_memory(),
                "hands": torch.empty((n, 4), dtype=torch.int64, device="cuda"),
                "out": torch.empty((n, 5, 4), dtype=torch.uint8, device="cuda"),
                "host_out": torch.empty((n, 5, 4), dtype=torch.uint8).pin_memory()}
    if do == "guided":
        n = case["n"]
        return {"case": c, "solver": ddg.Solver(), "guide": ddg.Guide(max_rows=4096, params=load_weights()),
                "hands": _device(_full(seed, n)),
                "seeds": torch.empty((n, 5, 4), dtype=torch.int8, device="cuda"),
                "hints": torch.empty((n, 5, 4), dtype=torch.int8, device="cuda"),
                "best": torch.empty((n, 5, 4), dtype=torch.int8, device="cuda"),
                "nodes": torch.empty((n, 5), dtype=torch.int64, device="cuda"),
                "out": torch.empty((n, 5, 4), dtype=torch.uint8, device="cuda")}
    if do == "graph":
        n = case["n"]
        return {"case": c, "solver": ddg.Solver(tt_log2=case["tt"], lanes=case["lanes"]),
                "hands": _device(ddg.make_deals_mixed(_seed(seed), 0, n, 5, case["k"], 0.3)),
                "out": torch.empty((n, 5, 4), dtype=torch.uint8, device="cuda")}
    if do == "stream":
        n, rng = case["n"], np.random.default_rng(_seed(seed) + 1)
        hands = ddg.make_deals_mixed(_seed(seed), 0, n, 7 if case["k"] >= 7 else 6, case["k"], 0.0)
        full = _full(seed, n)
        pick = rng.random(n) < 0.25
        hands[pick] = full[pick]
        return {"case": c, "solver": ddg.Solver(), "hands": np.ascontiguousarray(hands)}
    if do == "predict":
        n = case["n"]
        return {"case": c, "guide": ddg.Guide(max_rows=case["rows"], params=load_weights()),
                "hands": _device(ddg.make_deals(_seed(seed), 0, n, 13)),
                "seeds": torch.empty((n, 5, 4), dtype=torch.int8, device="cuda"),
                "hints": torch.empty((n, 5, 4), dtype=torch.int8, device="cuda")}
    data = _step_data(case, seed)
    return {"case": c, "guide": ddg.Guide(max_rows=4096, params=data["params"]), "params": data["params"],
            "hands": _device(data["hands"]), "tricks": torch.from_numpy(data["tricks"]).cuda(),
            "best": torch.from_numpy(data["best"]).cuda(), "rows": data["rows"]}


def _step_data(case, seed):
    """Examples as the trainer has them: a table of trick counts and best leads, some
    entries without a label, and a shuffled batch of their indices."""
    rng = np.random.default_rng(_seed(seed))
    deals = max(8, case["rows"] // 10)
    hands = ddg.make_deals(_seed(seed), 0, deals, 13)
    tricks = np.clip(np.rint(rng.normal(6.5, 2.5, (deals, 20))), 0, 13).astype(np.uint8)
    best = np.full((deals, 20), -1, np.int8)
    for d in range(deals):
        for e in range(20):
            own = int(hands[d, (e % 4 + 1) & 3])
            cards = [b for b in range(64) if own >> b & 1]
            best[d, e] = cards[rng.integers(len(cards))]
    hidden = rng.random((deals, 20))
    tricks[hidden < 0.1] = 255
    best[hidden < 0.2] = -1
    rows = rng.permutation(deals * 20)[:case["rows"]].astype(np.int64)
    params = load_weights() + rng.normal(0, 0.01, ddg.Guide.param_count()).astype(np.float32)
    return {"hands": hands, "tricks": tricks, "best": best, "rows": rows, "params": params}


def run(state):
    c, do = state["case"], state["case"]["do"]
    if do == "leads":
        return np.array([state["solver"].ns_tricks(state["hands"], strain, leader, state["guess"], c["stepping"])
                         for strain in range(5) for leader in range(4)])
    if do == "strains":
        return np.array([state["solver"].solve_strain(state["hands"], strain) for strain in range(5)])
    if do == "tables":
        return state["solver"].solve(state["hands"])
    if do == "device":
        state["solver"].solve_device(state["hands"].data_ptr(), c["n"], state["out"].data_ptr(),
                                     d_job_nodes=state["nodes"].data_ptr())
        return state["out"], state["nodes"]
    if do == "slices":
        s = state["solver"]
        s.begin(state["hands"].data_ptr(), c["n"], state["out"].data_ptr())
        done = False
        while not done:
            done, _ = s.resume(5.0, state["host"].data_ptr(), state["host_out"].data_ptr())
        return state["host_out"]
    if do == "guided":
        state["guide"].predict(state["hands"].data_ptr(), c["n"], state["seeds"].data_ptr(), state["hints"].data_ptr())
        state["solver"].solve_device(state["hands"].data_ptr(), c["n"], state["out"].data_ptr(),
                                     d_seeds=state["seeds"].data_ptr(), d_hints=state["hints"].data_ptr(),
                                     d_best=state["best"].data_ptr(), d_job_nodes=state["nodes"].data_ptr())
        return [state[k] for k in ("seeds", "hints", "out", "best", "nodes")]
    if do == "graph":
        state["solver"].solve_graph(state["hands"].data_ptr(), c["n"], state["out"].data_ptr())
        return state["out"]
    if do == "stream":
        n, sent, seen = c["n"], 0, 0
        tables = np.empty((n, 5, 4), np.uint8)
        st = ddg.Stream(state["solver"], ring_slots=1024, idle_timeout_s=10)
        while seen < n:
            if sent < n:
                sent += st.submit(state["hands"][sent:sent + 64])
            idx, tab = st.poll()
            tables[idx.astype(np.int64)] = tab
            seen += len(idx)
        st.close()
        return tables
    if do == "predict":
        state["guide"].predict(state["hands"].data_ptr(), c["n"], state["seeds"].data_ptr(), state["hints"].data_ptr())
        return state["seeds"], state["hints"]
    g = state["guide"]
    g.set_params(state["params"])
    loss, hits, labelled, grad = g.step(state["hands"].data_ptr(), state["tricks"].data_ptr(), state["best"].data_ptr(),
                                        state["rows"], 1e-3, want_grad=True)
    return {"loss": loss, "hits": int(hits), "labelled": int(labelled), "grad": grad}


def work(case):
    """Bytes: deals in, tables out, and the search's table traffic of a random deal of
    that size; for the guide, its inputs and outputs. Flops: the guide's products."""
    do = case["do"]
    mlp = 2 * (G_IN * G_HID + G_HID * G_HID + G_HID * G_OUT)
    if do in ("leads", "strains", "tables", "device"):
        return {"bytes": case.get("n", 1) * (DEAL_BYTES + NODES[case["k"]] * NODE_BYTES), "flops": 0}
    if do == "slices":
        return {"bytes": case["n"] * (DEAL_BYTES + NODES[13] * NODE_BYTES), "flops": 0}
    if do == "guided":
        return {"bytes": case["n"] * (DEAL_BYTES + NODES[13] * NODE_BYTES), "flops": case["n"] * 20 * mlp}
    if do == "graph":
        mean = np.mean([NODES[k] for k in range(5, case["k"] + 1)])
        return {"bytes": case["n"] * (DEAL_BYTES + mean * NODE_BYTES), "flops": 0}
    if do == "stream":
        mean = 0.75 * np.mean([NODES[k] for k in range(min(7, case["k"]), case["k"] + 1)]) + 0.25 * NODES[13]
        return {"bytes": case["n"] * (DEAL_BYTES + mean * NODE_BYTES), "flops": 0}
    if do == "predict":
        return {"bytes": case["n"] * (32 + 40) + 4 * mlp / 2, "flops": case["n"] * 20 * mlp}
    # forward, the gradients of the weights, and of the two hidden layers' inputs
    back = 2 * (G_HID * G_HID + G_HID * G_OUT)
    return {"bytes": case["rows"] * (8 + 32 + 2) + 8 * 4 * mlp / 2, "flops": case["rows"] * (2 * mlp + back)}


def exact(case, seed):
    if case["do"] != "step":
        return None  # trick counts, seeds and leads are whole numbers
    d = _step_data(case, seed)
    rows, padded = d["rows"], (case["rows"] + 127) // 128 * 128
    deal, e = rows // 20, rows % 20
    decl = e % 4
    bit = np.array([(c // 13) * 16 + c % 13 for c in range(52)])
    x = np.zeros((len(rows), 256))
    held = (d["hands"][deal][:, :, None] >> bit.astype(np.uint64)[None, None, :]) & np.uint64(1)  # (row, seat, card)
    x[:, :208] = np.moveaxis(held, 1, 2).reshape(len(rows), 208)
    x[np.arange(len(rows)), 208 + e // 4] = 1
    x[np.arange(len(rows)), 213 + (decl + 1) % 4] = 1
    x = torch.from_numpy(x).double().cuda()
    flat = torch.from_numpy(d["params"]).double().cuda().requires_grad_()
    parts = torch.split(flat, [256 * 256, 256, 256 * 256, 256, 80 * 256, 80])
    h = torch.nn.functional.gelu(x @ parts[0].view(256, 256).T + parts[1])
    h = torch.nn.functional.gelu(h @ parts[2].view(256, 256).T + parts[3])
    o = h @ parts[4].view(80, 256).T + parts[5]
    t = d["tricks"].reshape(-1)[rows].astype(np.int64)
    ok = t <= 13
    ns = np.where(decl % 2 == 0, t, 13 - t)
    logp = torch.log_softmax(o[:, :G_TRICKS], 1)
    on = torch.from_numpy(np.nonzero(ok)[0]).cuda()
    loss = -logp[on, torch.from_numpy(ns[ok]).cuda()].sum()
    best = d["best"].reshape(-1)[rows].astype(np.int64)
    own = held[np.arange(len(rows)), (decl + 1) % 4]  # the leader's cards
    lead = np.nonzero(ok & (best >= 0))[0]
    y = (best[lead] >> 4) * 13 + (best[lead] & 15)
    masked = o[torch.from_numpy(lead).cuda(), G_TRICKS:G_OUT].masked_fill(torch.from_numpy(own[lead] == 0).cuda(), -float("inf"))
    loss = loss - torch.log_softmax(masked, 1)[torch.arange(len(lead)).cuda(), torch.from_numpy(y).cuda()].sum()
    loss = loss / padded
    loss.backward()
    return {"loss": float(loss), "hits": None, "labelled": int(ok.sum()), "grad": flat.grad.cpu().numpy()}
