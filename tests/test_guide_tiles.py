"""The guide's kernels at the edges of their tiles: batches of one row to one past 32 tiles
(the weight gradients' splits then take two 128-row slices each), and inference of deal
counts that end inside a tile, against the numpy oracle and against themselves."""
import os
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "oracle"))
import guide_ref  # noqa: E402

pytestmark = pytest.mark.gpu


def to_dev(a, dtype):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a).view(dtype)).cuda()


def problem(ddg, deals, seed):
    rng = np.random.default_rng(seed)
    hands = ddg.make_deals(seed, 0, deals, 13)
    tricks = rng.integers(0, 14, (deals, 5, 4)).astype(np.uint8)
    tricks[rng.random(tricks.shape) < 0.1] = 255
    best = np.full((deals, 5, 4), -1, np.int8)
    for d in range(deals):
        for decl in range(4):
            cards = [b for b in range(64) if int(hands[d, (decl + 1) & 3]) >> b & 1]
            best[d, :, decl] = rng.choice(cards, 5)
    best[rng.random(best.shape) < 0.2] = -1
    return hands, tricks, best


@pytest.mark.parametrize("n_rows", [1, 127, 129, 4200])
def test_step_matches_oracle(ddg, n_rows):
    hands, tricks, best = problem(ddg, n_rows // 20 + 1, 31 + n_rows)
    rows = np.random.default_rng(n_rows).permutation(hands.shape[0] * 20)[:n_rows].astype(np.int64)
    params = guide_ref.init_params(5)
    params[guide_ref.OFF_B2:guide_ref.OFF_W3] = 0.03
    guide = ddg.Guide(max_rows=4224, params=params)
    try:
        d = to_dev(hands, np.int64), to_dev(tricks.reshape(-1), np.uint8), to_dev(best.reshape(-1), np.int8)
        loss, hits, labelled, grad = guide.step(*(x.data_ptr() for x in d), rows, 0.0, True)
        again = guide.step(*(x.data_ptr() for x in d), rows, 0.0, True)[3]
        before = guide.params()
        guide.step(*(x.data_ptr() for x in d), rows, 1e-3)
        after = guide.params()
    finally:
        guide.close()
    padded = np.concatenate([rows, np.full(-n_rows % 128, -1, np.int64)])
    ref_loss, ref, _ = guide_ref.loss_and_grads(params, hands, tricks, best, padded)
    assert labelled == (tricks.reshape(-1)[rows] <= 13).sum()
    assert abs(loss - ref_loss) <= 1e-3 * abs(ref_loss)
    assert (grad == again).all()  # the parts are added in a fixed order
    for a, b in ((guide_ref.OFF_W1, guide_ref.OFF_B1), (guide_ref.OFF_B1, guide_ref.OFF_W2),
                 (guide_ref.OFF_W2, guide_ref.OFF_B2), (guide_ref.OFF_B2, guide_ref.OFF_W3),
                 (guide_ref.OFF_W3, guide_ref.OFF_B3), (guide_ref.OFF_B3, guide_ref.N_PARAMS)):
        err = np.linalg.norm(grad[a:b] - ref[a:b]) / max(np.linalg.norm(ref[a:b]), 1e-12)
        assert err < 2e-2, (a, err)
    # the first Adam step moves every parameter that has a gradient by the learning rate
    assert (before == params).all()
    moved = np.abs(grad) > 1e-5
    assert np.allclose(np.abs(after - before)[moved], 1e-3, rtol=1e-2)
    assert (np.sign(before - after)[moved] == np.sign(grad[moved])).all()


def test_predict_ends_inside_a_tile(ddg):
    import torch
    params = guide_ref.init_params(9)
    hands = ddg.make_deals(77, 0, 129, 13)
    d_h = to_dev(hands, np.int64)
    guide = ddg.Guide(max_rows=128, params=params)
    try:
        out = {}
        for n in (1, 7, 32, 129):
            s = torch.full((129 * 20,), 99, dtype=torch.int8, device="cuda")
            h = torch.full((129 * 20,), 99, dtype=torch.int8, device="cuda")
            guide.predict(d_h.data_ptr(), n, s.data_ptr(), h.data_ptr())
            out[n] = s.cpu().numpy(), h.cpu().numpy()
            assert (out[n][0][n * 20:] == 99).all() and (out[n][1][n * 20:] == 99).all()
        only = torch.full((7 * 20,), 99, dtype=torch.int8, device="cuda")
        guide.predict(d_h.data_ptr(), 7, 0, only.data_ptr())
        assert (only.cpu().numpy() == out[7][1][:140]).all()
    finally:
        guide.close()
    for n in (1, 7, 32):
        assert (out[n][0][:n * 20] == out[129][0][:n * 20]).all()
        assert (out[n][1][:n * 20] == out[129][1][:n * 20]).all()
    rows = np.arange(129 * 20)
    blank = np.full((129, 5, 4), 255, np.uint8)
    _, _, L = guide_ref.loss_and_grads(params, hands, blank, blank.view(np.int8), rows)
    sure = lead_sure = 0
    for e in rows:
        t = np.sort(L[e, :14])
        if t[-1] - t[-2] > 2e-2:  # ten bf16 steps of a hidden unit times its weight
            sure += 1
            assert out[129][0][e] == int(L[e, :14].argmax())
        own = int(hands[e // 20, (e % 4 + 1) & 3])
        cards = [c for c in range(52) if own >> guide_ref.card_bit(c) & 1]
        m = L[e, 14:66][cards]
        o = np.sort(m)
        if o[-1] - o[-2] > 2e-2:
            lead_sure += 1
            assert out[129][1][e] == guide_ref.card_bit(cards[int(m.argmax())])
    assert sure > 500 and lead_sure > 500
