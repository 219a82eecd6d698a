"""Split scoring: the level kernel's choice and the stand-alone kernel's against scores in 64 bits from the same histograms."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("widths,depth", [
    ([17] * 8, 1), ([17] * 8, 3), ([3] * 28, 4),                 # few bins: a warp for every leaf
    ([129] * 12, 4), ([255] * 16, 2),                            # few columns
    ([129] * 28, 4), ([129] * 28, 6), ([255] * 39, 8),           # pairs of children: 4, 16 and 64 of them
    ([256] * 3 + [2] * 30 + [65] * 7, 7),
])
def test_best_split_has_the_best_score(widths, depth, n=20_011):
    from catboost_b200.data.quantization import FlatFeature, make_store, pack_columns_into
    from catboost_b200.ops import native
    from catboost_b200.train.gpu_engine import GpuObliviousEngine
    from catboost_b200.train.objectives import make_objective
    l2 = 3.0
    rng = np.random.default_rng(len(widths) + depth)
    cols = np.stack([rng.integers(0, w, n) for w in widths]).astype(np.uint8)
    feats = [FlatFeature("float", j, borders=np.arange(w - 1, dtype=np.float32), n_bins=w) for j, w in enumerate(widths)]
    store = make_store(feats, n, torch.device("cuda"))
    pack_columns_into(store, torch.from_numpy(cols).cuda(), 0)
    y = (sum(cols[j] / widths[j] for j in range(5)) + 0.3 * rng.standard_normal(n)).astype(np.float32)
    eng = GpuObliviousEngine(store, torch.from_numpy(y), None, torch.zeros(n), make_objective("RMSE", {}), depth=depth, iterations=2,
                             learning_rate=0.5, l2_leaf_reg=l2, random_strength=0.0, bootstrap_type="Bayesian", leaf_iterations=1,
                             seed=3, lane_hist=True)
    eng.step(1)
    torch.cuda.synchronize()
    level, W = depth - 1, eng.Wmax
    parents = max(1, 1 << (level - 1)) if level else 1
    got = eng.slots[: parents * 2 * W].view(parents, 2, W).cpu().numpy().astype(np.float64)
    prev = eng.hbuf[(level + 1) & 1][:parents].cpu().numpy().astype(np.float64)
    leaves = [got] if level == 0 else [got, prev - got]
    off, best, score = store.feat_off_host, -np.inf, {}
    for f, w in enumerate(widths):
        num, den = np.zeros(w - 1), np.zeros(w - 1)
        for h in leaves:
            s, g = h[:, 0, off[f]: off[f] + w].cumsum(1), h[:, 1, off[f]: off[f] + w].cumsum(1)
            for ss, ww in ((s[:, :-1], g[:, :-1]), (s[:, -1:] - s[:, :-1], g[:, -1:] - g[:, :-1])):
                ww = np.maximum(ww, 0.0)
                mu = np.where(ww > 1e-3, ss / (ww + l2), 0.0)
                num += (ss * mu).sum(0)
                den += (ww * mu * mu).sum(0)
        score[f] = num / np.sqrt(den + 1e-10)
        best = max(best, score[f].max())
    split = eng.splits[level].cpu().numpy()
    # fp32 prefix sums and terms of up to 128 leaves
    assert score[int(split[0])][int(split[1])] >= best * (1.0 - 1e-5)
    # the stand-alone kernel (its shared memory is all that a block has without asking for more)
    eng.best_key.zero_()
    src = (ctypes.c_void_p * 1)(eng.slots.data_ptr())
    P = lambda t: ctypes.c_void_p(t.data_ptr())
    native.cuda_check(eng.lib.cb_score(
        ctypes.c_void_p(store.handle), src, 1, P(eng.hbuf[(level + 1) & 1]), None, W, 0, 0, store.F, level, 2,
        P(eng.mask[level & 1]), l2, eng.score_fn, 0.0, P(eng.scal), P(eng.iter_ptr), eng.score_seed, 0.5, P(eng.best_key),
        eng._stream()), "cb_score")
    key = int(eng.best_key.cpu().numpy().view(np.uint64)[0])
    eng.best_key.zero_()
    col = 0xFFFFFFFF - (key & 0xFFFFFFFF)
    f = int(np.searchsorted(off, col, side="right")) - 1
    assert score[f][col - int(off[f])] >= best * (1.0 - 1e-5)
    eng.finish()
    eng.close()


@pytest.mark.parametrize("widths,depth", [([129] * 5, 2), ([255] * 16, 4)])
def test_best_split_of_few_columns_and_many_rows(widths, depth):
    """A warp for every leaf, whatever the number of bins, from 2^20 rows on."""
    test_best_split_has_the_best_score(widths, depth, n=(1 << 20) + 7)
