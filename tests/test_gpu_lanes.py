"""The feature-per-lane histogram pass against sums in 64 bits, at the sizes where its row blocks, lane widths, slot passes
and document blocks end."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _store(n, widths, seed, sparse=False):
    """A binned store with one column per entry of ``widths`` (number of bins); bins drawn, not quantised."""
    from catboost_b200.data.quantization import FlatFeature, make_store, pack_columns_into
    rng = np.random.default_rng(seed)
    feats = [FlatFeature("float", j, borders=np.arange(w - 1, dtype=np.float32), n_bins=w) for j, w in enumerate(widths)]
    store = make_store(feats, n, torch.device("cuda"))
    cols = np.stack([rng.integers(0, w, n) for w in widths]).astype(np.uint8)
    if sparse:
        cols[rng.random(cols.shape) < 0.7] = 0
    pack_columns_into(store, torch.from_numpy(cols).cuda(), 0)
    return store, cols


def _engine(store, y, depth, lane_hist, **kw):
    from catboost_b200.train.gpu_engine import GpuObliviousEngine
    from catboost_b200.train.objectives import make_objective
    args = dict(depth=depth, iterations=2, learning_rate=0.5, l2_leaf_reg=3.0, random_strength=0.0, bootstrap_type="Bayesian",
                leaf_iterations=1, seed=3, lane_hist=lane_hist)
    args.update(kw)
    return GpuObliviousEngine(store, torch.from_numpy(y), None, torch.zeros(len(y)), make_objective("RMSE", {}), **args)


@pytest.mark.parametrize("n,widths,depth,sparse", [
    (1, [5] * 5, 1, False),
    (255, [2, 3, 200, 7, 9], 3, False),
    (1023, [17] * 8, 4, False),                      # one row block of two groups: 16 documents a load
    (1025, [129] * 9, 6, False),                     # three groups: 8 documents a load
    (30_011, [129] * 28, 6, False),                  # seven groups: 4 documents a load, several slot passes
    (30_011, [129] * 28, 6, True),
    (260_003, [129] * 28, 6, False),                 # a chunk for every SM
    (5_000, [256] * 18, 6, False),                   # the widest columns, a row block of five groups
    (20_007, [255] * 33 + [2] * 6, 7, False),        # a second row block of two groups
    (9_999, [129] * 13 + [16] * 25 + [2] * 40, 8, True),     # narrow columns next to wide ones
])
def test_lane_histograms_equal_sums_in_64_bits(n, widths, depth, sparse, lane_seq_docs=None):
    store, cols = _store(n, widths, seed=n + len(widths), sparse=sparse)
    rng = np.random.default_rng(n)
    y = (cols[0] / widths[0] + 0.3 * rng.standard_normal(n) + (cols[-1] > 0)).astype(np.float32)
    eng = _engine(store, y, depth, True, lane_seq_docs=lane_seq_docs)
    assert (eng.lane_list is not None) == (lane_seq_docs == 0)
    eng.step(1)
    torch.cuda.synchronize()
    level = depth - 1
    nslots = 1 if level == 0 else 1 << (level - 1)
    W = eng.Wmax
    got = eng.slots[: nslots * 2 * W].view(nslots, 2, W).cpu().numpy().astype(np.float64)
    stats = eng.stats[:, :n].cpu().numpy().astype(np.float64)
    leaf = eng.leaf[:n].cpu().numpy().astype(np.int64) & 0xFFFF
    # leaf indices hold every split of the tree; those of the levels before this one decide the slot and the child
    sp = eng.splits[:depth].cpu().numpy()
    for d in range(depth):
        bit = (cols[sp[d, 0]] > sp[d, 1]) if sp[d, 0] >= 0 else np.zeros(n, dtype=bool)
        assert np.array_equal((leaf >> d) & 1, bit.astype(np.int64)), d
    take, slot = np.ones(n, dtype=bool), np.zeros(n, dtype=np.int64)
    if level > 0:
        slot = leaf & (nslots - 1)
        mask = eng.mask[level & 1].cpu().numpy().view(np.uint32)
        want = (mask[slot >> 5] >> (slot & 31).astype(np.uint32)) & 1
        take = ((leaf >> (level - 1)) & 1) == want
    # a value is rounded to half a quantum; a cell holds at most n documents, so the quantum is at most
    # max / (2^31 / n - 2), or max / 8388600 when that is coarser
    smax = np.abs(stats).max(1)
    quantum = smax / np.minimum(8388600.0, 2.0 ** 31 / (n + 2) - 2.0)
    off = store.feat_off_host
    for f, w in enumerate(widths):
        for s in range(2):
            oracle = np.zeros((nslots, w))
            count = np.zeros((nslots, w))
            mass = np.zeros((nslots, w))
            np.add.at(oracle, (slot[take], cols[f][take]), stats[s][take])
            np.add.at(count, (slot[take], cols[f][take]), 1.0)
            np.add.at(mass, (slot[take], cols[f][take]), np.abs(stats[s][take]))
            err = np.abs(got[:, s, off[f]: off[f] + w] - oracle)
            # rounding of the documents, of the scale (24 bits), and of the fp32 sums over the chunks
            tol = 0.5 * quantum[s] * count + mass * 2.0 ** -20 + 1e-30
            assert (err <= tol).all(), (f, s, float((err / tol).max()))
    eng.finish()
    eng.close()


@pytest.mark.parametrize("n,F,borders,depth", [(40_001, 30, 128, 6), (3_000, 12, 128, 6), (60_013, 39, 254, 8)])
def test_lane_pass_grows_the_trees_of_the_other_pass(n, F, borders, depth):
    store, cols = _store(n, [borders + 1] * F, seed=F)
    rng = np.random.default_rng(1)
    y = (np.sin(cols[0] / 20.0) + (cols[1] > 60) * (cols[2] > 40) + 0.01 * cols[5] + 0.2 * rng.standard_normal(n)).astype(np.float32)
    outs = []
    for lanes in (True, False):
        eng = _engine(store, y, depth, lanes, iterations=3, leaf_iterations=2)
        eng.step(3)
        outs.append([a.copy() for a in eng.finish()] + [eng.learn_loss_history()])
        eng.close()
    # the first tree sees the same statistics; a later level of it may meet two candidates equal to within the quantum
    same = (outs[0][0][0, :, :2] == outs[1][0][0, :, :2]).all(-1)
    assert same[: min(depth, 5)].all(), (outs[0][0][0], outs[1][0][0])
    assert np.allclose(outs[0][3], outs[1][3], rtol=5e-3)


@pytest.mark.parametrize("n,weighted,steps", [(1, False, 1), (33, True, 3), (40_001, False, 3), (40_001, True, 1)])
def test_logloss_leaf_steps_equal_newton_steps_in_64_bits(n, weighted, steps):
    """Logloss leaves: every step, the first included, adds fixed-point values scaled by the loss's own bounds."""
    from catboost_b200.train.objectives import make_objective
    from catboost_b200.train.gpu_engine import GpuObliviousEngine
    store, cols = _store(n, [33] * 6, seed=n)
    rng = np.random.default_rng(n)
    y = (rng.random(n) < 1.0 / (1.0 + np.exp(-(cols[0] / 8.0 - 2.0)))).astype(np.float32)
    w = (rng.random(n) * 1000.0).astype(np.float32) if weighted else np.ones(n, dtype=np.float32)
    start = (3.0 * rng.standard_normal(n)).astype(np.float32)
    eng = GpuObliviousEngine(store, torch.from_numpy(y), torch.from_numpy(w) if weighted else None, torch.from_numpy(start),
                             make_objective("Logloss", {}), depth=4, iterations=2, learning_rate=1.0, l2_leaf_reg=3.0,
                             random_strength=0.0, bootstrap_type="No", leaf_iterations=steps, leaf_backtracking="No", lane_hist=True)
    eng.step(1)
    torch.cuda.synchronize()
    leaf = eng.leaf[:n].cpu().numpy().astype(np.int64) & 0xFFFF
    delta = np.zeros(16)
    for _ in range(steps):
        p = 1.0 / (1.0 + np.exp(-(start.astype(np.float64) + delta[leaf])))
        der, hess = np.zeros(16), np.zeros(16)
        np.add.at(der, leaf, w * (y - p))
        np.add.at(hess, leaf, w * p * (1.0 - p))
        delta += der / (hess + 3.0)
    weights = np.zeros(16)
    np.add.at(weights, leaf, w.astype(np.float64))
    # a probability is right to a few 1e-7 (fast exponential), a sum of up to n of them to no more of its mass; the steps divide
    # two such sums
    assert np.allclose(eng.model_vals[0].cpu().numpy(), delta, rtol=5e-6, atol=5e-6 * max(1.0, np.abs(delta).max()))
    assert np.allclose(eng.model_wts[0].cpu().numpy(), weights, rtol=1e-6)
    eng.finish()
    eng.close()


@pytest.mark.parametrize("shift,spread,weights,steps", [
    (-13.0, 1.0, "", 1), (-13.0, 1.0, "", 3), (-15.0, 0.5, "", 3),       # documents that the model is sure of
    (0.0, 3.0, "lognormal", 1), (0.0, 3.0, "one heavy", 1),              # documents far lighter than the heaviest one
])
def test_logloss_leaf_steps_keep_small_derivatives_and_weights(shift, spread, weights, steps):
    """Leaf values and leaf weights of documents whose derivative or weight is orders below the largest possible one."""
    from catboost_b200.train.objectives import make_objective
    from catboost_b200.train.gpu_engine import GpuObliviousEngine
    n = 40_001
    store, _ = _store(n, [33] * 6, seed=5)
    rng = np.random.default_rng(6)
    y = np.zeros(n, dtype=np.float32) if shift < 0 else (rng.random(n) < 0.4).astype(np.float32)
    w = {"": np.ones(n), "lognormal": np.exp(3.0 * rng.standard_normal(n)),
         "one heavy": np.where(np.arange(n) == 7, 1.0e7, 1.0)}[weights].astype(np.float32)
    start = (shift + spread * rng.standard_normal(n)).astype(np.float32)
    eng = GpuObliviousEngine(store, torch.from_numpy(y), torch.from_numpy(w) if weights else None, torch.from_numpy(start),
                             make_objective("Logloss", {}), depth=4, iterations=2, learning_rate=1.0, l2_leaf_reg=3.0,
                             random_strength=0.0, bootstrap_type="No", leaf_iterations=steps, leaf_backtracking="No", lane_hist=True)
    eng.step(1)
    torch.cuda.synchronize()
    leaf = eng.leaf[:n].cpu().numpy().astype(np.int64) & 0xFFFF
    delta = np.zeros(16)
    for _ in range(steps):
        p = 1.0 / (1.0 + np.exp(-(start.astype(np.float64) + delta[leaf])))
        der = np.bincount(leaf, w * (y - p), 16)
        delta += der / (np.bincount(leaf, w * p * (1.0 - p), 16) + 3.0)
    # a fast exponential of a margin of 15 is right to 1e-6, the sums add fewer than 2^12 such values each
    got, wts = eng.model_vals[0].cpu().numpy(), eng.model_wts[0].cpu().numpy()
    light = np.bincount(leaf, w.astype(np.float64), 16)
    assert np.linalg.norm(got - delta) <= 5e-6 * np.linalg.norm(delta), np.abs(got / delta - 1.0).max()
    assert np.allclose(wts, light, rtol=1e-6), np.abs(wts / light - 1.0).max()
    eng.finish()
    eng.close()


def _sure_engine(store, n, depth=1, p=1.0e-4, positives=0.01, **kw):
    """Logloss at a constant cursor: every negative's derivative is -p, the positives' is 1 - p."""
    from catboost_b200.train.gpu_engine import GpuObliviousEngine
    from catboost_b200.train.objectives import make_objective
    y = (torch.rand(n, generator=torch.Generator(device="cuda").manual_seed(1), device="cuda") < positives).float()
    args = dict(depth=depth, iterations=2, learning_rate=0.5, l2_leaf_reg=3.0, random_strength=0.0, bootstrap_type="No",
                leaf_iterations=1, seed=3, lane_hist=True)
    args.update(kw)
    return GpuObliviousEngine(store, y, None, torch.full((n,), float(np.log(p / (1.0 - p)))), make_objective("Logloss", {}), **args), y


def _negative_mass_error(eng, store, y, n, features):
    """Level 0: largest error of a bin's derivative sum, over the mass of the bin's negatives."""
    der = eng.stats[0, :n].double()
    off, worst = store.feat_off_host, 0.0
    for f in features:
        nb = int(store.feat_nb_host[f])
        bins = store.column(f)[:n].long()
        exact = torch.bincount(bins, der, nb)
        mass = torch.bincount(bins, der.abs() * (y < 0.5), nb)
        got = eng.slots[off[f]: off[f] + nb].double()
        full = mass > 0
        worst = max(worst, float(((got - exact).abs()[full] / mass[full]).max()))
    return worst


@pytest.mark.parametrize("F", [5, 9, 30, 32])
def test_padding_columns_leave_the_scale_alone(F):
    """A last feature group of fewer than four columns: its padding columns hold every document in one bin."""
    n = 2_000_003
    store, _ = _store(n, [129] * F, seed=F)
    eng, y = _sure_engine(store, n)
    eng.step(1)
    torch.cuda.synchronize()
    steps = (n + 1663) // 1664
    cap = -(-steps // eng.level_geo[0][4]) * 52 + 1            # documents of a lane total: more than any of 129 bins gets
    quantum = 1.0 / (2.0 ** 31 / (cap + 1) - 1.0)
    # half a quantum a negative, and fp32 sums of positives that weigh 100 times as much
    assert _negative_mass_error(eng, store, y, n, (0, F - 1)) <= 0.5 * quantum / 1.0e-4 + 100 * 2.0 ** -20
    eng.finish()
    eng.close()


def test_a_two_valued_column_leaves_the_scale_of_wide_tables_alone():
    """Many columns leave few document chunks per row block; a column of two equally frequent values then fills a cell with a
    quarter of a million documents.  The negatives' derivative (5e-4 of the positives') must not vanish in the steps."""
    from catboost_b200.data.quantization import FlatFeature, make_store, pack_columns_into
    n, F, p = 2_000_003, 600, 5.0e-4
    widths = [2 if j % 32 == 7 else 129 for j in range(F)]
    feats = [FlatFeature("float", j, borders=np.arange(w - 1, dtype=np.float32), n_bins=w) for j, w in enumerate(widths)]
    store = make_store(feats, n, torch.device("cuda"))
    gen = torch.Generator(device="cuda").manual_seed(4)
    for f0 in range(0, F, 64):
        cols = torch.randint(0, 129, (min(64, F - f0), n), generator=gen, device="cuda", dtype=torch.uint8)
        for j in range(len(cols)):
            if widths[f0 + j] == 2:
                cols[j] &= 1
        pack_columns_into(store, cols, f0)
    eng, y = _sure_engine(store, n, p=p)
    eng.step(1)
    torch.cuda.synchronize()
    # at least 65534 steps to the largest derivative: half a step a negative, and fp32 sums of positives 20 times as heavy
    assert _negative_mass_error(eng, store, y, n, (0, 7, 300, 583)) <= 0.5 / 65534 / p + 20 * 2.0 ** -20
    eng.finish()
    eng.close()


def test_tables_whose_second_copy_does_not_fit_take_the_other_pass(monkeypatch):
    """The pass may take half of the free device memory; a fit that finds less grows its trees with the per-group pass."""
    from catboost_b200.train.gpu_engine import GpuObliviousEngine
    n, F = 30_011, 28
    store, cols = _store(n, [129] * F, seed=2)
    y = (cols[0] / 129.0 + 0.2 * np.random.default_rng(3).standard_normal(n)).astype(np.float32)
    trees = []
    for little in (False, True, None):
        if little:
            free = 2 * store.bins.numel() * 4            # room for the copy alone, not for the other half as well
            monkeypatch.setattr(GpuObliviousEngine, "LANE_BYTES_UNASKED", 0)
            monkeypatch.setattr(torch.cuda, "mem_get_info", lambda *a: (free, free))
            monkeypatch.setattr(torch.cuda, "memory_reserved", torch.cuda.memory_allocated)      # nothing cached
        else:
            monkeypatch.undo()
        eng = _engine(store, y, 6, little is not None)
        assert eng.lane_hist == (little is False) and (eng.lane_store is not None) == (little is False)
        eng.step(2)
        trees.append(eng.finish())
        eng.close()
    assert np.array_equal(trees[1][0][0], trees[2][0][0])           # the first tree, bit for bit
    assert np.array_equal(trees[0][0][0, :4, :2], trees[1][0][0, :4, :2])


def test_no_second_copy_for_one_feature_group():
    store, cols = _store(3_000, [129] * 4, seed=1)
    eng = _engine(store, cols[0].astype(np.float32), 3, True)
    assert eng.lane_store is None and not eng.lane_hist
    eng.step(1)
    eng.finish()
    eng.close()


@pytest.mark.parametrize("n,widths,depth,sparse", [
    (1665, [129] * 12, 6, False),                    # two chunks, the second of one document
    (5_000, [256] * 18, 6, False),                   # the widest columns
    (260_003, [129] * 28, 6, False),                 # three slot passes, a chunk for every SM and a short last one
    (100_003, [129] * 40 + [3] * 9, 7, True),        # bundles of different lane widths: two rounds from the counter
    (20_007, [255] * 33 + [2] * 6, 8, False),        # many slot passes
])
def test_work_items_with_all_slot_passes_equal_sums_in_64_bits(n, widths, depth, sparse):
    """Large tables: an item takes its chunk through all slot passes, the later ones read the list that the first one wrote."""
    test_lane_histograms_equal_sums_in_64_bits(n, widths, depth, sparse, lane_seq_docs=0)


@pytest.mark.parametrize("n", [1, 1663, 1665, 30_011])
@pytest.mark.parametrize("F", [5, 9, 12, 28, 41])
def test_level_0_equals_sums_in_64_bits(n, F):
    test_lane_histograms_equal_sums_in_64_bits(n, [129] * F, 1, False)


def test_allocation_failure_falls_back_to_the_other_pass(monkeypatch):
    """Tables too small to ask for the free memory first: the allocation itself decides (made to fail on the host)."""
    n, F = 3_001, 12
    store, cols = _store(n, [129] * F, seed=2)
    empty = torch.empty

    def no_room(size, *a, **kw):
        if size == words:
            raise torch.cuda.OutOfMemoryError("out of memory")
        return empty(size, *a, **kw)

    from catboost_b200.ops import native
    words = int(native.cuda_lib().cb_lane_store_words(n, 3))
    monkeypatch.setattr(torch, "empty", no_room)
    eng = _engine(store, cols[0].astype(np.float32), 4, True)
    monkeypatch.undo()
    assert not eng.lane_hist and eng.lane_store is None
    eng.step(2)
    assert (eng.finish()[0][:, :, 0] >= 0).any()
    eng.close()
