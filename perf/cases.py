"""Performance cases: whole ``fit`` and ``predict`` calls at the sizes the framework is used at.

Every case is one call of the public API as a program makes it: ``PackBoost(config).fit(...)``
(binning, packing, upload of host arrays, all boosting rounds, the trees and the training
predictions at the end) or ``PackBoost.predict(...)`` with a model in hand.  Shapes follow the five
benchmark configurations of the repository (``packboost_b200/workloads.py``), the default
configuration, and the options that change the path a fit takes: eras absent, interleaved or many,
few or many bins, threshold subsets, the directional term, era weights, evaluation sets.

Number of rounds: a fit of 1 000 rounds repeats one round, so the cases run as many as make the
rounds weigh next to the start of the fit.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from packboost_b200 import PackBoost, PackBoostConfig, PackBoostRegressor
from packboost_b200.booster import TreeBuilder

# data:    "gauss"   float32 columns (normal, log-normal and a tenth integer-valued), quantile-binned
#          "levels"  uint8 codes 0 .. bins - 1 declared as such (prebinned)
# source:  "numpy"   host arrays, the type the API was made for;  "cuda"  tensors already on the GPU
# order:   "sorted" contiguous eras;  "mixed" rows of all eras interleaved;  "none" no eras given
_FIT = dict(kind="fit", data="gauss", source="numpy", order="sorted", rows=20_000, features=64, eras=20, ragged=False,
            bins=63, depth=6, pack=8, rounds=20, fraction=1.0, min_leaf=20, l2=1e-6, dro=0.5, direction=0.0, alpha=0.0,
            k_cuts=0, cuts="mass", valid_rows=0)
_PREDICT = dict(kind="predict", data="gauss", source="numpy", rows=64, features=64, bins=128, depth=5, trees=20, pack=8)


def _fit(**over):
    return dict(_FIT, **over)


def _predict(**over):
    return dict(_PREDICT, **over)


# Each entry: the listed case and the ranges its size fields are drawn from.
_CASES = [
    # First contact and hyper-parameter searches on a small table (configuration 1): start-up cost,
    # launches and the host loop are what such a fit takes.
    (_fit(name="fit_small", rows=20_000, features=64, eras=20, bins=128, depth=5, rounds=20, l2=1.0),
     dict(rows=(2_000, 40_000), features=(16, 128), eras=(4, 40), rounds=(5, 30), depth=(4, 6), bins=(64, 128))),
    # An ordinary float table from host memory with many bins (configuration 2).
    (_fit(name="fit_table", rows=500_000, features=256, eras=100, bins=128, depth=6, pack=16, rounds=20),
     dict(rows=(60_000, 500_000), features=(48, 256), eras=(20, 100), rounds=(10, 20), depth=(5, 6), bins=(48, 128))),
    # The headline workload (configuration 3): a wide table of five-level codes, several hundred eras,
    # a tenth of the features sampled per depth.
    (_fit(name="fit_era_wide", data="levels", source="cuda", rows=2_700_000, features=2376, eras=574, bins=5, depth=6,
          pack=32, rounds=60, fraction=0.1),
     dict(rows=(150_000, 2_700_000), features=(400, 2376), eras=(40, 574), rounds=(20, 60), depth=(4, 6), bins=(4, 6))),
    # The same kind of table without eras and a deeper tree: the configuration of the demo notebook
    # (pack of 8, depth 7, a twentieth of the features, no eras).
    (_fit(name="fit_no_era", data="levels", source="cuda", order="none", rows=1_300_000, features=1051, eras=1, bins=5,
          depth=7, rounds=40, fraction=0.0538, dro=0.0),
     dict(rows=(100_000, 1_300_000), features=(300, 1100), rounds=(20, 40), depth=(5, 7), bins=(4, 6))),
    # Deep frontiers over many bins (configuration 4, at a fifth of its rows and features): hundreds
    # of live nodes at the last depths.
    (_fit(name="fit_deep", source="cuda", rows=200_000, features=100, eras=40, bins=128, depth=10, pack=64, rounds=4),
     dict(rows=(40_000, 200_000), features=(24, 100), eras=(8, 40), rounds=(2, 4), depth=(8, 10), bins=(64, 128))),
    # Directional term and era weights, the two options of the score that keep the histogram per era;
    # the codes are on the GPU as uint8.
    (_fit(name="fit_direction", data="levels", source="cuda", rows=330_001, features=511, eras=120, ragged=True, bins=5,
          depth=6, pack=8, rounds=20, fraction=0.2, direction=0.1, alpha=8.0),
     dict(rows=(50_000, 330_000), features=(100, 512), eras=(20, 120), rounds=(8, 20), depth=(4, 6), bins=(4, 7))),
    # Threshold subsets: 64 bins, 15 cuts at the mass quantiles.
    (_fit(name="fit_mass_cuts", source="cuda", rows=240_000, features=190, eras=60, bins=64, depth=6, pack=8, rounds=15,
          k_cuts=15, fraction=0.5),
     dict(rows=(40_000, 240_000), features=(40, 190), eras=(10, 60), rounds=(6, 15), depth=(4, 6), bins=(32, 64),
          k_cuts=(5, 16))),
    # A monitored fit of the estimator class with its defaults (63 bins, depth 6): rows in no order,
    # eras of unequal size, a validation set and a callback, so every round is looked at.
    (_fit(name="fit_monitored", order="mixed", rows=131_071, features=97, eras=53, ragged=True, rounds=20,
          valid_rows=30_011, dro=0.0),
     dict(rows=(10_000, 131_000), features=(24, 100), eras=(8, 60), rounds=(6, 20), valid_rows=(2_000, 30_000))),
    # A service that scores a handful of rows per request.
    (_predict(name="predict_request", rows=64, features=64),
     dict(rows=(1, 512), features=(20, 128), trees=(10, 60), depth=(4, 6), bins=(63, 128))),
    # The weekly live table scored by a model of 1 000 rounds, from host memory.
    (_predict(name="predict_live", data="levels", rows=5_417, features=2376, bins=5, depth=6, trees=1000, pack=32),
     dict(rows=(800, 9_000), features=(300, 2376), trees=(150, 1000), depth=(5, 7), bins=(4, 6))),
    # Scoring a long table of codes that is on the GPU (configuration 5: 2 000 rounds of 32 trees).
    (_predict(name="predict_codes", data="levels", source="cuda", rows=500_000, features=2376, bins=5, depth=6,
              trees=2000, pack=32),
     dict(rows=(60_000, 500_000), features=(300, 2376), trees=(300, 2000), depth=(5, 7), bins=(4, 6))),
    # Scoring a float table on the GPU: the binning of its columns is part of the call.
    (_predict(name="predict_floats", source="cuda", rows=300_007, features=256, depth=6, trees=100, pack=16),
     dict(rows=(20_000, 300_000), features=(48, 256), trees=(30, 100), depth=(5, 7), bins=(48, 128))),
]


def listed():
    return [dict(case) for case, _ in _CASES]


def _between(rng, lo, hi):
    """A whole number of [lo, hi], uniform over the logarithm when that spans more than a factor of ten."""
    if hi <= 10 * lo:
        return rng.randint(lo, hi)
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    base, ranges = rng.choice(_CASES)
    case = {k: v for k, v in base.items() if k != "name"}
    for field, (lo, hi) in ranges.items():
        case[field] = _between(rng, lo, hi)
    if case["kind"] == "fit" and case["order"] != "none":
        case["ragged"] = rng.random() < 0.5
    return case


# ---- inputs ------------------------------------------------------------------------------------------


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _table(g, data, rows, features, bins):
    """Feature matrix on the GPU: mixed float columns, or uniformly used levels."""
    if data == "levels":
        X = torch.empty((rows, features), dtype=torch.uint8, device="cuda")
        step = max(1, (1 << 29) // features)
        for a in range(0, rows, step):
            b = min(rows, a + step)
            X[a:b] = torch.randint(0, bins, (b - a, features), generator=g, device="cuda", dtype=torch.uint8)
        return X
    X = torch.randn((rows, features), generator=g, device="cuda")
    n_int = max(1, features // 10)
    n_log = features * 2 // 5
    X[:, :n_log].exp_()
    X[:, features - n_int:] = torch.randint(0, 10, (rows, n_int), generator=g, device="cuda").float()
    return X


def _eras(rng, rows, eras, ragged, order):
    """int16 era of every row, all of them used."""
    if order == "none":
        return None
    eras = max(1, min(eras, rows))
    if ragged:
        share = rng.gamma(4.0, size=eras)
        cuts = np.floor(np.cumsum(share) / share.sum() * (rows - eras)).astype(np.int64) + np.arange(1, eras + 1)
        era = np.searchsorted(cuts, np.arange(rows), side="right").clip(0, eras - 1).astype(np.int16)
    else:
        era = (np.arange(rows, dtype=np.int64) * eras // rows).astype(np.int16)
    return rng.permutation(era) if order == "mixed" else era


def _target(g, X, era, data):
    """Sparse linear signal with two interactions under noise; a third of the eras has its sign
    flipped.  Levels: a weak signal quantised to five values, as for the tables they stand for."""
    rows, features = X.shape
    pick = torch.randperm(features, generator=g, device="cuda")[:min(16, features)]
    Z = X[:, pick].float()
    Z = (Z - Z.mean(0)) / (Z.std(0) + 1e-6)
    w = torch.randn(Z.shape[1], generator=g, device="cuda")
    signal = Z @ w + 0.5 * Z[:, 0] * Z[:, 1] + 0.5 * Z[:, 2] * Z[:, 3]
    if era is not None:
        sign = 1.0 - 2.0 * (torch.rand(int(era.max()) + 1, generator=g, device="cuda") < 0.3).float()
        signal = signal * sign[torch.from_numpy(era).to("cuda").long()]
    noise = torch.randn(rows, generator=g, device="cuda")
    if data == "gauss":
        return signal + 0.5 * noise
    latent = 0.05 * signal / (signal.std() + 1e-6) + noise
    return torch.bucketize(latent, torch.tensor([-0.8416, -0.2533, 0.2533, 0.8416], device="cuda")).float() * 0.25


def _forest(rng, case):
    """Trees as a fit grows them: complete but for a few early leaves, small leaf values."""
    trees = []
    for _ in range(case["trees"]):
        n = 1 << case["depth"]
        feature = rng.integers(0, case["features"], n).tolist()
        threshold = rng.integers(0, case["bins"] - 1, n).tolist()
        early = (rng.random(n) < 0.03).tolist()
        tb = TreeBuilder()
        level, used = [0], 0
        for d in range(case["depth"]):
            nxt = []
            for node in level:
                if d and early[used]:
                    used += 1
                    continue
                nxt.extend(tb.split(node, feature[used], threshold[used]))
                used += 1
            level = nxt
        values = rng.normal(0.0, 0.01, len(tb.nodes)).astype(np.float32).tolist()
        for node, value in zip(tb.nodes, values):
            if node.is_leaf:
                node.value = value
        trees.append(tb.build())
    return trees


def _edges(X, bins):
    q = torch.linspace(0.0, 1.0, bins + 1, device=X.device)[1:-1]
    return torch.quantile(X[:20_000], q, dim=0).cpu().numpy().astype(np.float32)


def prepare(case, seed):
    g, rng = _generator(seed), np.random.default_rng(int(seed))
    X = _table(g, case["data"], case["rows"], case["features"], case["bins"])
    if case["kind"] == "predict":
        model = PackBoost(PackBoostConfig(pack_size=case["pack"], max_depth=case["depth"], max_bins=case["bins"],
                                          prebinned=case["data"] == "levels"))
        edges = None if case["data"] == "levels" else _edges(torch.randn((4_096, case["features"]), generator=g,
                                                                         device="cuda"), case["bins"])
        trees = _forest(rng, case)
        model.set_forest(trees, 0.4 / case["pack"], bin_edges=edges, repeats=[case["pack"]] * len(trees))
        return dict(kind="predict", model=model, X=X if case["source"] == "cuda" else X.cpu().numpy())
    era = _eras(rng, case["rows"], case["eras"], case["ragged"], case["order"])
    y = _target(g, X, era, case["data"])
    params = dict(pack_size=case["pack"], max_depth=case["depth"], learning_rate=0.4 / case["pack"],
                  lambda_l2=case["l2"], lambda_dro=case["dro"], direction_weight=case["direction"],
                  era_alpha=case["alpha"], min_samples_leaf=case["min_leaf"], max_bins=case["bins"],
                  k_cuts=case["k_cuts"], cut_selection=case["cuts"], layer_feature_fraction=case["fraction"],
                  random_state=int(seed) % 65_536, prebinned=case["data"] == "levels")
    state = dict(kind="fit", params=params, rounds=case["rounds"], pack=case["pack"], era=era)
    if case["source"] == "numpy":
        X, y = X.cpu().numpy(), y.cpu().numpy()
    n_valid = case["valid_rows"]
    if n_valid:
        Xv = _table(g, case["data"], n_valid, case["features"], case["bins"])
        ev = _eras(rng, n_valid, max(2, case["eras"] // 4), True, "sorted")
        yv = _target(g, Xv, ev, case["data"])
        state["valid"] = (Xv.cpu().numpy(), yv.cpu().numpy(), ev)
    state.update(X=X, y=y)
    return state


# ---- one pass ------------------------------------------------------------------------------------------


def run(state):
    if state["kind"] == "predict":
        return {"prediction": state["model"].predict(state["X"])}
    out = {}
    if "valid" in state:
        seen = []
        est = PackBoostRegressor(num_rounds=state["rounds"], **state["params"])
        est.fit(state["X"], state["y"], state["era"], eval_set=state["valid"],
                round_callback=lambda r, m: seen.append((m["train_corr"], m["valid_corr"])))
        booster = est.booster_
        out["correlations"] = np.asarray(seen, dtype=np.float64)
    else:
        booster = PackBoost(PackBoostConfig(**state["params"]))
        booster.fit(state["X"], state["y"], state["era"], num_rounds=state["rounds"])
    trees = [t.arrays() for t in booster.trees[::state["pack"]]]
    most = 2 ** state["params"]["max_depth"]
    sizes = [t["feature"].shape[0] for t in trees]
    for key, fill in (("feature", -1), ("threshold", -1), ("left", -1), ("right", -1), ("value", 0.0)):
        out[key] = _padded([t[key] for t in trees], sizes, 2 * most - 1, fill)
    splits = booster.split_records()
    for key in splits:
        out["split_" + key] = _padded([splits[key]], [splits[key].shape[0]], len(trees) * (most - 1), 0)
    out["train_predictions"] = booster.train_predictions()
    return out


def _padded(parts, sizes, most, fill):
    """The arrays as the rows of one table: trees differ in size from data set to data set."""
    flat = np.concatenate(parts)
    table = np.full((len(parts), most), fill, dtype=flat.dtype)
    table[np.arange(most) < np.asarray(sizes)[:, None]] = flat
    return table


# ---- what a pass cannot do without -----------------------------------------------------------------------


def work(case):
    n, f = case["rows"], case["features"]
    item = 1 if case["data"] == "levels" else 4
    code = 0.5 if case["bins"] <= 16 else 1.0
    if case["kind"] == "predict":
        nodes = case["trees"] * (2 ** (case["depth"] + 1) - 1)
        return {"bytes": float(n * f * item + nodes * 8 + n * 4),
                "flops": float(n * case["trees"] * (case["depth"] + case["pack"]))}
    # the table once, its codes written once; then every depth of every round the codes of the sampled
    # features with the node and the gradient of each row, and every round the target and predictions
    sampled = max(1, round(case["fraction"] * f))
    deep = case["rounds"] * case["depth"]
    thresholds = case["k_cuts"] if 0 < case["k_cuts"] < case["bins"] - 1 else case["bins"] - 1
    nodes = case["rounds"] * (2 ** case["depth"] - 1)
    table = (n + case["valid_rows"]) * f * (item + code)
    rounds = deep * n * (sampled * code + 2 + 4) + case["rounds"] * n * 12
    # a count and a gradient sum per row and sampled feature; a gain and its share of the mean and the
    # deviation (about 20 operations) per node, era, feature and threshold
    flops = deep * n * sampled * 2.0 + nodes * case["eras"] * sampled * thresholds * 20.0
    return {"bytes": float(table + rounds), "flops": float(flops)}


def tolerance(case):
    # trees, counts and splits are whole numbers that exact histogram sums decide; leaf values, scores
    # and predictions are float32 sums
    return {"rel": 1e-5}
