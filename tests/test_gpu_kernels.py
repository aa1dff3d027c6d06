"""Kernel-level parity through the C ABI: binning/packing, histograms, legacy predictors."""

import ctypes as C
import os

import numpy as np
import pytest
import torch

from oracle import packboost_oracle as po

pytestmark = pytest.mark.gpu


def _dev():
    return torch.device("cuda", 0)


@pytest.mark.parametrize("max_bins", [5, 16, 64, 128])
def test_bin_pack_matches_searchsorted(max_bins):
    from packboost_b200.data import pack_feature_major, pack_row_major, quantile_edges
    rng = np.random.default_rng(max_bins)
    X = rng.normal(size=(1537, 37)).astype(np.float32)
    X[::7, 3] = np.nan
    X[:, 5] = np.round(X[:, 5])
    edges = quantile_edges(np.nan_to_num(X), max_bins)
    want = po.bin_codes(X, edges, max_bins).astype(np.uint8)
    pm = pack_feature_major(X, edges, max_bins)
    np.testing.assert_array_equal(pm.unpack().cpu().numpy(), want.T)
    pr = pack_row_major(X, edges, max_bins)
    raw = pr.codes.cpu().numpy()
    if pr.code_bits == 4:
        got = np.stack([raw & 0xF, raw >> 4], axis=2).reshape(raw.shape[0], -1)[:, : X.shape[1]]
    else:
        got = raw[:, : X.shape[1]]
    np.testing.assert_array_equal(got, want)


def _hist_case(n, f, e, nb, n_nodes, seed, big_era=False):
    from packboost_b200 import backends as B
    from packboost_b200.data import pack_feature_major
    rng = np.random.default_rng(seed)
    codes = rng.integers(0, nb, size=(n, f), dtype=np.uint8)
    if big_era:
        cuts = np.sort(rng.choice(np.arange(1, n), size=e - 1, replace=False))
        cuts[0] = max(cuts[0], 40000) if n > 50000 else cuts[0]
        cuts = np.sort(cuts)
    else:
        cuts = np.sort(rng.choice(np.arange(1, n), size=e - 1, replace=False))
    era_off = np.concatenate([[0], cuts, [n]]).astype(np.int32)
    pm = pack_feature_major(codes, None, nb)
    npad = pm.rows_padded
    gq = np.zeros(npad, np.int32)
    slot = np.full(npad, 0xFFFF, np.uint16)
    slot[:n] = rng.integers(0, n_nodes + 1, size=n)
    slot[:n][slot[:n] == n_nodes] = 0xFFFF      # some rows sit in finished leaves
    dev = _dev()
    t = dict(gq=torch.from_numpy(gq).to(dev), slot=torch.from_numpy(slot.view(np.int16)).to(dev),
             era=torch.from_numpy(era_off).to(dev))
    st = B.TrainState()
    st.n_rows, st.n_features_total, st.n_features_local, st.n_eras = n, f, f, e
    st.max_bins, st.code_bits, st.pitch = nb, pm.code_bits, pm.pitch
    st.max_depth, st.pack_size, st.min_samples_leaf, st.n_thresholds, st.feature_block_size = 6, 1, 1, nb - 1, 32
    st.lambda_l2 = 1.0
    dummy = torch.zeros(max(npad, 4096), dtype=torch.float32, device=dev)
    ids = torch.arange(max(f, nb), dtype=torch.int32, device=dev)
    st.codes, st.era_offsets, st.thr_ids, st.feat_local = pm.codes.data_ptr(), t["era"].data_ptr(), ids.data_ptr(), ids.data_ptr()
    st.y = st.preds = dummy.data_ptr()
    st.gq, st.slot, st.leaf = t["gq"].data_ptr(), t["slot"].data_ptr(), t["slot"].data_ptr()
    ctl = torch.zeros(int(B.lib().pb_ctl_bytes()), dtype=torch.uint8, device=dev)
    ws = torch.zeros(int(B.lib().pb_workspace_min_bytes(C.byref(st))) + 1024, dtype=torch.uint8, device=dev)
    st.ctl, st.workspace, st.workspace_bytes = ctl.data_ptr(), ws.data_ptr(), ws.numel()
    B.check(B.lib().pb_train_prepare(C.byref(st), era_off.ctypes.data))
    lim = 1 << int(st.gq_bits)
    gq[:n] = rng.integers(-lim, lim + 1, size=n)     # the full range the quantiser may produce
    t["gq"].copy_(torch.from_numpy(gq))
    feat = rng.permutation(f)[: max(1, f // 2)].astype(np.int32)
    feat_t = torch.from_numpy(feat).to(dev)
    cnt = torch.full((feat.shape[0], e, n_nodes, nb), -1, dtype=torch.int32, device=dev)
    gs = torch.full((feat.shape[0], e, n_nodes, nb), -1, dtype=torch.int64, device=dev)
    B.check(B.lib().pb_hist_build(C.byref(st), feat_t.data_ptr(), feat.shape[0], n_nodes, n_nodes, cnt.data_ptr(),
                                  gs.data_ptr(), torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    # numpy reference (exact integers)
    era_of = np.repeat(np.arange(e), np.diff(era_off))
    live = slot[:n] != 0xFFFF
    want_c = np.zeros((feat.shape[0], n_nodes, e, nb), np.int64)
    want_g = np.zeros_like(want_c)
    for i, fid in enumerate(feat):
        key = (slot[:n][live].astype(np.int64) * e + era_of[live]) * nb + codes[live, fid]
        want_c[i] = np.bincount(key, minlength=n_nodes * e * nb).reshape(n_nodes, e, nb)
        pos = np.bincount(key, weights=np.maximum(gq[:n][live], 0).astype(np.float64), minlength=n_nodes * e * nb)
        # float64 bincount is not exact at this magnitude; accumulate exactly instead
        acc = np.zeros(n_nodes * e * nb, np.int64)
        np.add.at(acc, key, gq[:n][live].astype(np.int64))
        want_g[i] = acc.reshape(n_nodes, e, nb)
    # device layout is [feature][era][node][bin]
    np.testing.assert_array_equal(cnt.cpu().numpy().astype(np.int64).transpose(0, 2, 1, 3), want_c)
    np.testing.assert_array_equal(gs.cpu().numpy().transpose(0, 2, 1, 3), want_g)


@pytest.mark.parametrize("n,f,e,nb,nodes", [
    (5000, 12, 7, 5, 1), (5000, 12, 7, 5, 32), (4097, 9, 3, 16, 4), (6000, 10, 5, 128, 8),
    (3001, 6, 4, 200, 3), (20000, 5, 2, 64, 300), (1000, 3, 1, 2, 1), (16000, 4, 2, 5, 2),
    (7000, 70, 3, 5, 2), (7000, 41, 3, 5, 8), (7000, 33, 2, 5, 50), (5000, 9, 2, 16, 1), (5000, 9, 2, 3, 9),
    (5000, 20, 2, 16, 17),
])
def test_histogram_exact(n, f, e, nb, nodes):
    _hist_case(n, f, e, nb, nodes, seed=n + nb)


def test_histogram_exact_when_an_era_spans_several_tiles():
    _hist_case(120_000, 6, 3, 5, 4, seed=5, big_era=True)
    _hist_case(90_000, 4, 1, 32, 2, seed=6)
    _hist_case(30_000, 3, 2, 128, 40, seed=7)


def test_legacy_predictors_match_oracle_router():
    from packboost_b200 import backends as B
    rng = np.random.default_rng(3)
    n, f = 3000, 40
    codes = rng.integers(0, 16, size=(n, f), dtype=np.uint8)
    # three random (not complete) trees with BFS-compact numbering
    trees = []
    for t in range(3):
        tr = po.OracleTree()
        frontier = [0]
        for depth in range(4):
            nxt = []
            for nid in frontier:
                if rng.random() < 0.8:
                    l, r = tr.split(nid, int(rng.integers(0, f)), int(rng.integers(0, 15)))
                    tr.set_leaf(l, float(rng.normal()))
                    tr.set_leaf(r, float(rng.normal()))
                    nxt += [l, r]
            frontier = nxt
        trees.append(tr.arrays())
    dev = _dev()
    fm = torch.from_numpy(np.ascontiguousarray(codes.T)).to(dev)
    for tr in trees:
        got = B.predict_bins_cuda(fm, *(torch.from_numpy(tr[k].astype(np.int32)).to(dev) for k in ("feature", "threshold", "left", "right")),
                                  torch.from_numpy(tr["value"].astype(np.float32)).to(dev),
                                  torch.from_numpy(tr["is_leaf"].astype(np.uint8)).to(dev))
        np.testing.assert_array_equal(got.cpu().numpy().view(np.int32), po.route_tree(tr, codes.astype(np.int8)).view(np.int32))
    # pack: absolute child ids, out = w * sum of leaves
    off = np.cumsum([0] + [t["feature"].shape[0] for t in trees]).astype(np.int32)
    cat = {k: np.concatenate([t[k] for t in trees]) for k in trees[0]}
    la = np.concatenate([np.where(t["left"] >= 0, t["left"] + o, -1) for t, o in zip(trees, off[:-1])]).astype(np.int32)
    ra = np.concatenate([np.where(t["right"] >= 0, t["right"] + o, -1) for t, o in zip(trees, off[:-1])]).astype(np.int32)
    got = B.predict_pack_cuda(fm, torch.from_numpy(cat["feature"]).to(dev), torch.from_numpy(cat["threshold"]).to(dev),
                              torch.from_numpy(la).to(dev), torch.from_numpy(ra).to(dev),
                              torch.from_numpy(cat["value"].astype(np.float32)).to(dev),
                              torch.from_numpy(cat["is_leaf"].astype(np.uint8)).to(dev), torch.from_numpy(off).to(dev), 0.25)
    want = np.zeros(n, np.float32)
    for tr in trees:
        want = want + po.route_tree(tr, codes.astype(np.int8))
    np.testing.assert_allclose(got.cpu().numpy(), np.float32(0.25) * want, rtol=1e-6, atol=1e-7)


def test_superseded_frontier_calls_say_so():
    from packboost_b200 import backends as B
    assert B.cuda_available() and not B.cpu_available()
    for fn in (B.find_best_splits_batched_cuda, B.partition_frontier_cuda, B.find_best_splits_batched):
        with pytest.raises(RuntimeError):
            fn()


def test_era_correlation_matches_host_formula():
    """Device per-era correlation against the reference's numpy loop, with the eras it skips:
    a single-row era, an era of constant predictions and an era of constant targets."""
    import ctypes as C
    from packboost_b200 import backends as B
    from packboost_b200.booster import _era_correlation_np
    rng = np.random.default_rng(5)
    sizes = [700, 1, 333, 50, 1200, 64]
    era = np.repeat(np.arange(len(sizes)), sizes).astype(np.int16)
    n = era.shape[0]
    y = rng.integers(0, 5, size=n).astype(np.float32) / 4
    p = (0.05 * y + 0.02 * rng.standard_normal(n)).astype(np.float32)
    p[era == 3] = 0.125          # constant predictions
    y[era == 5] = 0.5            # constant targets
    offs = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int32)
    dev = torch.device("cuda", 0)
    yd, pd, od = (torch.from_numpy(a).to(dev) for a in (y, p, offs))
    out = torch.empty(len(sizes), dtype=torch.float64, device=dev)
    B.check(B.lib().pb_era_correlation(yd.data_ptr(), pd.data_ptr(), od.data_ptr(), len(sizes), out.data_ptr(),
                                       torch.cuda.current_stream().cuda_stream))
    c = out.cpu().numpy()
    assert np.isnan(c[[1, 3, 5]]).all() and np.isfinite(c[[0, 2, 4]]).all()
    want = _era_correlation_np(era, y, p)
    np.testing.assert_allclose(c[np.isfinite(c)].mean(), want, rtol=1e-5)


def test_device_quantile_edges_equal_host_quantile_edges():
    from packboost_b200.data import quantile_edges, quantile_edges_device
    rng = np.random.default_rng(3)
    X = rng.normal(size=(60_001, 33)).astype(np.float32)
    X[:, 4] = np.round(X[:, 4] * 2)
    X[:, 9] = np.exp(X[:, 9])
    for nb in (5, 128):
        want = quantile_edges(X, nb)
        assert np.array_equal(quantile_edges_device(X, nb), want)
        assert np.array_equal(quantile_edges_device(torch.from_numpy(X).cuda(), nb), want)


def _oracle_candidates(trace, K):
    """Best threshold of every (sampled position, frontier node) from the oracle's per-candidate
    scores: highest score, then largest left count, then largest threshold index
    (packboost/booster.py:1912-1919 restricted to one feature)."""
    out = {}
    pos = 0
    for blk in trace["blocks"]:
        score = blk["score"].numpy()          # [node, feature in block, K], -inf where min_samples_leaf fails
        lc = blk["left_count"].numpy()
        for j in range(score.shape[1]):
            for n in range(score.shape[0]):
                s, c = score[n, j], lc[n, j]
                best = None
                for k in range(K):
                    if np.isnan(s[k]):
                        continue
                    if best is None or s[k] > s[best] or (s[k] == s[best] and c[k] >= c[best]):
                        best = k
                out[(pos + j, n)] = (np.float32(s[best]), best, int(c[best]))
        pos += score.shape[1]
    return out


@pytest.mark.parametrize("case,round_idx,depth", [("prebinned5", 0, 0), ("prebinned5", 1, 3), ("prebinned5", 3, 4),
                                                  ("config1", 0, 2), ("config1", 4, 4), ("ragged_eras", 2, 3),
                                                  ("kcuts_even", 1, 2), ("interleaved", 2, 3)])
def test_scorer_candidates_match_oracle_bit_for_bit(case, round_idx, depth):
    """Kernel-level check of the histogram + DES scorer pass: the candidate table it writes (best
    threshold of every sampled feature at every frontier node: float32 score, threshold index,
    left count) against the oracle's per-candidate scores in its exact-sum variant, for frontiers
    of one to sixteen nodes in the first and in later rounds."""
    import cases
    from gpu_util import gpu_candidates_at
    X, y, era, cfg, rounds, _ = cases.CASES[case]()
    table, subset, n_ctx = gpu_candidates_at(X, y, era, cfg, round_idx, depth)
    model = po.fit(X, y, era, po.OracleParams(exact_sums=True, **cfg), round_idx + 1, trace_at=(round_idx, depth))
    tr = model.trace
    assert tr, "the oracle did not reach this frontier"
    np.testing.assert_array_equal(tr["subset"].numpy(), subset)
    K = tr["blocks"][0]["K"]
    want = _oracle_candidates(tr, K)
    assert n_ctx == len(tr["context_nodes"])
    bad = []
    for (p, n), (s, k, c) in want.items():
        g = table[p, n]
        if (np.float32(g["score"]).view(np.int32) != s.view(np.int32)) or int(g["k"]) != k or int(g["left_count"]) != c:
            bad.append((p, n, float(g["score"]), int(g["k"]), int(g["left_count"]), float(s), k, c))
    assert not bad, f"{len(bad)} of {len(want)} candidates differ, first: {bad[:5]}"


_SHAPE_SCRIPT = """
import sys
sys.path.insert(0, {root!r})
from tests.test_gpu_kernels import _hist_case
_hist_case(7000, 70, 3, 5, 2, seed=11)
_hist_case(5000, 40, 2, 16, 1, seed=12)
_hist_case(9000, 300, 4, 5, 4, seed=13)
_hist_case(6000, 24, 3, 3, 9, seed=14)
_hist_case(4100, 16, 2, 5, 30, seed=15)
print("ok")
"""


@pytest.mark.parametrize("shape", ["1 8 1", "1 4 2", "1 1 4", "2 4 1", "2 2 2", "2 1 4", "2 4 2", "1 8 2", "1 2 1"])
def test_histogram_exact_in_every_launch_shape(shape):
    """The launcher picks the shape <features per joint code, tuples per lane, row phases> of the
    lane kernel by a cost model, so a given test size exercises one shape only.  The tuning
    override forces each shape in turn (it is read once per process, hence the child process) and
    the same exact-integer comparison runs on several sizes; the launch log must show that the
    forced shape really ran."""
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, PACKBOOST_HIST_SHAPE=shape)
    res = subprocess.run([sys.executable, "-c", _SHAPE_SCRIPT.format(root=root)], env=env, capture_output=True,
                         text=True, timeout=600)
    assert res.returncode == 0, res.stdout[-2000:] + res.stderr[-4000:]
    assert res.stdout.strip().endswith("ok")
    assert "hist_lane_kernel<%s>" % shape.replace(" ", ",") in res.stderr, res.stderr[-2000:]


_MMA_SCRIPT = """
import sys
sys.path.insert(0, {root!r})
from tests.test_gpu_kernels import _hist_case
for n, f, e, nb, nodes, big in {cases!r}:
    _hist_case(n, f, e, nb, nodes, seed=n + nodes, big_era=big)
print("ok")
"""


@pytest.mark.parametrize("cases,kernels", [
    ([(8_161, 2, 1, 5, 1, False), (20_001, 270, 1, 5, 1, False), (33_000, 258, 2, 4, 2, True)], {"2,4,0,0", "4,4,0,0"}),   # two and four thresholds a lane
    ([(17_000, 262, 1, 5, 4, False), (16_500, 20, 1, 2, 3, False), (40_000, 70, 3, 8, 4, True)], {"4,2,0,0", "2,4,0,0"}),
    ([(20_001, 130, 1, 5, 5, False), (17_000, 24, 1, 6, 16, False), (26_000, 9, 2, 3, 9, True)], {"2,4,1,0"}),   # two
    ([(20_001, 65, 1, 5, 17, False), (17_000, 24, 1, 8, 32, False), (30_000, 8, 2, 5, 33, True), (17_000, 70, 1, 7, 64, False)],
     {"1,4,1,0", "1,4,1,1"})])  # one
def test_histogram_exact_on_the_tensor_cores(cases, kernels):
    """Exact sums of the contraction for eras of several tiles: every number of thresholds a lane holds, either
    layout of the nodes' columns, more than 256 columns, features past a whole block of lanes, tiles that start
    and end anywhere.  (The switch that takes it at every size is read once per process.)"""
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    res = subprocess.run([sys.executable, "-c", _MMA_SCRIPT.format(root=root, cases=cases)], env=dict(os.environ, PACKBOOST_HIST_MMA="1"),
                         capture_output=True, text=True, timeout=600)
    assert res.returncode == 0 and res.stdout.strip().endswith("ok"), res.stdout[-2000:] + res.stderr[-4000:]
    ran = [line for line in res.stderr.splitlines() if line.startswith("hist_mma_kernel<")]
    assert len(ran) >= len(cases) and {line.split("<")[1].split(">")[0] for line in ran} == kernels, ran


@pytest.mark.parametrize("n,f,eras,bins,depth,extra", [
    (6_001, 300, 7, 5, 4, {}), (5_003, 40, 40, 5, 6, {}), (700, 33, 1, 2, 3, {}), (9_000, 70, 200, 8, 6, {}),
    (6_000, 150, 9, 4, 6, dict(direction_weight=0.3)), (6_000, 35, 11, 5, 5, dict(era_alpha=4.0)),
    (6_000, 35, 5, 7, 5, dict(k_cuts=3, cut_selection="even")), (20_001, 45, 2, 5, 7, {}), (17_000, 200, 1, 6, 7, {}),
    (6_001, 300, 7, 5, 4, dict(workspace=460_000))])
def test_fit_on_the_tensor_cores_equals_the_one_by_atomics(n, f, eras, bins, depth, extra, tmp_path):
    """Trees, scores and predictions bit for bit: gains made in the flush, every form of the score, eras shorter
    than a step of the rows and longer than a tile."""
    import json
    import subprocess
    import sys
    script = r"""
import json, sys
import numpy as np
from packboost_b200 import PackBoost, PackBoostConfig
n, f, eras, bins, depth, extra, out = json.loads(sys.argv[1])
rng = np.random.default_rng(n + f)
X = rng.integers(0, bins, size=(n, f)).astype(np.uint8)
y = (X[:, 0] + X[:, 1] * (X[:, 2] > 1) + rng.normal(size=n)).astype(np.float32)
era = np.sort((rng.random(n) ** 2 * eras).astype(np.int16))
cfg = dict(pack_size=2, max_depth=depth, learning_rate=0.2, lambda_l2=1.0, lambda_dro=0.4, min_samples_leaf=5, max_bins=bins,
           random_state=1, prebinned=True)
cfg.update(extra)
b = PackBoost(PackBoostConfig(**cfg)).fit(X, y, era, num_rounds=3)
np.savez(out, preds=b.train_predictions().view(np.int32), **{k: v.view(np.int32) if v.dtype == np.float32 else v for k, v in b.split_records().items()})
"""
    got, ran = [], []
    extra = dict(extra)
    env = {"PACKBOOST_WORKSPACE_BYTES": str(extra.pop("workspace"))} if "workspace" in extra else {}
    for mma in ("1", "0"):
        path = str(tmp_path / f"{mma}.npz")
        res = subprocess.run([sys.executable, "-c", script, json.dumps([n, f, eras, bins, depth, extra, path])],
                             env=dict(os.environ, PACKBOOST_HIST_MMA=mma, **env), cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                             capture_output=True, text=True)
        assert res.returncode == 0, res.stderr[-2000:]
        ran.append([dict(kv.split("=") for kv in line.split()[1:]) for line in res.stderr.splitlines() if line.startswith("hist_mma_kernel<")])
        got.append(np.load(path))
    # the kernel ran at every depth it takes, made the gains where an era is one tile, and never with the switch off
    one_tile = np.max(np.diff(np.sqrt(np.arange(eras + 1) / eras))) * n < 8_000
    nodes = {int(r["nodes"]) for r in ran[0]}
    assert nodes >= {1 << d for d in range(min(depth, 6))} and not ran[1], ran
    assert {r["fused"] for r in ran[0]} == {"1" if one_tile else "0"}
    assert (min(int(r["features"]) for r in ran[0]) < f) == bool(env)
    assert len(got[0]["node"]) > 3
    for key in got[0].files:
        np.testing.assert_array_equal(got[0][key], got[1][key], err_msg=key)


_LIMIT_SCRIPT = r"""
import json, sys
import numpy as np, torch
from packboost_b200 import PackBoost, PackBoostConfig
for n, f, eras, bins, depth in json.loads(sys.argv[1]):
    rng = np.random.default_rng(n + f)
    X = rng.integers(0, bins, size=(n, f)).astype(np.uint8)
    y = (X[:, 0] + rng.normal(size=n)).astype(np.float32)
    era = np.sort(rng.integers(0, eras, n)).astype(np.int16)
    cfg = PackBoostConfig(pack_size=2, max_depth=depth, lambda_l2=1.0, min_samples_leaf=5, max_bins=bins, prebinned=True)
    try:
        PackBoost(cfg).fit(X, y, era, num_rounds=3)
        print("no error")
    except RuntimeError as e:
        print("error" if "ran into its limit" in str(e) else e)
    torch.cuda.synchronize()
    assert int(torch.arange(1000, device="cuda").sum().item()) == 499500
"""


@pytest.mark.parametrize("fails,says", [(True, "error"), (False, "no error")])
def test_waits_that_run_out_end_the_launch_and_are_reported(fails, says):
    """Launches of the contraction that are marked as failed from the start, so that no product is issued and whatever
    waits for one gives up: they end, the fit says why, and the device goes on working.  One and two issuing warps, batches of 64 and 128 rows, gains made
    in the flush and a stored histogram, eras shorter than a batch."""
    import json
    import subprocess
    import sys
    shapes = [(6_001, 300, 7, 5, 4), (5_003, 40, 40, 5, 6), (700, 33, 1, 2, 3), (20_001, 45, 2, 5, 7), (17_000, 200, 1, 6, 7), (3_000, 70, 900, 8, 5)]
    env = dict(os.environ, PACKBOOST_HIST_MMA="1")
    if fails:
        env["PACKBOOST_WAIT_FAILS"] = "1"
    res = subprocess.run([sys.executable, "-c", _LIMIT_SCRIPT, json.dumps(shapes)], env=env, capture_output=True, text=True, timeout=300,
                         cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    assert res.returncode == 0, res.stderr[-2000:]
    assert res.stdout.split("\n")[:-1] == [says] * len(shapes), res.stdout


_RAW_SCRIPT = r"""
import torch
from packboost_b200 import kernels
n, f = 20_001, 45
X = torch.randint(0, 5, (n, f), dtype=torch.uint8)
node = torch.randint(0, 3, (n,))
try:
    cnt, sums, _ = kernels.histograms_nodes(X, torch.randn(n), torch.ones(n), torch.zeros(n, dtype=torch.int64), node, 3, 1, 5)
    assert torch.equal(cnt.sum((2, 3)).cpu(), torch.bincount(node).expand(f, 3))
    print("no error")
except RuntimeError as e:
    print("error" if "ran into its limit" in str(e) else e)
"""


@pytest.mark.parametrize("fails,says", [(True, "error"), (False, "no error")])
def test_histograms_whose_waits_ran_out_are_refused(fails, says):
    """The histogram entry only enqueues and has no log: its caller looks at the control block."""
    import subprocess
    import sys
    env = dict(os.environ, PACKBOOST_HIST_MMA="1")
    if fails:
        env["PACKBOOST_WAIT_FAILS"] = "1"
    res = subprocess.run([sys.executable, "-c", _RAW_SCRIPT], env=env, capture_output=True, text=True, timeout=300,
                         cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    assert res.returncode == 0 and res.stdout.strip() == says, res.stdout + res.stderr[-2000:]


def test_threads_that_launch_a_kernel_at_different_sizes_do_not_disturb_each_other():
    """Two threads, each with a state of its own, launch the same instantiations at sizes that need different
    amounts of shared memory: neither lowers the limit between the other's asking and its launch."""
    import threading
    from packboost_b200 import backends as B
    lib, dev = B.lib(), _dev()
    errors, keep = [], []

    def state(n_bins):
        n, f, nb = 4_096, 8, n_bins
        codes = torch.zeros((f, n), dtype=torch.uint8, device=dev)
        row = torch.zeros(4 * n, dtype=torch.float32, device=dev)
        eo = torch.tensor([0, n], dtype=torch.int32, device=dev)
        ids = torch.arange(256, dtype=torch.int32, device=dev)
        ctl = torch.zeros(int(lib.pb_ctl_bytes()), dtype=torch.uint8, device=dev)
        out = (torch.empty(f * 512 * nb, dtype=torch.int32, device=dev), torch.empty(f * 512 * nb, dtype=torch.int64, device=dev))
        st = B.TrainState()
        st.n_rows, st.n_features_total, st.n_features_local, st.n_eras = n, f, f, 1
        st.max_bins, st.code_bits, st.pitch = nb, 8, n
        st.max_depth, st.pack_size, st.min_samples_leaf, st.n_thresholds, st.feature_block_size = 6, 1, 1, nb - 1, 32
        st.lambda_l2 = 1.0
        st.codes, st.era_offsets, st.thr_ids, st.feat_local = codes.data_ptr(), eo.data_ptr(), ids.data_ptr(), ids.data_ptr()
        st.y = st.preds = st.gq = st.slot = st.leaf = row.data_ptr()
        st.ctl = ctl.data_ptr()
        eo_host = np.array([0, n], np.int32)
        B.check(lib.pb_train_prepare(C.byref(st), eo_host.ctypes.data))
        keep.append((codes, row, eo, ids, ctl, out))
        return st, ids, out

    def launch(st, ids, out, nodes, stream):
        try:
            for _ in range(4_000):
                B.check(lib.pb_hist_build(C.byref(st), ids.data_ptr(), 8, nodes, nodes, out[0].data_ptr(), out[1].data_ptr(), stream))
        except Exception as e:   # noqa: BLE001
            errors.append(str(e))

    streams = [torch.cuda.Stream() for _ in range(2)]
    jobs = [(*state(128), nodes, s.cuda_stream) for nodes, s in zip((60, 180), streams)]
    torch.cuda.synchronize()
    threads = [threading.Thread(target=launch, args=j) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors, errors[0]


@pytest.mark.parametrize("max_bins,n_nodes", [(96, 64), (12, 512), (191, 32), (47, 128)])
def test_histogram_whose_cells_take_just_the_shared_memory_given_without_asking(max_bins, n_nodes):
    """48 KB of cells or a little less beside the kernel's own arrays: such a launch has to ask for more
    (in a child process, where no larger launch has asked before)."""
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    script = (f"import sys; sys.path.insert(0, {root!r})\nfrom tests.test_gpu_kernels import _hist_case\n"
              f"_hist_case(3000, 5, 2, {max_bins}, {n_nodes}, seed=3)\nprint('ok')\n")
    res = subprocess.run([sys.executable, "-c", script], capture_output=True, text=True, timeout=600)
    assert res.returncode == 0 and res.stdout.strip().endswith("ok"), res.stdout[-2000:] + res.stderr[-4000:]


@pytest.mark.parametrize("n,f,max_bins", [(1, 1, 5), (255, 127, 5), (256, 128, 5), (257, 129, 16), (1030, 301, 5),
                                          (513, 131, 64), (300, 33, 2), (259, 97, 128)])
def test_pack_kernels_at_tile_edges(n, f, max_bins):
    """Byte and float packers (both layouts, rows in order and gathered) where rows start on odd bytes
    and tiles are partly filled; padding rows are code 0 and the range check sees the largest byte."""
    from packboost_b200.data import pack_feature_major, pack_row_major
    rng = np.random.default_rng(n * f)
    codes = rng.integers(0, max_bins, size=(n, f), dtype=np.uint8)
    order = rng.permutation(n)
    X = rng.normal(size=(n, f)).astype(np.float32)
    edges = np.sort(rng.normal(size=(max_bins - 1, f)).astype(np.float32), axis=0)
    binned = po.bin_codes(X, edges, max_bins).astype(np.uint8)

    def rows_of(pr):
        raw = pr.codes.cpu().numpy()
        return (np.stack([raw & 0xF, raw >> 4], axis=2).reshape(raw.shape[0], -1) if pr.code_bits == 4 else raw)[:, :f]

    for src, e, want in ((codes, None, codes), (X, edges, binned)):
        for device in (False, True):
            table = torch.from_numpy(src).to(_dev()) if device else src
            for row_order in (None, order):
                pm = pack_feature_major(table, e, max_bins, row_order=row_order, validate_codes=e is None)
                np.testing.assert_array_equal(pm.unpack().cpu().numpy(), (want if row_order is None else want[order]).T)
                if pm.code_bits == 8:
                    assert not pm.codes[:, n:].any()
                if e is None:
                    assert pm.max_code == int(codes.max())
            np.testing.assert_array_equal(rows_of(pack_row_major(table, e, max_bins)), want)


@pytest.mark.parametrize("n_edges,max_bins", [(15, 16), (20, 16), (127, 128), (300, 100), (300, 256), (3, 64)])
def test_rows_are_binned_with_more_or_fewer_edges_than_bins(n_edges, max_bins):
    """A model may bring any number of edges: codes are cut to max_bins - 1."""
    from packboost_b200.data import pack_row_major
    rng = np.random.default_rng(n_edges)
    X = rng.normal(size=(333, 21)).astype(np.float32)
    X[::9, 4], X[1, 5], X[2, 5] = np.nan, np.inf, -np.inf
    edges = np.sort(rng.normal(size=(n_edges, 21)).astype(np.float32), axis=0)
    raw = pack_row_major(X, edges, max_bins).codes.cpu().numpy()
    got = (np.stack([raw & 0xF, raw >> 4], axis=2).reshape(333, -1) if max_bins <= 16 else raw)[:, :21]
    want = np.stack([np.searchsorted(edges[:, j], X[:, j]) for j in range(21)], axis=1).clip(0, max_bins - 1)
    np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("nbytes", [1, (384 << 10) + 1, (1 << 20) - 3, (16 << 20) + 5, (37 << 20) + 1])
def test_upload_moves_every_byte(nbytes):
    """The page-locked ring below, at and beyond its size."""
    from packboost_b200.data import Uploads
    src = np.random.default_rng(nbytes).integers(0, 256, nbytes, dtype=np.uint8)
    uploads = Uploads()
    for _ in range(2):
        got = uploads(src, torch.uint8)
        np.testing.assert_array_equal(got.cpu().numpy(), src)


@pytest.mark.parametrize("rows,features,bins,depth,trees", [
    (1, 1, 2, 0, 1), (31, 7, 5, 1, 3), (33, 8, 16, 3, 9), (257, 300, 5, 6, 40), (500, 2376, 5, 6, 17),
    (64, 33, 64, 5, 8), (999, 257, 128, 7, 33), (4099, 20, 5, 7, 5), (20_000, 64, 5, 4, 12)])
def test_small_tree_predictor_equals_the_general_one(rows, features, bins, depth, trees):
    """Bit for bit, with partial row groups and batches, uneven repeats, early leaves and a start value."""
    from packboost_b200 import PackBoost, PackBoostConfig
    from packboost_b200.booster import TreeBuilder
    rng = np.random.default_rng(rows + features)
    X = torch.from_numpy(rng.integers(0, bins, size=(rows, features), dtype=np.uint8)).to(_dev())
    forest = []
    for t in range(trees):
        tb = TreeBuilder()
        level = [0]
        for d in range(depth):
            keep = [n for n in level if d == 0 or rng.random() > 0.1]
            level = [c for n in keep for c in tb.split(n, int(rng.integers(features)), int(rng.integers(bins - 1)))]
        for node in tb.nodes:
            node.value = float(np.float32(rng.normal()))
        forest.append(tb.build())
    model = PackBoost(PackBoostConfig(max_bins=bins, prebinned=True))
    model.set_forest(forest, 0.3, repeats=[int(v) for v in rng.integers(0, 20, trees)])
    packed, _ = model._pack_rows(X)
    small = model._pack_forest(model._distinct)
    assert "slots" in small
    large = {k: v for k, v in small.items() if k != "slots"}
    init = torch.from_numpy(rng.normal(size=rows).astype(np.float32)).to(_dev())
    for start in (None, init):
        got = model._predict_packed(packed, small, init=start)
        want = model._predict_packed(packed, dict(large), init=start)
        assert torch.equal(got.view(torch.int32), want.view(torch.int32))


@pytest.mark.parametrize("dtype", [torch.uint16, torch.int32, torch.int64])
def test_fit_takes_codes_of_any_integer_type_on_the_device(dtype):
    from packboost_b200 import PackBoost, PackBoostConfig
    rng = np.random.default_rng(3)
    X = rng.integers(0, 5, size=(900, 12), dtype=np.uint8)
    y = (X[:, 0] - X[:, 3] + rng.normal(size=900)).astype(np.float32)
    cfg = PackBoostConfig(pack_size=2, max_depth=3, learning_rate=0.2, lambda_l2=1.0, min_samples_leaf=5, max_bins=5, random_state=1)
    want = PackBoost(cfg).fit(X, y, None, num_rounds=2).train_predictions()
    got = PackBoost(cfg).fit(torch.from_numpy(X).to(_dev()).to(dtype), y, None, num_rounds=2).train_predictions()
    np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("trees", [1, 40])
def test_prediction_takes_device_bytes_up_to_max_bins(trees):
    """More than 128 bins: bytes on the device count up to max_bins, host arrays and int8 up to 128."""
    from packboost_b200 import PackBoost, PackBoostConfig
    from packboost_b200.booster import TreeBuilder
    rng = np.random.default_rng(trees)
    X = rng.integers(0, 200, size=(300, 9), dtype=np.uint8)
    X[0, 0] = 199
    forest = []
    for _ in range(trees):
        tb = TreeBuilder()
        for node in tb.split(0, int(rng.integers(9)), int(rng.integers(199))):
            tb.split(node, int(rng.integers(9)), int(rng.integers(199)))
        for node in tb.nodes:
            node.value = float(np.float32(rng.normal()))
        forest.append(tb.build())
    model = PackBoost(PackBoostConfig(max_bins=200, prebinned=True)).set_forest(forest, 1.0)
    on_device = torch.from_numpy(X).to(_dev())
    got = model.predict(on_device)
    want = torch.zeros(300, device=_dev())
    for tree in forest:
        want += tree.predict_bins(on_device)
    np.testing.assert_array_equal(got, want.cpu().numpy())
    np.testing.assert_array_equal(model.predict(on_device[:, :9].t().contiguous().t()), got)   # (the general way)
    for refused in (X, on_device.view(torch.int8), X.view(np.int8)):
        with pytest.raises(ValueError, match="prebinned"):
            model.predict(refused)
    on_device[5, 5] = 200
    with pytest.raises(ValueError, match="prebinned"):
        model.predict(on_device)


def test_a_forest_laid_out_on_one_stream_is_there_for_another(monkeypatch):
    """The first call's stream is busy when the copies are made; a second stream reads them right after."""
    from packboost_b200 import PackBoost, PackBoostConfig
    from packboost_b200.booster import TreeBuilder

    def install(model, sign):
        forest = []
        for t in range(12):
            tb = TreeBuilder()
            tb.split(0, t, 1)
            tb.nodes[1].value, tb.nodes[2].value = sign * (1.0 + t), -sign * (1.0 + t)
            forest.append(tb.build())
        model.set_forest(forest, 1.0)

    plain = torch.Tensor.repeat

    def late(self, *sizes):
        torch.cuda._sleep(200_000_000)           # (about a tenth of a second)
        return plain(self, *sizes)

    model = PackBoost(PackBoostConfig(max_bins=5, prebinned=True))
    install(model, 1.0)
    first, second = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(first):
        shape = model._current_forest()["slots"].shape
    with torch.cuda.stream(second):              # (everything the second stream needs is there before)
        got = torch.zeros(shape, dtype=torch.int32, device=_dev())
        got.copy_(torch.ones_like(got))
    torch.cuda.synchronize()
    install(model, -1.0)
    with torch.cuda.stream(first), monkeypatch.context() as m:
        m.setattr(torch.Tensor, "repeat", late)
        laid = model._current_forest()
    with torch.cuda.stream(second):
        got.copy_(laid["slots"])
    torch.cuda.synchronize()
    assert laid["copies"] > 1 and torch.equal(got, laid["slots"])


@pytest.mark.parametrize("n,f,eras,bins,depth,extra", [
    (700, 32, 1, 17, 3, {}), (5_003, 33, 7, 64, 6, {}), (9_000, 40, 40, 128, 5, dict(era_alpha=4.0)),
    (20_001, 32, 2, 33, 4, {}), (6_000, 35, 9, 100, 5, dict(direction_weight=0.3)),
    (4_000, 32, 5, 64, 4, dict(k_cuts=7, cut_selection="even")), (8_000, 36, 11, 64, 6, dict(k_cuts=9, cut_selection="mass")),
    (3_000, 32, 6, 70, 4, dict(y_scale=1e-12)), (3_000, 32, 6, 70, 4, dict(lambda_l2=1e-9)),
    (3_000, 32, 6, 70, 4, dict(y_scale=2.0 ** -20)), (3_000, 32, 6, 70, 4, dict(y_scale=2.0 ** 33)),   # (scale of the sums: its ends)
    (3_000, 32, 6, 70, 4, dict(lambda_l2=2.0 ** -24)), (3_000, 32, 6, 70, 4, dict(lambda_l2=2.0 ** 24))])
def test_era_walk_equals_the_stored_histogram_path(n, f, eras, bins, depth, extra, tmp_path):
    """Trees, scores and predictions bit for bit between the kernel that walks the eras and the two-step
    path (run in a child process, which the switch is read in): partly filled node groups, eras longer
    than a tile, every form of the score, thresholds in lists, gradients too small for the division table."""
    import json
    import os
    import subprocess
    import sys
    script = r"""
import json, sys
import numpy as np
from packboost_b200 import PackBoost, PackBoostConfig
n, f, eras, bins, depth, extra, out = json.loads(sys.argv[1])
rng = np.random.default_rng(n + f)
X = rng.normal(size=(n, f)).astype(np.float32)
X[:, ::5] = rng.integers(0, 6, size=X[:, ::5].shape)
y = ((X[:, 0] + X[:, 1] * X[:, 2] + 0.3 * rng.normal(size=n)) * extra.pop("y_scale", 1.0)).astype(np.float32)
era = np.sort(rng.integers(0, eras, n)).astype(np.int16)
cfg = dict(pack_size=2, max_depth=depth, learning_rate=0.2, lambda_l2=1.0, lambda_dro=0.4, min_samples_leaf=5, max_bins=bins, random_state=1)
cfg.update(extra)
b = PackBoost(PackBoostConfig(**cfg)).fit(X, y, era, num_rounds=3)
np.savez(out, preds=b.train_predictions().view(np.int32), **{k: v.view(np.int32) if v.dtype == np.float32 else v for k, v in b.split_records().items()})
"""
    got = []
    for walk in ("1", "0"):
        path = str(tmp_path / f"{walk}.npz")
        res = subprocess.run([sys.executable, "-c", script, json.dumps([n, f, eras, bins, depth, extra, path])],
                             env=dict(os.environ, PACKBOOST_WALK=walk), cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                             capture_output=True, text=True)
        assert res.returncode == 0, res.stderr[-2000:]
        got.append(np.load(path))
    assert len(got[0]["node"]) > 3
    for key in got[0].files:
        np.testing.assert_array_equal(got[0][key], got[1][key], err_msg=key)


@pytest.mark.parametrize("n,f,eras,bins,depth,extra", [
    (4_801, 3, 3, 128, 6, {}),                       # a node per warp from sixteen nodes on, thirty-two warps before
    (1_701, 150, 1, 65, 6, {}), (3_333, 4, 2, 17, 8, {}),   # one and two eras; groups of nodes, most rows another's
    (5_003, 33, 7, 64, 8, {}), (2_600, 9, 37, 33, 6, {}),   # eras that start and end anywhere in a warp's rows
    (2_403, 3, 3, 128, 6, dict(y_scale=1e15)),       # sums past the range of the division table
    (2_403, 3, 3, 100, 6, dict(k_cuts=9, cut_selection="mass")), (2_403, 3, 3, 100, 6, dict(lambda_l2=1e-9))])
def test_era_walk_with_a_warp_per_node(n, f, eras, bins, depth, extra, tmp_path):
    """The same comparison at the sizes where the walk changes its form: the number of warps, a warp per
    node, nodes in groups, the division table left out."""
    test_era_walk_equals_the_stored_histogram_path(n, f, eras, bins, depth, extra, tmp_path)


_WALK_FORMS = [                                          # eras, groups of nodes that are partly filled
    (4_801, 5, 7, 128, 7, {}), (5_003, 9, 9, 64, 6, {}), (1_900, 4, 37, 17, 6, {}),
    (2_600, 6, 11, 33, 6, dict(y_scale=1e15)), (3_000, 6, 6, 100, 6, dict(lambda_l2=1e-9)),     # divisions without the table
    (3_403, 5, 5, 100, 6, dict(k_cuts=9, cut_selection="mass")), (3_403, 5, 5, 64, 6, dict(k_cuts=7, cut_selection="even"))]
_WALK_FORMS_SCRIPT = r"""
import json, sys
import numpy as np
from packboost_b200 import PackBoost, PackBoostConfig
out = {}
for i, (n, f, eras, bins, depth, extra) in enumerate(json.loads(sys.argv[1])):
    rng = np.random.default_rng(n + f)
    X = rng.normal(size=(n, f)).astype(np.float32)
    X[:, ::5] = rng.integers(0, 6, size=X[:, ::5].shape)
    y = ((X[:, 0] + X[:, 1] * X[:, 2] + 0.3 * rng.normal(size=n)) * extra.pop("y_scale", 1.0)).astype(np.float32)
    era = np.sort(rng.integers(0, eras, n)).astype(np.int16)
    cfg = dict(pack_size=2, max_depth=depth, learning_rate=0.2, lambda_l2=1.0, lambda_dro=0.4, min_samples_leaf=5, max_bins=bins, random_state=1)
    cfg.update(extra)
    b = PackBoost(PackBoostConfig(**cfg)).fit(X, y, era, num_rounds=2)
    out[f"preds{i}"] = b.train_predictions().view(np.int32)
    for k, v in b.split_records().items():
        out[f"{k}{i}"] = v.view(np.int32) if v.dtype == np.float32 else v
np.savez(sys.argv[2], **out)
"""


def _walk_forms(path, **env):
    import json
    import subprocess
    import sys
    res = subprocess.run([sys.executable, "-c", _WALK_FORMS_SCRIPT, json.dumps(_WALK_FORMS), str(path)], env=dict(os.environ, **env),
                         cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))), capture_output=True, text=True)
    assert res.returncode == 0, res.stderr[-2000:]
    return np.load(path), [line for line in res.stderr.splitlines() if line.startswith("walk_")]


@pytest.fixture(scope="module")
def stored_histogram_fits(tmp_path_factory):
    return _walk_forms(tmp_path_factory.mktemp("walk") / "stored.npz", PACKBOOST_WALK="0", PACKBOOST_WALK_FORM="0")


@pytest.mark.parametrize("form,kernel", list(enumerate(["walk_kernel<{}> warps=16", "walk_kernel<{}> warps=32", "walk_nodes_kernel<{}> warps=16",
                                                   "walk_nodes_kernel<{}> warps=32"])))
def test_every_form_of_the_era_walk_equals_the_stored_histogram_path(form, kernel, stored_histogram_fits, tmp_path):
    """Trees, scores and predictions bit for bit, each form taken at every depth of every fit."""
    want, none = stored_histogram_fits
    got, ran = _walk_forms(tmp_path / "walk.npz", PACKBOOST_WALK="1", PACKBOOST_WALK_FORM=str(form))
    assert not none
    assert {" ".join(line.split()[:2]) for line in ran} == {kernel.format(bpl) for bpl in (1, 2, 4)}, ran
    shapes = [dict(kv.split("=") for kv in line.split()[1:]) for line in ran]
    assert {int(r["nodes"]) for r in shapes} == {1 << d for d in range(7)} and {r["mass"] for r in shapes} == {"0", "1"}
    assert max(int(r["groups"]) for r in shapes) > 1
    assert sum(len(want[f"node{i}"]) for i in range(len(_WALK_FORMS))) > 200
    for key in want.files:
        np.testing.assert_array_equal(got[key], want[key], err_msg=key)


@pytest.mark.parametrize("form", range(4))
def test_era_walk_with_a_byte_that_is_no_bin(form):
    """Bytes of 255 in a column that packing did not check stay within the cells of their node: to the right of every
    threshold, so nothing changes.  (Four rows are fewer than min_samples_leaf: the column, constant but for
    them, is never split.)"""
    import subprocess
    import sys
    script = r"""
import sys
import numpy as np, torch
from packboost_b200.booster import _DeviceTrainer
from packboost_b200.config import PackBoostConfig
from packboost_b200.data import pack_feature_major
from packboost_b200.sharding import feature_map
rng = np.random.default_rng(2)
n, f, eras, depth = 6_000, 6, 8, 6
X = rng.integers(0, 17, size=(n, f), dtype=np.uint8)
y = (X[:, 1] + X[:, 2] * (X[:, 3] > 4) + rng.normal(size=n)).astype(np.float32)
X[:, 0] = 16
logs = []
for bad in (False, True):
    if bad:
        X[[5, 2_500, 4_900, 5_999], 0] = 255         # (the last: in the eighth era, whose cells are the last)
    cfg = PackBoostConfig(device="cuda", pack_size=1, max_depth=depth, learning_rate=0.2, lambda_l2=1.0, min_samples_leaf=30,
                          max_bins=17, prebinned=True)
    tr = _DeviceTrainer(cfg, pack_feature_major(X, None, 17), y, np.linspace(0, n, eras + 1).astype(np.int32), f, feature_map(f, 0, 1), 0, 1)
    ticket = tr.run_round([np.arange(f, dtype=np.int32)] * depth)
    head, winners = tr.read_log(ticket)
    logs.append((head.copy(), winners.copy()))
(h0, w0), (h1, w1) = logs
assert np.array_equal(h0["n_ctx"], h1["n_ctx"]) and h0["n_ctx"].reshape(-1)[4] == 16 and h0["n_ctx"].reshape(-1)[5] > 16
for d in range(depth):
    a, b = (1 << d) - 1, (1 << d) - 1 + int(h0["n_ctx"].reshape(-1)[d])
    assert np.array_equal(w0[a:b], w1[a:b]) and (w1["feature"][a:b] != 0).all(), d
print("ok")
"""
    res = subprocess.run([sys.executable, "-c", script], env=dict(os.environ, PACKBOOST_WALK="1", PACKBOOST_WALK_FORM=str(form)),
                         cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))), capture_output=True, text=True)
    assert res.returncode == 0 and res.stdout.strip().endswith("ok"), res.stderr[-2000:]
    assert ("walk_nodes_kernel<1>" if form >= 2 else "walk_kernel<1>") in res.stderr


@pytest.mark.parametrize("form", ["frontier", "helper"])
@pytest.mark.parametrize("n,eras,bins", [(3_000, 7, 5), (20_000, 1, 5), (17_000, 2, 4), (6_000, 9, 14)])
def test_directional_term_streamed_with_the_gains_matches_the_oracle(form, n, eras, bins, monkeypatch):
    """Few-bin codes: agreement left by the fused flush (one tile per era), by the gain kernel behind
    several tiles and by its many-bin form; era weights on."""
    if form == "helper":
        monkeypatch.setenv("PACKBOOST_DIRECTION_FORM", "helper")
    from packboost_b200 import PackBoost, PackBoostConfig
    rng = np.random.default_rng(n + bins)
    X = rng.integers(0, bins, size=(n, 11), dtype=np.uint8)
    y = (0.3 * X[:, 1] - 0.2 * X[:, 3] * (X[:, 5] > 1) + rng.normal(size=n)).astype(np.float32)
    era = np.sort(rng.integers(0, eras, n)).astype(np.int16)
    cfg = dict(pack_size=2, max_depth=4, learning_rate=0.2, lambda_l2=1.0, lambda_dro=0.3, direction_weight=0.2, era_alpha=3.0,
               min_samples_leaf=10, max_bins=bins, prebinned=True, random_state=5)
    b = PackBoost(PackBoostConfig(device="cuda", **cfg)).fit(X, y, era, num_rounds=2)
    got = b.split_records()
    assert len(got["node"]) > 8
    # every split of both rounds (below the root the parent's direction differs by node): float32 scores bit for bit
    exact = po.fit(X, y, era, po.OracleParams(exact_sums=True, direction_form=form, **cfg), 2, record_depths=True)
    for key in ("node", "feature", "threshold"):
        np.testing.assert_array_equal(got[key], [r[key] for r in exact.depth_records], err_msg=key)
    want = np.asarray([r["score"] for r in exact.depth_records], dtype=np.float32)
    np.testing.assert_array_equal(got["score"].view(np.int32), want.view(np.int32))
    np.testing.assert_array_equal(b.train_predictions().view(np.int32), exact.train_preds.view(np.int32))
    # and the first root re-scored by the general scorer
    root = b._find_best_split(_root_shard(era, eras), torch.from_numpy(-y), torch.ones(n), torch.from_numpy(X.astype(np.int64)),
                              torch.arange(11))
    assert (got["feature"][0], got["threshold"][0]) == (root.feature, root.threshold)
    np.testing.assert_allclose(got["score"][0], root.score, rtol=2e-6)


@pytest.mark.parametrize("bins,eras,n", [(5, 7, 3_000), (14, 2, 17_000), (40, 5, 3_000)])
def test_directional_term_of_child_values_that_round_to_zero(bins, eras, n):
    """A lambda so large that -G / (H + lambda) is no float32: such a child points nowhere.  Codes of 4 and
    of 8 bits, bit for bit with the oracle."""
    from packboost_b200 import PackBoost, PackBoostConfig
    rng = np.random.default_rng(bins)
    X = rng.integers(0, bins, size=(n, 11), dtype=np.uint8)
    y = (5e-10 * (0.3 * X[:, 1] - 0.2 * X[:, 3] + rng.normal(size=n))).astype(np.float32)
    era = np.sort(rng.integers(0, eras, n)).astype(np.int16)
    cfg = dict(pack_size=2, max_depth=3, learning_rate=0.2, lambda_l2=1e37, lambda_dro=0.3, direction_weight=0.2,
               min_samples_leaf=10, max_bins=bins, prebinned=True, random_state=5)
    got = PackBoost(PackBoostConfig(device="cuda", **cfg)).fit(X, y, era, num_rounds=1).split_records()
    exact = po.fit(X, y, era, po.OracleParams(exact_sums=True, **cfg), 1, record_depths=True)
    for key in ("node", "feature", "threshold"):
        np.testing.assert_array_equal(got[key], [r[key] for r in exact.depth_records], err_msg=key)
    want = np.asarray([r["score"] for r in exact.depth_records], dtype=np.float32)
    assert len(want) > 3 and len(set(want.tolist())) > 1
    np.testing.assert_array_equal(got["score"].view(np.int32), want.view(np.int32))


def _root_shard(era, eras):
    from packboost_b200.booster import NodeShard
    return NodeShard(tree_id=0, node_id=0, depth=0, era_rows=[torch.from_numpy(np.flatnonzero(era == e)) for e in range(eras)])


@pytest.mark.parametrize("alpha", [0.0, 3.0])
def test_a_wait_that_ran_out_reaches_every_device(alpha):
    """A device's fault goes out with its candidates, and a candidate that brings one marks the round's log: the
    bit is set by the host, once where a kernel leaves it and once as the exchange brings it from elsewhere."""
    import ctypes as C
    from packboost_b200 import backends as B
    from packboost_b200.booster import _HEADER_DT, _DeviceTrainer
    from packboost_b200.config import PackBoostConfig
    from packboost_b200.data import pack_feature_major
    from packboost_b200.sharding import feature_map
    rng = np.random.default_rng(11)
    n, f, eras, depth = 3_000, 40, 7, 2
    X = rng.integers(0, 5, size=(n, f), dtype=np.uint8)
    y = (X[:, 0] - X[:, 3] + rng.normal(size=n)).astype(np.float32)
    offsets = np.linspace(0, n, eras + 1).astype(np.int32)
    cfg = PackBoostConfig(device="cuda", pack_size=1, max_depth=depth, learning_rate=0.2, lambda_l2=1.0, min_samples_leaf=5,
                          max_bins=5, prebinned=True, era_alpha=alpha)
    lib = B.lib()
    tr = _DeviceTrainer(cfg, pack_feature_major(X, None, 5), y, offsets, f, feature_map(f, 0, 1), 0, 1)
    st, stream = C.byref(tr.st), torch.cuda.current_stream().cuda_stream
    feats = torch.arange(f, dtype=torch.int32, device=_dev())
    ctl = next(t for t in vars(tr).values() if isinstance(t, torch.Tensor) and t.data_ptr() == tr.st.ctl)
    ptr, nbytes, flags = C.c_void_p(), C.c_int64(), C.c_uint32()

    def word_of_flags():         # (the only word of the control block that the getter follows)
        head = ctl.view(torch.int32)
        for i in range(64):
            old = head[i].item()
            head[i] = old ^ 8
            B.check(lib.pb_debug_flags(st, C.byref(flags)))
            head[i] = old
            if flags.value & 8:
                return i
        raise AssertionError("no such word")

    def round_(own: bool, other: bool):
        head = ctl.view(torch.int32)
        head[at] = 0
        B.check(lib.pb_round_begin(st, 0, stream))
        carried = []
        for d in range(depth):
            if own and d == 1:
                head[at] = 8
            B.check(lib.pb_depth_hist_score(st, d, feats.data_ptr(), feats.data_ptr(), f, f, stream))
            B.check(lib.pb_candidates_buffer(st, d, f, C.byref(ptr), C.byref(nbytes)))
            off = ptr.value - tr.workspace.data_ptr()
            cand = tr.workspace[off: off + nbytes.value].view(torch.int32).view(f, 1 << d, 6)
            carried.append((cand[:, :, 3] & 2).ne(0).cpu().numpy())
            if other and d == 0:
                cand[7, 0, 3] |= 2
            B.check(lib.pb_depth_select(st, d, feats.data_ptr(), f, stream))
            B.check(lib.pb_depth_partition(st, d, stream))
        B.check(lib.pb_round_end(st, stream))
        log = tr.log_dev[: _HEADER_DT.itemsize].cpu().numpy().view(_HEADER_DT)[0]
        assert log["n_ctx"][1] == 2                  # (both nodes of the second depth are there)
        return carried, int(log["faults"])

    at = word_of_flags()
    carried, faults = round_(False, False)
    assert not any(c.any() for c in carried) and faults == 0
    carried, faults = round_(True, False)
    assert not carried[0].any() and carried[1].all() and faults == 8
    carried, faults = round_(False, True)
    assert faults == 8
