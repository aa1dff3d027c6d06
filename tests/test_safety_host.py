"""Host-side refusals that keep malformed input away from the GPU (no device needed)."""

import ctypes as C
import os

import numpy as np
import pytest

from packboost_b200.forest import validate_forest


def _tree(left, right, is_leaf, feature=None, threshold=None):
    n = len(left)
    feature = feature if feature is not None else [0 if not l else -1 for l in is_leaf]
    threshold = threshold if threshold is not None else [1] * n
    return (np.asarray(feature, np.int32), np.asarray(threshold, np.int32), np.asarray(left, np.int32),
            np.asarray(right, np.int32), np.asarray(is_leaf, np.uint8))


def test_well_formed_trees_pass_and_report_the_largest_tree():
    f, t, l, r, il = _tree([1, -1, 3, -1, -1], [2, -1, 4, -1, -1], [0, 1, 0, 1, 1])
    assert validate_forest(f, t, l, r, il, [0, 5]) == 5
    # two trees back to back, the second a single leaf
    f2 = np.concatenate([f, [-1]]).astype(np.int32)
    assert validate_forest(f2, np.append(t, 0), np.append(l, -1), np.append(r, -1), np.append(il, 1), [0, 5, 6]) == 5
    # children need not be adjacent, only later than their parent
    f, t, l, r, il = _tree([2, -1, 4, -1, -1], [1, -1, 3, -1, -1], [0, 1, 0, 1, 1])
    assert validate_forest(f, t, l, r, il, [0, 5]) == 5


@pytest.mark.parametrize("left,right,why", [
    ([0, -1, -1], [2, -1, -1], "a node that is its own child (cycle)"),
    ([1, 0, -1], [2, 2, -1], "a child that points back to the root (cycle)"),
    ([1, -1, -1], [7, -1, -1], "a child outside the tree"),
    ([1, -1, -1], [-3, -1, -1], "a negative child of an internal node"),
])
def test_cyclic_and_out_of_range_children_are_refused(left, right, why):
    is_leaf = [0, 1 if left[1] < 0 else 0, 1]
    f, t, l, r, il = _tree(left, right, is_leaf)
    with pytest.raises(ValueError, match="children"):
        validate_forest(f, t, l, r, il, [0, 3])


def test_children_must_stay_inside_their_own_tree():
    # tree 0 = nodes 0..2, tree 1 = nodes 3..5; node 0 points at relative index 4 (a node of tree 1)
    f, t, l, r, il = _tree([1, -1, -1, 1, -1, -1], [4, -1, -1, 2, -1, -1], [0, 1, 1, 0, 1, 1])
    with pytest.raises(ValueError, match="children"):
        validate_forest(f, t, l, r, il, [0, 3, 6])
    # the same ensemble with absolute child ids is fine when they stay in range ...
    f, t, l, r, il = _tree([1, -1, -1, 4, -1, -1], [2, -1, -1, 5, -1, -1], [0, 1, 1, 0, 1, 1])
    assert validate_forest(f, t, l, r, il, [0, 3, 6], absolute_children=True) == 3
    # ... and refused when a child crosses into the other tree
    f, t, l, r, il = _tree([1, -1, -1, 4, -1, -1], [3, -1, -1, 5, -1, -1], [0, 1, 1, 0, 1, 1])
    with pytest.raises(ValueError, match="children"):
        validate_forest(f, t, l, r, il, [0, 3, 6], absolute_children=True)


def test_feature_threshold_and_offset_ranges():
    f, t, l, r, il = _tree([1, -1, -1], [2, -1, -1], [0, 1, 1], feature=[9, -1, -1])
    assert validate_forest(f, t, l, r, il, [0, 3], n_features=10) == 3
    with pytest.raises(ValueError, match="feature"):
        validate_forest(f, t, l, r, il, [0, 3], n_features=9)
    f, t, l, r, il = _tree([1, -1, -1], [2, -1, -1], [0, 1, 1], feature=[-1, -1, -1])
    with pytest.raises(ValueError, match="feature"):
        validate_forest(f, t, l, r, il, [0, 3])
    f, t, l, r, il = _tree([1, -1, -1], [2, -1, -1], [0, 1, 1], threshold=[300, 0, 0])
    with pytest.raises(ValueError, match="threshold"):
        validate_forest(f, t, l, r, il, [0, 3])
    f, t, l, r, il = _tree([1, -1, -1], [2, -1, -1], [0, 1, 1])
    for offs in ([1, 3], [0, 2], [0, 3, 2, 3], [0, 0, 3]):
        with pytest.raises(ValueError):
            validate_forest(f, t, l, r, il, offs)


def test_predictor_refuses_a_malformed_file_before_touching_the_device(tmp_path):
    from packboost_b200.wrapper import PackBoostPredictor
    path = str(tmp_path / "bad.npz")
    np.savez(path, tree_offsets=np.array([0, 3]), repeats=np.array([1], np.int32), tree_weight=np.float64(1.0),
             max_bins=np.int64(5), pack_size=np.int64(1), has_edges=np.bool_(False),
             bin_edges=np.zeros((0, 0), np.float32), feature=np.array([0, -1, -1], np.int32),
             threshold=np.array([1, 0, 0], np.int32), left=np.array([0, -1, -1], np.int32),
             right=np.array([2, -1, -1], np.int32), value=np.zeros(3), is_leaf=np.array([0, 1, 1], np.uint8))
    with pytest.raises(ValueError, match="children"):
        PackBoostPredictor.load(path)


# ---- training state: alignment and the no-workspace mode, through the C ABI ------------------------

@pytest.fixture(scope="module")
def lib():
    from packboost_b200 import build
    build.build()
    from packboost_b200 import backends as B
    return B.lib()


def _state(B, base=1 << 20):
    """A shape-valid training state over made-up addresses (never dereferenced: pb_train_prepare
    does no device work)."""
    st = B.TrainState()
    st.n_rows, st.n_features_total, st.n_features_local, st.n_eras = 1000, 4, 4, 2
    st.max_bins, st.code_bits, st.pitch = 5, 4, 512
    st.max_depth, st.pack_size, st.min_samples_leaf, st.n_thresholds, st.feature_block_size = 3, 2, 5, 4, 32
    st.lambda_l2, st.learning_rate = 1e-3, 0.1
    for i, name in enumerate(("codes", "era_offsets", "thr_ids", "feat_local", "y", "preds", "gq", "slot", "leaf", "ctl")):
        setattr(st, name, base * (i + 1))
    st.workspace = base * 20
    st.workspace_bytes = 1 << 30
    return st


def test_codes_must_be_32_byte_aligned(lib):
    from packboost_b200 import backends as B
    eo = np.array([0, 600, 1000], np.int32)
    st = _state(B)
    B.check(lib.pb_train_prepare(C.byref(st), eo.ctypes.data))
    st.codes = (1 << 20) + 16          # 16-byte aligned only: the 256-bit code loads would fault
    with pytest.raises(ValueError, match="32-byte"):
        B.check(lib.pb_train_prepare(C.byref(st), eo.ctypes.data))


def test_a_state_without_workspace_is_accepted_and_workspace_entries_say_so(lib):
    from packboost_b200 import backends as B
    eo = np.array([0, 600, 1000], np.int32)
    st = _state(B)
    st.workspace = None
    st.workspace_bytes = 0
    B.check(lib.pb_train_prepare(C.byref(st), eo.ctypes.data))
    with pytest.raises(ValueError, match="needs pb_train_state.workspace"):
        B.check(lib.pb_depth_hist_score(C.byref(st), 0, None, None, 0, 1, None))
    with pytest.raises(ValueError, match="needs pb_train_state.workspace"):
        B.check(lib.pb_depth_select(C.byref(st), 0, None, 1, None))
    ptr, nbytes = C.c_void_p(), C.c_int64()
    with pytest.raises(ValueError, match="needs pb_train_state.workspace"):
        B.check(lib.pb_candidates_buffer(C.byref(st), 0, 1, C.byref(ptr), C.byref(nbytes)))
    st.workspace_bytes = 64            # a size without a pointer is a caller error
    with pytest.raises(ValueError, match="workspace is null"):
        B.check(lib.pb_train_prepare(C.byref(st), eo.ctypes.data))
    st = _state(B)
    st.workspace_bytes = 16            # a pointer with too few bytes still is, too
    with pytest.raises(ValueError, match="workspace too small"):
        B.check(lib.pb_train_prepare(C.byref(st), eo.ctypes.data))


@pytest.mark.parametrize("rows,feats,eras,depth,walks", [
    (4_000_000, 32, 20, 0, 0), (4_000_000, 32, 20, 5, 0), (1_000_000, 64, 100, 0, 0), (262_144, 16, 100, 0, 0),
    (262_144, 64, 20, 3, 0), (500_000, 200, 100, 5, 1), (131_072, 200, 574, 0, 1), (131_072, 8, 574, 5, 1),
    (2_000_000, 148, 574, 5, 1)])
def test_many_bins_take_the_path_that_measured_faster(lib, rows, feats, eras, depth, walks):
    """Sizes at which one of the two equal paths measured 1.4 to 6 times as fast as the other; and a
    workspace too small for the stored histogram leaves the walk."""
    from packboost_b200 import backends as B
    if "PACKBOOST_WALK" in os.environ:
        pytest.skip("the path is forced")
    st = _state(B)
    st.n_rows, st.n_eras, st.max_bins, st.code_bits, st.pitch = rows, eras, 128, 8, (rows + 255) // 256 * 256
    st.n_features_total = st.n_features_local = feats
    st.max_depth, st.n_thresholds, st.workspace_bytes = 6, 127, 8 << 30
    eo = (np.arange(eras + 1, dtype=np.int64) * rows // eras).astype(np.int32)
    B.check(lib.pb_train_prepare(C.byref(st), eo.ctypes.data))
    got = C.c_int64(-1)
    B.check(lib.pb_depth_walks(C.byref(st), depth, feats, feats, C.byref(got)))
    assert got.value == walks
    st.workspace_bytes = (24 * feats << depth) + 512
    B.check(lib.pb_depth_walks(C.byref(st), depth, feats, feats, C.byref(got)))
    assert got.value == 1
    st.max_bins, st.n_thresholds, st.code_bits = 5, 4, 4
    st.workspace_bytes = 8 << 30
    B.check(lib.pb_depth_walks(C.byref(st), depth, feats, feats, C.byref(got)))
    assert got.value == 0


_ROWS = """#include "rows.cuh"
#include <cstdio>
int main() {
    long long b, e, i, t, n;
    while (std::scanf("%lld %lld %lld %lld %lld", &b, &e, &i, &t, &n) == 5) {
        int r0, r1;
        pb::tile_range((int)b, (int)e, (int)i, (int)t, r0, r1);
        std::printf("%d %d %d\\n", r0, r1, pb::tiles_of(n, t));
    }
    return 0;
}
"""


def test_row_ranges_of_tiles_up_to_the_largest_table(tmp_path):
    """Tiles of an era that ends at the last row of the largest table (2^31 - 513 rows), and the tiles past the
    end of a short era behind a very long one, where 32-bit sums would come out negative."""
    import subprocess
    csrc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "packboost_b200", "csrc")
    (tmp_path / "rows.cpp").write_text(_ROWS)
    subprocess.run(["g++", "-std=c++17", "-O2", "-fsanitize=undefined", "-fno-sanitize-recover", "-I", csrc,
                    str(tmp_path / "rows.cpp"), "-o", str(tmp_path / "rows")], check=True)
    last = 2 ** 31 - 513
    asked = [(b, e, i, t, n) for t in (512, 8160, 32256) for b, e in ((0, 0), (0, 10), (0, last), (last - 7, last), (2 ** 30 + 9, last), (last, last))
             for i in (0, 1, -(-(last) // t) - 1, -(-(e - b) // t)) for n in (0, 1, t, t + 1, last)]
    out = subprocess.run([str(tmp_path / "rows")], input="\n".join(" ".join(map(str, a)) for a in asked), capture_output=True,
                         text=True, check=True).stdout.split()
    for k, (b, e, i, t, n) in enumerate(asked):
        r0 = min(b + i * t, e)
        assert [int(v) for v in out[3 * k: 3 * k + 3]] == [r0, min(r0 + t, e), -(-n // t)], (b, e, i, t, n)


_SHARES = """#include "rows.cuh"
#include <cstdio>
#include <vector>
using namespace pb;
int main() {                             // eras, feature blocks, shares, whole, tile, offsets -> shares; share, block, era, r0, r1, b0, b1
    int E, blocks, grid, whole, tile;
    while (std::scanf("%d %d %d %d %d", &E, &blocks, &grid, &whole, &tile) == 5) {
        std::vector<int> off(E + 1);
        for (int& o : off) std::scanf("%d", &o);
        const int64_t work = off[E] + (whole ? (int64_t)512 * E : 0);
        const Shares s = shares_of(blocks, work, grid, !whole);
        std::printf("%d\\n", s.count);
        auto cut = [&](int share, int* c) {
            int fb, hits = 0, row = 0;
            const int64_t at = share_begin(s, share, fb);
            for (int e = 0; e <= E; ++e)
                if (fb == blocks ? e == 0 : whole ? cut_in_era<true>(off.data(), E, at, 512, e, row) : cut_in_era<false>(off.data(), E, at, 0, e, row)) {
                    ++hits;
                    c[0] = e == E ? fb + 1 : fb;
                    c[1] = e == E ? 0 : e;
                    c[2] = e == E || fb == blocks ? 0 : row;
                }
            return hits == 1;
        };
        for (int i = 0; i < s.count; ++i) {
            int from[3], to[3];
            if (!cut(i, from) || !cut(i + 1, to)) return 1;
            RowTask x{from[0], 0, 0, from[2], 0, 0, from[1]};
            while (next_row_task(off.data(), E, whole != 0, to, tile, x))
                std::printf("%d %d %d %d %d %d %d\\n", i, x.fb, x.era, x.r0, x.r1, x.b0, x.b1);
        }
        std::printf("-1\\n");
    }
    return 0;
}
"""


def test_shares_of_rows_are_even_and_complete(tmp_path):
    """Shares of a histogram launch: every row of every feature block in one of them, and none longer than its part by
    more than an era (eras kept whole; half a one at each end) or a block of rows (eras divided), whatever the lengths."""
    import subprocess
    csrc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "packboost_b200", "csrc")
    (tmp_path / "shares.cpp").write_text(_SHARES)
    subprocess.run(["g++", "-std=c++17", "-O2", "-fsanitize=undefined", "-fno-sanitize-recover", "-I", csrc,
                    str(tmp_path / "shares.cpp"), "-o", str(tmp_path / "shares")], check=True)
    rng = np.random.default_rng(5)
    last = 2 ** 31 - 513
    lengths = [[1], [700], [9_000], [0, 5, 0, 0, 9_000, 0], [1_000_000, 100_000], [10] * 300 + [40_000] + [0] * 7, [last - 70_000, 0, 70_000],
               [4_700] * 574, rng.gamma(4.0, 1_175.0, 574).astype(int).tolist(), np.linspace(2_500, 6_900, 574).astype(int).tolist(),
               rng.gamma(4.0, 700.0, 120).astype(int).tolist(), [0] * 40 + [3] * 40]
    asked = [(n, blocks, grid, whole) for n in lengths for blocks in (1, 2, 7) for whole in (0, 1) for grid in (1, 3, 148)
             if grid <= blocks * (len(n) if whole else -(-sum(n) // 512)) and (not whole or sum(n) < 1 << 30)]
    text = "\n".join(" ".join(map(str, [len(n), blocks, grid, whole, 32_256] + np.concatenate([[0], np.cumsum(n)]).tolist())) for n, blocks, grid, whole in asked)
    out = subprocess.run([str(tmp_path / "shares")], input=text, capture_output=True, text=True, check=True).stdout
    for (n, blocks, grid, whole), part in zip(asked, out.split("-1\n")):
        off = np.concatenate([[0], np.cumsum(n)]).astype(np.int64)
        head, *lines = part.splitlines()
        shares = int(head)
        assert grid - 4 * (not whole) <= shares <= grid
        t = np.array([line.split() for line in lines], dtype=np.int64).reshape(-1, 7)
        share, fb, era, r0, r1, b0, b1 = t.T
        assert ((off[era] <= r0) & (r0 <= r1) & (r1 <= off[era + 1]) & (b0 == r0 // 512) & (b1 == np.where(r0 < r1, -(-r1 // 512), b0))).all()
        assert (np.diff(share) >= 0).all()
        if whole:                                   # every era of every block once, in order
            assert (fb * len(n) + era).tolist() == list(range(blocks * len(n))) and (r0 == off[era]).all() and (r1 == off[era + 1]).all()
            most = max(n) + 512
        else:                                       # the rows follow on one another
            assert (r0 < r1).all() and (r1 - r0 <= 32_256).all()
            place = fb * off[-1] + r0
            assert (place[1:] == (fb * off[-1] + r1)[:-1]).all() and place[0] == 0 and fb[-1] * off[-1] + r1[-1] == blocks * off[-1]
            most = 512
            if shares % blocks == 0:                # a share has rows of one block
                assert all(len(set(fb[share == i])) == 1 for i in set(share.tolist()))
        loads = np.bincount(share, weights=(r1 - r0) + 512 * whole, minlength=grid)
        assert loads.max() <= blocks * (off[-1] + 512 * whole * len(n)) / shares + most, (n[:5], blocks, grid, whole)


_RULE = """#include "hist_rule.h"
#include <cstdio>
int main() {
    long long fused, nodes, feats, bins, rows, eras;
    while (std::scanf("%lld %lld %lld %lld %lld %lld", &fused, &nodes, &feats, &bins, &rows, &eras) == 6)
        std::printf("%d\\n", (int)pb::mma_pays(fused != 0, (int)nodes, (int)feats, (int)bins, rows, eras));
    return 0;
}
"""


def test_few_bins_take_the_kernel_that_measured_faster(tmp_path):
    """us of the contraction and of the atomics, measured side by side, by number of bins and nodes: where they are
    a tenth apart or more in favour of the atomics, the rule is with them, and with the contraction where it saves a quarter
    of a launch of up to four nodes and five bins."""
    import subprocess
    csrc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "packboost_b200", "csrc")
    (tmp_path / "rule.cpp").write_text(_RULE)
    subprocess.run(["g++", "-std=c++17", "-I", csrc, str(tmp_path / "rule.cpp"), "-o", str(tmp_path / "rule")], check=True)
    measured = [      # gains in the flush, rows, features, eras, bins, (nodes, contraction, atomics) ...
        (1, 2_700_000, 238, 574, 2, [(1, 122, 180), (2, 129, 182), (4, 154, 199), (8, 244, 227), (32, 577, 381)]),
        (1, 2_700_000, 238, 574, 4, [(1, 123, 187), (2, 129, 190), (4, 158, 211)]),
        (1, 2_700_000, 238, 574, 5, [(1, 123, 171), (2, 129, 172), (4, 158, 188), (8, 248, 231), (16, 323, 256), (32, 553, 393)]),
        (1, 2_700_000, 238, 574, 6, [(1, 226, 192), (2, 232, 199), (4, 291, 240)]),
        (1, 1_000_000, 238, 574, 3, [(1, 68, 140), (2, 83, 132), (4, 109, 149), (16, 251, 225), (32, 517, 372)]),
        (1, 1_000_000, 238, 574, 5, [(1, 67, 118), (2, 89, 122), (8, 183, 130), (16, 250, 159), (32, 494, 243)]),
        (1, 1_500_000, 200, 300, 5, [(1, 85, 136), (2, 90, 137), (8, 154, 139), (16, 187, 154), (32, 286, 211)]),
        (1, 253_890, 218, 308, 4, [(1, 33, 66), (2, 39, 58), (4, 54, 72), (16, 122, 92), (32, 230, 125)]),
        (1, 253_890, 218, 308, 5, [(4, 55, 39), (8, 75, 49), (16, 116, 75)]),
        (1, 250_000, 218, 1000, 2, [(2, 74, 66), (4, 111, 88), (8, 176, 138), (16, 292, 234)]),
        (1, 250_000, 218, 1000, 5, [(1, 54, 49), (2, 76, 51), (4, 117, 64)]),
        (1, 600_000, 300, 2000, 4, [(1, 142, 420), (8, 457, 343), (16, 806, 512)]),
        (1, 700_000, 100, 300, 5, [(1, 37, 59), (2, 39, 57), (8, 68, 53), (16, 89, 62), (32, 160, 94)]),
        (1, 150_000, 70, 150, 5, [(2, 25, 22), (4, 31, 22), (8, 35, 24), (16, 50, 29), (32, 71, 36)]),
        (1, 300_000, 60, 60, 5, [(1, 25, 20), (2, 27, 18), (4, 31, 20), (8, 31, 27), (16, 37, 27), (32, 39, 29)]),
        (0, 1_300_000, 57, 1, 2, [(1, 33, 48), (32, 64, 53)]),
        (0, 1_300_000, 57, 1, 5, [(1, 35, 47), (32, 66, 74)]),
        (0, 2_600_000, 238, 200, 2, [(1, 109, 203), (2, 111, 207), (4, 137, 216), (32, 401, 312), (64, 646, 418)]),
        (0, 2_600_000, 238, 200, 3, [(1, 109, 203), (2, 113, 207), (4, 139, 221), (32, 401, 362)]),
        (0, 2_600_000, 238, 200, 5, [(1, 111, 200), (2, 115, 206), (4, 145, 210)]),
        (0, 2_600_000, 238, 200, 6, [(8, 397, 307), (32, 724, 480), (64, 1190, 678)]),
        (0, 1_000_000, 128, 20, 2, [(32, 92, 62), (64, 127, 78)]),
        (0, 1_000_000, 128, 20, 6, [(4, 61, 53), (8, 88, 59), (32, 164, 100), (64, 242, 141)]),
        (0, 1_000_000, 100, 20, 5, [(1, 33, 56), (2, 35, 55), (4, 41, 57), (32, 93, 78)]),
        (0, 300_000, 40, 1, 5, [(1, 19, 35), (2, 23, 35), (16, 34, 29), (64, 39, 29)]),
        (0, 300_000, 40, 1, 8, [(64, 61, 43)]),
        (0, 248_795, 33, 1, 5, [(1, 18, 27), (2, 21, 30), (4, 23, 21), (8, 24, 21)]),
        (0, 461_197, 55, 1, 5, [(1, 20, 33), (2, 26, 35)]),
        (0, 160_630, 42, 1, 5, [(1, 17, 27), (2, 20, 18), (4, 21, 18), (8, 23, 20), (16, 27, 23), (64, 33, 24)]),
        (0, 1_000_000, 60, 1, 6, [(1, 33, 46), (32, 86, 78), (64, 111, 92)]),
        (0, 100_000, 30, 1, 3, [(1, 15, 25), (8, 25, 16), (16, 27, 16), (32, 25, 14), (64, 35, 16)]),
        (0, 100_000, 30, 1, 5, [(4, 22, 20), (8, 20, 18), (32, 25, 18), (64, 31, 20)]),
        (0, 30_000, 100, 3, 5, [(1, 16, 11), (2, 16, 10), (4, 18, 12), (8, 18, 12), (16, 23, 12), (32, 28, 14)]),
        (0, 150_000, 16, 2, 5, [(2, 16, 14), (4, 20, 16), (8, 18, 14), (16, 23, 16), (32, 29, 16), (64, 43, 20)])]
    flat = [(fused, n, feats, bins, rows, eras, a, b) for fused, rows, feats, eras, bins, at in measured for n, a, b in at]
    out = subprocess.run([str(tmp_path / "rule")], input="\n".join(" ".join(map(str, c[:6])) for c in flat), capture_output=True, text=True,
                         check=True).stdout.split()
    for c, takes in zip(flat, out):
        if c[6] >= 1.1 * c[7]:
            assert takes == "0", c
        if c[6] <= 0.75 * c[7] and c[1] <= 4 and c[3] <= 5:
            assert takes == "1", c


@pytest.mark.parametrize("flags", [[], ["-U__SSE2__"]])
def test_host_sources_need_no_x86(flags, tmp_path):
    """The ring copy builds without x86 intrinsics (``-U__SSE2__``: as on another host) and moves every
    byte either way; no other source includes an intrinsics header."""
    import glob
    import re
    import subprocess
    csrc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "packboost_b200", "csrc")
    for path in glob.glob(os.path.join(csrc, "*")):
        if os.path.isfile(path) and os.path.basename(path) != "stream_copy.h":
            assert not re.search(r"#include\s*<\w*intrin\.h>", open(path).read()), path
    deps = subprocess.run(["g++", "-std=c++17", *flags, "-M", "-x", "c++", os.path.join(csrc, "stream_copy.h")],
                          capture_output=True, text=True, check=True).stdout
    assert ("intrin.h" in deps) == (not flags and "__SSE2__" in subprocess.run(
        ["g++", "-dM", "-E", "-x", "c++", os.devnull], capture_output=True, text=True, check=True).stdout)
    src = tmp_path / "copy.cpp"
    src.write_text("""#include "stream_copy.h"
#include <vector>
int main() {
    alignas(16) static char dst[5000];
    std::vector<char> src(5000);
    for (int i = 0; i < 5000; ++i) src[i] = (char)(i * 7 + 1);
    for (int n : {0, 1, 15, 63, 64, 65, 127, 128, 1000, 4093}) {
        memset(dst, 0, sizeof(dst));
        pb::stream_copy(dst, src.data() + 3, n);
        if (memcmp(dst, src.data() + 3, n) || dst[n]) return 1;
    }
    return 0;
}
""")
    subprocess.run(["g++", "-std=c++17", "-O2", *flags, "-I", csrc, str(src), "-o", str(tmp_path / "copy")], check=True)
    assert subprocess.run([str(tmp_path / "copy")]).returncode == 0


_NO_MEMORY = """
import ctypes as C, resource, sys
import numpy as np
lib = C.CDLL({lib!r})
n = 20_000_000
one = np.ones(n, np.uint8)
ints = np.zeros(n, np.int32)
value = np.zeros(n, np.float32)
offs = np.array([0, n], np.int32)
src, dst, ring = np.ones(2 << 20, np.uint8), np.zeros(2 << 20, np.uint8), np.zeros((2 << 20) + 16, np.uint8)
slot, depth, out = C.c_int64(), C.c_int64(), np.zeros(4, np.uint32)
lib.pb_last_error.restype = C.c_char_p
i64, p = C.c_int64, lambda a: C.c_void_p(a.ctypes.data)
tree = [p(ints), p(ints), p(ints), p(ints), p(value), p(one), p(offs)]
pages = int(open("/proc/self/statm").read().split()[0])
resource.setrlimit(resource.RLIMIT_AS, (pages * 4096 + (4 << 20),) * 2)
if {what!r} == "shape":
    rc = lib.pb_forest_shape(*tree, i64(1), C.byref(slot), C.byref(depth))
elif {what!r} == "words":
    rc = lib.pb_forest_words(*tree, i64(1), i64(4), i64(0), p(out))
elif {what!r} == "negative":
    rc = lib.pb_forest_shape(*tree, i64(-1), C.byref(slot), C.byref(depth))
else:   # no thread can be had (and without a device the copy itself is refused)
    at = ring.ctypes.data + 15 & ~15
    rc = lib.pb_upload(p(dst), p(src), i64(2 << 20), C.c_void_p(at), i64(2 << 20), None)
print("rc", rc, lib.pb_last_error().decode())
"""


@pytest.mark.parametrize("what,rc", [("shape", (-5,)), ("words", (-5,)), ("negative", (-1,)), ("threads", (0, -2, -5))])
def test_a_host_out_of_memory_or_threads_is_an_error_code(lib, what, rc):
    """No C++ exception leaves an entry point (it would end the process): address space runs out in a child
    process."""
    import subprocess
    import sys
    from packboost_b200 import backends as B
    res = subprocess.run([sys.executable, "-c", _NO_MEMORY.format(lib=B._LIB_PATH, what=what)], capture_output=True, text=True)
    assert res.returncode == 0 and int(res.stdout.split()[1]) in rc, (res.returncode, res.stdout, res.stderr[-2000:])


_DIVIDE = """#include "divide.cuh"
#include <cstdio>
#include <cstring>
#include <random>
int main() {
    std::mt19937_64 rng(7);
    long long n = 0, bad = 0;
    auto check = [&](float a, float d) {
        volatile float num = a, den = d;
        const float y = 1.0f / den, want = num / den, got = pb::divide_by(a, d, y);
        ++n;
        if (memcmp(&want, &got, 4)) { if (bad++ < 5) std::printf("%a / %a: %a, not %a\\n", a, d, got, want); }
    };
    for (int es = -48; es <= 5; es += es < -40 || es >= -2 ? 1 : 7)
        for (int el : {-24, -23, -20, -10, -3, -1, 0, 1, 5, 12, 13, 20, 23, 24}) {
            const float inv = ldexpf(1.0f, es);
            for (int i = 0; i < 30000; ++i) {
                // lambda anywhere in its binade (the ends: the powers themselves), rows of an era, a sum of theirs
                float lam = ldexpf(1.0f, el);
                if (i % 3 && el < 24) lam += ldexpf((float)(rng() >> 40), el - 24);
                if (!pb::division_in_range(inv, lam)) return 2;
                const int rows = i % 5 == 0 ? (int)(rng() % 4) + 1 : (int)(rng() % 8192) + 1;
                long long g = (long long)(rng() >> (20 + rng() % 43)) | 1;
                if (i % 7 == 0) g = 1;
                if (i % 11 == 0) g = (1ll << 44) - (long long)(rng() % 3);
                const float s = (float)g * inv, d = (float)rows + lam, sq = s * s;
                check(sq, d);
                check(0.5f * sq, d);
                check(0.0f, i % 2 ? d : lam);
            }
        }
    const float tiny = ldexpf(1.0f, -48), lo = ldexpf(1.0f, -24), hi = ldexpf(1.0f, 24);
    const bool ends = pb::division_in_range(tiny, lo) && pb::division_in_range(32.0f, hi) && !pb::division_in_range(0.5f * tiny, 1.0f) &&
                      !pb::division_in_range(64.0f, 1.0f) && !pb::division_in_range(1.0f, 0.5f * lo) && !pb::division_in_range(1.0f, 2.0f * hi);
    std::printf("%lld divisions, %lld differ\\n", n, bad);
    return bad || !ends;
}
"""


def test_division_by_a_known_reciprocal_is_the_division(tmp_path):
    """Every quotient of the era walk's gains is the correctly rounded one (the host's division): squares of
    gradient sums over row counts plus lambda, up to the ends of the range in which the table is used."""
    import subprocess
    csrc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "packboost_b200", "csrc")
    (tmp_path / "divide.cpp").write_text(_DIVIDE)
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", csrc, str(tmp_path / "divide.cpp"),
                    "-o", str(tmp_path / "divide")], check=True)
    res = subprocess.run([str(tmp_path / "divide")], capture_output=True, text=True)
    assert res.returncode == 0, (res.returncode, res.stdout)


def test_comm_entries_validate_their_arguments_without_a_gpu(lib):
    """The NCCL-backed exchange entries refuse bad arguments before touching NCCL or a device."""
    from packboost_b200 import backends as B
    comm = C.c_void_p()
    ident = (C.c_ubyte * 128)()
    for n_ranks, rank in ((0, 0), (2, 2), (2, -1)):
        with pytest.raises(ValueError, match="out of range"):
            B.check(lib.pb_comm_init(C.byref(comm), ident, n_ranks, rank))
    with pytest.raises(ValueError, match="null"):
        B.check(lib.pb_comm_init(None, ident, 2, 0))
    with pytest.raises(ValueError, match="null"):
        B.check(lib.pb_comm_unique_id(None))
    with pytest.raises(ValueError, match="communicator is null"):
        B.check(lib.pb_comm_allreduce_mask(None, 1 << 20, 16, None))
    st = _state(B)
    with pytest.raises(ValueError, match="communicator is null"):
        B.check(lib.pb_comm_allreduce_candidates(None, C.byref(st), 0, 4, None))
    assert lib.pb_comm_destroy(None) == 0
