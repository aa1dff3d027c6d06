// Where a histogram of few bins is faster as a contraction on the tensor cores (hist_mma_kernel) than by atomics
// (hist_lane_kernel).  Plain host code.
#pragma once

#include <stdint.h>

namespace pb {

// Thresholds of a feature that take lanes of a block (4 or 8), how many of them a lane holds, and features of a block.
inline int mma_thresholds(int max_bins) { return max_bins <= 5 ? 4 : 8; }
inline int mma_per_lane(int n_nodes, int n_feat, int max_bins) {
    return n_nodes <= 4 && n_feat > 128 * 2 / mma_thresholds(max_bins) ? 4 : n_nodes <= 16 ? 2 : 1;
}
inline int mma_features(int n_nodes, int n_feat, int max_bins) {
    return 128 * mma_per_lane(n_nodes, n_feat, max_bins) / mma_thresholds(max_bins);
}

// Measured, us of the contraction / us by atomics, at 1, 2, 4, 8, 16, 32 nodes; (2) .. (8): bins, else five.
// Eras of one tile, whose flush makes the gains:
//   2 700 000 x 238, 574 eras  123/171 129/172 158/188 248/231 323/256 553/393;  (2) 122/180 129/182 154/199 244/227 288/278
//                              (4) 123/187 129/190 158/211 250/258 325/368 583/625;  (6) 226/192 232/199 291/240
//   the same, growing eras     133/186 137/186 168/203 277/240 359/265;          (3) 131/197 137/201 166/217 276/254 370/315
//                              (4) 132/201 137/203 168/223 273/266 372/374 740/627
//   1 500 000 x 200, 300       85/136 90/137 109/125 154/139 187/154 286/211;    (3) 85/147 88/148 106/162 152/190 182/207
//   1 000 000 x 238, 574       67/118 89/122 118/113 183/130;                    (4) 68/130 88/132 114/157 181/182 248/270 515/493
//   253 890 x 218, 308         33/38 39/39 55/39 75/49 116/75;                   (4) 33/66 39/58 54/72 76/88 122/92
//   250 000 x 218, 1 000       54/49 76/51;                  (2) 55/69 74/66 111/88;  (4) 56/84 77/78 121/114 198/188
//   700 000 x 100, 300         37/59 39/57 51/58 68/53 89/62;   330 001 x 102, 120  23/29 25/31 29/49 35/35
//   150 000 x 70, 150          23/21 25/22 31/22;  (3) 23/33 25/32 31/33;   300 000 x 60, 60  25/20 27/18 31/20
// So: up to five bins and four nodes (more nodes take two thresholds a lane or one, and the rows' operand is made for 64
// or 32 features at a time where it was 128), with four bins, the worst for the atomics, up to sixteen; features for
// most of a block's lanes; more than 100 tasks; and eras long enough to hide the flush, which has more to do with
// more nodes, and longer ones with five bins, the best for the atomics.
// Eras of several tiles, whose sums both add to a stored histogram (then also 64 nodes):
//   1 300 000 x 57, one era    35/47 39/47 43/55 47/61 47/59 66/74 86/108;       (2) 33/48 37/43 45/47 45/51 53/62 64/53
//                              (3) .. 68/96 86/102;  (4) .. 65/99 84/104;  (6) 39/49 43/49 51/53 62/68 66/94 110/106
//   2 600 000 x 238, 200       111/200 115/206 145/210 215/244 229/278 404/424 647/631;  (2) .. 211/235 219/273 401/312
//                              (6) 197/215 201/232 252/248 397/307;  (7) .. 254/274 397/336;  (8) .. 254/287 397/352
//   1 000 000 x 128, 20        35/42 35/43 43/47 55/51 57/57;   (6) 50/48 51/49 61/53 88/59;  (8) 50/52 50/55 62/57
//   461 197 x 55, one era      20/33 26/35 27/35 29/31 31/37 36/41 47/51;    865 141 x 41  (4) 27/38 31/42 33/43 35/45 37/45 49/66
//   495 200 x 27, one era      21/23 22/25 27/29 27/29 31/33 33/35 42/44;    300 000 x 40  19/35 23/35 25/22 29/29 34/29 29/31
//   248 795 x 33, one era      18/27 21/30 23/21 24/21 27/25 28/29 35/33;    160 630 x 42  17/27 20/18 21/18 23/20
//   100 000 x 30  17/19 20/20 22/20;  (2) 15/21 16/25;  (7) 16/32 18/18;     30 000 x 100, three eras  16/11 16/10 18/12
// So: by rows x features for the fixed 15 us of it, more of them with more nodes or bins; above four nodes one block of
// features or very many rows; and at 32 and 64 nodes the bins where the atomics meet least often.
inline bool mma_pays(bool fused, int n_nodes, int n_feat, int max_bins, int64_t rows, int64_t n_eras) {
    const int features = mma_features(n_nodes, n_feat, max_bins);
    const int64_t blocks = (n_feat + features - 1) / features, work = rows * n_feat;
    if (fused) {
        if (max_bins > 5 || n_feat <= 64 || n_nodes > (n_feat <= 128 ? 2 : max_bins == 4 ? 16 : 4)) return false;
        if (n_eras * blocks < (n_feat > 128 ? 444 : 100)) return false;
        const int era = max_bins == 5 ? (n_nodes == 1 && n_feat > 128 ? 800 : n_nodes <= 2 ? 1500 : 2500)
                                      : n_nodes == 1 ? 0 : n_nodes <= 4 ? 400 : n_nodes <= 8 ? 800 : 1700;
        return rows >= era * n_eras;
    }
    if (rows < 100000) return false;
    if (n_nodes <= 2) return work >= (max_bins > 5 ? 10000000 : n_nodes == 1 ? 3000000 : 8000000);
    const bool one_block = n_feat <= 64 && work >= 13000000;   // (at two thresholds a lane, up to five bins)
    const bool many = work >= 200000000;
    // (more than five bins: but where the atomics have a feature on every lane)
    if (n_nodes <= 4) return work >= 13000000 && (max_bins <= 5 || n_feat * 100 < (n_feat + 31) / 32 * 32 * 95);
    if (n_nodes <= 16) return one_block || (max_bins <= 5 && many);
    if (max_bins < 3 || max_bins > 5) return false;
    return one_block || (n_nodes <= 32 && max_bins > 3 && work >= 50000000 && n_feat * 100 >= blocks * features * 85);
}

}  // namespace pb
