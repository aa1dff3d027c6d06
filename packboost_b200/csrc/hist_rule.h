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
//   2 700 000 x 238, 574 eras  123/170 129/171 160/187 248/229 289/256 572/393;  (2) 122/179 125/182 156/198 248/227
//                              (6) 226/192 232/199 291/240
//   the same, growing eras     132/185 137/186 171/203 270/238 382/264 813/402;  (3) 132/196 135/199 168/215 260/254
//   1 500 000 x 200, 300       86/136 90/137 111/125 156/138 176/154 296/211;    (3) 85/147 88/148 108/162 156/189
//   1 000 000 x 238, 574       68/119 88/121 121/113 180/131;                    (4) 68/135 88/137 120/158 182/177
//   700 000 x 100, 300         37/57 39/57 51/57 66/53 94/61 167/96
//   330 001 x 102, 120         25/29 25/31 29/49 35/34;   150 000 x 70, 150  24/21 25/22 31/22;  (3) 24/33 25/33 31/33
//   300 000 x 60, 60           25/20 27/18 31/20
// So: up to four nodes (more take two thresholds a lane or one, and the rows' operand is made for 64 or 32 features at
// a time where it was 128) and up to five bins; features for most of a block's lanes; more than 100 tasks; and with
// five bins, where the atomics are at their best, eras long enough to hide the flush.
// Eras of several tiles, whose sums both add to a stored histogram (then also 64 nodes):
//   1 300 000 x 57, one era    35/47 39/47 43/55 47/61 47/59 66/74 86/108;       (2) 33/48 37/43 45/47 45/51 53/62 64/53
//                              (3) .. 68/96 86/102;  (4) .. 65/99 84/104;  (6) 39/49 43/49 51/53 62/68 66/94 110/106
//   2 600 000 x 238, 200       111/200 115/206 145/210 215/244 229/278 404/424 647/631;  (2) .. 211/235 219/273 401/312
//                              (6) 197/215 201/232 252/248 397/307;  (7) .. 254/274 397/336;  (8) .. 254/287 397/352
//   1 000 000 x 128, 20        35/42 35/43 43/47 55/51 57/57;   (6) 50/48 51/49 61/53 88/59;  (8) 50/52 50/55 62/57
//   300 000 x 40, one era      19/35 23/35 25/22 29/29 34/29 29/31;  (3) .. 27/38 29/29 31/31;  (8) .. 27/37 27/29 28/33
//   100 000 x 30, one era      17/19 20/20 22/20 20/18;  (2) 15/21 16/25;  (7) 16/32 18/18 18/18
//   30 000 x 100, three eras   16/11 16/10 18/12;   10 000 x 20  12/11 14/10
// So: by rows x features for the fixed 15 us of it, more of them with more nodes or bins; above four nodes one block of
// features or very many rows; and at 32 and 64 nodes the bins where the atomics meet least often.
inline bool mma_pays(bool fused, int n_nodes, int n_feat, int max_bins, int64_t rows, int64_t n_eras) {
    const int features = mma_features(n_nodes, n_feat, max_bins);
    const int64_t blocks = (n_feat + features - 1) / features, work = rows * n_feat;
    if (fused) {
        if (max_bins > 5 || n_nodes > (n_feat > 128 ? 4 : 2) || n_feat <= 64) return false;
        if (n_eras * blocks < (n_feat > 128 ? 444 : 100)) return false;
        return max_bins < 5 || rows >= (n_nodes <= 2 ? 1500 : 2500) * n_eras;
    }
    if (rows < 100000) return false;
    if (n_nodes <= 2) return work >= (max_bins <= 5 ? 3000000 : 10000000);
    const bool one_block = n_feat <= 64;                     // (at two thresholds a lane, up to five bins)
    if (n_nodes <= 4) return work >= 12000000 && (max_bins <= 5 || one_block || (max_bins >= 7 && work >= 200000000));
    if (n_nodes <= 8) return work >= (one_block ? 12000000 : 200000000) && (one_block || max_bins <= 5);
    if (n_nodes <= 16) return work >= (one_block ? 40000000 : 200000000) && (one_block || max_bins <= 5);
    return (max_bins == 4 || max_bins == 5) && work >= 50000000 && n_feat * 100 >= blocks * features * 85 && (n_nodes <= 32 || one_block);
}

}  // namespace pb
