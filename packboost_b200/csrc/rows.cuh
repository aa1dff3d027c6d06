// Row ranges of tiles, for host and device.  Tables have up to 2^31 - 513 rows: the rows themselves fit 32 bits,
// "rows + tile - 1" and "first row of the tile after the last" do not.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define PB_ROWS_FN __host__ __device__ __forceinline__
#else
#define PB_ROWS_FN inline
#endif

namespace pb {

// Tiles of `tile` rows that `rows` rows make.
PB_ROWS_FN int tiles_of(int64_t rows, int64_t tile) { return (int)((rows + tile - 1) / tile); }

// Rows [r0, r1) of the index-th tile of an era; a tile past the end of the era is empty and starts there.
PB_ROWS_FN void tile_range(int era_begin, int era_end, int index, int tile, int& r0, int& r1) {
    const int64_t at = (int64_t)era_begin + (int64_t)index * tile;
    r0 = at < era_end ? (int)at : era_end;
    r1 = era_end - r0 > tile ? r0 + tile : era_end;
}

// Shares of the rows of all feature blocks, the block the slowest.
struct Shares {
    int64_t block_work, share;           // work of a block, of a share (rounded down)
    int blocks, more;                    // (blocks;) shares with one more, of a block's where it has its own
    int per_block;                       // shares of a block, 0: a share may begin in one block and end in another
    int count;
};

// At most `count` shares.  `own`: none of two blocks, where that leaves four of `count` out at most.
inline Shares shares_of(int blocks, int64_t block_work, int count, bool own) {
    Shares s;
    s.block_work = block_work;
    s.blocks = blocks;
    s.per_block = own && count / blocks * blocks + 4 >= count ? count / blocks : 0;
    s.count = s.per_block ? s.per_block * blocks : count;
    const int64_t work = block_work * (s.per_block ? 1 : blocks);
    const int parts = s.per_block ? s.per_block : count;
    s.share = work / parts;
    s.more = (int)(work % parts);
    return s;
}

// Where share i begins: the feature block, and the work of it that lies before.  (A few subtractions: a 64-bit
// division by every warp is 2 us a launch.)
PB_ROWS_FN int64_t share_begin(const Shares& s, int i, int& fb) {
    fb = s.per_block ? i / s.per_block : 0;
    i -= fb * s.per_block;
    int64_t at = s.share * i + (i < s.more ? i : s.more);
    if (!s.per_block)
        for (; at >= s.block_work; at -= s.block_work) ++fb;
    return at;
}

// Where a share of the work of a feature block ends.  `at` counts rows (WHOLE: and era_rows more for each era, which
// stand for its flush).  WHOLE: between two eras, at the nearest place, so that a share differs from its part of the
// work by half an era at each end at most; otherwise at any multiple of kCutRows.  True for exactly one e of
// [0, n_eras], the era in which the rows after the cut begin, at `row`; n_eras: none is left (WHOLE alone).
constexpr int kCutRows = 512;
template <bool WHOLE>
PB_ROWS_FN bool cut_in_era(const int* offsets, int n_eras, int64_t at, int era_rows, int e, int& row) {
    row = WHOLE ? offsets[e] : (int)(at / kCutRows * kCutRows);
    if (!WHOLE) return e < n_eras && offsets[e] <= row && row < offsets[e + 1];
    // twice the work before the middle of an era
    auto middle = [&](int i) { return (int64_t)offsets[i] + offsets[i + 1] + (int64_t)era_rows * (2 * i + 1); };
    return (e == 0 || middle(e - 1) < 2 * at) && (e == n_eras || middle(e) >= 2 * at);
}

// A step through the rows of a share: rows [r0, r1), blocks [b0, b1) of kCutRows rows, of an era, or (not `whole`) of
// as much of it as a tile may have.  Eras without rows are steps where they are whole: their gains have to be written.
struct RowTask {
    int fb, era, r0, r1, b0, b1;
    int next;                            // era of the rows from r1 on
};

// The step after x up to the cut at `end` = {feature block, era, row}; false: none.  x starts as {fb, next, r1} of a cut.
PB_ROWS_FN bool next_row_task(const int* offsets, int n_eras, bool whole, const int* end, int tile, RowTask& x) {
    for (;;) {
        if (x.next == n_eras) {
            ++x.fb;
            x.next = x.r1 = 0;
        }
        const bool last_block = x.fb == end[0];
        if (x.fb > end[0] || (last_block && (x.next > end[1] || (x.next == end[1] && x.r1 >= end[2])))) return false;
        const int era_end = offsets[x.next + 1];
        x.era = x.next;
        x.r0 = x.r1;
        x.r1 = era_end;
        if (!whole) {
            if (era_end - x.r0 > tile) x.r1 = (x.r0 + tile) / kCutRows * kCutRows;
            if (last_block && x.era == end[1] && end[2] < x.r1) x.r1 = end[2];
        }
        if (x.r1 == era_end) ++x.next;
        x.b0 = x.r0 / kCutRows;
        x.b1 = x.r0 < x.r1 ? (x.r1 + kCutRows - 1) / kCutRows : x.b0;
        if (x.r0 < x.r1 || whole) return true;
    }
}

}  // namespace pb
