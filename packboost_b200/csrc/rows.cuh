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

}  // namespace pb
