// Window lists: the plan's second layout of the sparse entries, made for the tensor-core kernels.
//
// A window is 32 consecutive rows x 64 consecutive k: one warp's share (lane = row) of a 64-k block of a weight tile.
// Its entries lie together, so that a warp takes 32 of them with one coalesced load; two neighbouring windows (128 k) of a
// row group are neighbours in the list too.  An entry is {f16 value | place}, the place being the byte offset of
// (row, k) in a 128-byte swizzled FP16 tile of 32 rows x 64 k, plus kWinTile for the odd windows: a warp that scatters
// entries adds the low half of the word to its tile's address.  Inside a window the entries are ordered by round, then
// row: round r holds the r-th entry of every row that has more than r.
// win_off[group * (kblocks + 1) + kb] is the first entry of a window and the next element its end.
// Long rows are not listed.
#pragma once

#include "common.cuh"

namespace ob {

constexpr int kWinRows = 32, kWinK = 64;
constexpr uint32_t kWinTile = 128 * 128;        // bytes between the tiles of two neighbouring k blocks (128 rows each)
__host__ __device__ __forceinline__ uint32_t window_entry(uint32_t packed, int row) {      // packed: {f16 | column}
    const uint32_t k = packed & 127u, r = (uint32_t)(row & (kWinRows - 1));
    return (packed & 0xFFFF0000u) | ((k >> 6) * kWinTile + r * 128u + ((((k >> 3) & 7u) ^ (r & 7u)) << 4) + (k & 7u) * 2u);
}

}  // namespace ob
