// Window lists: the plan's second layout of the sparse entries, made for the tensor-core kernels.
//
// A window is 32 consecutive rows x 64 consecutive k: one warp's share (lane = row) of a 64-k block of a weight tile.
// Its entries lie together, {f16 value | row inside the group | k inside 128}, so that a warp takes 32 of them with one
// coalesced load; two neighbouring windows (128 k) of a row group are neighbours in the list too.  Inside a window the
// entries are ordered by round, then row: round r holds the r-th entry of every row that has more than r, and a list
// of 32-bit row masks, one per round, lets each lane find its own entry by a popcount.
// win_off[group * (kblocks + 1) + kb] is the first entry of a window and the next element its end; mask_off likewise.
// Long rows are not listed.
#pragma once

#include "common.cuh"

namespace ob {

constexpr int kWinRows = 32, kWinK = 64;
__host__ __device__ __forceinline__ uint32_t window_entry(uint32_t packed, int row) {      // packed: {f16 | column}
    return (packed & 0xFFFF0000u) | ((uint32_t)(row & (kWinRows - 1)) << 7) | (packed & 127u);
}
__device__ __forceinline__ int window_k(uint32_t e) { return (int)(e & 127u); }
__device__ __forceinline__ int window_row(uint32_t e) { return (int)((e >> 7) & 31u); }

}  // namespace ob
