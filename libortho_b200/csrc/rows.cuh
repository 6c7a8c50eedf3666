// Rows of a matrix through shared memory: a CTA of 256 threads walks the rows n, n + grid, ...; while it works on one, the next is
// on its way by an untiled bulk copy, so that HBM is never waited for from the registers.  For element-wise kernels that need a
// whole row before its first output (the packer's and the sieve's row scales).
#pragma once

#include "common.cuh"
#include "tma.cuh"

namespace ob {

constexpr int kRowBufs = 2;
constexpr int kRowBytesMax = 32768;              // longer rows are read from global memory
constexpr size_t row_smem_bytes(size_t row_bytes) { return row_bytes * kRowBufs + kRowBufs * sizeof(uint64_t); }
// CTAs per SM that shared memory (227 KB, 1 KB of it per CTA taken by the system, `fixed` bytes static) has room for, at most 8
static inline int row_ctas_per_sm(int64_t row_bytes, int fixed)
{
    const int64_t n = (227 * 1024) / ((int64_t)row_smem_bytes((size_t)row_bytes) + 1024 + fixed);
    return n < 1 ? 1 : n > 8 ? 8 : (int)n;
}

struct RowPipe {
    unsigned char *buf;
    uint64_t *bar;
    const unsigned char *src;
    size_t bytes;
    int64_t next, N, step;                       // next row to fetch (thread 0)
    int at;
    uint32_t phase;
    bool ok;

    __device__ __forceinline__ void fetch(int b)
    {
        if (next >= N) return;
        mbar_arrive_expect_tx(&bar[b], (uint32_t)bytes);
        bulk_load_1d(buf + (size_t)b * bytes, src + (size_t)next * bytes, (uint32_t)bytes, &bar[b]);
        next += step;
    }
    // row_bytes: a multiple of 16, at most kRowBytesMax; smem: row_smem_bytes(row_bytes), 16-byte aligned
    __device__ __forceinline__ RowPipe(unsigned char *smem, const void *matrix, size_t row_bytes, int64_t rows)
        : buf(smem), bar(reinterpret_cast<uint64_t *>(smem + row_bytes * kRowBufs)), src((const unsigned char *)matrix), bytes(row_bytes),
          next(blockIdx.x), N(rows), step(gridDim.x), at(0), phase(0), ok(true)
    {
        if (threadIdx.x == 0) {
            for (int b = 0; b < kRowBufs; b++) mbar_init(&bar[b], 1);
            fence_mbar_init();
            for (int b = 0; b < kRowBufs; b++) fetch(b);
        }
        __syncthreads();
    }
    // the current row, complete; the wait is bounded (a copy that never completes sets the status word)
    __device__ __forceinline__ const float4 *row(int *status)
    {
        if (ok && !mbar_wait(&bar[at], phase, 1u << 22)) { ok = false; atomicExch(status, 1); }
        return reinterpret_cast<const float4 *>(buf + (size_t)at * bytes);
    }
    // every thread is done with the row (the caller's barrier): its buffer takes the next one
    __device__ __forceinline__ void release()
    {
        if (threadIdx.x == 0) fetch(at);
        if (++at == kRowBufs) { at = 0; phase ^= 1u; }
    }
};

}  // namespace ob
