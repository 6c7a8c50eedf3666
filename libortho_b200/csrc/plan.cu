// Plan: one-time GPU-side re-layout of a layer's sparse ortho component, and the two probe
// kernels that let a test prove the integer/index handling bit-exact.
//
// The reference kernels read CSR as three separate streams per row (row_ptr, then col_indices
// and float values; src/dual_gemm.cu:106-130).  The re-layout keeps the CSR row-major order
// (tools/sieve.py:131-136) but fuses column and value into one 32-bit word per entry
// ({f16 value bits | 16-bit column}; an entry outside [0, K) becomes an explicit zero) and keeps its own
// copy of the row pointers, so that every kernel reads one word per entry instead of two.
#include <new>
#include <vector>

#include "common.cuh"
#include "windows.cuh"

namespace ob {

// one warp per output row: pack the row's entries, track the longest row, the largest magnitude of every row
// (NaN counts as infinite) and whether every row lists its columns in strictly ascending order inside [0, K)
// (info[0] = longest row, info[1] != 0: some row does not)
__global__ void relayout_rows_kernel(const int32_t *__restrict__ row_ptr, const int32_t *__restrict__ col,
                                     const __half *__restrict__ val, int N, int K,
                                     uint32_t *__restrict__ entries, int32_t *__restrict__ row_ptr_copy,
                                     float *__restrict__ row_max, int *__restrict__ info)
{
    const int warps_per_block = blockDim.x >> 5;
    const int lane = threadIdx.x & 31;
    for (int n = blockIdx.x * warps_per_block + (threadIdx.x >> 5); n <= N; n += gridDim.x * warps_per_block) {
        const int e0 = row_ptr[n];
        if (lane == 0) row_ptr_copy[n] = e0;
        if (n == N) continue;
        const int e1 = row_ptr[n + 1];
        float vmax = 0.f;
        bool unordered = false;
        for (int e = e0 + lane; e < e1; e += 32) {
            int c = col[e];
            unsigned short vb = __half_as_ushort(val[e]);
            if (e > e0 && col[e - 1] >= c) unordered = true;
            // an entry outside [0,K) is skipped by the reference (src/ortho.c:394); store it as an
            // explicit zero so that it contributes nothing
            if ((unsigned)c >= (unsigned)K) { c = 0; vb = 0; unordered = true; }
            const float av = fabsf(__half2float(__ushort_as_half(vb)));
            vmax = (av != av) ? __int_as_float(0x7f800000) : fmaxf(vmax, av);
            entries[e] = ((uint32_t)vb << 16) | (uint32_t)c;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) vmax = fmaxf(vmax, __shfl_xor_sync(0xffffffffu, vmax, o));
        unordered = __any_sync(0xffffffffu, unordered);
        if (lane == 0) {
            row_max[n] = vmax;
            atomicMax(&info[0], e1 - e0);
            if (unordered) atomicExch(&info[1], 1);
        }
    }
}

// Window lists (windows.cuh).  One CTA per group of 32 rows, lane = row: every warp walks an eighth of the k blocks with a
// cursor per row, once to size the windows and, after a scan over the sizes, once to write the entries, round by round.  The
// group's entries start at the index of its first CSR entry.
// Rows of more than `heavy` entries (0: no limit) are left out; a plan found unordered (info[1]) gets no lists.
__global__ void __launch_bounds__(256)
window_lists_kernel(const uint32_t *__restrict__ entries, const int32_t *__restrict__ row_ptr, int N, int kblocks, int heavy,
                    const int *__restrict__ info, uint32_t *__restrict__ off, uint32_t *__restrict__ words)
{
    __shared__ uint32_t size[65536 / kWinK + 1];
    if (info[1] != 0) return;
    const int g = (int)blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n = g * kWinRows + lane;
    int e0 = 0, e1 = 0;
    if (n < N) { e0 = row_ptr[n]; e1 = row_ptr[n + 1]; }
    if (heavy > 0 && e1 - e0 > heavy) e1 = e0;
    const int kb0 = kblocks * warp / 8, kb1 = kblocks * (warp + 1) / 8;
    int start = e0;                                      // first entry at or past this warp's first column
    for (int hi = e1; start < hi;) {
        const int mid = (start + hi) >> 1;
        if ((int)(entries[mid] & 0xFFFFu) < kb0 * kWinK) start = mid + 1; else hi = mid;
    }
    for (int kb = kb0, e = start; kb < kb1; kb++) {
        int c = 0;
        while (e < e1 && (int)(entries[e] & 0xFFFFu) < (kb + 1) * kWinK) { e++; c++; }
        __syncwarp();
        const int sum = __reduce_add_sync(0xffffffffu, c);
        if (lane == 0) size[kb] = (uint32_t)sum;
    }
    __syncthreads();
    if (warp == 0) {                                     // exclusive scan, 32 at a time
        uint32_t run = (uint32_t)row_ptr[g * kWinRows];
        for (int b = 0; b < kblocks; b += 32) {
            const uint32_t v = b + lane < kblocks ? size[b + lane] : 0u;
            uint32_t s = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t t = __shfl_up_sync(0xffffffffu, s, o);
                if (lane >= o) s += t;
            }
            if (b + lane < kblocks) size[b + lane] = run + s - v;
            run += __shfl_sync(0xffffffffu, s, 31);
        }
        if (lane == 0) size[kblocks] = run;
    }
    __syncthreads();
    for (int kb = threadIdx.x; kb <= kblocks; kb += 256) off[(size_t)g * (size_t)(kblocks + 1) + kb] = size[kb];
    for (int kb = kb0, e = start; kb < kb1; kb++) {
        uint32_t at = size[kb];
        for (;;) {
            uint32_t pk = 0;
            bool has = e < e1;
            if (has) { pk = entries[e]; has = (int)(pk & 0xFFFFu) < (kb + 1) * kWinK; }
            const uint32_t mask = __ballot_sync(0xffffffffu, has);
            if (mask == 0u) break;
            if (has) { words[at + __popc(mask & ((1u << lane) - 1u))] = window_entry(pk, lane); e++; }
            at += __popc(mask);
        }
    }
}

// one warp per output row: the row of an entry is recovered from the plan's own row pointers
__global__ void plan_decode_dump_kernel(const uint32_t *__restrict__ entries, const int32_t *__restrict__ row_ptr,
                                        int N, int32_t *__restrict__ rows, int32_t *__restrict__ cols,
                                        __half *__restrict__ vals)
{
    const int warps_per_block = blockDim.x >> 5;
    const int lane = threadIdx.x & 31;
    for (int n = blockIdx.x * warps_per_block + (threadIdx.x >> 5); n < N; n += gridDim.x * warps_per_block) {
        const int e0 = row_ptr[n], e1 = row_ptr[n + 1];
        for (int e = e0 + lane; e < e1; e += 32) {
            const uint32_t pk = entries[e];
            rows[e] = n;
            cols[e] = (int32_t)(pk & 0xFFFFu);
            vals[e] = __ushort_as_half((unsigned short)(pk >> 16));
        }
    }
}

// every thread unpacks one 32-bit word (8 elements) with the forward kernels' own converters:
// elements 0..7 come back from the pair-order converter, and the natural-order converter of the tensor-core
// kernels must agree with it, otherwise a poison value is written.
__global__ void dequant_dump_kernel(const uint32_t *__restrict__ w32, const __half *__restrict__ scales,
                                    int64_t N, int64_t K, int8_t *__restrict__ w_int, float *__restrict__ w_deq)
{
    const int64_t words_per_row = K >> 3;
    const int64_t total = N * words_per_row;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t n = i / words_per_row;
        const uint32_t w = w32[i];
        uint32_t hp[4], hn[4];
        int4x8_to_half2x4(w, hp);
        int4x8_to_half2x4_natural(w, hn);
        float e[8];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const __half2 pr = *reinterpret_cast<const __half2 *>(&hp[q]);
            e[q] = __low2float(pr);        // pair q = (e_q, e_{q+4})
            e[q + 4] = __high2float(pr);
        }
        bool agree = true;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const __half2 pr = *reinterpret_cast<const __half2 *>(&hn[q]);
            agree = agree && (__low2float(pr) == e[2 * q]) && (__high2float(pr) == e[2 * q + 1]);
        }
        const float s = __half2float(scales[n]);
#pragma unroll
        for (int q = 0; q < 8; q++) {
            const float v = agree ? e[q] : 127.f;
            if (w_int) w_int[i * 8 + q] = (int8_t)v;
            if (w_deq) w_deq[i * 8 + q] = __fmul_rn(v, s);
        }
    }
}

}  // namespace ob

using namespace ob;

extern "C" int ortho_b200_plan_create(ortho_b200_plan **plan_out, const int32_t *row_ptr,
                                      const int32_t *col_indices, const void *values_f16, int64_t nnz,
                                      int64_t in_features, int64_t out_features, void *stream)
{
    if (!plan_out) return ORTHO_B200_ERR_NULL;
    *plan_out = nullptr;
    const int64_t K = in_features, N = out_features;
    if (K <= 0 || N <= 0 || nnz < 0 || K > 65536 || (K % 32) != 0 || nnz > 0x7fffffffLL || N > 0x7fffff00LL)
        return ORTHO_B200_ERR_SHAPE;
    if (nnz > 0 && (!row_ptr || !col_indices || !values_f16)) return ORTHO_B200_ERR_NULL;
    Plan *pl = new (std::nothrow) Plan();
    if (!pl) return ORTHO_B200_ERR_ALLOC;
    pl->magic = kPlanMagic; pl->K = K; pl->N = N; pl->nnz = nnz; pl->max_row_nnz = 0;
    pl->row_ptr = nullptr; pl->entries = nullptr; pl->row_max = nullptr; pl->ordered = false;
    pl->heavy = kLongRowMin; pl->n_long = 0; pl->n_pad = 0;
    pl->hrow = nullptr; pl->hdense = nullptr;
    pl->win_off = pl->win_words = nullptr;
    pl->rows_block = pl->lists_block = nullptr;
    cudaStream_t st = (cudaStream_t)stream;
    cudaError_t e = cudaGetDevice(&pl->device);
    if (e == cudaSuccess && nnz > 0) {
        // the stream is synchronised below, and memory from the pool would become a node of the graph
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
        e = cudaStreamIsCapturing(st, &cap);
        if (e == cudaSuccess && cap != cudaStreamCaptureStatusNone) e = cudaErrorStreamCaptureUnsupported;
    }
    if (e != cudaSuccess) { note_cuda_error(e); delete pl; return ORTHO_B200_ERR_CUDA; }
    if (nnz > 0) {
        // Device memory: {entries, row pointers, row maxima, two result words} and {list offsets, list entries}, from the device's
        // memory pool.  cudaMalloc maps memory 2 MB at a time for pieces of up to 1 MB, some 300 us each, and with the lists nearly
        // every plan paid for one: a plan of 4096->4096 with 1 % took 376 us (median of 12) and takes 50, 8192->57344 with 0.3 %
        // 464 and 119.  (The pool's first use in a process costs some 6 ms.)
        const int kblocks = (int)ceil_div(K, kWinK);
        const int64_t groups = ceil_div(N, kWinRows);
        const size_t noff = (size_t)groups * (size_t)(kblocks + 1);
        e = cudaMallocAsync(&pl->rows_block, sizeof(uint32_t) * ((size_t)nnz + 2 * (size_t)N + 3), st);
        if (e == cudaSuccess) e = cudaMallocAsync(&pl->lists_block, sizeof(uint32_t) * (noff + (size_t)nnz), st);
        int *d_info = nullptr;
        if (e == cudaSuccess) {
            pl->entries = reinterpret_cast<uint32_t *>(pl->rows_block);
            pl->row_ptr = reinterpret_cast<int32_t *>(pl->entries + nnz);
            pl->row_max = reinterpret_cast<float *>(pl->row_ptr + N + 1);
            d_info = reinterpret_cast<int *>(pl->row_max + N);
            pl->win_off = reinterpret_cast<uint32_t *>(pl->lists_block);
            pl->win_words = pl->win_off + noff;
            e = cudaMemsetAsync(d_info, 0, 2 * sizeof(int), st);
        }
        auto build_windows = [&](int heavy) -> cudaError_t {
            window_lists_kernel<<<(unsigned)groups, 256, 0, st>>>(pl->entries, pl->row_ptr, (int)N, kblocks, heavy, d_info,
                                                                  pl->win_off, pl->win_words);
            count_launch();
            return cudaGetLastError();
        };
        if (e == cudaSuccess) {
            const int threads = 256, wpb = threads / 32;
            int64_t blocks = ceil_div(N + 1, wpb);
            if (blocks > 148 * 16) blocks = 148 * 16;
            relayout_rows_kernel<<<(unsigned)blocks, threads, 0, st>>>(
                row_ptr, col_indices, (const __half *)values_f16, (int)N, (int)K, pl->entries, pl->row_ptr, pl->row_max, d_info);
            count_launch();
            e = cudaGetLastError();
        }
        if (e == cudaSuccess) e = build_windows(0);      // again below in the rarer case that there are long rows to leave out
        int h_info[2] = {0, 0};
        if (e == cudaSuccess) e = cudaMemcpyAsync(h_info, d_info, 2 * sizeof(int), cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) {
            note_cuda_error(e);
            ortho_b200_plan_destroy(reinterpret_cast<ortho_b200_plan *>(pl));
            return ORTHO_B200_ERR_CUDA;
        }
        const int h_max = h_info[0];
        pl->max_row_nnz = h_max;
        pl->ordered = h_info[1] == 0;
        const int64_t mean = (nnz + N - 1) / N;
        const int lmin = tuning_snapshot().long_row_min;
        pl->heavy = (int)(4 * mean > lmin ? (4 * mean > 65536 ? 65536 : 4 * mean) : lmin);
        if (h_max > pl->heavy) {
            // list the long rows on the host (one pass over the row pointers); the threshold doubles until their
            // dense copy fits its budget
            std::vector<int32_t> rp((size_t)N + 1), hr;
            e = cudaMemcpy(rp.data(), row_ptr, sizeof(int32_t) * (N + 1), cudaMemcpyDeviceToHost);
            if (e == cudaSuccess) {
                for (;;) {
                    hr.clear();
                    for (int64_t n = 0; n < N; n++)
                        if (rp[n + 1] - rp[n] > pl->heavy) hr.push_back((int32_t)n);
                    const int64_t n_pad = ((int64_t)hr.size() + 127) / 128 * 128;
                    if (n_pad * K * 2 <= kLongDenseMaxBytes || pl->heavy >= 65536) break;
                    pl->heavy *= 2;
                }
                const size_t nl = hr.size();
                if (nl > 0 && (int64_t)((nl + 127) / 128 * 128) * K * 2 <= kLongDenseMaxBytes) {
                    e = cudaMallocAsync(reinterpret_cast<void **>(&pl->hrow), sizeof(int32_t) * nl, st);
                    if (e == cudaSuccess) e = cudaStreamSynchronize(st);      // (the copy below is on another stream)
                    if (e == cudaSuccess) e = cudaMemcpy(pl->hrow, hr.data(), sizeof(int32_t) * nl, cudaMemcpyHostToDevice);
                    if (e == cudaSuccess) {
                        pl->n_long = (int64_t)nl;
                        bool dup = false;
                        e = (cudaError_t)plan_build_long_rows(pl, st, &dup);
                        if (e == cudaSuccess && dup) {         // a repeated column: every row stays with the in-kernel pass
                            cudaFreeAsync(pl->hdense, st); pl->hdense = nullptr;
                            cudaFreeAsync(pl->hrow, st); pl->hrow = nullptr;
                            pl->n_long = 0; pl->n_pad = 0;
                        }
                    }
                }
            }
            if (e != cudaSuccess) {
                note_cuda_error(e);
                ortho_b200_plan_destroy(reinterpret_cast<ortho_b200_plan *>(pl));
                return ORTHO_B200_ERR_CUDA;
            }
        }
        if (!pl->ordered) {
            pl->win_off = pl->win_words = nullptr;
            cudaFreeAsync(pl->lists_block, st);
            pl->lists_block = nullptr;
        }
        if (pl->ordered && pl->n_long > 0) {
            e = build_windows(pl->heavy);
            if (e == cudaSuccess) e = cudaStreamSynchronize(st);
            if (e != cudaSuccess) {
                note_cuda_error(e);
                ortho_b200_plan_destroy(reinterpret_cast<ortho_b200_plan *>(pl));
                return ORTHO_B200_ERR_CUDA;
            }
        }
    }
    *plan_out = reinterpret_cast<ortho_b200_plan *>(pl);
    return ORTHO_B200_OK;
}

extern "C" int ortho_b200_plan_destroy(ortho_b200_plan *plan)
{
    Plan *pl = reinterpret_cast<Plan *>(plan);
    if (!pl) return ORTHO_B200_OK;
    if (pl->magic != kPlanMagic) return ORTHO_B200_ERR_PLAN;
    void *const blocks[] = {pl->rows_block, pl->lists_block, pl->hrow, pl->hdense};
    if (pl->nnz > 0) {
        // cudaFree of pool memory does not wait for kernels that may still read it, as it does for cudaMalloc's
        int dev = pl->device;
        cudaGetDevice(&dev);
        if (dev != pl->device) cudaSetDevice(pl->device);
        if (cudaDeviceSynchronize() == cudaSuccess) {    // (refused while a stream is captured: the blocks then stay allocated)
            for (void *b : blocks)
                if (b) cudaFree(b);
        }
        if (dev != pl->device) cudaSetDevice(dev);
    }
    pl->magic = 0;
    delete pl;
    return ORTHO_B200_OK;
}

extern "C" int64_t ortho_b200_plan_nnz(const ortho_b200_plan *plan)
{
    const Plan *pl = reinterpret_cast<const Plan *>(plan);
    return (pl && pl->magic == kPlanMagic) ? pl->nnz : -1;
}

extern "C" int64_t ortho_b200_plan_max_row_nnz(const ortho_b200_plan *plan)
{
    const Plan *pl = reinterpret_cast<const Plan *>(plan);
    return (pl && pl->magic == kPlanMagic) ? pl->max_row_nnz : -1;
}

extern "C" int ortho_b200_plan_rows_ordered(const ortho_b200_plan *plan)
{
    const Plan *pl = reinterpret_cast<const Plan *>(plan);
    if (!pl || pl->magic != kPlanMagic) return -1;
    return (pl->nnz == 0 || pl->ordered) ? 1 : 0;
}

extern "C" int64_t ortho_b200_plan_workspace_bytes(const ortho_b200_plan *plan, int64_t M)
{
    const Plan *pl = reinterpret_cast<const Plan *>(plan);
    if (!pl || pl->magic != kPlanMagic) return -1;
    const int64_t plain = ortho_b200_workspace_bytes(M, pl->K, pl->N);      // base-only calls too: partial sums of cut tiles
    if (pl->nnz == 0) return plain;
    // the tensor-core kernels take the sums of the plan's long rows from a pre-pass
    return plain + (decode_regime(M, pl->N, pl->K) && !mid_range(M, pl->N, pl->K) ? 0 : long_rows_workspace_bytes(pl, M));
}

extern "C" int ortho_b200_plan_decode_dump(const ortho_b200_plan *plan, int32_t *rows_out, int32_t *cols_out,
                                           void *values_f16_out, void *stream)
{
    const Plan *pl = reinterpret_cast<const Plan *>(plan);
    if (!pl || pl->magic != kPlanMagic) return ORTHO_B200_ERR_PLAN;
    if (pl->nnz == 0) return ORTHO_B200_OK;
    if (!rows_out || !cols_out || !values_f16_out) return ORTHO_B200_ERR_NULL;
    int64_t blocks = ceil_div(pl->N, 8);
    if (blocks > 148 * 16) blocks = 148 * 16;
    plan_decode_dump_kernel<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(
        pl->entries, pl->row_ptr, (int)pl->N, rows_out, cols_out, (__half *)values_f16_out);
    count_launch();
    OB_CUDA(cudaGetLastError());
    return ORTHO_B200_OK;
}

extern "C" int ortho_b200_dequant_dump(const void *q_weight, const void *q_scales_f16, int64_t out_features,
                                       int64_t in_features, int8_t *w_int_out, float *w_deq_out, void *stream)
{
    if (!q_weight || !q_scales_f16) return ORTHO_B200_ERR_NULL;
    if (out_features <= 0 || in_features <= 0 || (in_features % 8) != 0) return ORTHO_B200_ERR_SHAPE;
    if (((uintptr_t)q_weight & 3u) != 0) return ORTHO_B200_ERR_ALIGN;
    if (!w_int_out && !w_deq_out) return ORTHO_B200_OK;
    const int64_t total = out_features * (in_features / 8);
    int64_t blocks = ceil_div(total, 256);
    if (blocks > 148 * 16) blocks = 148 * 16;
    dequant_dump_kernel<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(
        (const uint32_t *)q_weight, (const __half *)q_scales_f16, out_features, in_features, w_int_out, w_deq_out);
    count_launch();
    OB_CUDA(cudaGetLastError());
    return ORTHO_B200_OK;
}
