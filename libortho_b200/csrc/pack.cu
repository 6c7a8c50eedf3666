// Device-side producer of the layout the forward consumes: INT4 quantise + nibble-pack of the base and
// CSR build of the ortho residual.  Follows OrthoLinear.load_from_weights
// (torch_bind/ortho_linear.py:79-128) and pack_ortho_sparse(..., "csr") (tools/sieve.py:119-152) of the
// reference operation by operation, so the results are bit-identical to that torch chain:
//   scale   = max(rowmax|W| / 7, 1e-6)                 (IEEE FP32 division; stored as FP16, round to nearest)
//   w_int   = clamp(round_half_even(W / scale_fp32), -8, 7)
//   byte    = (w_int[2i] & 15) | (w_int[2i+1] & 15) << 4       (even flat index in the low nibble)
//   CSR     = positions with W_ortho != 0 in row-major order, int32 indices, values rounded to FP16
// All of it is element-wise work bound by HBM: one pass over W (the second read of a row hits L1 or L2) per step.
// 4096->11008 by kernel: pack 49 us (203 MB; 57 with the row read twice from global memory), CSR with 1 % entries: count with marks
// 42, scan 10, fill from the marks 13 (whole rows again: about 40).
#include "common.cuh"
#include "rows.cuh"

namespace ob {

// W != 0 exactly as IEEE compares it (no flush of subnormals; NaN counts as non-zero)
__device__ __forceinline__ bool is_nonzero(float v) { return (__float_as_uint(v) << 1) != 0u; }
__device__ __forceinline__ int quantise_one(float w, float scale, float rscale) {
    const float q = quant_clamped(w, scale, rscale);
    return q != q ? -8 : (int)q;                // NaN -> -8 here; torch leaves NaN undefined after the int8 cast
}

// One CTA per output row.  Bound by HBM (4.5 bytes per weight).  PIPE: rows come through shared memory, the next one while this one
// is packed; longer ones are read twice, the second time from L2.
template <bool PIPE>
__global__ void __launch_bounds__(256)
pack_base_kernel(const float *__restrict__ w, const float *__restrict__ scales_in, int64_t N, int K,
                 uint32_t *__restrict__ packed, __half *__restrict__ scales_out, int *__restrict__ status)
{
    extern __shared__ __align__(16) unsigned char row_smem[];
    __shared__ float wmax[8];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    RowPipe pipe(row_smem, w, PIPE ? (size_t)K * 4 : 0, PIPE ? N : 0);
    for (int64_t n = blockIdx.x; n < N; n += gridDim.x) {
        const float4 *row = PIPE ? pipe.row(status) : reinterpret_cast<const float4 *>(w + (size_t)n * K);
        float scale;
        if (scales_in) {
            scale = scales_in[n];
        } else {
            float m = 0.f;
#pragma unroll 4
            for (int i = tid; i < K / 4; i += 256) {
                const float4 v = row[i];
                m = fmaxf(m, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
            }
#pragma unroll
            for (int o = 16; o >= 1; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
            if (lane == 0) wmax[warp] = m;
            __syncthreads();
            float mm = wmax[0];
#pragma unroll
            for (int i = 1; i < 8; i++) mm = fmaxf(mm, wmax[i]);
            scale = fmaxf(div_ieee(mm, 7.0f), 1e-6f);
        }
        if (tid == 0) scales_out[n] = __float2half_rn(scale);
        const float rscale = quant_rscale(scale);
        uint32_t *out = packed + (size_t)n * (K / 8);
#pragma unroll 2
        for (int i = tid; i < K / 8; i += 256) {          // 8 weights -> one 32-bit word
            const float4 a = row[2 * i], b = row[2 * i + 1];
            const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
            uint32_t word = 0;
#pragma unroll
            for (int e = 0; e < 8; e++) word |= ((uint32_t)quantise_one(v[e], scale, rscale) & 0xFu) << (4 * e);
            out[i] = word;
        }
        __syncthreads();      // wmax is reused by the next row; the row has been read
        if (PIPE) pipe.release();
    }
}

// nnz per row (one warp per row, four 16-byte loads in flight per lane), then an exclusive scan by one CTA.  MARKS: the non-zero
// positions as well, four words per 128 weights: bit l of word e is weight 4 l + e.
template <bool MARKS>
__global__ void __launch_bounds__(256)
csr_count_kernel(const float *__restrict__ w, int64_t N, int K, int32_t *__restrict__ row_ptr, uint4 *__restrict__ marks)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, groups = (K + 127) / 128;
    for (int64_t n = (int64_t)blockIdx.x * 8 + warp; n < N; n += (int64_t)gridDim.x * 8) {
        const float4 *row = reinterpret_cast<const float4 *>(w + (size_t)n * K);
        int c = 0;
        for (int k0 = 0; k0 < K / 4; k0 += 128) {
            float4 v[4];
#pragma unroll
            for (int j = 0; j < 4; j++) v[j] = k0 + 32 * j + lane < K / 4 ? row[k0 + 32 * j + lane] : make_float4(0.f, 0.f, 0.f, 0.f);
            if (MARKS) {
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    uint4 m;
                    m.x = __ballot_sync(0xffffffffu, is_nonzero(v[j].x)); m.y = __ballot_sync(0xffffffffu, is_nonzero(v[j].y));
                    m.z = __ballot_sync(0xffffffffu, is_nonzero(v[j].z)); m.w = __ballot_sync(0xffffffffu, is_nonzero(v[j].w));
                    if (lane == j && k0 / 32 + j < groups) {
                        marks[(size_t)n * groups + k0 / 32 + j] = m;
                        c += __popc(m.x) + __popc(m.y) + __popc(m.z) + __popc(m.w);
                    }
                }
            } else {
#pragma unroll
                for (int j = 0; j < 4; j++)
                    c += (is_nonzero(v[j].x) ? 1 : 0) + (is_nonzero(v[j].y) ? 1 : 0) + (is_nonzero(v[j].z) ? 1 : 0) + (is_nonzero(v[j].w) ? 1 : 0);
            }
        }
        c = __reduce_add_sync(0xffffffffu, c);
        if (lane == 0) row_ptr[n + 1] = c;
    }
}

// The same from the marks: a warp per row, a lane per 128 weights.  Reads the marks and the sectors with entries only.
__global__ void __launch_bounds__(256)
csr_fill_marks_kernel(const float *__restrict__ w, int64_t N, int K, const int32_t *__restrict__ row_ptr, const uint4 *__restrict__ marks,
                      int32_t *__restrict__ col, __half *__restrict__ val)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, groups = (K + 127) / 128;
    for (int64_t n = (int64_t)blockIdx.x * 8 + warp; n < N; n += (int64_t)gridDim.x * 8) {
        int at = row_ptr[n];
        if (row_ptr[n + 1] == at) continue;
        const float *row = w + (size_t)n * K;
        for (int g0 = 0; g0 < groups; g0 += 32) {
            const uint4 m = g0 + lane < groups ? marks[(size_t)n * groups + g0 + lane] : make_uint4(0u, 0u, 0u, 0u);
            const int mine = __popc(m.x) + __popc(m.y) + __popc(m.z) + __popc(m.w);
            int upto = mine;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, upto, o);
                if (lane >= o) upto += t;
            }
            int pos = at + upto - mine;
            at += __shfl_sync(0xffffffffu, upto, 31);
            for (uint32_t any = m.x | m.y | m.z | m.w; any; any &= any - 1u) {
                const uint32_t bit = any & (0u - any);
                const int c0 = (g0 + lane) * 128 + 4 * (__ffs(any) - 1);
                const uint32_t mm[4] = {m.x, m.y, m.z, m.w};
#pragma unroll
                for (int e = 0; e < 4; e++)
                    if (mm[e] & bit) {
                        col[pos] = c0 + e;
                        val[pos] = __float2half_rn(row[c0 + e]);
                        pos++;
                    }
            }
        }
    }
}

// four rows per thread and round
__global__ void __launch_bounds__(1024)
csr_scan_kernel(int64_t N, int32_t *__restrict__ row_ptr, int *__restrict__ overflow)
{
    __shared__ long long warp_sum[32];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) row_ptr[0] = 0;
    long long carry = 0;
    for (int64_t base = 0; base < N; base += 4096) {
        const int64_t i = base + 4 * tid;
        long long v[4];
#pragma unroll
        for (int j = 0; j < 4; j++) v[j] = i + j < N ? row_ptr[i + j + 1] : 0;
        v[1] += v[0]; v[2] += v[1]; v[3] += v[2];
        long long s = v[3];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const long long t = __shfl_up_sync(0xffffffffu, s, o); if (lane >= o) s += t; }
        if (lane == 31) warp_sum[warp] = s;
        __syncthreads();
        long long before = 0, all = 0;
        for (int k = 0; k < 32; k++) { if (k < warp) before += warp_sum[k]; all += warp_sum[k]; }
        before += carry + s - v[3];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            if (i + j < N) {
                if (before + v[j] > 0x7fffffffLL) atomicExch(overflow, 1);
                row_ptr[i + j + 1] = (int32_t)(before + v[j]);
            }
        }
        carry += all;
        __syncthreads();
    }
}

// one warp per row, a lane holds four neighbouring columns: ballots per column of the quad keep the column order
__global__ void __launch_bounds__(256)
csr_fill_kernel(const float *__restrict__ w, int64_t N, int K, const int32_t *__restrict__ row_ptr,
                int32_t *__restrict__ col, __half *__restrict__ val)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    for (int64_t n = (int64_t)blockIdx.x * 8 + warp; n < N; n += (int64_t)gridDim.x * 8) {
        const float4 *row = reinterpret_cast<const float4 *>(w + (size_t)n * K);
        int at = row_ptr[n];
        if (row_ptr[n + 1] == at) continue;
        for (int k0 = 0; k0 < K / 4; k0 += 128) {
            float4 v[4];
#pragma unroll
            for (int j = 0; j < 4; j++) v[j] = k0 + 32 * j + lane < K / 4 ? row[k0 + 32 * j + lane] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float e[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
                unsigned m[4];
#pragma unroll
                for (int i = 0; i < 4; i++) m[i] = __ballot_sync(0xffffffffu, is_nonzero(e[i]));
                if ((m[0] | m[1] | m[2] | m[3]) == 0u) continue;
                int pos = at + __popc(m[0] & below) + __popc(m[1] & below) + __popc(m[2] & below) + __popc(m[3] & below);
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    if (is_nonzero(e[i])) {
                        col[pos] = (k0 + 32 * j + lane) * 4 + i;
                        val[pos] = __float2half_rn(e[i]);
                        pos++;
                    }
                }
                at += __popc(m[0]) + __popc(m[1]) + __popc(m[2]) + __popc(m[3]);
            }
        }
    }
}

int *kernel_status_word();   // api.cu

}  // namespace ob

using namespace ob;

static int check_pack_args(const void *w, int64_t N, int64_t K)
{
    if (!w) return ORTHO_B200_ERR_NULL;
    if (N <= 0 || K <= 0 || (K % 8) != 0 || K > 0x7fffffffLL || N > 0x7fffff00LL) return ORTHO_B200_ERR_SHAPE;
    if (((uintptr_t)w & 15u) != 0) return ORTHO_B200_ERR_ALIGN;
    return ORTHO_B200_OK;
}

extern "C" int ortho_b200_pack_base(const float *w, int64_t N, int64_t K, const float *scales_in,
                                    void *q_weight_out, void *q_scales_f16_out, void *stream)
{
    int st = check_pack_args(w, N, K);
    if (st != ORTHO_B200_OK) return st;
    if (!q_weight_out || !q_scales_f16_out) return ORTHO_B200_ERR_NULL;
    if (((uintptr_t)q_weight_out & 3u) != 0 || ((uintptr_t)q_scales_f16_out & 1u) != 0) return ORTHO_B200_ERR_ALIGN;
    int *status = ob::kernel_status_word();
    const int dev = current_device_index();
    if (!status || dev < 0) return ORTHO_B200_ERR_CUDA;
    const int64_t sms = device_sm_count(dev);
    if (K * 4 <= kRowBytesMax) {
        static bool attr_set[kMaxDevices] = {};
        if (!attr_set[dev]) {
            OB_CUDA(cudaFuncSetAttribute(pack_base_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)row_smem_bytes(kRowBytesMax)));
            attr_set[dev] = true;
        }
        const int64_t grid = sms * row_ctas_per_sm(K * 4, 64);
        pack_base_kernel<true><<<(unsigned)(grid < N ? grid : N), 256, row_smem_bytes((size_t)K * 4), (cudaStream_t)stream>>>(
            w, scales_in, N, (int)K, (uint32_t *)q_weight_out, (__half *)q_scales_f16_out, status);
    } else {
        pack_base_kernel<false><<<(unsigned)(sms * 8 < N ? sms * 8 : N), 256, kRowBufs * sizeof(uint64_t), (cudaStream_t)stream>>>(
            w, scales_in, N, (int)K, (uint32_t *)q_weight_out, (__half *)q_scales_f16_out, status);
    }
    OB_CUDA(cudaGetLastError());
    count_launch();
    return ORTHO_B200_OK;
}

static int csr_count(const float *w_ortho, int64_t N, int64_t K, int32_t *row_ptr_out, void *marks, void *stream)
{
    int st = check_pack_args(w_ortho, N, K);
    if (st != ORTHO_B200_OK) return st;
    if (!row_ptr_out) return ORTHO_B200_ERR_NULL;
    int *status = ob::kernel_status_word();
    if (!status) return ORTHO_B200_ERR_CUDA;
    const int64_t blocks = ceil_div(N, 8);
    const unsigned grid = (unsigned)(blocks < 148 * 16 ? blocks : 148 * 16);
    if (marks) csr_count_kernel<true><<<grid, 256, 0, (cudaStream_t)stream>>>(w_ortho, N, (int)K, row_ptr_out, (uint4 *)marks);
    else csr_count_kernel<false><<<grid, 256, 0, (cudaStream_t)stream>>>(w_ortho, N, (int)K, row_ptr_out, nullptr);
    OB_CUDA(cudaGetLastError());
    csr_scan_kernel<<<1, 1024, 0, (cudaStream_t)stream>>>(N, row_ptr_out, status);
    OB_CUDA(cudaGetLastError());
    count_launch(2);
    return ORTHO_B200_OK;
}

extern "C" int ortho_b200_csr_count(const float *w_ortho, int64_t N, int64_t K, int32_t *row_ptr_out, void *stream)
{
    return csr_count(w_ortho, N, K, row_ptr_out, nullptr, stream);
}

extern "C" int64_t ortho_b200_csr_marks_bytes(int64_t N, int64_t K) { return N > 0 && K > 0 ? N * ceil_div(K, 128) * 16 : -1; }

extern "C" int ortho_b200_csr_count_marks(const float *w_ortho, int64_t N, int64_t K, int32_t *row_ptr_out, void *marks, void *stream)
{
    const int st = check_pack_args(w_ortho, N, K);
    if (st != ORTHO_B200_OK) return st;
    if (!marks) return ORTHO_B200_ERR_NULL;
    if (((uintptr_t)marks & 15u) != 0) return ORTHO_B200_ERR_ALIGN;
    return csr_count(w_ortho, N, K, row_ptr_out, marks, stream);
}

extern "C" int ortho_b200_csr_fill_marks(const float *w_ortho, int64_t N, int64_t K, const int32_t *row_ptr, const void *marks,
                                         int32_t *col_out, void *val_f16_out, void *stream)
{
    int st = check_pack_args(w_ortho, N, K);
    if (st != ORTHO_B200_OK) return st;
    if (!row_ptr || !marks) return ORTHO_B200_ERR_NULL;
    if (((uintptr_t)marks & 15u) != 0) return ORTHO_B200_ERR_ALIGN;
    const int64_t blocks = ceil_div(N, 8);
    csr_fill_marks_kernel<<<(unsigned)(blocks < 148 * 16 ? blocks : 148 * 16), 256, 0, (cudaStream_t)stream>>>(
        w_ortho, N, (int)K, row_ptr, (const uint4 *)marks, col_out, (__half *)val_f16_out);
    OB_CUDA(cudaGetLastError());
    count_launch();
    return ORTHO_B200_OK;
}

extern "C" int ortho_b200_csr_fill(const float *w_ortho, int64_t N, int64_t K, const int32_t *row_ptr,
                                   int32_t *col_out, void *val_f16_out, void *stream)
{
    int st = check_pack_args(w_ortho, N, K);
    if (st != ORTHO_B200_OK) return st;
    if (!row_ptr) return ORTHO_B200_ERR_NULL;
    const int64_t blocks = ceil_div(N, 8);
    csr_fill_kernel<<<(unsigned)(blocks < 148 * 16 ? blocks : 148 * 16), 256, 0, (cudaStream_t)stream>>>(
        w_ortho, N, (int)K, row_ptr, col_out, (__half *)val_f16_out);
    OB_CUDA(cudaGetLastError());
    count_launch();
    return ORTHO_B200_OK;
}
