// Device-side Hessian sieve: the split of a full-precision weight matrix into the INT4-representable base
// and the sparse residual that the packer (pack.cu) then turns into the operator's buffers.
//
// Follows hessian_sieve / quantize_int4 of the reference (tools/sieve.py:13-23, 25-76) operation by
// operation in IEEE FP32, so that the two outputs are bit-identical to that torch chain:
//   scale[n]  = max(rowmax|W|, 1e-8) / 7
//   base      = clamp(round_half_even(W / scale), -8, 7) * scale        (non-finite -> 0)
//   residual  = W - base
//   score     = residual^2 / (diag(H_inv) + 1e-6)
//   ortho     = residual * (score > threshold)
// The threshold is a given constant (curvature threshold) or the k-th largest score ("keep the top
// fraction", tools/sieve.py:61-66), found by a radix select over the scores' order-preserving keys: the first pass over W
// takes the row scales and counts the keys' top 12 bits; the second counts the next 10 bits of the keys in the
// selected bin and lists those keys (in an output buffer, which is written later); the last 10 bits are
// counted from that short list.  The last CTA of each pass selects the bin.  An output may be W itself (an element is read
// before it is written): the list then goes to the other output, and without either the last 10 bits take a pass over W too.
// Everything is element-wise work; with the IEEE divisions (two of some 15 instructions per weight and pass) spelled out
// each pass was bound by instructions, so they are only done where an approximate quotient cannot decide:
// near a rounding tie (quant_clamped), near the edge of a bin or near the threshold.
// 4096->11008, keep the top 1 %: 344 us for the call (rows 115, bin 126, list 8, split 94); six passes with the divisions
// spelled out took about 700.
#include <cstring>

#include "common.cuh"

namespace ob {

__device__ __forceinline__ bool sv_finite(float v) { return (__float_as_uint(v) & 0x7f800000u) != 0x7f800000u; }

// base value and residual of one weight; returns residual^2
__device__ __forceinline__ float sieve_one(float w, float scale, float rscale, float &base, float &res)
{
    const float q = quant_clamped(w, scale, rscale);
    base = __fmul_rn(q, scale);
    if (q != q || !sv_finite(base)) base = 0.f;
    res = __fsub_rn(w, base);
    return __fmul_rn(res, res);
}
// The score is r2 / hs in IEEE arithmetic.  r2 * rcp(hs) is within 2^-21 of it relatively while everything is in the normal
// range with room: the callers use it only then.
__device__ __forceinline__ bool approx_ok(float r2, float hs) { return r2 >= 1e-30f && r2 <= 1e30f && hs >= 1e-30f && hs <= 1e4f; }
// order-preserving map of a float to an unsigned key (larger float <-> larger key)
__device__ __forceinline__ uint32_t score_key(float s)
{
    const uint32_t b = __float_as_uint(s);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float key_score(uint32_t k)
{
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

constexpr int kBins0 = 4096, kBins = 1024;       // 12 + 10 + 10 bits
// radix-select state in device memory, cleared before the first pass
struct SelectState {
    unsigned int hist0[kBins0], hist1[kBins], hist2[kBins];
    unsigned int done[3];                        // CTAs of a pass that have added their counts
    unsigned int prefix[3];                      // selected bin of each pass
    unsigned int listed;                         // keys in the list
    unsigned long long krem[3];                  // rank inside the selected bin
    float threshold;
};

// Adds the CTA's counts h[BINS] to the global ones; the last CTA then finds the bin that holds the k-th largest key
// (k counted from the top bin downwards).  Called by all 256 threads.
template <int BINS>
__device__ __forceinline__ void add_and_select(const unsigned int *h, unsigned int *hist, SelectState *st, int pass, unsigned long long k)
{
    __shared__ unsigned int is_last;
    __shared__ unsigned long long warp_sum[8];
    __syncthreads();
    for (int i = threadIdx.x; i < BINS; i += 256)
        if (h[i]) atomicAdd(&hist[i], h[i]);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) is_last = atomicAdd(&st->done[pass], 1u) == gridDim.x * gridDim.y - 1 ? 1u : 0u;
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    // thread t owns bins [t * PER, (t + 1) * PER); keys in the bins above its own: a suffix sum over the threads
    constexpr int PER = BINS / 256;
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    unsigned long long mine = 0;
    for (int i = 0; i < PER; i++) mine += __ldcg(&hist[t * PER + i]);
    unsigned long long suf = mine;               // inclusive over lanes >= lane
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long u = __shfl_down_sync(0xffffffffu, suf, o);
        if (lane + o < 32) suf += u;
    }
    if (lane == 0) warp_sum[warp] = suf;
    __syncthreads();
    unsigned long long above = suf - mine;
    for (int w2 = warp + 1; w2 < 8; w2++) above += warp_sum[w2];
    for (int i = PER - 1; i >= 0; i--) {
        const unsigned long long cnt = __ldcg(&hist[t * PER + i]);
        if (above < k && k <= above + cnt) { st->prefix[pass] = (unsigned)(t * PER + i); st->krem[pass] = k - above; }
        above += cnt;
    }
    if (pass == 2) {
        __syncthreads();
        if (t == 0) st->threshold = key_score((st->prefix[0] << 20) | (st->prefix[1] << 10) | st->prefix[2]);
    }
}

// First pass, one CTA per row at a time: scale[n] = max(rowmax|W|, 1e-8) / 7, and with k > 0 the counts of the keys' top
// 12 bits (the row's second reading hits L1)
__global__ void __launch_bounds__(256)
sieve_rows_kernel(const float *__restrict__ w, const float *__restrict__ hinv, int64_t N, int K, float *__restrict__ scales,
                  SelectState *__restrict__ st, unsigned long long k)
{
    __shared__ float wmax[8];
    __shared__ unsigned int h[kBins0];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (k)
        for (int i = tid; i < kBins0; i += 256) h[i] = 0;
    for (int64_t n = blockIdx.x; n < N; n += gridDim.x) {
        const float4 *row = reinterpret_cast<const float4 *>(w + (size_t)n * K);
        float m = 0.f;
        for (int i = tid; i < K / 4; i += 1024) {
            float4 v[4];
#pragma unroll
            for (int j = 0; j < 4; j++) v[j] = i + 256 * j < K / 4 ? row[i + 256 * j] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int j = 0; j < 4; j++) m = fmaxf(m, fmaxf(fmaxf(fabsf(v[j].x), fabsf(v[j].y)), fmaxf(fabsf(v[j].z), fabsf(v[j].w))));
        }
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        if (lane == 0) wmax[warp] = m;
        __syncthreads();
        float mm = wmax[0];
#pragma unroll
        for (int i = 1; i < 8; i++) mm = fmaxf(mm, wmax[i]);
        const float scale = div_ieee(fmaxf(mm, 1e-8f), 7.0f), rscale = quant_rscale(scale);
        if (tid == 0) scales[n] = scale;
        if (k) {
            for (int i = tid; i < K / 4; i += 256) {
                const float4 v = row[i];
                const float4 hv = *reinterpret_cast<const float4 *>(hinv + 4 * i);
                const float ww[4] = {v.x, v.y, v.z, v.w}, hh[4] = {hv.x, hv.y, hv.z, hv.w};
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    float b, r;
                    const float hs = __fadd_rn(hh[e], 1e-6f), r2 = sieve_one(ww[e], scale, rscale, b, r);
                    uint32_t bits = __float_as_uint(r2 * rcp_approx(hs));
                    uint32_t key = bits | 0x80000000u;
                    if (!approx_ok(r2, hs) || (((bits + 16u) ^ (bits - 16u)) >> 20) != 0u) key = score_key(div_ieee(r2, hs));
                    atomicAdd(&h[key >> 20], 1u);
                }
            }
        }
        __syncthreads();                         // wmax is reused by the next row
    }
    if (k) add_and_select<kBins0>(h, st->hist0, st, 0, k);
}

// the quads of a row that are this CTA's: a row is cut into gridDim.y pieces of whole 1024 quads
struct Piece { int begin, end; };
__device__ __forceinline__ Piece piece_of(int quads)
{
    const int rounds = (quads + 1023) / 1024, per = (rounds + (int)gridDim.y - 1) / (int)gridDim.y * 1024;
    return Piece{(int)blockIdx.y * per, min(quads, ((int)blockIdx.y + 1) * per)};
}

// Second pass (PASS 1): the keys in the selected bin, counted by their next 10 bits and listed.  PASS 2, for want of
// a list: the keys that agree in these bits too, counted by the last 10.  PASS 0: the first pass's counts, where rows are cut
template <int PASS, bool LIST>
__global__ void __launch_bounds__(256)
sieve_bin_kernel(const float *__restrict__ w, const float *__restrict__ hinv, const float *__restrict__ scales,
                 int64_t N, int K, SelectState *__restrict__ st, uint32_t *__restrict__ list, unsigned long long k)
{
    constexpr int BINS = PASS == 0 ? kBins0 : kBins;
    __shared__ unsigned int h[BINS];
    for (int i = threadIdx.x; i < BINS; i += 256) h[i] = 0;
    __syncthreads();
    const Piece pc = piece_of(K / 4);
    const uint32_t bin = PASS == 0 ? 0u : st->prefix[0], mid = PASS == 2 ? st->prefix[1] : 0u;
    const int lane = threadIdx.x & 31;
    for (int64_t n = blockIdx.x; n < N; n += gridDim.x) {
        const float4 *row = reinterpret_cast<const float4 *>(w + (size_t)n * K);
        const float sc = scales[n], rs = quant_rscale(sc);
        for (int i0 = pc.begin; i0 < pc.end; i0 += 1024) {
            float4 v[4];
#pragma unroll
            for (int j = 0; j < 4; j++) v[j] = i0 + 256 * j + threadIdx.x < K / 4 ? row[i0 + 256 * j + threadIdx.x] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int i = i0 + 256 * j + threadIdx.x;
                const bool on = i < K / 4;
                const float4 hv = on ? *reinterpret_cast<const float4 *>(hinv + 4 * i) : make_float4(1.f, 1.f, 1.f, 1.f);
                const float ww[4] = {v[j].x, v[j].y, v[j].z, v[j].w}, hh[4] = {hv.x, hv.y, hv.z, hv.w};
                uint32_t key[4];
                bool in[4];
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    float b, r;
                    const float hs = __fadd_rn(hh[e], 1e-6f), r2 = sieve_one(ww[e], sc, rs, b, r);
                    const uint32_t bits = __float_as_uint(r2 * rcp_approx(hs)) | 0x80000000u;
                    if (PASS == 0) {
                        key[e] = bits;
                        if (!approx_ok(r2, hs) || (((bits + 16u) ^ (bits - 16u)) >> 20) != 0u) key[e] = score_key(div_ieee(r2, hs));
                        if (on) atomicAdd(&h[key[e] >> 20], 1u);
                        in[e] = false;
                        continue;
                    }
                    // clearly outside the bin: nothing to do; else the exact key
                    key[e] = 0;
                    in[e] = on && !(approx_ok(r2, hs) && (bits + 16u) >> 20 != bin && (bits - 16u) >> 20 != bin);
                    if (in[e]) {
                        key[e] = score_key(div_ieee(r2, hs));
                        in[e] = PASS == 1 ? (key[e] >> 20) == bin : (key[e] >> 10) == (bin << 10 | mid);
                    }
                }
                if (!__any_sync(0xffffffffu, in[0] || in[1] || in[2] || in[3])) continue;
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const unsigned m = __ballot_sync(0xffffffffu, in[e]);
                    if (m == 0u) continue;
                    unsigned at = 0;
                    if (LIST) {
                        if (lane == __ffs(m) - 1) at = atomicAdd(&st->listed, (unsigned)__popc(m));
                        at = __shfl_sync(0xffffffffu, at, __ffs(m) - 1);
                    }
                    if (in[e]) {
                        if (LIST) list[at + __popc(m & ((1u << lane) - 1u))] = key[e];
                        atomicAdd(&h[(PASS == 1 ? key[e] >> 10 : key[e]) & 1023u], 1u);
                    }
                }
            }
        }
    }
    if constexpr (PASS == 0) add_and_select<kBins0>(h, st->hist0, st, 0, k);
    else add_and_select<kBins>(h, PASS == 1 ? st->hist1 : st->hist2, st, PASS, st->krem[PASS - 1]);
}

// Third pass: the last 10 bits, from the list
__global__ void __launch_bounds__(256)
sieve_list_kernel(SelectState *__restrict__ st, const uint32_t *__restrict__ list)
{
    __shared__ unsigned int h[kBins];
    for (int i = threadIdx.x; i < kBins; i += 256) h[i] = 0;
    __syncthreads();
    const unsigned n = st->listed, mid = st->prefix[1];
    for (unsigned i = blockIdx.x * 256 + threadIdx.x; i < n; i += gridDim.x * 256) {
        const uint32_t key = list[i];
        if (((key >> 10) & 1023u) == mid) atomicAdd(&h[key & 1023u], 1u);
    }
    add_and_select<kBins>(h, st->hist2, st, 2, st->krem[1]);
}

__global__ void __launch_bounds__(256)
sieve_split_kernel(const float *__restrict__ w, const float *__restrict__ hinv, const float *__restrict__ scales,
                   int64_t N, int K, const float *__restrict__ thr_dev, float thr_host,
                   float *__restrict__ w_base, float *__restrict__ w_ortho)
{
    const float thr = thr_dev ? *thr_dev : thr_host;
    const bool thr_ok = thr >= 1e-20f && thr <= 1e20f;
    const float thr_lo = thr * 0.99999f, thr_hi = thr * 1.00001f;
    const Piece pc = piece_of(K / 4);
    for (int64_t n = blockIdx.x; n < N; n += gridDim.x) {
        const size_t at = (size_t)n * (K / 4);
        const float sc = scales[n], rs = quant_rscale(sc);
        for (int i0 = pc.begin + threadIdx.x; i0 < pc.end; i0 += 1024) {
            float4 v[4];
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (i0 + 256 * j < K / 4) v[j] = __ldcs(reinterpret_cast<const float4 *>(w) + at + i0 + 256 * j);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int i = i0 + 256 * j;
                if (i >= K / 4) break;
                const float4 hv = *reinterpret_cast<const float4 *>(hinv + 4 * i);
                const float ww[4] = {v[j].x, v[j].y, v[j].z, v[j].w}, hh[4] = {hv.x, hv.y, hv.z, hv.w};
                float bo[4], oo[4];
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    float r;
                    const float hs = __fadd_rn(hh[e], 1e-6f), r2 = sieve_one(ww[e], sc, rs, bo[e], r);
                    const float s = r2 * rcp_approx(hs);
                    bool keep = s > thr_hi;
                    if (!thr_ok || !approx_ok(r2, hs) || (s >= thr_lo && s <= thr_hi)) keep = div_ieee(r2, hs) > thr;
                    oo[e] = __fmul_rn(r, keep ? 1.f : 0.f);         // residual * mask, signed zeros as torch produces them
                }
                reinterpret_cast<float4 *>(w_base)[at + i] = make_float4(bo[0], bo[1], bo[2], bo[3]);
                reinterpret_cast<float4 *>(w_ortho)[at + i] = make_float4(oo[0], oo[1], oo[2], oo[3]);
            }
        }
    }
}

// Eight CTAs per SM at most, a row each.  A matrix of fewer rows than two per SM has its rows cut (into pieces of 4096
// weights or more) so that it still fills the GPU; its first pass then is two, the row scales and the counts.
// Keep the top 1 %, whole / cut rows: 1 x 4194304 8.8 / 0.33 ms, 64 x 65536 200 / 106 us, 295 x 8192 82 / 75 us.
static dim3 sieve_grid(int64_t N, int64_t K)
{
    const int64_t sms = device_sm_count(current_device_index()), cap = sms * 8, rounds = ceil_div(K / 4, 1024);
    if (N >= 2 * sms) return dim3((unsigned)(N > cap ? cap : N));
    const int64_t pieces = ceil_div(cap, N);
    return dim3((unsigned)N, (unsigned)(pieces < rounds ? pieces : rounds));
}

}  // namespace ob

using namespace ob;

extern "C" int64_t ortho_b200_sieve_scratch_bytes(int64_t N) { return N > 0 ? ((N * 4 + 255) / 256) * 256 + (int64_t)sizeof(SelectState) + 256 : -1; }

extern "C" int ortho_b200_sieve(const float *w, const float *h_inv_diag, int64_t N, int64_t K,
                                float curvature_thresh, int64_t keep_top_k,
                                float *w_base_out, float *w_ortho_out,
                                void *scratch, int64_t scratch_bytes, void *stream)
{
    if (!w || !h_inv_diag || !w_base_out || !w_ortho_out || !scratch) return ORTHO_B200_ERR_NULL;
    if (N <= 0 || K <= 0 || (K % 4) != 0 || keep_top_k < -1 || keep_top_k > N * K) return ORTHO_B200_ERR_SHAPE;
    if ((((uintptr_t)w | (uintptr_t)h_inv_diag | (uintptr_t)w_base_out | (uintptr_t)w_ortho_out) & 15u) != 0 ||
        ((uintptr_t)scratch & 255u) != 0)
        return ORTHO_B200_ERR_ALIGN;
    if (scratch_bytes < ortho_b200_sieve_scratch_bytes(N)) return ORTHO_B200_ERR_WORKSPACE;
    cudaStream_t st = (cudaStream_t)stream;
    float *scales = reinterpret_cast<float *>(scratch);
    SelectState *sel = reinterpret_cast<SelectState *>(reinterpret_cast<unsigned char *>(scratch) + ((N * 4 + 255) / 256) * 256);
    const dim3 grid = sieve_grid(N, K);
    const float *thr_dev = nullptr;
    float thr_host = curvature_thresh;
    const unsigned long long k = keep_top_k > 0 ? (unsigned long long)keep_top_k : 0ull;
    if (k) OB_CUDA(cudaMemsetAsync(sel, 0, sizeof(SelectState), st));
    const bool cut = grid.y > 1;
    sieve_rows_kernel<<<grid.x, 256, 0, st>>>(w, h_inv_diag, N, (int)K, scales, sel, cut ? 0ull : k);
    if (k && cut) sieve_bin_kernel<0, false><<<grid, 256, 0, st>>>(w, h_inv_diag, scales, N, (int)K, sel, nullptr, k);
    count_launch(k && cut ? 2 : 1);
    OB_CUDA(cudaGetLastError());
    if (k) {
        // the list: room for every key in an output that is not read on the way to the split, which writes both
        auto apart = [&](const float *out) {
            const uintptr_t o = (uintptr_t)out, n = (uintptr_t)(N * K) * 4, a = (uintptr_t)w, b = (uintptr_t)h_inv_diag;
            return (o + n <= a || a + n <= o) && (o + n <= b || b + (uintptr_t)K * 4 <= o);
        };
        uint32_t *list = reinterpret_cast<uint32_t *>(apart(w_ortho_out) ? w_ortho_out : apart(w_base_out) ? w_base_out : nullptr);
        if (list) {
            sieve_bin_kernel<1, true><<<grid, 256, 0, st>>>(w, h_inv_diag, scales, N, (int)K, sel, list, k);
            sieve_list_kernel<<<(unsigned)device_sm_count(current_device_index()), 256, 0, st>>>(sel, list);
        } else {
            sieve_bin_kernel<1, false><<<grid, 256, 0, st>>>(w, h_inv_diag, scales, N, (int)K, sel, nullptr, k);
            sieve_bin_kernel<2, false><<<grid, 256, 0, st>>>(w, h_inv_diag, scales, N, (int)K, sel, nullptr, k);
        }
        count_launch(2);
        OB_CUDA(cudaGetLastError());
        thr_dev = &sel->threshold;
    } else if (keep_top_k == 0) {
        thr_host = __builtin_inff();          // "keep nothing" (tools/sieve.py:65-66)
    }
    sieve_split_kernel<<<grid, 256, 0, st>>>(w, h_inv_diag, scales, N, (int)K, thr_dev, thr_host, w_base_out, w_ortho_out);
    count_launch();
    OB_CUDA(cudaGetLastError());
    return ORTHO_B200_OK;
}
