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
// (4096->11008, keep the top 1 %: 344 us by these passes: rows 115, bin 126, list 8, split 94.)
// Matrices of whole rows, of 10 million weights or more, take one pass over W where the scratch holds a list of candidates: a sample of the rows brackets the
// k-th largest score, the pass splits every weight at once (a row's scale first, its second reading comes from registers or L1),
// counts the scores above the bracket and lists those inside it, a radix select over that short list finds the threshold, and the
// listed residuals above it are written.  When the bracket turns out not to hold the k-th score, or the list overflows, the passes
// above run behind it (they look at a flag), so the result never depends on the sample.
#include <cstddef>
#include <cstring>

#include "common.cuh"
#include "rows.cuh"

namespace ob {

int *kernel_status_word();   // api.cu

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
// the same for the one-pass form: keys in the bins lo_bin .. hi_bin (top 12 bits) are listed and counted by 4096 bins of
// 2^shift keys
struct OnePass {
    unsigned int hist_sample[kBins0], hist1[kBins0], hist2[kBins0];
    unsigned int done[3];
    unsigned int lo_bin, hi_bin;
    int shift, bracket;                          // bracket: it could be set
    unsigned int listed, overflow;
    unsigned int prefix;
    int ok;                                      // the k-th score is in the list: what the other form would do is done
    unsigned long long above, krem;
    float threshold;
};
static_assert(offsetof(OnePass, ok) == 3 * kBins0 * 4 + 40, "the tests read it in the scratch, behind the other form's");
struct Candidate { uint32_t at, key; };          // flat position, key

// Adds the CTA's counts h[BINS] to the global ones; true in the last CTA to do so.  Called by all 256 threads.
template <int BINS>
__device__ __forceinline__ bool add_counts(const unsigned int *h, unsigned int *hist, unsigned int *done)
{
    __shared__ unsigned int is_last;
    __syncthreads();
    if (h)
        for (int i = threadIdx.x; i < BINS; i += 256)
            if (h[i]) atomicAdd(&hist[i], h[i]);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) is_last = atomicAdd(done, 1u) == gridDim.x * gridDim.y - 1 ? 1u : 0u;
    __syncthreads();
    if (is_last) __threadfence();
    return is_last != 0u;
}
// The bin that holds the k-th largest key (k counted from the top bin downwards) and the rank inside it, for all 256 threads;
// bin -1: there are fewer than k keys.
struct Found { int bin; unsigned long long rank; };
template <int BINS>
__device__ __forceinline__ Found find_rank(const unsigned int *hist, unsigned long long k)
{
    __shared__ unsigned long long warp_sum[8], f_rank;
    __shared__ int f_bin;
    // thread t owns bins [t * PER, (t + 1) * PER); keys in the bins above its own: a suffix sum over the threads
    constexpr int PER = BINS / 256;
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    __syncthreads();
    if (t == 0) { f_bin = -1; f_rank = 0; }
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
        if (above < k && k <= above + cnt) { f_bin = t * PER + i; f_rank = k - above; }
        above += cnt;
    }
    __syncthreads();
    return Found{f_bin, f_rank};
}
template <int BINS>
__device__ __forceinline__ void add_and_select(const unsigned int *h, unsigned int *hist, SelectState *st, int pass, unsigned long long k)
{
    if (!add_counts<BINS>(h, hist, &st->done[pass])) return;
    const Found f = find_rank<BINS>(hist, k);
    if (threadIdx.x != 0 || f.bin < 0) return;
    st->prefix[pass] = (unsigned)f.bin;
    st->krem[pass] = f.rank;
    if (pass == 2) st->threshold = key_score((st->prefix[0] << 20) | (st->prefix[1] << 10) | (unsigned)f.bin);
}

// First pass, one CTA per row at a time: scale[n] = max(rowmax|W|, 1e-8) / 7, and with k > 0 the counts of the keys' top
// 12 bits (the row's second reading hits L1)
// (SAMPLE: of N rows, `step` apart; the last CTA brackets the k-th largest score of the whole matrix, of which k_sample is
// the sample's share)
template <bool SAMPLE>
__global__ void __launch_bounds__(256)
sieve_rows_kernel(const float *__restrict__ w, const float *__restrict__ hinv, int64_t N, int K, float *__restrict__ scales,
                  SelectState *__restrict__ st, unsigned long long k, const int *__restrict__ done, int64_t step,
                  OnePass *__restrict__ op, float k_sample)
{
    if (!SAMPLE && done && *done) return;
    __shared__ float wmax[8];
    __shared__ unsigned int h[kBins0];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (k)
        for (int i = tid; i < kBins0; i += 256) h[i] = 0;
    for (int64_t n = blockIdx.x; n < N; n += gridDim.x) {
        const float4 *row = reinterpret_cast<const float4 *>(w + (size_t)(SAMPLE ? n * step : n) * K);
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
        if (!SAMPLE && tid == 0) scales[n] = scale;
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
    if (!SAMPLE) {
        if (k) add_and_select<kBins0>(h, st->hist0, st, 0, k);
        return;
    }
    if (!add_counts<kBins0>(h, op->hist_sample, &op->done[0])) return;
    // ranks between which the k-th is expected: a quarter to either side for rows that differ, and six standard deviations of
    // the count; no more than 16 bins
    const float slack = 6.f * sqrtf(k_sample) + 8.f, lo_rank = 1.25f * k_sample + slack, hi_rank = 0.75f * k_sample - slack;
    const Found lo = find_rank<kBins0>(op->hist_sample, (unsigned long long)lo_rank);
    const Found hi = find_rank<kBins0>(op->hist_sample, (unsigned long long)fmaxf(hi_rank, 1.f));
    if (tid == 0 && lo.bin >= 0 && hi.bin >= lo.bin) {
        int span = 15, shift = 12;
        if (hi_rank >= 1.f && hi.bin - lo.bin < span) span = hi.bin - lo.bin;
        while (shift > 8 && (span + 1) << 1 <= 1 << (shift - 8)) shift--;
        if (lo.bin + span >= kBins0) span = kBins0 - 1 - lo.bin;
        op->lo_bin = (unsigned)lo.bin; op->hi_bin = (unsigned)(lo.bin + span); op->shift = shift;
        op->bracket = 1;
    }
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
                 int64_t N, int K, SelectState *__restrict__ st, uint32_t *__restrict__ list, unsigned long long k,
                 const int *__restrict__ done)
{
    if (done && *done) return;
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
sieve_list_kernel(SelectState *__restrict__ st, const uint32_t *__restrict__ list, const int *__restrict__ done)
{
    if (done && *done) return;
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
                   float *__restrict__ w_base, float *__restrict__ w_ortho, const int *__restrict__ done)
{
    if (done && *done) return;
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

// One pass: scale of a row, then its split.  SELECT: against the bracket; what falls into it is listed with a zero residual for
// now.  Else: against the threshold `thr`.  An output may be W itself without SELECT (a thread reads a quad before it writes it, a
// row is read for its scale before any of it is written; with PIPE, rows that come through shared memory, W is nobody's output).
// Bound by HBM: 4 bytes read and 8 written per weight, some 30 instructions.  The list is kept in shared memory and handed over
// some hundred entries at a time (an atomic per warp and quad on one counter cost the bin pass above 100 us).
// 4096->11008 on one B200: 140 us for 540 MB (3.9 TB/s), 116 at a given threshold; the whole call, top 1 %, 344 -> about
// 210 (sample 16, pass 140, threshold 11, kept residuals 13, launches that find nothing to do), at a threshold 162 -> 126.
constexpr int kListBuf = 1024;
template <bool SELECT, bool PIPE>
__global__ void __launch_bounds__(256, 5)
sieve_onepass_kernel(const float *__restrict__ w, const float *__restrict__ hinv, int64_t N, int K, float thr_given,
                     OnePass *__restrict__ op, Candidate *__restrict__ list, unsigned cap, unsigned long long k,
                     float *__restrict__ w_base, float *__restrict__ w_ortho, int *__restrict__ status)
{
    extern __shared__ __align__(16) unsigned char row_smem[];
    __shared__ float wmax[8];
    __shared__ Candidate buf[SELECT ? kListBuf : 1];
    __shared__ unsigned int buffered, list_at;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, quads = K / 4;
    unsigned lo_bin = 0, hi_bin = 0;
    int shift = 0;
    float thr_lo, thr_hi;                        // a score clearly below / above what has to be looked at exactly
    bool thr_ok;
    if (SELECT) {
        if (!op->bracket) return;
        lo_bin = op->lo_bin; hi_bin = op->hi_bin; shift = op->shift;
        const float a = key_score(lo_bin << 20), b = hi_bin + 1 < kBins0 ? key_score((hi_bin + 1) << 20) : __builtin_inff();
        thr_ok = a >= 1e-20f && b <= 1e20f;
        thr_lo = a * 0.99999f; thr_hi = b * 1.00001f;
        if (tid == 0) buffered = 0;
    } else {
        thr_ok = thr_given >= 1e-20f && thr_given <= 1e20f;
        thr_lo = thr_given * 0.99999f; thr_hi = thr_given * 1.00001f;
    }
    unsigned above = 0;
    // an undecided score, exactly: into the list (key 0 leaves a gap there) or clearly above the bracket (true)
    auto decide = [&](unsigned slot, uint32_t pos, float r2) -> bool {
        const float exact = div_ieee(r2, __fadd_rn(hinv[pos % (unsigned)K], 1e-6f));
        const uint32_t key = score_key(exact), bin = key >> 20;
        const bool in = bin >= lo_bin && bin <= hi_bin;
        if (slot < cap) {
            list[slot] = Candidate{pos, in ? key : 0u};
            if (in) atomicAdd(&op->hist1[(key - (lo_bin << 20)) >> shift], 1u);
        } else {
            op->overflow = 1u;
        }
        above += bin > hi_bin ? 1u : 0u;
        return bin > hi_bin && exact == exact;                        // (the threshold is below, NaN is not above it)
    };
    RowPipe pipe(row_smem, w, PIPE ? (size_t)K * 4 : 0, PIPE ? N : 0);
    for (int64_t n = blockIdx.x; n < N; n += gridDim.x) {
        const size_t at = (size_t)n * quads;
        const float4 *row = PIPE ? pipe.row(status) : reinterpret_cast<const float4 *>(w) + at;
        float4 v[4];
        float m = 0.f;
        for (int i0 = tid; i0 < quads; i0 += 1024) {
#pragma unroll
            for (int j = 0; j < 4; j++) v[j] = i0 + 256 * j < quads ? row[i0 + 256 * j] : make_float4(0.f, 0.f, 0.f, 0.f);
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
        const float sc = div_ieee(fmaxf(mm, 1e-8f), 7.0f), rs = quant_rscale(sc);
        for (int i0 = tid; i0 < quads; i0 += 1024) {
            if (!PIPE) {
#pragma unroll
                for (int j = 0; j < 4; j++)
                    if (i0 + 256 * j < quads) v[j] = row[i0 + 256 * j];
            }
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int i = i0 + 256 * j;
                if (i >= quads) break;
                if (PIPE) v[j] = row[i];
                const float4 hv = *reinterpret_cast<const float4 *>(hinv + 4 * i);
                const float ww[4] = {v[j].x, v[j].y, v[j].z, v[j].w}, hh[4] = {hv.x, hv.y, hv.z, hv.w};
                float bo[4], oo[4];
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    float r;
                    const float hs = __fadd_rn(hh[e], 1e-6f), r2 = sieve_one(ww[e], sc, rs, bo[e], r);
                    const float s = r2 * rcp_approx(hs);
                    bool keep = s > thr_hi;
                    const bool unsure = !thr_ok || !approx_ok(r2, hs) || (s >= thr_lo && s <= thr_hi);
                    if (SELECT) {
                        if (!unsure) {
                            above += keep ? 1u : 0u;
                        } else {                 // few, but some lane of most warps: the division waits until there are enough
                            const uint32_t pos = (uint32_t)((at + i) * 4 + e);
                            const unsigned slot = atomicAdd(&buffered, 1u);
                            keep = false;
                            if (slot < kListBuf) buf[slot] = Candidate{pos, __float_as_uint(r2)};
                            else keep = decide(atomicAdd(&op->listed, 1u), pos, r2);
                        }
                    } else if (unsure) {
                        keep = div_ieee(r2, hs) > thr_given;
                    }
                    oo[e] = __fmul_rn(r, keep ? 1.f : 0.f);         // residual * mask, signed zeros as torch produces them
                }
                reinterpret_cast<float4 *>(w_base)[at + i] = make_float4(bo[0], bo[1], bo[2], bo[3]);
                reinterpret_cast<float4 *>(w_ortho)[at + i] = make_float4(oo[0], oo[1], oo[2], oo[3]);
            }
        }
        __syncthreads();                         // wmax is reused by the next row; the buffer is complete; the row has been read
        if (PIPE) pipe.release();
        if (SELECT) {
            const unsigned have = min(buffered, (unsigned)kListBuf);
            if (have >= kListBuf / 4 || (have > 0 && n + gridDim.x >= N)) {
                if (tid == 0) list_at = atomicAdd(&op->listed, have);
                __syncthreads();
                for (unsigned i = tid; i < have; i += 256) {
                    const uint32_t pos = buf[i].at;
                    if (decide(list_at + i, pos, __uint_as_float(buf[i].key))) w_ortho[pos] = __fsub_rn(w[pos], w_base[pos]);
                }
                __syncthreads();
                if (tid == 0) buffered = 0;
                __syncthreads();
            }
        }
    }
    if (!SELECT) return;
    above = __reduce_add_sync(0xffffffffu, above);
    if (lane == 0 && above) atomicAdd(&op->above, (unsigned long long)above);
    if (!add_counts<kBins0>(nullptr, nullptr, &op->done[1])) return;
    const unsigned long long over = __ldcg(&op->above);
    if (__ldcg(&op->overflow) || over >= k) return;
    const Found f = find_rank<kBins0>(op->hist1, k - over);
    if (tid == 0 && f.bin >= 0) { op->prefix = (unsigned)f.bin; op->krem = f.rank; op->ok = 1; }
}

// The listed keys of the selected bin, counted one by one: the threshold
__global__ void __launch_bounds__(256)
sieve_candidates_kernel(OnePass *__restrict__ op, const Candidate *__restrict__ list)
{
    if (!op->ok) return;
    const unsigned n = op->listed, prefix = op->prefix, base = op->lo_bin << 20;
    const int shift = op->shift;
    for (unsigned i = blockIdx.x * 256 + threadIdx.x; i < n; i += gridDim.x * 256) {
        const uint32_t key = list[i].key;
        if ((key - base) >> shift == prefix) atomicAdd(&op->hist2[key & ((1u << shift) - 1u)], 1u);
    }
    if (!add_counts<kBins0>(nullptr, nullptr, &op->done[2])) return;
    const Found f = find_rank<kBins0>(op->hist2, op->krem);
    if (threadIdx.x == 0) op->threshold = key_score(base + (prefix << shift) + (unsigned)f.bin);
}

// the listed residuals above the threshold
__global__ void __launch_bounds__(256)
sieve_keep_kernel(const OnePass *__restrict__ op, const Candidate *__restrict__ list, const float *__restrict__ w,
                  const float *__restrict__ w_base, float *__restrict__ w_ortho)
{
    if (!op->ok) return;
    const unsigned n = op->listed;
    const float thr = op->threshold;
    for (unsigned i = blockIdx.x * 256 + threadIdx.x; i < n; i += gridDim.x * 256) {
        const Candidate c = list[i];
        if (key_score(c.key) > thr) w_ortho[c.at] = __fsub_rn(w[c.at], w_base[c.at]);
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

// `apart`: no output is W, so rows may be fetched ahead of the ones being written
template <bool SELECT>
static int launch_onepass(const float *w, const float *h, int64_t N, int K, float thr, OnePass *op, Candidate *list, unsigned cap,
                          unsigned long long k, float *base, float *ortho, bool apart, cudaStream_t st)
{
    const int dev = current_device_index();
    if (dev < 0) return ORTHO_B200_ERR_CUDA;
    int *status = kernel_status_word();
    if (!status) return ORTHO_B200_ERR_CUDA;
    const int64_t sms = device_sm_count(dev);
    if (apart && K * 4 <= kRowBytesMax) {
        static bool attr_set[kMaxDevices] = {};
        if (!attr_set[dev]) {
            OB_CUDA(cudaFuncSetAttribute(sieve_onepass_kernel<SELECT, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)row_smem_bytes(kRowBytesMax)));
            attr_set[dev] = true;
        }
        const int64_t grid = sms * row_ctas_per_sm((int64_t)K * 4, SELECT ? kListBuf * (int)sizeof(Candidate) : 64);
        sieve_onepass_kernel<SELECT, true><<<(unsigned)(grid < N ? grid : N), 256, row_smem_bytes((size_t)K * 4), st>>>(w, h, N, K, thr, op, list, cap, k, base, ortho, status);
    } else {
        const int64_t grid = sms * 8;
        sieve_onepass_kernel<SELECT, false><<<(unsigned)(grid < N ? grid : N), 256, kRowBufs * sizeof(uint64_t), st>>>(w, h, N, K, thr, op, list, cap, k, base, ortho, status);
    }
    OB_CUDA(cudaGetLastError());
    return ORTHO_B200_OK;
}

// one-pass form: state and the list of candidates, behind the other form's scratch
static unsigned candidate_cap(int64_t N, int64_t K) { return (unsigned)(N * K / 16 > 65536 ? N * K / 16 : 65536); }
// Whole rows; below 10 million weights its ten launches cost as much as the passes: 2048 x 1024 93 us against 84, whole layers of
// 8.6 million 209 / 202, 10.2 million 217 / 238
static bool onepass_shape(int64_t N, int64_t K) { return N <= 0xffffffffLL / K && N * K >= 10000000 && sieve_grid(N, K).y == 1; }
extern "C" int64_t ortho_b200_sieve_scratch_bytes(int64_t N);
extern "C" int64_t ortho_b200_sieve_onepass_scratch_bytes(int64_t N, int64_t K)
{
    if (N <= 0 || K <= 0) return -1;
    if (K > 0x7fffffffLL || !onepass_shape(N, K)) return ortho_b200_sieve_scratch_bytes(N);
    return (ortho_b200_sieve_scratch_bytes(N) + 255) / 256 * 256 + (int64_t)(sizeof(OnePass) + 255) / 256 * 256 + (int64_t)candidate_cap(N, K) * (int64_t)sizeof(Candidate);
}

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
    const bool cut = grid.y > 1;
    auto apart_from = [](const void *x, int64_t nx, const void *y, int64_t ny) {
        const uintptr_t a = (uintptr_t)x, b = (uintptr_t)y;
        return a + (uintptr_t)nx <= b || b + (uintptr_t)ny <= a;
    };
    const int64_t wbytes = N * K * 4, hbytes = K * 4;
    const bool outs_apart = apart_from(w_base_out, wbytes, w_ortho_out, wbytes) && apart_from(w_base_out, wbytes, h_inv_diag, hbytes) &&
                            apart_from(w_ortho_out, wbytes, h_inv_diag, hbytes);
    const bool base_apart = apart_from(w_base_out, wbytes, w, wbytes), ortho_apart = apart_from(w_ortho_out, wbytes, w, wbytes);
    const int *done = nullptr;
    if (!k && !cut && outs_apart && (base_apart || w_base_out == w) && (ortho_apart || w_ortho_out == w)) {
        // a given threshold ("keep nothing": infinite, tools/sieve.py:65-66)
        const int rc = launch_onepass<false>(w, h_inv_diag, N, (int)K, keep_top_k == 0 ? __builtin_inff() : curvature_thresh, nullptr, nullptr, 0u,
                                             0ull, w_base_out, w_ortho_out, base_apart && ortho_apart, st);
        if (rc != ORTHO_B200_OK) return rc;
        count_launch();
        OB_CUDA(cudaGetLastError());
        return ORTHO_B200_OK;
    }
    // One pass where the list can hold what a bracket of the k-th score holds (half of k and two bins' worth) and W outlives
    // the pass
    const bool onepass = k && onepass_shape(N, K) && outs_apart && base_apart && ortho_apart && k <= (unsigned long long)(N * K / 25) &&
                         scratch_bytes >= ortho_b200_sieve_onepass_scratch_bytes(N, K);
    if (onepass) {
        OnePass *op = reinterpret_cast<OnePass *>(reinterpret_cast<unsigned char *>(scratch) + (ortho_b200_sieve_scratch_bytes(N) + 255) / 256 * 256);
        Candidate *list = reinterpret_cast<Candidate *>(reinterpret_cast<unsigned char *>(op) + (sizeof(OnePass) + 255) / 256 * 256);
        const int64_t sms = device_sm_count(current_device_index());
        // two rows per SM, or as many as hold half a million weights
        int64_t rows = 2 * sms > ((int64_t)1 << 19) / K ? 2 * sms : ((int64_t)1 << 19) / K;
        if (rows > N) rows = N;
        OB_CUDA(cudaMemsetAsync(op, 0, sizeof(OnePass), st));
        sieve_rows_kernel<true><<<(unsigned)(rows < 8 * sms ? rows : 8 * sms), 256, 0, st>>>(w, h_inv_diag, rows, (int)K, nullptr, nullptr, k,
            nullptr, N / rows, op, (float)((double)k * (double)rows / (double)N));
        const int rc = launch_onepass<true>(w, h_inv_diag, N, (int)K, 0.f, op, list, candidate_cap(N, K), k, w_base_out, w_ortho_out, true, st);
        if (rc != ORTHO_B200_OK) return rc;
        sieve_candidates_kernel<<<(unsigned)sms, 256, 0, st>>>(op, list);
        sieve_keep_kernel<<<(unsigned)(4 * sms), 256, 0, st>>>(op, list, w, w_base_out, w_ortho_out);
        count_launch(4);
        OB_CUDA(cudaGetLastError());
        done = &op->ok;                          // what follows returns at once where that worked
    }
    if (k) OB_CUDA(cudaMemsetAsync(sel, 0, sizeof(SelectState), st));
    sieve_rows_kernel<false><<<grid.x, 256, 0, st>>>(w, h_inv_diag, N, (int)K, scales, sel, cut ? 0ull : k, done, 1, nullptr, 0.f);
    if (k && cut) sieve_bin_kernel<0, false><<<grid, 256, 0, st>>>(w, h_inv_diag, scales, N, (int)K, sel, nullptr, k, nullptr);
    count_launch(k && cut ? 2 : 1);
    OB_CUDA(cudaGetLastError());
    if (k) {
        // the list: room for every key in an output that is not read on the way to the split, which writes both
        auto apart = [&](const float *out) { return apart_from(out, wbytes, w, wbytes) && apart_from(out, wbytes, h_inv_diag, hbytes); };
        uint32_t *list = reinterpret_cast<uint32_t *>(apart(w_ortho_out) ? w_ortho_out : apart(w_base_out) ? w_base_out : nullptr);
        if (list) {
            sieve_bin_kernel<1, true><<<grid, 256, 0, st>>>(w, h_inv_diag, scales, N, (int)K, sel, list, k, done);
            sieve_list_kernel<<<(unsigned)device_sm_count(current_device_index()), 256, 0, st>>>(sel, list, done);
        } else {
            sieve_bin_kernel<1, false><<<grid, 256, 0, st>>>(w, h_inv_diag, scales, N, (int)K, sel, nullptr, k, done);
            sieve_bin_kernel<2, false><<<grid, 256, 0, st>>>(w, h_inv_diag, scales, N, (int)K, sel, nullptr, k, done);
        }
        count_launch(2);
        OB_CUDA(cudaGetLastError());
        thr_dev = &sel->threshold;
    } else if (keep_top_k == 0) {
        thr_host = __builtin_inff();          // "keep nothing" (tools/sieve.py:65-66)
    }
    sieve_split_kernel<<<grid, 256, 0, st>>>(w, h_inv_diag, scales, N, (int)K, thr_dev, thr_host, w_base_out, w_ortho_out, done);
    count_launch();
    OB_CUDA(cudaGetLastError());
    return ORTHO_B200_OK;
}
