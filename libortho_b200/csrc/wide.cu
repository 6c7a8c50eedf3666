// Forward for more than 128 tokens on the 5th-generation tensor cores: the pipeline of mid.cu with the token block cut
// into tiles of up to 192.
//
//     D[n, m] = sum_k w[n, k] * x[m, k]            (tcgen05.mma, A in tensor memory, B in shared memory, FP32 in TMEM)
//     y[m, n] = scale[n] * D[n, m] + bias[n]       with w = w_int + v * alpha / scale where row n has an entry v
//
// Replaces the reference's WMMA kernels (src/dual_gemm_tensor_core.cu:70-174, 215-337) for base-only calls and for plans
// with window lists; prefill.cu keeps the calls whose sparse term has to be gathered and the peer exchange.
//
// Tile: 128 weight rows x nt tokens, nt <= 192, for base-only calls.  Tensor memory holds two accumulators of 192 columns
// and four stages of 32 columns of converted weights, so a tile's epilogue (which a single accumulator of 256 columns
// exposed, about 7 of 66 us per tile) runs under the next tile's MMAs.  With a sparse term a tile is 128 x 2 nt tokens,
// nt <= 176, both accumulators at once: a converted k block then serves 352 tokens, since its entries cost the converters
// about as much again as the conversion (one token tile per k block: 8192->8192 at 2048 tokens and 0.3 % 276 us against
// 190 base-only); the epilogue is exposed instead, some 2 of 50 us.  Tokens are cut into tiles of equal size rounded up to 16.
// The pipeline's unit is a k block (128 rows x 64 k): a token tile of nt x 64 by TMA, one barrier for both operands of a
// stage (what a second wait and commit cost is told in mid.cu), four MMAs of nt / 2 cycles each.  Packed INT4 comes four
// k blocks at a time (128 rows x 128 B: a row of a box costs the TMA unit about 2 cycles however short it is, and with
// 32-byte rows the weights cost as much of it as the tokens).  Sixteen converter warps form four groups, one per k block of a
// box (thread = row); K is rounded up to whole boxes (zeros).
// Sparse entries are added to the weights in the converters' registers: a warp takes its window's list (windows.cuh)
// with one coalesced load a turn ahead and goes through it round by round.  The contraction of scattered tiles that mid.cu
// uses would double the MMAs, which are the bound here; a round costs about 75 instructions of a warp, and the
// converters have about twice the time that the base needs.
// One B200, us, base-only / fused, against the 128 x 256 tile of prefill.cu: 8192->8192 at 2048 tokens, 0.3 % 190 / 204
// (265 / 295; 1440 / 1350 TFLOP/s now), at 8192 tokens 783 / 900 (963 / 1174); 4096->4096 at 2048, 1 % 54 / 70 (76 / 108);
// 8192->8192 with Zipf rows at 512 tokens 53 / 65 (71 / 81).  Bounds: the power cap (cuBLAS sustains 1400) at many tokens; in the
// fused form the converters (4096->4096 at 2048 tokens, 1 %, by counters: tensor pipe busy in 55 % of the active cycles, issue
// slots in 56 %, integer pipe in 47 %, DRAM 5 %).
//
// Work split: as many whole waves of tiles as there are, tile after tile with the token tiles of a row tile next to each
// other (a wave then reads few weight rows, and the activations from L2); the tiles left over are cut along K into
// equal contiguous shares as in mid.cu (partial sums to the workspace, collected in CTA order) when the caller's
// workspace has room, else they are one more wave.
#include <cstring>

#include "common.cuh"
#include "umma.cuh"
#include "windows.cuh"

namespace ob {

int *kernel_status_word();

namespace wd {
constexpr int TN = 128;                 // weight rows per tile (MMA M)
template <bool SPARSE> constexpr int kTMax = SPARSE ? 176 : 192;      // most tokens per MMA: two accumulators and four stages fill
                                                                      // tensor memory, and with two token tiles per stage shared memory
template <bool SPARSE> constexpr int kHalves = SPARSE ? 2 : 1;        // token tiles (and accumulators) that share a k block
constexpr int KB = 64;                  // k block: the pipeline's unit
constexpr int GROUPS = 4;               // converter groups = k blocks of a box
constexpr int KC = GROUPS * KB;         // k of a box, the unit of the work split
constexpr int W_BYTES = TN * KC / 2;    // 16 KB
constexpr int A_STAGE_COLS = KB / 2;
// By the rule told in mid.cu a group, which comes back after four units, needs four stages or more; of the boxes it is
// one ahead of one it has stored a block of, which took the MMAs of a block of the box two before: three slots or more.
constexpr int ST_MAX = 6, WST_MAX = 6;
constexpr int CONV_WARPS = 4 * GROUPS;
constexpr int EPI_WARP0 = 2 + CONV_WARPS;
constexpr int EPI_WARPS = 4;
constexpr int XPROD_WARP = EPI_WARP0 + EPI_WARPS;
constexpr int NWARPS = XPROD_WARP + 1;
constexpr int TMEM_COLS = 512;
constexpr int kSmemData = 225 * 1024;   // packed-weight slots and token stages

struct Params {
    const __half *scales; const float *bias; __half *y;
    int y_type;                 // kTypeF16 ..: what y points to
    int M, K, N;
    long long ldy;
    int tiles_n, tiles_m, kblocks, boxes;       // boxes = ceil(K / 256)
    int nt, acc_cols;           // tokens of an MMA, tensor-memory columns of an accumulator (nt rounded up to 32)
    int tt;                     // tokens of a tile (nt, or 2 nt with a sparse term)
    int xtile, nst, wst;        // bytes of a token tile, stages, packed-weight slots
    int band;                   // token tiles of a band (see tile_of)
    int full;                   // whole tiles per CTA: tiles cta, cta + grid, ...
    int tail0, tail_ctas;       // first tile of those behind the whole waves, the CTAs that share their units:
    int share, extra;           // `share` each, one more for the first `extra` CTAs
    float *slots; unsigned long long *flags; unsigned long long tag;     // as in mid.cu
    float alpha;
    const uint32_t *win_off, *win_words; int ngroups;
    OrthoView ov; const float *row_max; const __half *x;                  // rows that FP16 cannot hold are gathered from x
    float *rest; int rest_mp; const int32_t *hrow; int n_long, heavy;     // long rows: their FP32 values go to `rest` (longrows.cu)
    int *status;
};

struct Smem {
    uint64_t w_full[WST_MAX], w_empty[WST_MAX];
    uint64_t full[ST_MAX], empty[ST_MAX];
    uint64_t d_full[2], d_empty[2];
    uint64_t all_done;          // the CTA's last piece is complete (one phase: the converters have not followed d_full)
    uint32_t tmem_base;
};
constexpr size_t kSmemBytes = 1024 + (size_t)kSmemData + sizeof(Smem);
static_assert(kSmemBytes <= 232448, "shared memory per CTA");

// Tiles are numbered in bands of token tiles whose activations stay in L2: inside a band the token tiles of a row tile come
// one after the other, then the next row tile's.
struct Tile { int row, mt; };
__device__ __forceinline__ Tile tile_of(const Params &p, int t)
{
    const int per = p.band * p.tiles_n, b = t / per, r = t - b * per;
    const int width = min(p.band, p.tiles_m - b * p.band);
    Tile x;
    x.row = r / width;
    x.mt = b * p.band + r - x.row * width;
    return x;
}
// The CTA's pieces in order: whole tiles, then its share of the cut ones.  Boxes [b0, b1) of tile t.
struct Pieces {
    int t, b0, b1;
    int whole, next_tile, step;          // whole tiles left
    int tail_t, tail_b, tail_units, boxes;
    __device__ __forceinline__ Pieces(const Params &p, int cta, int G) : t(0), b0(0), b1(0), whole(p.full), next_tile(cta), step(G), boxes(p.boxes)
    {
        const int at = p.share * cta + min(cta, p.extra);
        tail_units = cta < p.tail_ctas ? p.share + (cta < p.extra ? 1 : 0) : 0;
        tail_t = p.tail0 + at / p.boxes;
        tail_b = at % p.boxes;
    }
    __device__ __forceinline__ bool last() const { return whole <= 0 && tail_units <= 0; }
    __device__ __forceinline__ bool next()
    {
        if (whole > 0) {
            t = next_tile; b0 = 0; b1 = boxes;
            whole--; next_tile += step;
            return true;
        }
        if (tail_units <= 0) return false;
        t = tail_t; b0 = tail_b;
        b1 = boxes - b0 < tail_units ? boxes : b0 + tail_units;
        tail_units -= b1 - b0;
        tail_t++; tail_b = 0;
        return true;
    }
};
// box after box
struct Walk {
    Pieces pc; int b; bool ok;
    __device__ __forceinline__ Walk(const Params &p, int cta, int G) : pc(p, cta, G), b(0), ok(true) { ok = pc.next(); b = pc.b0; }
    __device__ __forceinline__ void step()
    {
        if (++b >= pc.b1) { ok = pc.next(); b = pc.b0; }
    }
};

// adds v * rsc (rounded to FP16) of a window's entries to the 64 converted weights of the lane's row, pairs (2i, 2i + 1) in
// h[i].  `mine` = entry `lane` of the list, `count` entries at `list`; every 32 of them are taken round by round:
// a new round starts where the row does not grow.
__device__ __forceinline__ void add_entries(uint32_t (&h)[32], uint32_t mine, uint32_t count, const uint32_t *list, float rsc, int lane)
{
    const uint32_t below = (1u << lane) - 1u;
    for (uint32_t at = 0; at < count; at += 32) {
        const uint32_t n = min(32u, count - at);
        if (at > 0) mine = (uint32_t)lane < n ? __ldg(list + at + lane) : 0u;
        const uint32_t row = (mine >> 7) & 31u;
        const uint32_t prev = __shfl_up_sync(0xffffffffu, row, 1);
        const bool in = (uint32_t)lane < n;
        uint32_t starts = __ballot_sync(0xffffffffu, in && (lane == 0 || row <= prev));
        while (starts) {
            const int s = __ffs(starts) - 1;
            starts &= starts - 1;
            const int e = starts ? __ffs(starts) - 1 : (int)n;
            const uint32_t rows = __reduce_or_sync(0xffffffffu, lane >= s && lane < e ? 1u << row : 0u);
            const uint32_t ent = __shfl_sync(0xffffffffu, mine, (s + __popc(rows & below)) & 31);
            const bool has = ((rows >> lane) & 1u) != 0u && rsc != 0.f;
            const float d = __half2float(__ushort_as_half((unsigned short)(ent >> 16))) * rsc;
            const uint32_t hb = (uint32_t)__half_as_ushort(__float2half_rn(d));
            const uint32_t dv = (ent & 2u) ? hb << 16 : hb;
            const uint32_t chunk = ((ent >> 4) ^ (uint32_t)lane) & 7u;            // 8 weights = 4 pairs
            const uint32_t bit = has ? 1u << ((chunk & 3u) * 4 + ((ent >> 2) & 3u)) : 0u;
            const uint32_t lo = (chunk & 4u) ? 0u : bit, hi = (chunk & 4u) ? bit : 0u;
            const __half2 d2 = *reinterpret_cast<const __half2 *>(&dv);
#pragma unroll
            for (int i = 0; i < 16; i++)
                if (lo & (1u << i)) {
                    const __half2 r = __hadd2(*reinterpret_cast<const __half2 *>(&h[i]), d2);
                    h[i] = *reinterpret_cast<const uint32_t *>(&r);
                }
#pragma unroll
            for (int i = 0; i < 16; i++)
                if (hi & (1u << i)) {
                    const __half2 r = __hadd2(*reinterpret_cast<const __half2 *>(&h[16 + i]), d2);
                    h[16 + i] = *reinterpret_cast<const uint32_t *>(&r);
                }
        }
    }
}
}  // namespace wd

// TYPED: as in mid.cu
template <bool SPARSE, bool TYPED>
__global__ void __launch_bounds__(wd::NWARPS * 32, 1)
wide_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap wmap, const wd::Params p)
{
    using namespace wd;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char *base = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    unsigned char *xs = base;                                          // token stages, 1 KB aligned (nt is a multiple of 16)
    constexpr int H = kHalves<SPARSE>;
    unsigned char *ws = xs + (size_t)(p.nst * H) * p.xtile;
    Smem *sm = reinterpret_cast<Smem *>(base + (size_t)kSmemData);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int cta = blockIdx.x, G = gridDim.x;

    if (threadIdx.x == 0) {
        for (int s = 0; s < WST_MAX; s++) { mbar_init(&sm->w_full[s], 1); mbar_init(&sm->w_empty[s], CONV_WARPS); }
        for (int s = 0; s < ST_MAX; s++) { mbar_init(&sm->full[s], 5); mbar_init(&sm->empty[s], 1); }
        for (int s = 0; s < 2; s++) { mbar_init(&sm->d_full[s], 1); mbar_init(&sm->d_empty[s], EPI_WARPS); }
        mbar_init(&sm->all_done, 1);
        fence_mbar_init();
        prefetch_tensormap(&xmap);
        prefetch_tensormap(&wmap);
    }
    if (warp == 1) { tmem_alloc(&sm->tmem_base, TMEM_COLS); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sm->tmem_base;
    // programmatic dependent launch: barriers, tensor memory and descriptors are set up beside the predecessor's tail; nothing is loaded
    // before its end
    if (!SPARSE || p.n_long == 0) asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    bool dead = false;
    auto wait = [&](uint64_t *bar, uint32_t parity) {
        if (mbar_try_wait(bar, parity) || dead) return;
        if (!mbar_wait(bar, parity, 1u << 24)) { dead = true; atomicExch(p.status, 1); }
    };

    if (warp == 0) {
        // ================= TMA producer: packed weights =================
        if (elect_one()) {
            int wi = 0; uint32_t wph = 0;
            Pieces pc(p, cta, G);
            while (pc.next()) {
                const int row0 = tile_of(p, pc.t).row * TN;
                for (int b = pc.b0; b < pc.b1; b++) {
                    wait(&sm->w_empty[wi], wph ^ 1u);
                    mbar_arrive_expect_tx(&sm->w_full[wi], W_BYTES);
                    tma_load_2d(ws + (size_t)wi * W_BYTES, &wmap, &sm->w_full[wi], b * (KC / 2), row0);
                    if (++wi == p.wst) { wi = 0; wph ^= 1u; }
                }
            }
        }
    } else if (warp == XPROD_WARP) {
        // ================= TMA producer: token tiles =================
        if (elect_one()) {
            int st = 0; uint32_t ph = 0;
            Pieces pc(p, cta, G);
            while (pc.next()) {
                const int m0 = tile_of(p, pc.t).mt * p.tt;
                const bool two = H == 2 && m0 + p.nt < p.M;
                for (int kb = pc.b0 * GROUPS; kb < pc.b1 * GROUPS; kb++) {                 // past K: zeros
                    wait(&sm->empty[st], ph ^ 1u);
                    unsigned char *dst = xs + (size_t)(st * H) * p.xtile;
                    mbar_arrive_expect_tx(&sm->full[st], (uint32_t)(two ? 2 * p.xtile : p.xtile));
                    tma_load_2d(dst, &xmap, &sm->full[st], kb * KB, m0);
                    if (two) tma_load_2d(dst + p.xtile, &xmap, &sm->full[st], kb * KB, m0 + p.nt);
                    if (++st == p.nst) { st = 0; ph ^= 1u; }
                }
            }
        }
    } else if (warp == 1) {
        // ================= MMA issuer =================
        if (elect_one()) {
            const uint32_t idesc = umma_idesc_f16(TN, p.nt);
            const uint64_t bdesc0 = umma_desc_sw128(smem_u32(xs));
            int st = 0; uint32_t ph = 0;
            bool ready = false;
            Pieces pc(p, cta, G);
            for (int it = 0; pc.next(); it++) {
                const int a = H == 1 ? it & 1 : 0, use = H == 1 ? it >> 1 : it;
                wait(&sm->d_empty[a], (uint32_t)((use & 1) ^ 1));            // the epilogue has drained this accumulator (both)
                const uint32_t d_tmem = tmem + (uint32_t)(a * p.acc_cols);
                const bool two = H == 2 && tile_of(p, pc.t).mt * p.tt + p.nt < p.M;
                uint32_t acc = 0u;
                for (int kb = pc.b0 * GROUPS; kb < pc.b1 * GROUPS; kb++) {
                    if (!ready) wait(&sm->full[st], ph);
                    tc_fence_after();
                    const uint32_t at = tmem + (uint32_t)(2 * p.acc_cols + st * A_STAGE_COLS);
                    const uint64_t bd = bdesc0 + (uint64_t)((st * H * p.xtile) >> 4);
                    const uint32_t acc0 = acc;
                    uint64_t *done = &sm->empty[st];
                    if (++st == p.nst) { st = 0; ph ^= 1u; }
                    ready = mbar_try_wait(&sm->full[st], ph);
#pragma unroll
                    for (int kk = 0; kk < KB / 16; kk++) {
                        umma_f16_ts(d_tmem, at + (uint32_t)(kk * 8), bd + (uint64_t)(2 * kk), idesc, acc);
                        acc = 1u;
                    }
                    if (two) {
                        const uint64_t bd2 = bd + (uint64_t)(p.xtile >> 4);
#pragma unroll
                        for (int kk = 0; kk < KB / 16; kk++)
                            umma_f16_ts(d_tmem + (uint32_t)p.acc_cols, at + (uint32_t)(kk * 8), bd2 + (uint64_t)(2 * kk), idesc, kk == 0 ? acc0 : 1u);
                    }
                    umma_commit(done);
                }
                umma_commit(&sm->d_full[a]);
            }
            umma_commit(&sm->all_done);
        }
    } else {
        const int grp = (warp - 2) >> 2;                 // converter group; GROUPS: the epilogue warps
        if (grp < GROUPS) {
        // ================= converters: packed INT4 (smem) -> FP16 (+ sparse entries) -> A operand in tensor memory =================
        const int q = warp & 3;                          // tensor-memory lane quarter this warp may touch
        const int row = q * 32 + lane;                   // weight row inside the tile
        const uint32_t swz = (uint32_t)((2 * grp) ^ (row & 7)) << 4;      // 128-byte swizzle: 16-byte chunk c sits at c ^ (row & 7)
        const uint32_t ta = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(2 * p.acc_cols);
        const unsigned char *wrow = ws + row * 128;
        int wi = 0, st = grp;                            // slot of the box, stage of the group's unit
        uint32_t wph = 0, ph = 0;
        Walk cur(p, cta, G);
        // the list of the next unit is on its way while this one is converted, its extent is fetched a turn earlier
        Walk ahead = cur;
        int ahead_t = -1;
        const uint32_t *ahead_off = nullptr;             // extents of the row group in that tile
        uint32_t x0 = 0, x1 = 0, n0 = 0, nn = 0, nw = 0;
        auto fetch_extent = [&]() {
            x0 = x1 = 0;
            if (!ahead.ok) return;
            if (ahead.pc.t != ahead_t) {
                ahead_t = ahead.pc.t;
                const int g = tile_of(p, ahead_t).row * 4 + q;
                ahead_off = g < p.ngroups ? p.win_off + (size_t)g * (size_t)(p.kblocks + 1) : nullptr;
            }
            const int kb = ahead.b * GROUPS + grp;
            if (ahead_off && kb < p.kblocks) { x0 = __ldg(ahead_off + kb); x1 = __ldg(ahead_off + kb + 1); }
            ahead.step();
        };
        auto fetch_list = [&]() {
            n0 = x0; nn = x1 - x0;
            if ((uint32_t)lane < nn) nw = __ldg(p.win_words + n0 + lane);
        };
        float rsc = 0.f;
        int cur_t = -1;
        if (SPARSE) { fetch_extent(); fetch_list(); fetch_extent(); }
        for (; cur.ok; cur.step()) {
            uint32_t l0 = 0, ln = 0, lw = 0;
            if (SPARSE) {
                if (cur.pc.t != cur_t) {
                    cur_t = cur.pc.t;
                    const int n = tile_of(p, cur_t).row * TN + row;
                    rsc = n < p.N ? patch_rscale(p.alpha, __half2float(p.scales[n]), p.row_max[n]) : 0.f;
                }
                l0 = n0; ln = nn; lw = nw;
                fetch_list();
                fetch_extent();
            }
            wait(&sm->w_full[wi], wph);
            const uint4 w0 = *reinterpret_cast<const uint4 *>(wrow + (size_t)wi * W_BYTES + swz);
            const uint4 w1 = *reinterpret_cast<const uint4 *>(wrow + (size_t)wi * W_BYTES + (swz ^ 16u));
            const uint32_t ww[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
            uint32_t h[32];
#pragma unroll
            for (int j = 0; j < 8; j++) {
                uint32_t o[4];
                int4x8_to_half2x4_natural(ww[j], o);
                h[4 * j] = o[0]; h[4 * j + 1] = o[1]; h[4 * j + 2] = o[2]; h[4 * j + 3] = o[3];
            }
            if (SPARSE) add_entries(h, lw, ln, p.win_words + l0, rsc, lane);
            wait(&sm->empty[st], ph ^ 1u);
            tc_fence_after();
            __syncwarp();
            tmem_st_32x32b_x32(ta + (uint32_t)(st * A_STAGE_COLS), h);
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) { mbar_arrive(&sm->full[st]); mbar_arrive(&sm->w_empty[wi]); }      // (not before the store: mid.cu)
            if (++wi == p.wst) { wi = 0; wph ^= 1u; }
            st += GROUPS;
            if (st >= p.nst) { st -= p.nst; ph ^= 1u; }
        }
        }
        // The CTA's last piece is finished by the converters too, which have nothing left to do: five sets of four warps take
        // every fifth chunk of 16 tokens.  (Collecting the other pieces of a cut tile is a chain of loads from L2 per chunk: by
        // the four epilogue warps alone it took 15-25 us at the end of a forward.)
        // ================= epilogue: TMEM -> (+ partials) -> scale, bias -> FP16 -> global =================
        if (SPARSE && p.n_long > 0) asm volatile("griddepcontrol.wait;" ::: "memory");       // the long rows' pre-pass
        const int q = warp & 3;                          // TMEM lane quarter of this warp
        const int et = (warp - EPI_WARP0) * 32 + lane;   // 0..127 among the epilogue threads, negative in the converters
        Pieces pc(p, cta, G);
        for (int it = 0; pc.next(); it++) {
            const int a = H == 1 ? it & 1 : 0, use = H == 1 ? it >> 1 : it;
            const bool owner = pc.b0 == 0, last = pc.last();
            if (!last && grp < GROUPS) continue;
            const int set = last ? (grp + 1) % (GROUPS + 1) : 0, sets = last ? GROUPS + 1 : 1;
            auto sync_sets = [&]() { if (last) named_bar_sync(2, (CONV_WARPS + EPI_WARPS) * 32); else named_bar_sync(1, EPI_WARPS * 32); };
            const Tile tile = tile_of(p, pc.t);
            const int n = tile.row * TN + q * 32 + lane;             // weight row of this thread
            const int m0 = tile.mt * p.tt;
            const bool n_ok = n < p.N;
            // contributors: the CTAs behind this one whose share starts inside the same tile
            int c_last = cta;
            if (owner && pc.b1 < p.boxes) {
                const int tile_end = (pc.t - p.tail0 + 1) * p.boxes;
                while (c_last + 1 < p.tail_ctas && p.share * (c_last + 1) + min(c_last + 1, p.extra) < tile_end) c_last++;
            }
            float sc = 0.f, bs = 0.f;
            int e0 = 0, e1 = 0, li = -1;                 // li: this row's index among the long rows; e1 > e0: gather it here
            if (owner && n_ok) {
                sc = __half2float(p.scales[n]);
                if (p.bias) bs = p.bias[n];
                if (SPARSE) {
                    e0 = p.ov.row_ptr[n]; e1 = p.ov.row_ptr[n + 1];
                    if (p.n_long > 0 && e1 - e0 > p.heavy) {
                        int lo = 0, hi = p.n_long - 1;
                        while (lo < hi) {
                            const int mid2 = (lo + hi) >> 1;
                            if (p.hrow[mid2] < n) lo = mid2 + 1; else hi = mid2;
                        }
                        li = lo; e1 = e0;
                    } else if (patch_rscale(p.alpha, sc, p.row_max[n]) != 0.f) {
                        e1 = e0;                         // folded into the weight tile
                    }
                }
            }
            const bool gathers = SPARSE && __any_sync(0xffffffffu, e1 > e0), longs = SPARSE && __any_sync(0xffffffffu, li >= 0);
            const bool n_st = n_ok && li < 0;            // this row goes to y from here
            if (grp < GROUPS) wait(&sm->all_done, 0u); else wait(&sm->d_full[a], (uint32_t)(use & 1));
            __syncwarp();
            tc_fence_after();
            const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(a * p.acc_cols);
            auto col = [&](int c) -> uint32_t { return (uint32_t)(H == 2 && c >= p.nt ? p.acc_cols + c - p.nt : c); };      // of token m0 + c
            if (!owner) {
                // the first piece of a share that starts inside a tile: raw FP32 sums to this CTA's slot, then the flag
                float *dst = p.slots + ((size_t)cta * p.tt + set * 16) * TN + q * 32 + lane;
                for (int c = set * 16; c < p.tt; c += sets * 16, dst += sets * 16 * TN) {
                    uint32_t r[16];
                    tmem_ld_32x32b_x16(taddr + col(c), r);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 16; j++) dst[j * TN] = __uint_as_float(r[j]);
                }
                tc_fence_before();
                __syncwarp();
                if (!last && lane == 0) mbar_arrive(&sm->d_empty[a]);
                __threadfence();
                sync_sets();
                if (et == 0) asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(p.flags + cta), "l"(p.tag) : "memory");
                continue;
            }
            if (c_last > cta) {                          // bounded wait for the contributors' flags, one lane per contributor
                bool ok = true;
                for (int c = cta + 1 + lane; c <= c_last && !dead; c += 32) {
                    unsigned long long seen = 0;
                    for (unsigned spin = 0; spin < (1u << 22); spin++) {
                        asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(seen) : "l"(p.flags + c) : "memory");
                        if (seen == p.tag) break;
                        __nanosleep(32);
                    }
                    ok = ok && seen == p.tag;
                }
                if (!ok) { dead = true; atomicExch(p.status, 1); }
                dead = __any_sync(0xffffffffu, dead);
            }
            const float *part = p.slots + ((size_t)(cta + 1) * p.tt + set * 16) * TN + q * 32 + lane;
            const size_t part_cta = (size_t)p.tt * TN;
            for (int c = set * 16; c < p.tt && m0 + c < p.M; c += sets * 16, part += sets * 16 * TN) {
                __syncwarp();
                uint32_t r[16];
                tmem_ld_32x32b_x16(taddr + col(c), r);
                tmem_ld_wait();
                const float *src = part;
                for (int cc = cta + 1; cc <= c_last; cc++, src += part_cta) {        // the other pieces of the tile, in CTA order
                    float t[16];
#pragma unroll
                    for (int j = 0; j < 16; j++) t[j] = __ldcg(src + j * TN);
#pragma unroll
                    for (int j = 0; j < 16; j++) r[j] = __float_as_uint(__uint_as_float(r[j]) + t[j]);
                }
#pragma unroll
                for (int j = 0; j < 16; j++) r[j] = __float_as_uint(fmaf(__uint_as_float(r[j]), sc, bs));
                if (longs && li >= 0) {                  // a long row: its other sums are added by long_finish_kernel
                    float4 *dst = reinterpret_cast<float4 *>(p.rest + (size_t)li * p.rest_mp + m0 + c);      // (rows of 256 tokens a time)
#pragma unroll
                    for (int j = 0; j < 4; j++)
                        dst[j] = make_float4(__uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1]), __uint_as_float(r[4 * j + 2]),
                                             __uint_as_float(r[4 * j + 3]));
                }
                if (gathers && e1 > e0) {                // outside the FP16 range of the weight tile: straight from x
#pragma unroll 1
                    for (int e = e0; e < e1; e++) {
                        int k; float ev;
                        ortho_entry(p.ov, e, p.K, k, ev);
                        ev *= p.alpha;
#pragma unroll
                        for (int j = 0; j < 16; j++)
                            if (m0 + c + j < p.M)
                                r[j] = __float_as_uint(fmaf(ev, __half2float(p.x[(size_t)(m0 + c + j) * p.K + k]), __uint_as_float(r[j])));
                    }
                }
                if (TYPED) {
                    store_column<16>(p.y, (size_t)(m0 + c) * (size_t)p.ldy + n, p.ldy, p.y_type, p.M - m0 - c, n_st,
                                     [&](int j) { return __uint_as_float(r[j]); });
                    continue;
                }
                __half *yp = p.y + (size_t)(m0 + c) * (size_t)p.ldy + n;
#pragma unroll
                for (int j = 0; j < 16; j++) {
                    if (n_st && m0 + c + j < p.M) *yp = __float2half_rn(__uint_as_float(r[j]));
                    yp += p.ldy;
                }
            }
            __syncwarp();
            tc_fence_before();
            if (!last && lane == 0) mbar_arrive(&sm->d_empty[a]);
            if (c_last > cta) {                          // every reader is past the flags: clear them (a replayed graph brings the same tag)
                sync_sets();
                if (et >= 0)
                    for (int c = cta + 1 + et; c <= c_last; c += EPI_WARPS * 32) p.flags[c] = 0ull;
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem, TMEM_COLS); }
}

// partial sums of the cut tiles, then the flags
constexpr int kWideMaxSms = 148;
constexpr int64_t kWideSlotBytes = (int64_t)kWideMaxSms * (wd::kTMax<true> * wd::kHalves<true>) * wd::TN * 4;
int64_t wide_split_bytes() { return kWideSlotBytes + 2048; }

// A call without peer exchange whose sparse term is inactive or listed; `long_off` = offset of the long rows' shares in the
// workspace (launch_prefill has checked that they fit).
int launch_wide(const FwdArgs &a, int64_t long_off)
{
    using namespace wd;
    const int dev = current_device_index();
    if (dev < 0) return ORTHO_B200_ERR_CUDA;
    int num_sms = device_sm_count(dev);
    if (num_sms > kWideMaxSms) num_sms = kWideMaxSms;
    Params p;
    memset(&p, 0, sizeof(p));
    p.scales = a.scales; p.bias = a.bias; p.y = a.y; p.M = (int)a.M; p.K = (int)a.K; p.N = (int)a.N; p.ldy = a.pitch_y(); p.y_type = a.y_type;
    const bool sparse = a.has_ortho != 0;
    const int halves = sparse ? kHalves<true> : kHalves<false>, tmax = sparse ? kTMax<true> : kTMax<false>;
    p.tiles_m = (int)ceil_div(a.M, halves * tmax);
    p.nt = (int)(ceil_div(ceil_div(a.M, p.tiles_m * halves), 16) * 16);
    p.tt = halves * p.nt;
    p.tiles_m = (int)ceil_div(a.M, p.tt);                // (the rounding may have saved one)
    p.tiles_n = (int)ceil_div(a.N, TN); p.kblocks = (int)ceil_div(a.K, KB); p.boxes = (int)ceil_div(a.K, KC);
    // a band's activations take up to 48 of the 126 MB of L2
    p.band = (int)((48ll << 20) / ((int64_t)p.tt * a.K * 2));
    if (p.band < 1) p.band = 1;
    if (p.band > p.tiles_m) p.band = p.tiles_m;
    p.acc_cols = (p.nt + 31) / 32 * 32;
    p.xtile = p.nt * 128;
    p.nst = (TMEM_COLS - 2 * p.acc_cols) / A_STAGE_COLS;
    if (p.nst > ST_MAX) p.nst = ST_MAX;
    while (p.nst > GROUPS && kSmemData - p.nst * halves * p.xtile < 3 * W_BYTES) p.nst--;
    p.wst = (kSmemData - p.nst * halves * p.xtile) / W_BYTES;
    if (p.wst > WST_MAX) p.wst = WST_MAX;
    if (p.nst < GROUPS || p.wst < 3) return ORTHO_B200_ERR_SHAPE;                    // not reached for nt in 16..192 / 16..176
    p.alpha = a.alpha;
    p.status = kernel_status_word();
    if (!p.status) return ORTHO_B200_ERR_CUDA;
    int64_t off = 0;                                     // workspace already spoken for
    if (sparse) {
        p.win_off = a.plan->win_off; p.win_words = a.plan->win_words; p.ngroups = (int)ceil_div(a.N, kWinRows);
        p.ov = a.ortho; p.row_max = a.plan->row_max; p.x = a.x;
        if (a.plan->n_long > 0) {
            p.hrow = a.plan->hrow; p.n_long = (int)a.plan->n_long; p.heavy = a.plan->heavy;
            off = long_off + long_rows_workspace_bytes(a.plan, a.M);
        }
    }
    const int64_t tiles = (int64_t)p.tiles_n * p.tiles_m;
    if (tiles > 0x7fffffffLL) return ORTHO_B200_ERR_SHAPE;
    const int rest = (int)(tiles % num_sms);             // tiles beyond whole waves
    const bool room = a.workspace && ((uintptr_t)a.workspace & 255u) == 0 && a.workspace_bytes >= off + wide_split_bytes();
    p.full = (int)(tiles / num_sms);
    p.tail0 = (int)(tiles - rest);
    p.tail_ctas = rest; p.share = p.boxes; p.extra = 0;            // one more wave, a tile each
    if (rest > 0 && room) {
        // at most eight pieces per tile, of two boxes at the least: the collecting CTA reads nt x 512 bytes per piece
        const int64_t units = (int64_t)rest * p.boxes, least = p.boxes / 8 > 2 ? p.boxes / 8 : 2;
        const int64_t cut = units / least < num_sms ? units / least : num_sms;
        if (cut > rest) {
            p.tail_ctas = (int)cut; p.share = (int)(units / cut); p.extra = (int)(units % cut);
            unsigned char *b = reinterpret_cast<unsigned char *>(a.workspace) + off;
            p.slots = reinterpret_cast<float *>(b);
            p.flags = reinterpret_cast<unsigned long long *>(b + kWideSlotBytes);
            p.tag = next_launch_tag();
        }
    }
    const int grid = p.full > 0 ? num_sms : p.tail_ctas;
    CUtensorMap xmap, wmap;
    if (!make_tensor_map_2d(&xmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, a.x, (uint64_t)a.M, (uint64_t)a.K,
                            (uint64_t)a.K * 2, (uint32_t)p.nt, KB, CU_TENSOR_MAP_SWIZZLE_128B))
        return ORTHO_B200_ERR_CUDA;
    if (!make_tensor_map_2d(&wmap, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, a.w, (uint64_t)a.N, (uint64_t)(a.K / 2),
                            (uint64_t)(a.K / 2), TN, KC / 2, CU_TENSOR_MAP_SWIZZLE_128B))
        return ORTHO_B200_ERR_CUDA;
    static bool attr_set[kMaxDevices] = {};
    if (!attr_set[dev]) {
        for (auto k : {wide_kernel<false, false>, wide_kernel<true, false>, wide_kernel<false, true>, wide_kernel<true, true>})
            OB_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes));
        attr_set[dev] = true;
    }
    if (p.n_long > 0) {
        void *lw = reinterpret_cast<unsigned char *>(a.workspace) + long_off;
        p.rest_mp = (int)(ceil_div(a.M, 256) * 256);
        p.rest = long_rows_rest(a, p.rest_mp, lw);
        const int st = launch_long_rows(a, p.rest_mp, lw, nullptr);
        if (st != ORTHO_B200_OK) return st;
    }
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3((unsigned)grid); cfg.blockDim = dim3(NWARPS * 32); cfg.dynamicSmemBytes = kSmemBytes; cfg.stream = a.stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
    const bool typed = p.y_type != kTypeF16;
    OB_CUDA(cudaLaunchKernelEx(&cfg, sparse ? (typed ? wide_kernel<true, true> : wide_kernel<true, false>)
                                            : (typed ? wide_kernel<false, true> : wide_kernel<false, false>), xmap, wmap, p));
    count_launch();
    if (p.n_long > 0) return launch_long_finish(a, p.rest_mp, reinterpret_cast<unsigned char *>(a.workspace) + long_off);
    return ORTHO_B200_OK;
}

}  // namespace ob
