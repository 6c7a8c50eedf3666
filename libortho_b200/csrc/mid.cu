// Forward for a few tokens up to 128 on the 5th-generation tensor cores.  The WEIGHT tile is the M operand of the MMA
// (128 rows, converted into tensor memory) and the token block its N operand (M rounded up to 16).
//
//     D[n, m] = sum_k w_int[n, k] * x[m, k]        (tcgen05.mma, A in tensor memory, B in shared memory, FP32 in TMEM)
//     y[m, n] = scale[n] * D[n, m] + alpha * O[m, n] + bias[n]
//
// Why this way round: a 128 x N x 16 tcgen05.mma with A in tensor memory takes N / 2 cycles (N = 16: 10, 32: 16, 64: 32,
// 128: 64 measured, issued from an elected lane), so few tokens cost few cycles and the pipe is never the bound below
// 64 tokens: HBM delivers the 4 KB of a k block (128 rows x 64 k) in about 180 cycles per SM.  Converted weights go
// from registers straight to tensor memory; the form before this one (tokens as the M operand, weights converted into
// a shared-memory B tile of 256 rows) spent 512 cycles of tensor pipe per 256 x 64 weights whatever the token count
// and 4 bytes of shared-memory traffic per weight.
// What bounds it, by the counters of one launch on 8192->10240 at 32 tokens with 0.3 % entries (base-only): no pipe is full.  Of
// the active cycles the integer pipe is busy in 49 % (48), the issue slots in 59 % (54), the tensor pipe in 26 % (16), HBM in
// 20 % (24) of the whole time; a unit's MMAs take some 450 cycles to go through (8 from shared memory at 40, 8 at 16), 45 % of the active cycles.
// The rest is ramp, the waits between the warp roles and the collecting of cut tiles.
// One B200, us, base-only / with entries, weights rotating over more than L2; in brackets with one issuer, weights loaded behind
// the predecessor and the cut tiles collected 16 tokens and one piece at a time: 8192->10240 at 32 tokens 16.0 / 20.3 (17.4 / 22.4),
// 4096->22016 at 16 14.1 / 19.0 (16.1 / 20.8), 4096->4096 at 24 7.8 / 10.0 (10.6 / 12.1), 28672->8192 at 32 37 / 49 (41 / 52).
// 33 tokens on with entries, as 65 on without, one issuer is enough: 4096->22016 with 0.5 % at 48 / 96 / 128 24.3 / 35 / 43 (27.5 / 36 / 43),
// 4096->4096 at 64 / 128 11.8 / 15.7 (13.4 / 17.3).
// Long calls run into the power cap: 28672->8192 at 100 tokens 46 / 73-78 for the first milliseconds at 1.9 GHz, 56 / 85 after that at
// 1.43 GHz, of which the 97 units of both contractions (960 cycles each) take 47 and 65 with entries.
// Replaces, for this token range, the reference's one-thread-per-output kernel (src/dual_gemm.cu:176-225) and its WMMA
// variant (src/dual_gemm_tensor_core.cu:215-337).
//
// The pipeline's unit is a k pair (two k blocks, 128 rows x 128 k): 8 KB of packed INT4 come in by TMA (64-byte rows and
// swizzle), two token tiles of 64 k with them, and the result is 64 tensor-memory columns of weights and 8 MMAs.  Sixteen
// converter warps form groups that take units in turn (thread = weight row), so several units are in work at any time
// and no warp waits for another group's conversion.  Two accumulators alternate, so the epilogue of one piece runs under
// the MMAs of the next.  Epilogue thread = weight row, columns = tokens: a warp stores 32 consecutive outputs of a token
// at a time, no transposition.
//
// Work split (stream-K): the sequence of all (row tile, k pair) units is cut into one contiguous share per
// CTA, so every SM does the same number of k pairs however few row tiles the layer has.  A CTA whose share starts
// inside a row tile leaves that tile's partial FP32 sums in its slot of the workspace and raises a flag; the CTA
// that holds the tile's first k pair adds the partials of the CTAs behind it, in CTA order (fixed order:
// reproducible), in its epilogue.  A share's partial piece is processed first and the piece that collects partials
// last, so the bounded flag wait does not normally wait for long.
//
// The sparse term is a second contraction over the same token tiles, E[n, m] = sum_k v[n, k] * x[m, k], with its own
// accumulator: y = scale * D + alpha * E + bias, so the stored FP16 values enter exactly.  With a plan whose rows are in
// column order four warps scatter the entries of a unit (window lists, windows.cuh) as FP16 into a zeroed
// shared-memory tile of 128 rows x 128 k, lane = entry, and take them out again once the MMAs have read it; the A operand
// of those MMAs comes from that tile (40 to 64 cycles per K = 16, whatever the density).  Adding the entries to the
// converted weights in registers, a round of predicated additions per entry and row, doubled the work of the
// converters, whose integer and FP16 pipes are the bound: 8192->57344 at 32 tokens and 0.3 % took 122 us that way against
// 64 base-only, 84 with the scattered tiles.  The plan's long rows come from the tensor-core pre-pass of longrows.cu.
// Without such a plan the term is computed ahead into O[m][n] (token-major FP32, in the workspace) by
// ortho_tokens_kernel from the once-transposed activations (a warp per 8 weight rows, lanes = tokens) and added in
// the FP32 epilogue.
#include <cstring>

#include "common.cuh"
#include "gather.cuh"
#include "umma.cuh"
#include "windows.cuh"

namespace ob {

int *kernel_status_word();
int launch_transpose_x(const __half *x, __half *xt, int M, int K, int Mp, cudaStream_t stream);   // transpose.cu

namespace md {
constexpr int TN = 128;                 // weight rows per tile (MMA M)
constexpr int TMK = 128;                // most tokens (MMA N)
constexpr int KB = 64;                  // k block: one 128-byte swizzled token tile, one window of the sparse lists
constexpr int KP = 128;                 // k pair: the pipeline's unit and the unit of the work split
constexpr int W_BYTES = TN * KP / 2;    // 8 KB
constexpr int A_STAGE_COLS = KP / 2;    // tensor-memory columns of a stage's converted weights
constexpr int ST_MAX = 7, ST_SPARSE_MAX = 4, WST_MAX = 20;
static_assert(kWinTile == TN * KB * 2 && kWinRows == 32, "places of the window lists");
constexpr int S_BYTES = TN * KP * 2;    // 32 KB: a stage's sparse tile, two k blocks of 128 rows x 128 B (128-byte swizzle)
constexpr int kSmemData = 224 * 1024;   // packed-weight slots, token stages, sparse tiles
// Converter warps form groups of four (thread = row) that take the CTA's units in turn, as many groups (Params::groups)
// as the stages allow.  A parity wait is only sound for a waiter at most one phase ahead of the barrier.  A group comes
// back after `groups` units, so stages must be at least that many (the unit before it in its stage is one whose
// MMAs its own last store had waited for), and weight slots at least stages + groups: having stored unit i, a group knows
// that units up to i - stages have been multiplied, hence loaded, and waits for unit i + groups next, whose slot's previous
// load (i + groups - slots) must be one of those -- loads may complete out of order.  With two issuers it knows so only of
// every other unit: numbers of slots, stages and groups are even then, and i + groups - slots is one of those.
constexpr int MAX_GROUPS = 4;
constexpr int CONV_WARPS = 4 * MAX_GROUPS;
constexpr int EPI_WARP0 = 2 + CONV_WARPS;
constexpr int EPI_WARPS = 4;
constexpr int XPROD_WARP = EPI_WARP0 + EPI_WARPS;   // token tiles have a producer of their own: the packed weights run ahead of them
constexpr int SCAT_WARP0 = XPROD_WARP + 1;
constexpr int SCAT_WARPS = 8;           // two sets of four that take the units in turn; a warp of a set has 32 rows of the tile
template <bool SPARSE> constexpr int kIssue2Warp = SCAT_WARP0 + (SPARSE ? SCAT_WARPS : 0);    // the second MMA issuer, where there are two
template <bool SPARSE, int ISSUERS> constexpr int kWarps = kIssue2Warp<SPARSE> + ISSUERS - 1;
constexpr int TMEM_COLS = 512;
constexpr int kTwoIssuers = 64, kTwoIssuersSparse = 32;      // two issuers up to this many columns of D (with more, shared
                                        // memory does not hold four stages with their sparse tiles)

struct Params {
    const __half *scales; const float *bias; __half *y;
    int y_type;                 // kTypeF16 ..: what y points to
    int M, K, N;
    long long ldy;
    int tiles_n, kblocks, kpairs;
    int share, extra;           // units per CTA: share, and one more for the first `extra` CTAs
    int nt;                     // token columns of an MMA: M rounded up to 16
    int nt32;                   // nt rounded up to 32: columns kept for D, and for E behind it
    int nacc, acc_cols;         // accumulators (2 where tensor memory allows) and the columns of one
    int issuers;                // threads that issue MMAs, in turns, each with accumulators of its own (host side: ISSUERS)
    int xtile;                  // bytes of a token tile (nt x 128); a stage holds two
    int nst;                    // stages: a unit's converted weights and tokens
    int wst;                    // packed-weight slots
    int groups;                 // converter groups at work
    int sets;                   // scatter sets at work: 2 with two or four stages, else 1
    float *slots;               // slots[cta][nt][128]: partial sums handed to another CTA ...
    unsigned long long *flags;  // ... and flags[cta] = tag once they are there (see launch_mid)
    unsigned long long tag;
    const float *o; float alpha; int has_ortho;    // O[m][n], row pitch N
    // sparse instantiation (a plan with ordered rows): the window lists; long rows are read from the pre-pass's sums
    const uint32_t *win_off, *win_words; int ngroups;
    const int32_t *row_ptr; const float *ol; int ol_mp; const int32_t *hrow; int n_long, heavy;
    const uint32_t *entries; const __half *x;      // the plan's entries, for sums that an infinite activation made NaN
    int *status;
    int gather;
    GatherView gv;
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

// the pieces of a CTA's share, in order: row tile t, k pairs [kp0, kp1)
struct Pieces {
    int t, kp0, kp1, left, kpairs;
    __device__ __forceinline__ Pieces(int t0, int kp, int units, int kpairs_) : t(t0 - 1), kp0(0), kp1(kp), left(units), kpairs(kpairs_) {}
    __device__ __forceinline__ bool next()
    {
        if (left <= 0) return false;
        t++;
        kp0 = kp1 == kpairs ? 0 : kp1;
        kp1 = kpairs - kp0 < left ? kpairs : kp0 + left;
        left -= kp1 - kp0;
        return true;
    }
};
}  // namespace md

// SPARSE: the entries of an ordered plan are contracted from the scattered tiles; at most 4 stages then.  TYPED: y is of another type
// than FP16 (an instantiation of its own: the branch cost the others 1-2 %).  ISSUERS: threads that issue MMAs; with the number as a
// parameter of the launch, calls of one issuer paid for the second one's code (4096->22016 with 0.5 % at 96 / 128 tokens 37.9 / 45.5 us
// against 37.3 / 44.8) and had its narrow epilogue.
template <bool SPARSE, bool TYPED, int ISSUERS>
__global__ void __launch_bounds__(md::kWarps<SPARSE, ISSUERS> * 32, 1)
mid_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap wmap, const md::Params p)
{
    using namespace md;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char *base = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    unsigned char *ws = base;
    unsigned char *xs = ws + (size_t)p.wst * W_BYTES;
    unsigned char *ss = base + (size_t)kSmemData - (size_t)p.nst * S_BYTES;      // SPARSE only
    Smem *sm = reinterpret_cast<Smem *>(base + (size_t)kSmemData);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int cta = blockIdx.x, G = gridDim.x;
    const int units = p.share + (cta < p.extra ? 1 : 0);
    const int r_begin = p.share * cta + min(cta, p.extra);
    const int t_begin = r_begin / p.kpairs, kp_begin = r_begin - t_begin * p.kpairs;

    if (threadIdx.x == 0) {
        for (int s = 0; s < WST_MAX; s++) { mbar_init(&sm->w_full[s], 1); mbar_init(&sm->w_empty[s], 4); }
        // full: the four warps of a converter group, the token producer with its bytes, a set of scatter warps
        for (int s = 0; s < ST_MAX; s++) { mbar_init(&sm->full[s], 5 + (SPARSE ? 4 : 0)); mbar_init(&sm->empty[s], 1); }
        for (int s = 0; s < 2; s++) { mbar_init(&sm->d_full[s], ISSUERS); mbar_init(&sm->d_empty[s], EPI_WARPS); }
        mbar_init(&sm->all_done, ISSUERS);
        fence_mbar_init();
        prefetch_tensormap(&xmap);
        prefetch_tensormap(&wmap);
    }
    if (warp == 1) { tmem_alloc(&sm->tmem_base, TMEM_COLS); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sm->tmem_base;
    // The kernel is a programmatic dependent of whatever precedes it on the stream and runs beside that kernel's tail: weights
    // and window lists, constants of the layer, are loaded and converted at once; the token producer and the epilogue wait.
    // Behind the long rows' pre-pass (an ordinary launch, so all earlier work is done) only the epilogue does.
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    // The roles that run ahead come to wait for units that the predecessor's end holds up, and it may take any time: a wait that runs
    // out starts anew behind that end (here, off the roles' loops: a wait for the predecessor inside them cost 1-2 %).
    bool dead = false;
    auto wait = [&](uint64_t *bar, uint32_t parity) {
        if (mbar_try_wait(bar, parity) || dead) return;
#pragma unroll 1
        for (uint32_t i = 0; !mbar_try_wait(bar, parity); i++) {
            if ((i & 0xFFFFFFu) == 0xFFFFFFu) {
                asm volatile("griddepcontrol.wait;" ::: "memory");
                if (i >> 24) { dead = true; atomicExch(p.status, 1); return; }       // the second time
            }
        }
    };

    if (warp == 0) {
        // ================= TMA producer: packed weights =================
        if (elect_one()) {
            int wi = 0; uint32_t wph = 0;
            int t = t_begin, kp = kp_begin;
            for (int i = 0; i < units; i++) {
                wait(&sm->w_empty[wi], wph ^ 1u);
                mbar_arrive_expect_tx(&sm->w_full[wi], W_BYTES);
                tma_load_2d(ws + (size_t)wi * W_BYTES, &wmap, &sm->w_full[wi], kp * (KP / 2), t * TN);
                if (++wi == p.wst) { wi = 0; wph ^= 1u; }
                if (++kp == p.kpairs) { kp = 0; t++; }
            }
        }
    } else if (warp == XPROD_WARP) {
        // ================= TMA producer: token tiles =================
        if (elect_one()) {
            if (!SPARSE || p.n_long == 0) asm volatile("griddepcontrol.wait;" ::: "memory");
            int st = 0; uint32_t ph = 0;
            int kp = kp_begin;
            for (int i = 0; i < units; i++) {
                wait(&sm->empty[st], ph ^ 1u);
                unsigned char *dst = xs + (size_t)(2 * st) * p.xtile;
                mbar_arrive_expect_tx(&sm->full[st], (uint32_t)(2 * p.xtile));
                tma_load_2d(dst, &xmap, &sm->full[st], kp * KP, 0);
                tma_load_2d(dst + p.xtile, &xmap, &sm->full[st], kp * KP + KB, 0);         // past K: zeros
                if (++st == p.nst) { st = 0; ph ^= 1u; }
                if (++kp == p.kpairs) kp = 0;
            }
        }
    } else if (warp == 1 || (ISSUERS == 2 && warp == kIssue2Warp<SPARSE>)) {
        // ================= MMA issuers =================
        // A ready mbarrier takes this one thread 60-100 cycles to see and a commit 35-60: with a wait each for tokens
        // and weights and two commits per 64 k the loop took 490 cycles per k block whatever the token count.  Hence one
        // barrier for all operands, two k blocks per turn, a look at the next stage's barrier before this stage's MMAs are issued,
        // and up to 64 tokens two threads that take the units in turn, each into accumulators of its own: by clocks at 32 tokens
        // one thread took 500-530 cycles a unit base-only (750 with the sparse term) while converted units piled up, for MMAs
        // of 130 (450).  (One thread for D and one for E: slower than one for both.  A loop that the whole warp runs, with an
        // elected lane for the MMAs alone: 8192->57344 at 32 tokens 65 us against 60.)  The number of stages is even then, so that a
        // stage is always the same thread's and its waits stay within one phase.
        const int who = ISSUERS == 1 || warp == 1 ? 0 : 1;
        if (elect_one()) {
            constexpr int step = ISSUERS;
            const uint32_t idesc = umma_idesc_f16(TN, p.nt);
            const uint64_t bdesc0 = umma_desc_sw128(smem_u32(xs)), sdesc0 = umma_desc_sw128(smem_u32(ss));
            const uint32_t a_tmem = tmem + (uint32_t)(p.nacc * p.acc_cols);
            int st = who; uint32_t ph = 0;
            bool ready = false;
            Pieces pc(t_begin, kp_begin, units, p.kpairs);
            int skip = st;                               // units to pass over: every other one belongs to the other thread
            for (int it = 0; pc.next(); it++) {
                const int a = p.nacc == 2 ? it & 1 : 0, use = p.nacc == 2 ? it >> 1 : it;
                wait(&sm->d_empty[a], (uint32_t)((use & 1) ^ 1));            // the epilogue has drained this accumulator
                const uint32_t d_tmem = tmem + (uint32_t)(a * p.acc_cols + who * (SPARSE ? 2 : 1) * p.nt32);
                uint32_t acc = 0u;
                int kp = pc.kp0 + skip;
                for (; kp < pc.kp1; kp += step) {
                    if (!ready) wait(&sm->full[st], ph);
                    tc_fence_after();
                    const uint32_t at = a_tmem + (uint32_t)(st * A_STAGE_COLS);
                    const uint64_t sd = sdesc0 + (uint64_t)((st * S_BYTES) >> 4);
                    const uint64_t bd = bdesc0 + (uint64_t)((2 * st * p.xtile) >> 4);
                    const uint64_t bd2 = bd + (uint64_t)(p.xtile >> 4);
                    uint64_t *done = &sm->empty[st];
                    st += step;
                    if (st >= p.nst) { st -= p.nst; ph ^= 1u; }
                    ready = mbar_test_wait(&sm->full[st], ph);
                    const uint32_t acc_e = acc;
#pragma unroll
                    for (int kk = 0; kk < KB / 16; kk++) {
                        umma_f16_ts(d_tmem, at + (uint32_t)(kk * 8), bd + (uint64_t)(2 * kk), idesc, acc);
                        acc = 1u;
                    }
#pragma unroll
                    for (int kk = 0; kk < KB / 16; kk++)
                        umma_f16_ts(d_tmem, at + (uint32_t)(KB / 2 + kk * 8), bd2 + (uint64_t)(2 * kk), idesc, 1u);
                    if constexpr (SPARSE) {
#pragma unroll
                        for (int kk = 0; kk < KB / 16; kk++)
                            umma_f16_ss(d_tmem + (uint32_t)p.nt32, sd + (uint64_t)(2 * kk), bd + (uint64_t)(2 * kk), idesc, kk == 0 ? acc_e : 1u);
#pragma unroll
                        for (int kk = 0; kk < KB / 16; kk++)
                            umma_f16_ss(d_tmem + (uint32_t)p.nt32, sd + (uint64_t)(S_BYTES / 32 + 2 * kk), bd2 + (uint64_t)(2 * kk), idesc, 1u);
                    }
                    umma_commit(done);
                }
                skip = kp - pc.kp1;
                umma_commit(&sm->d_full[a]);
            }
            umma_commit(&sm->all_done);
        }
    } else if (SPARSE && warp >= SCAT_WARP0) {
        // ================= scatter: the unit's sparse entries -> zeroed FP16 tile in shared memory (A operand) =================
        // A warp's loop is a chain of dependent instructions, so the entries come with their place in the tile worked out,
        // are fetched a turn ahead (their extent a turn before that), and stay in registers until they are taken out again.
        // With three stages a stage would pass from set to set, so one set does it all (Params::sets).
        const int q = (warp - SCAT_WARP0) & 3, set = (warp - SCAT_WARP0) >> 2, sets = p.sets;
        int t = t_begin, kp = kp_begin + set, left = units - set;        // unit whose extent is fetched next
        while (kp >= p.kpairs) { kp -= p.kpairs; t++; }
        uint32_t x0 = 0, x1 = 0;                         // that extent
        auto fetch_extent = [&]() {
            x0 = x1 = 0;
            const int g = 4 * t + q;
            if (left > 0 && g < p.ngroups) {
                const uint32_t *o = p.win_off + (size_t)g * (size_t)(p.kblocks + 1) + 2 * kp;
                x0 = __ldg(o);
                x1 = __ldg(o + (2 * kp + 1 < p.kblocks ? 2 : 1));
            }
            left -= sets;
            kp += sets;
            while (kp >= p.kpairs) { kp -= p.kpairs; t++; }
        };
        uint32_t n0 = 0, nn = 0, na = 0, nb = 0;         // the next unit: first entry, count, this lane's first two
        auto fetch_entries = [&]() {
            n0 = x0; nn = x1 - x0;
            if ((uint32_t)lane < nn) na = __ldg(p.win_words + n0 + lane);
            if ((uint32_t)lane + 32u < nn) nb = __ldg(p.win_words + n0 + 32 + lane);
        };
        fetch_extent();
        fetch_entries();
        fetch_extent();
        // what the last three visits put into their stages; a stage comes round after nst / sets visits, 1 to 3
        const int back = p.nst / sets;
        uint32_t o1n = 0, o1a = 0, o1b = 0, o2n = 0, o2a = 0, o2b = 0, o3n = 0, o3a = 0, o3b = 0;
        const uint32_t tiles = smem_u32(ss) + (uint32_t)(q * (32 * 128));
        auto put = [&](uint32_t addr, uint32_t v) { asm volatile("st.shared.u16 [%0], %1;" ::"r"(addr), "h"((unsigned short)v) : "memory"); };
        int st = set; uint32_t ph = 0;                   // nst is 2 or more
        for (int i = set; i < units && set < sets; i += sets) {
            const uint32_t first = n0, count = nn, a = na, b = nb;
            fetch_entries();
            fetch_extent();
            const uint32_t tile = tiles + (uint32_t)(st * S_BYTES);
            auto clear_all = [&]() {
                for (int j = lane; j < 2 * 32 * 8; j += 32)
                    *reinterpret_cast<uint4 *>(ss + (size_t)st * S_BYTES + q * (32 * 128) + (j >> 8) * kWinTile + (j & 255) * 16) = make_uint4(0, 0, 0, 0);
            };
            if (i < p.nst) clear_all();                  // the stage's first use
            const uint32_t on = back == 1 ? o1n : back == 2 ? o2n : o3n, oa = back == 1 ? o1a : back == 2 ? o2a : o3a;
            const uint32_t ob2 = back == 1 ? o1b : back == 2 ? o2b : o3b;
            wait(&sm->empty[st], ph ^ 1u);
            __syncwarp();
            if ((uint32_t)lane < on) put(tile + (oa & 0xFFFFu), 0u);
            if (on > 32u) {
                if (on <= 64u) {
                    if ((uint32_t)lane + 32u < on) put(tile + (ob2 & 0xFFFFu), 0u);
                } else {
                    clear_all();
                }
            }
            __syncwarp();
            if ((uint32_t)lane < count) put(tile + (a & 0xFFFFu), a >> 16);
            if (count > 32u) {
                if ((uint32_t)lane + 32u < count) put(tile + (b & 0xFFFFu), b >> 16);
                for (uint32_t j = 64 + lane; j < count; j += 32) {
                    const uint32_t e = __ldg(p.win_words + first + j);
                    put(tile + (e & 0xFFFFu), e >> 16);
                }
            }
            fence_proxy_async();                         // the tensor core reads shared memory through the async proxy
            __syncwarp();
            if (lane == 0) mbar_arrive(&sm->full[st]);
            o3n = o2n; o3a = o2a; o3b = o2b; o2n = o1n; o2a = o1a; o2b = o1b; o1n = count; o1a = a; o1b = b;
            st += sets;
            if (st >= p.nst) { st -= p.nst; ph ^= 1u; }
        }
    } else {
        const int grp = (warp - 2) >> 2;                 // converter group; MAX_GROUPS: the epilogue warps
        if (grp < p.groups) {
        // ================= converters: packed INT4 (smem) -> FP16 -> A operand in tensor memory =================
        const int q = warp & 3;                          // tensor-memory lane quarter this warp may touch
        const int row = q * 32 + lane;                   // weight row inside the tile
        const uint32_t swz = (uint32_t)((row >> 1) & 3) << 4;     // 64-byte swizzle: 16-byte chunk c sits at c ^ ((row >> 1) & 3)
        const uint32_t ta = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(p.nacc * p.acc_cols);
        const unsigned char *wrow = ws + row * (KP / 2);
        int wi = grp, st = grp;                          // slot and stage of the group's unit
        uint32_t wph = 0, ph = 0;
        for (int i = grp; i < units; i += p.groups) {
            wait(&sm->w_full[wi], wph);
#pragma unroll
            for (int half = 0; half < 2; half++) {
                const uint4 w0 = *reinterpret_cast<const uint4 *>(wrow + (size_t)wi * W_BYTES + ((uint32_t)(32 * half) ^ swz));
                const uint4 w1 = *reinterpret_cast<const uint4 *>(wrow + (size_t)wi * W_BYTES + ((uint32_t)(32 * half + 16) ^ swz));
                const uint32_t ww[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
                uint32_t h[32];
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    uint32_t o[4];
                    int4x8_to_half2x4_natural(ww[j], o);
                    h[4 * j] = o[0]; h[4 * j + 1] = o[1]; h[4 * j + 2] = o[2]; h[4 * j + 3] = o[3];
                }
                if (half == 0) {
                    wait(&sm->empty[st], ph ^ 1u);
                    tc_fence_after();
                }
                __syncwarp();
                tmem_st_32x32b_x32(ta + (uint32_t)(st * A_STAGE_COLS + half * (KB / 2)), h);
            }
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            // The slot is given back here and not right behind the loads above: an arrive does not wait for loads in flight,
            // and with the tensor core reading shared memory hard the next TMA box was seen to overtake them.
            if (lane == 0) { mbar_arrive(&sm->full[st]); mbar_arrive(&sm->w_empty[wi]); }
            wi += p.groups;
            if (wi >= p.wst) { wi -= p.wst; wph ^= 1u; }
            st += p.groups;
            if (st >= p.nst) { st -= p.nst; ph ^= 1u; }
        }
        }
        // The CTA's last piece is finished by the converters too, which have nothing left to do: five sets of four warps take
        // every fifth chunk of tokens.  (Collecting the other pieces of a cut tile is a chain of loads from L2 per chunk: by
        // the four epilogue warps alone it took 15-25 us at the end of a forward.)
        // ================= epilogue: TMEM -> (+ partials) -> scale, sparse term, bias -> FP16 -> global =================
        asm volatile("griddepcontrol.wait;" ::: "memory");
        const int q = warp & 3;                          // TMEM lane quarter of this warp
        const int et = (warp - EPI_WARP0) * 32 + lane;   // 0..127 among the epilogue threads, negative in the converters
        Pieces pc(t_begin, kp_begin, units, p.kpairs);
        int pos = r_begin;                               // first unit of the current piece
        for (int it = 0; pc.next(); it++) {
            const int a = p.nacc == 2 ? it & 1 : 0, use = p.nacc == 2 ? it >> 1 : it;
            const bool owner = pc.kp0 == 0, last = pc.left == 0;
            if (!last && grp < MAX_GROUPS) { pos += pc.kp1 - pc.kp0; continue; }
            const int set = last ? (grp + 1) % (MAX_GROUPS + 1) : 0, sets = last ? MAX_GROUPS + 1 : 1;
            auto sync_sets = [&]() { if (last) named_bar_sync(2, (CONV_WARPS + EPI_WARPS) * 32); else named_bar_sync(1, EPI_WARPS * 32); };
            const int n = pc.t * TN + q * 32 + lane;     // weight row of this thread
            const bool n_ok = n < p.N;
            // contributors: the CTAs behind this one whose share starts inside the same row tile
            int c_last = cta;
            if (owner && pc.kp1 < p.kpairs) {
                const int tile_end = pos + p.kpairs;
                while (c_last + 1 < G && p.share * (c_last + 1) + min(c_last + 1, p.extra) < tile_end) c_last++;
            }
            // with two issuers: the accumulators that have been written (a piece of one unit fills one thread's)
            const uint32_t own_cols = (uint32_t)((SPARSE ? 2 : 1) * p.nt32);
            const bool both = ISSUERS == 2 && pc.kp1 - pc.kp0 > 1;
            const uint32_t d_off = ISSUERS == 2 && !both && ((pos - r_begin) & 1) ? own_cols : 0u;
            pos += pc.kp1 - pc.kp0;
            float sc = 0.f, bs = 0.f;
            int li = -1;                                 // this row's index among the plan's long rows
            if (n_ok) {
                sc = __half2float(p.scales[n]);
                if (p.bias && owner) bs = p.bias[n];
                if (SPARSE && p.n_long > 0 && owner && p.row_ptr[n + 1] - p.row_ptr[n] > p.heavy) {
                    int lo = 0, hi = p.n_long - 1;
                    while (lo < hi) {
                        const int mid2 = (lo + hi) >> 1;
                        if (p.hrow[mid2] < n) lo = mid2 + 1; else hi = mid2;
                    }
                    li = lo;
                }
            }
            // every row of this warp goes to one plain matrix; some row of it is a long one
            const bool plain = !p.has_ortho && !p.gather, longs = SPARSE && __any_sync(0xffffffffu, li >= 0);
            if (grp < MAX_GROUPS) wait(&sm->all_done, 0u); else wait(&sm->d_full[a], (uint32_t)(use & 1));
            __syncwarp();
            tc_fence_after();
            const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(a * p.acc_cols);
            // scale * D + bias (+ alpha * E) of C tokens.  The zeros of the scattered tile times an infinite activation make E NaN for every
            // row: such a sum is taken again from the row's entries in this piece.
            // One issuer: 16 columns, of both accumulators under one wait.  Short rows are bound by this: 512->38230 with 1 % at 67 / 100 /
            // 128 tokens 13.6 / 16.9 / 18.7 us against 17.2 / 21.7 / 24.2 with 8 columns and a wait each, base-only 9.5 / 11.9 / 12.5 against
            // 10.6 / 12.8 / 13.8; 4096->22016 at 96 34.9 / 37.2.  (Tiles cut eight times lose at 81-112 tokens, where 16 columns divide
            // less evenly over the sets: 8192->2048 at 100 17.6 against 16.4.)  Two issuers' four accumulators: registers for 8.
            constexpr int C = ISSUERS == 2 ? 8 : 16;
            auto columns = [&](uint32_t col, uint32_t (&r)[C]) {          // C accumulator columns, once tmem_ld_wait has been called
                if constexpr (C == 8) tmem_ld_32x32b_x8(taddr + col, r); else tmem_ld_32x32b_x16(taddr + col, r);
            };
            auto both_columns = [&](uint32_t col, uint32_t (&r)[C]) {     // two issuers: of both
                columns(d_off + col, r);
                tmem_ld_wait();
                if (both) {
                    uint32_t r2[C];
                    columns(own_cols + col, r2);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < C; j++) r[j] = __float_as_uint(__uint_as_float(r[j]) + __uint_as_float(r2[j]));
                }
            };
            auto load = [&](int c, float (&v)[C]) {
                uint32_t r[C], e[SPARSE ? C : 1];
                if constexpr (ISSUERS == 2) {
                    both_columns((uint32_t)c, r);
                } else {
                    columns((uint32_t)c, r);
                    if constexpr (SPARSE) columns((uint32_t)(p.nt32 + c), e);
                    tmem_ld_wait();
                }
#pragma unroll
                for (int j = 0; j < C; j++) v[j] = fmaf(__uint_as_float(r[j]), sc, bs);
                if constexpr (SPARSE) {
                    if constexpr (ISSUERS == 2) both_columns((uint32_t)(p.nt32 + c), e);
                    bool nan = false;
#pragma unroll
                    for (int j = 0; j < C; j++) {
                        v[j] = fmaf(p.alpha, __uint_as_float(e[j]), v[j]);
                        nan = nan || v[j] != v[j];
                    }
                    if (__any_sync(0xffffffffu, nan)) {
                        uint32_t bad = 0;
#pragma unroll
                        for (int j = 0; j < C; j++) bad |= v[j] != v[j] ? 1u << j : 0u;
                        int e0 = 0, e1 = 0;
                        if (n_ok) { e0 = p.row_ptr[n]; e1 = p.row_ptr[n + 1]; } else bad = 0;
                        if (p.n_long > 0 && e1 - e0 > p.heavy) e1 = e0;               // a long row is not listed
#pragma unroll 1
                        for (int j = 0; j < C && c + j < p.M; j++) {
                            uint32_t d, d2 = 0;
                            __syncwarp();
                            tmem_ld_32x32b_x1(taddr + d_off + (uint32_t)(c + j), d);
                            if (both) tmem_ld_32x32b_x1(taddr + own_cols + (uint32_t)(c + j), d2);
                            tmem_ld_wait();
                            if (!((bad >> j) & 1u)) continue;
                            const float es = entries_sum(p.entries, e0, e1, pc.kp0 * KP, pc.kp1 * KP, p.x + (size_t)(c + j) * p.K);
                            const float base = both ? __uint_as_float(d) + __uint_as_float(d2) : __uint_as_float(d);
                            const float t = fmaf(p.alpha, es, fmaf(base, sc, bs));
#pragma unroll
                            for (int i = 0; i < C; i++) v[i] = i == j ? t : v[i];
                        }
                        __syncwarp();
                    }
                }
            };
            if (!owner) {
                // the first piece of a share that starts inside a tile: its FP32 sums to this CTA's slot, then the flag.  One fence
                // behind the barrier covers every thread's stores.
                float *dst = p.slots + ((size_t)cta * p.nt + set * C) * TN + q * 32 + lane;
                for (int c = set * C; c < p.nt; c += sets * C, dst += sets * C * TN) {
                    float v[C];
                    load(c, v);
#pragma unroll
                    for (int j = 0; j < C; j++) dst[j * TN] = v[j];
                }
                tc_fence_before();
                __syncwarp();
                if (!last && lane == 0) mbar_arrive(&sm->d_empty[a]);
                sync_sets();
                if (et == 0) {
                    __threadfence();
                    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p.flags + cta), "l"(p.tag) : "memory");
                }
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
            const float *part = p.slots + ((size_t)(cta + 1) * p.nt + set * C) * TN + q * 32 + lane;
            const size_t part_cta = (size_t)p.nt * TN;
            constexpr int H = SPARSE ? C : 8, FLY = SPARSE ? 1 : 3;     // tokens and pieces in flight (registers)
            for (int c = set * C; c < p.nt; c += sets * C, part += sets * C * TN) {
                __syncwarp();
                float v[C];
                load(c, v);
#pragma unroll
                for (int h = 0; h < C; h += H) {
                    const float *src = part + h * TN;
                    for (int cc = cta + 1; cc <= c_last; cc += FLY, src += FLY * part_cta) { // the other pieces of the tile, in CTA order
                        float t[FLY][H];
#pragma unroll
                        for (int i = 0; i < FLY; i++)
                            if (cc + i <= c_last) {
#pragma unroll
                                for (int j = 0; j < H; j++) t[i][j] = __ldcg(src + i * part_cta + j * TN);
                            }
#pragma unroll
                        for (int i = 0; i < FLY; i++)
                            if (cc + i <= c_last) {
#pragma unroll
                                for (int j = 0; j < H; j++) v[h + j] += t[i][j];
                            }
                    }
                }
                if (longs && li >= 0) {                           // a long row's sums from the pre-pass
                    const float4 *o4 = reinterpret_cast<const float4 *>(p.ol + (size_t)li * p.ol_mp + c);
#pragma unroll
                    for (int j = 0; j < C / 4; j++) {
                        const float4 t = __ldcg(o4 + j);
                        v[4 * j] = fmaf(p.alpha, t.x, v[4 * j]); v[4 * j + 1] = fmaf(p.alpha, t.y, v[4 * j + 1]);
                        v[4 * j + 2] = fmaf(p.alpha, t.z, v[4 * j + 2]); v[4 * j + 3] = fmaf(p.alpha, t.w, v[4 * j + 3]);
                    }
                }
                if (TYPED && plain) {
                    store_column<C>(p.y, (size_t)c * (size_t)p.ldy + n, p.ldy, p.y_type, p.M - c, n_ok, [&](int j) { return v[j]; });
                    continue;
                }
                if (plain) {
                    __half *yp = p.y + (size_t)c * (size_t)p.ldy + n;
#pragma unroll
                    for (int j = 0; j < C; j++) {
                        if (n_ok && c + j < p.M) *yp = __float2half_rn(v[j]);
                        yp += p.ldy;
                    }
                    continue;
                }
                if (!n_ok) continue;
#pragma unroll
                for (int j = 0; j < C; j++) {
                    const int m = c + j;
                    if (m >= p.M) break;
                    float o = v[j];
                    if (p.has_ortho) o = fmaf(p.alpha, p.o[(size_t)m * p.N + n], o);
                    const __half hv = __float2half_rn(o);
                    const size_t at = (size_t)m * (size_t)p.ldy + n;
                    if (!p.gather) p.y[at] = hv;
                    else for (int rk = 0; rk < p.gv.world; rk++) p.gv.y[rk][at] = hv;
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

    if (p.gather) {
        if (!gather_signal_and_wait(p.gv, gridDim.x)) atomicExch(p.status, 2);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem, TMEM_COLS); }
}

// O[m][n] = sum over the entries of row n of v * x[m, c]   (FP32, token-major with row pitch N; alpha is applied
// in the epilogue).  A warp takes 8 consecutive weight rows; a lane holds TPL consecutive tokens (Mp = 32 * TPL) and
// reads them from the transposed activations Xt[k][Mp] with one load per entry, up to 32 / TPL entries in flight;
// entries are fetched 32 at a time with one coalesced load and broadcast by shuffles.
template <int TPL>
__global__ void __launch_bounds__(256)
ortho_tokens_kernel(const OrthoView ov, const __half *__restrict__ xt, float *__restrict__ o, int M, int K, int N)
{
    constexpr int Mp = 32 * TPL;
    constexpr int U = 32 / TPL;                          // activation loads in flight per lane
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n_first = (blockIdx.x * 8 + warp) * 8;     // a warp takes 8 consecutive weight rows, one after the other
    if (n_first >= N) return;
    float res[8][TPL];
#pragma unroll
    for (int r = 0; r < 8; r++) {
#pragma unroll
        for (int i = 0; i < TPL; i++) res[r][i] = 0.f;
        const int n = n_first + r;
        if (n >= N) continue;
        const int e0 = ov.row_ptr[n], e1 = ov.row_ptr[n + 1];
        float acc[TPL];
#pragma unroll
        for (int i = 0; i < TPL; i++) acc[i] = 0.f;
        for (int eb = e0; eb < e1; eb += 32) {
            int cl = 0; float vl = 0.f;
            if (eb + lane < e1) ortho_entry(ov, eb + lane, K, cl, vl);
            const int nb = min(32, e1 - eb);
            for (int j0 = 0; j0 < nb; j0 += U) {
                float vv[U];
                if constexpr (TPL == 1) {
                    __half h[U];
#pragma unroll
                    for (int j = 0; j < U; j++) {
                        const int c = __shfl_sync(0xffffffffu, cl, (j0 + j) & 31);
                        vv[j] = __shfl_sync(0xffffffffu, vl, (j0 + j) & 31);      // slots past the row hold v = 0, c = 0
                        h[j] = xt[(size_t)c * Mp + lane];
                    }
#pragma unroll
                    for (int j = 0; j < U; j++) acc[0] = fmaf(vv[j], __half2float(h[j]), acc[0]);
                } else if constexpr (TPL == 2) {
                    __half2 h[U];
#pragma unroll
                    for (int j = 0; j < U; j++) {
                        const int c = __shfl_sync(0xffffffffu, cl, (j0 + j) & 31);
                        vv[j] = __shfl_sync(0xffffffffu, vl, (j0 + j) & 31);
                        h[j] = *reinterpret_cast<const __half2 *>(xt + (size_t)c * Mp + lane * 2);
                    }
#pragma unroll
                    for (int j = 0; j < U; j++) {
                        const float2 f = __half22float2(h[j]);
                        acc[0] = fmaf(vv[j], f.x, acc[0]); acc[1] = fmaf(vv[j], f.y, acc[1]);
                    }
                } else {
                    uint2 u[U];
#pragma unroll
                    for (int j = 0; j < U; j++) {
                        const int c = __shfl_sync(0xffffffffu, cl, (j0 + j) & 31);
                        vv[j] = __shfl_sync(0xffffffffu, vl, (j0 + j) & 31);
                        u[j] = *reinterpret_cast<const uint2 *>(xt + (size_t)c * Mp + lane * 4);
                    }
#pragma unroll
                    for (int j = 0; j < U; j++) {
                        const float2 f0 = __half22float2(*reinterpret_cast<const __half2 *>(&u[j].x));
                        const float2 f1 = __half22float2(*reinterpret_cast<const __half2 *>(&u[j].y));
                        acc[0] = fmaf(vv[j], f0.x, acc[0]); acc[1] = fmaf(vv[j], f0.y, acc[1]);
                        acc[2] = fmaf(vv[j], f1.x, acc[2]); acc[3] = fmaf(vv[j], f1.y, acc[3]);
                    }
                }
            }
        }
#pragma unroll
        for (int i = 0; i < TPL; i++) res[r][i] = acc[i];
    }
    // a lane writes the 8 rows' sums of each of its tokens as one 32-byte run
    const bool vec = (N % 4) == 0 && n_first + 8 <= N;
#pragma unroll
    for (int i = 0; i < TPL; i++) {
        const int m = lane * TPL + i;
        if (m >= M) continue;
        float *dst = o + (size_t)m * N + n_first;
        if (vec) {
            reinterpret_cast<float4 *>(dst)[0] = make_float4(res[0][i], res[1][i], res[2][i], res[3][i]);
            reinterpret_cast<float4 *>(dst)[1] = make_float4(res[4][i], res[5][i], res[6][i], res[7][i]);
        } else {
#pragma unroll
            for (int r = 0; r < 8; r++)
                if (n_first + r < N) dst[r] = res[r][i];
        }
    }
}

// workspace: [ Xt : K * Mp halves ][ O : M * N floats ][ partial slots : SMs * nt * 128 floats ][ flags ][ long rows' shares ]
constexpr int kMidMaxSms = 148;         // the partial-sum slots are sized for this many CTAs; the grid never exceeds it
static int64_t mid_mp(int64_t M) { return M <= 32 ? 32 : M <= 64 ? 64 : 128; }
static int64_t mid_nt(int64_t M) { return (M + 15) / 16 * 16; }
static int64_t mid_xt_bytes(int64_t M, int64_t K) { return ((K * mid_mp(M) * 2 + 255) / 256) * 256; }
static int64_t mid_o_bytes(int64_t M, int64_t N) { return ((M * N * 4 + 255) / 256) * 256; }
static int64_t mid_slot_bytes(int64_t M) { return (int64_t)kMidMaxSms * mid_nt(M) * md::TN * 4; }
static_assert(kMidMaxSms * 8 <= 2048, "flag words");
int64_t mid_workspace_bytes(int64_t M, int64_t K, int64_t N)
{
    return mid_xt_bytes(M, K) + mid_o_bytes(M, N) + mid_slot_bytes(M) + 2048;
}

bool mid_has_lists(const FwdArgs &a)
{
    const int64_t long_bytes = a.plan && a.plan->n_long > 0 ? long_rows_workspace_bytes(a.plan, a.M) : 0;
    return a.has_ortho && a.plan && a.ortho.entries && a.plan->win_off && a.workspace_bytes >= mid_workspace_bytes(a.M, a.K, a.N) + long_bytes &&
           tuning_snapshot().patch_weights;
}

int launch_mid(const FwdArgs &a)
{
    using namespace md;
    if (a.M > TMK || a.M < 1) return ORTHO_B200_ERR_SHAPE;
    const int64_t own_bytes = mid_workspace_bytes(a.M, a.K, a.N);
    if (!a.workspace || a.workspace_bytes < own_bytes) return ORTHO_B200_ERR_WORKSPACE;
    if (((uintptr_t)a.workspace & 255u) != 0) return ORTHO_B200_ERR_ALIGN;
    const int dev = current_device_index();
    if (dev < 0) return ORTHO_B200_ERR_CUDA;
    const int num_sms = device_sm_count(dev);
    unsigned char *wsb = reinterpret_cast<unsigned char *>(a.workspace);
    __half *xt = reinterpret_cast<__half *>(wsb);
    float *o = reinterpret_cast<float *>(wsb + mid_xt_bytes(a.M, a.K));
    float *slots = reinterpret_cast<float *>(wsb + mid_xt_bytes(a.M, a.K) + mid_o_bytes(a.M, a.N));
    unsigned long long *flags = reinterpret_cast<unsigned long long *>(wsb + mid_xt_bytes(a.M, a.K) + mid_o_bytes(a.M, a.N) + mid_slot_bytes(a.M));

    Params p;
    memset(&p, 0, sizeof(p));
    p.scales = a.scales; p.bias = a.bias; p.y = a.y; p.M = (int)a.M; p.K = (int)a.K; p.N = (int)a.N; p.ldy = a.pitch_y();
    p.tiles_n = (int)ceil_div(a.N, TN); p.kblocks = (int)ceil_div(a.K, KB);
    p.kpairs = (int)ceil_div(a.K, KP);
    p.nt = (int)mid_nt(a.M);
    p.xtile = p.nt * 128;
    p.slots = slots; p.flags = flags;
    p.alpha = a.alpha; p.has_ortho = 0; p.o = nullptr;
    p.status = kernel_status_word();
    if (!p.status) return ORTHO_B200_ERR_CUDA;
    bool sparse = false;
    const bool long_rows = a.plan && a.plan->n_long > 0;
    p.y_type = a.y_type;
    if (mid_has_lists(a)) {
        sparse = true;
        p.win_off = a.plan->win_off; p.win_words = a.plan->win_words; p.ngroups = (int)ceil_div(a.N, kWinRows);
        p.row_ptr = a.plan->row_ptr; p.entries = a.ortho.entries; p.x = a.x;
        if (long_rows) {
            p.hrow = a.plan->hrow; p.n_long = (int)a.plan->n_long; p.heavy = a.plan->heavy;
        }
    } else if (a.has_ortho) {
        const int Mp = (int)mid_mp(a.M);
        int st = launch_transpose_x(a.x, xt, (int)a.M, (int)a.K, Mp, a.stream);
        if (st != ORTHO_B200_OK) return st;
        const unsigned blocks = (unsigned)ceil_div(a.N, 64);
        if (Mp == 32) ortho_tokens_kernel<1><<<blocks, 256, 0, a.stream>>>(a.ortho, xt, o, (int)a.M, (int)a.K, (int)a.N);
        else if (Mp == 64) ortho_tokens_kernel<2><<<blocks, 256, 0, a.stream>>>(a.ortho, xt, o, (int)a.M, (int)a.K, (int)a.N);
        else ortho_tokens_kernel<4><<<blocks, 256, 0, a.stream>>>(a.ortho, xt, o, (int)a.M, (int)a.K, (int)a.N);
        count_launch();
        OB_CUDA(cudaGetLastError());
        p.o = o; p.has_ortho = 1;
    }
    // Tensor memory: accumulators D (and E behind it), then the converted stages.  Shared memory: token stages and sparse
    // tiles of the same number, the rest for packed weights (8 KB slots): 64 KB or more in flight per SM, but 48 KB with entries at
    // 33-48 tokens and 40-56 KB above 64, where a stage with its sparse tiles is worth more than a slot.
    p.nt32 = (p.nt + 31) / 32 * 32;
    p.issuers = p.nt32 <= (sparse ? kTwoIssuersSparse : kTwoIssuers) ? 2 : 1;
    p.acc_cols = (sparse ? 2 : 1) * p.issuers * p.nt32;
    p.nacc = 2 * p.acc_cols + 4 * A_STAGE_COLS <= TMEM_COLS ? 2 : 1;
    p.nst = (TMEM_COLS - p.nacc * p.acc_cols) / A_STAGE_COLS;
    if (p.nst > (sparse ? ST_SPARSE_MAX : ST_MAX)) p.nst = sparse ? ST_SPARSE_MAX : ST_MAX;
    // The issuers, and the two sets of scatter warps, take turns: even numbers of stages then, and of weight slots.  Above 64 tokens,
    // where shared memory holds three stages, three and one set are better than two and two (28672->8192 at 100: 73 us against 77).
    // With entries at 33-48 tokens four stages, two converter groups and six slots against three, three and eleven (one set): 8192->10240
    // at 33 / 48 22.8 / 23.0 us against 25.9 / 25.8, 4096->22016 at 48 25.5 / 27.5, 28672->8192 at 48 58.6 / 64.7; at 49-64 two, two and
    // sixteen against three, three and ten: 8192->10240 at 49 / 64 25.8 / 27.9 against 26.9 / 28.8, 28672->8192 at 64 66 / 70; at
    // 113-128, two stages, one set instead of two makes no difference (4096->22016 at 128 45.2 / 45.4).
    const int down = p.issuers == 2 || (sparse && p.nt <= 64) ? 2 : 1;
    const int nst_max = p.nst - p.nst % down;
    for (p.groups = MAX_GROUPS;; p.groups -= down) {         // most groups first, then most stages, by the rule above MAX_GROUPS
        for (p.nst = nst_max; p.nst >= p.groups; p.nst -= down) {
            p.wst = (kSmemData - p.nst * (2 * p.xtile + (sparse ? S_BYTES : 0))) / W_BYTES;
            if (p.wst > WST_MAX) p.wst = WST_MAX;
            p.wst -= p.wst % down;
            if (p.wst >= p.nst + p.groups) break;
        }
        if (p.nst >= p.groups) break;
        if (p.groups <= 2) return ORTHO_B200_ERR_SHAPE;      // not reached for up to 128 tokens
    }
    p.sets = p.nst % 2 == 0 ? 2 : 1;
    CUtensorMap xmap, wmap;
    if (!make_tensor_map_2d(&xmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, a.x, (uint64_t)a.M, (uint64_t)a.K,
                            (uint64_t)a.K * 2, (uint32_t)p.nt, KB, CU_TENSOR_MAP_SWIZZLE_128B))
        return ORTHO_B200_ERR_CUDA;
    if (!make_tensor_map_2d(&wmap, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, a.w, (uint64_t)a.N, (uint64_t)(a.K / 2),
                            (uint64_t)(a.K / 2), TN, KP / 2, CU_TENSOR_MAP_SWIZZLE_64B))
        return ORTHO_B200_ERR_CUDA;
    p.gather = 0;
    if (a.gv && a.gv->world > 1) {
        p.gv = *a.gv;
        p.gather = 1;
        if (a.gather_fused) *a.gather_fused = true;
    }
    static bool attr_set[kMaxDevices] = {};
    if (!attr_set[dev]) {
        for (auto k : {mid_kernel<false, false, 1>, mid_kernel<true, false, 1>, mid_kernel<false, true, 1>, mid_kernel<true, true, 1>,
                       mid_kernel<false, false, 2>, mid_kernel<true, false, 2>, mid_kernel<false, true, 2>, mid_kernel<true, true, 2>})
            OB_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes));
        attr_set[dev] = true;
    }
    // every CTA gets at least kMinShare units: a narrow layer cut into shares of a few would spend its time adding
    // dozens of partial tiles
    constexpr long long kMinShare = 8;
    const long long total = (long long)p.tiles_n * p.kpairs;
    if (total > 0x7fffffffLL) return ORTHO_B200_ERR_SHAPE;
    long long grid = (total + kMinShare - 1) / kMinShare;
    if (grid > num_sms) grid = num_sms;
    if (grid > kMidMaxSms) grid = kMidMaxSms;
    if (grid < 1) grid = 1;
    p.share = (int)(total / grid); p.extra = (int)(total % grid);
    // A contributor's flag is "this launch's tag is in my word".  The workspace comes as it is (clearing the words on the
    // stream first would be one more node per forward, and no programmatic launch past it), so a tag is a 64-bit value that no other launch of any process has and that
    // a stale word holds with probability 2^-64; the collecting CTA clears the words it has seen, so that a replay of
    // a captured graph, which brings the same tag again, finds them cleared.
    p.tag = next_launch_tag();
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3((unsigned)grid); cfg.blockDim = dim3((unsigned)((sparse ? kWarps<true, 1> : kWarps<false, 1>) + p.issuers - 1) * 32); cfg.dynamicSmemBytes = kSmemBytes; cfg.stream = a.stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
    if (p.n_long > 0) {                                  // the long rows' pre-pass right in front
        p.ol_mp = (int)(ceil_div(a.M, 256) * 256);
        const int st = launch_long_rows(a, p.ol_mp, wsb + own_bytes, &p.ol);
        if (st != ORTHO_B200_OK) return st;
    }
    const bool typed = p.y_type != kTypeF16;
    auto pick = [&](auto one, auto two) { return p.issuers == 2 ? two : one; };
    auto kern = sparse ? (typed ? pick(mid_kernel<true, true, 1>, mid_kernel<true, true, 2>) : pick(mid_kernel<true, false, 1>, mid_kernel<true, false, 2>))
                       : (typed ? pick(mid_kernel<false, true, 1>, mid_kernel<false, true, 2>) : pick(mid_kernel<false, false, 1>, mid_kernel<false, false, 2>));
    OB_CUDA(cudaLaunchKernelEx(&cfg, kern, xmap, wmap, p));
    count_launch();
    return ORTHO_B200_OK;
}

}  // namespace ob
