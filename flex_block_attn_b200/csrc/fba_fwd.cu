// Block-sparse attention forward for sm_100a.
//
// Computes what the reference's fwd_attend_ker (flex_block_attn_h100.cu:52-318) computes --
// O = softmax(QK^T / sqrt(128) restricted to the active blocks) V and the row log-sum-exp -- but
// is organised around Blackwell's tensor memory instead of Hopper register accumulators:
//
//   * a CTA owns two 128-row query tiles (A and B) of one (batch, head) and ping-pongs between
//     them, so the tensor core works on one tile while the softmax warps work on the other;
//   * one warp per query tile issues that tile's tcgen05.mma.  S = Q K^T goes to TMEM (128 fp32 columns), the
//     softmax warps read it with tcgen05.ld (one thread = one row, so row max / row sum need no shuffles), write
//     P as bf16 to the tile's own 64 columns, and O += P V consumes P straight from TMEM; O (128 fp32 columns per
//     tile) never leaves TMEM until the epilogue.  The score buffer is needed only from the MMA to the load into
//     registers, a fraction of a step, so ONE buffer serves both tiles in turn (A(0) B(0) A(1) B(1) ...) and the
//     scores of step i + 1 are computed while the softmax of step i runs.  Columns: [0,64) P of tile A, [64,192) S,
//     [192,256) P of tile B, [256,384) O_A, [384,512) O_B.
//     What bounds it: the softmax warps (1024 exp2 clocks per tile and the instructions around them) and the tensor
//     core (1024 clocks per tile) side by side.  All-ones mask, S = 9216, 24 heads: 2 x 128 keys take 2850 clocks
//     here; with S and P of a tile sharing 128 columns, so that S of step i + 1 had to wait for P V of step i, they
//     took 3310.  Inference pass, S = 30720, keep 0.4: 4.43 -> 3.89 ms;
//   * one thread streams only the listed K / V tiles through a 5-stage shared-memory ring with
//     TMA + mbarrier; the list comes from the compaction kernel, not from scanning the mask;
//   * rescaling of O is lazy (only when the running row max grew by more than 2^8), done by the
//     softmax warps between two MMAs of their tile.  A share of the exponentials by a
//     degree-5 polynomial on the FMA pipe costs 5 % (1 / 8) and 13 % (1 / 4).  (Counters, S = 23040, 8 heads, keep 0.4:
//     tensor pipe 74 %, exp2 unit 76 %, issue slots 42 % busy.)
//
// If both query tiles map to the same list row they share every K / V stage; otherwise each tile
// streams its own list ("split" mode) in a fixed interleaving that loader and issuer both follow.
#include "fba_common.cuh"

namespace fba {

constexpr int kFwdThreads = 384;  // warpgroup 0: softmax A, 1: softmax B, 2: {MMA A, TMA, MMA B, idle}
constexpr int kFwdStages = 5;
constexpr uint32_t kFwdSmemQ = 0;
constexpr uint32_t kFwdSmemRing = 2 * kTileBytes;
constexpr uint32_t kFwdSmemBars = kFwdSmemRing + kFwdStages * kTileBytes;
constexpr uint32_t kFwdSmemBytes = kFwdSmemBars + 256 + 1024;  // + alignment slack

// P is handed to the MMA issuer in this many pieces per 128-key step, so that O += P V starts while
// the later exponentials are still being computed (2 pieces of 96 + 32 keys: 8 % more clocks).
constexpr int kFwdPieces = 4;
constexpr int kFwdPiecePairs = 64 / kFwdPieces;   // bf16x2 words (= TMEM columns) per piece
// The next step's scores are issued before this piece of O += P V.
constexpr int kFwdScoresAt = 1;
// TMEM columns: P of tile A, one score buffer for both tiles, P of tile B, O of A, O of B.
constexpr uint32_t kTmemPA = 0, kTmemS = 64, kTmemPB = 192, kTmemO = 256;

struct FwdParams {
    ListDev list;
    float* lse;            // may be null: no log-sum-exp is written (inference)
    uint32_t* status;
    int n_mtiles, Sq, Hq, Hkv;
    float scale_log2;      // softmax scale * log2(e)
};

// Barrier slots (8 bytes each) inside the barrier block.
enum FwdBar : uint32_t {
    kBarQFull = 0,                         // 2
    kBarRingFull = 2,                      // kFwdStages
    kBarRingEmpty = 2 + kFwdStages,        // kFwdStages
    kBarSFull = 2 + 2 * kFwdStages,        // 2
    kBarP = 4 + 2 * kFwdStages,            // 2 x 4: piece q of tile t's P is in TMEM (slot 4 t + q)
    kBarSLoaded = 12 + 2 * kFwdStages,     // 2: tile t's warps hold the scores in registers, the S buffer is free
    kBarPvDone = 14 + 2 * kFwdStages,      // 2: O += P V of a step has completed (P and O may be touched)
    kBarCount = 16 + 2 * kFwdStages
};
static_assert(8 * kBarCount + 16 <= 256, "barrier block overflows its 256-byte slot");
static_assert(kFwdSmemBytes <= 232448, "exceeds the 227 KiB shared memory of an sm_100 CTA");

// One piece (8 / kFwdPieces k-steps of 16 keys) of O += P V.
__device__ __forceinline__ void mma_pv_piece(uint32_t d_tmem, uint32_t p_tmem, uint32_t v_smem, int piece,
                                             bool accumulate) {
    const uint32_t b = desc_lo_mnmajor(v_smem);
    constexpr int kSteps = 8 / kFwdPieces;
#pragma unroll
    for (int k = 0; k < kSteps; ++k) {
        const int kk = piece * kSteps + k;
        umma_ts(d_tmem, p_tmem + static_cast<uint32_t>(kk) * 8u, b + kstep_mnmajor(kk), kIdescKM,
                (accumulate || kk > 0) ? 1u : 0u);
    }
}

__global__ void __launch_bounds__(kFwdThreads, 1)
fba_fwd_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
               const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_o,
               const FwdParams p) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t* base_ptr = smem_raw + (base - raw);
    const uint32_t bars = base + kFwdSmemBars;
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(base_ptr + kFwdSmemBars + 8 * kBarCount);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(base_ptr + kFwdSmemBars + 8 * kBarCount + 4);
    auto bar = [&](uint32_t slot) { return bars + 8u * slot; };

    const int warp = warp_uniform(static_cast<int>(threadIdx.x >> 5));
    const int lane = threadIdx.x & 31;
    const int bh = blockIdx.y;
    // Work item of this CTA: the blockIdx.x-th entry of the (batch, head)'s longest-first order when
    // one is given (CTAs are dispatched in blockIdx order, so the shortest items of the grid run
    // last and the tail of the launch stays short), else blockIdx.x itself.
    const int pair = p.list.order
                         ? p.list.order[static_cast<long long>(p.list.bh_stride ? bh : 0) * gridDim.x + blockIdx.x]
                         : static_cast<int>(blockIdx.x);
    const int hr = p.Hq / p.Hkv;
    const int bhk = (bh / p.Hq) * p.Hkv + (bh % p.Hq) / hr;

    // Per-tile list rows and lengths (identical in every thread).
    const int mt0 = 2 * pair, mt1 = 2 * pair + 1;
    const bool tile1_valid = mt1 < p.n_mtiles;
    const long long lrow0 = static_cast<long long>(bh) * p.list.bh_stride + mt0 / p.list.rows_div;
    const long long lrow1 = static_cast<long long>(bh) * p.list.bh_stride + (tile1_valid ? mt1 / p.list.rows_div : 0);
    const int sub = p.list.sub;
    const int n0 = warp_uniform(p.list.cnt[lrow0] * sub);
    const int n1 = warp_uniform(tile1_valid ? p.list.cnt[lrow1] * sub : 0);
    const bool shared_mode = tile1_valid && lrow0 == lrow1;

    if (threadIdx.x == 0) {
        *abort_flag = 0;
        mbar_init(bar(kBarQFull + 0), 1);
        mbar_init(bar(kBarQFull + 1), 1);
        for (int s = 0; s < kFwdStages; ++s) {
            mbar_init(bar(kBarRingFull + s), 1);
            mbar_init(bar(kBarRingEmpty + s), 2);
        }
        for (int t = 0; t < 2; ++t) {
            mbar_init(bar(kBarSFull + t), 1);
            for (int q = 0; q < kFwdPieces; ++q) mbar_init(bar(kBarP + 4 * t + q), 128);
            mbar_init(bar(kBarSLoaded + t), 128);
            mbar_init(bar(kBarPvDone + t), 1);
        }
        mbar_fence_init();
    }
    if (warp == 8) {
        tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), 512);
        tmem_relinquish();
    }
    if (warp == 9 && lane == 0) {
        tma_prefetch_desc(&tm_q);
        tma_prefetch_desc(&tm_k);
        tma_prefetch_desc(&tm_v);
        tma_prefetch_desc(&tm_o);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = warp_uniform(*tmem_slot);
    const uint32_t sQ0 = base + kFwdSmemQ, sQ1 = base + kFwdSmemQ + kTileBytes;
    auto ring = [&](int s) { return base + kFwdSmemRing + static_cast<uint32_t>(s) * kTileBytes; };
    auto kv_tile_of = [&](int t, int i) {
        const int e = i / sub;
        return p.list.idx[(t ? lrow1 : lrow0) * p.list.stride + e] * sub + (i - e * sub);
    };

    if (warp >= 8) {
        // Register pool of the CTA = 384 threads x 168 at launch = 3 x 128 x 168.  The budgets set
        // below must not add up to more than that (216 + 216 + 72 = 504), or the increase would
        // wait for registers that are never released.
        reg_dec<72>();
        if (warp == 9) {
            // -------------------------------------------------------------- TMA loader
            if (lane == 0) {
                bool ok = true;
                uint32_t prod = 0;
                if (n0 > 0) {
                    mbar_expect_tx(bar(kBarQFull + 0), kTileBytes);
                    tma_load_3d(sQ0, &tm_q, 0, mt0 * 128, bh, bar(kBarQFull + 0));
                    tma_load_3d(sQ0 + kPanelBytes, &tm_q, 64, mt0 * 128, bh, bar(kBarQFull + 0));
                }
                if (n1 > 0) {
                    mbar_expect_tx(bar(kBarQFull + 1), kTileBytes);
                    tma_load_3d(sQ1, &tm_q, 0, mt1 * 128, bh, bar(kBarQFull + 1));
                    tma_load_3d(sQ1 + kPanelBytes, &tm_q, 64, mt1 * 128, bh, bar(kBarQFull + 1));
                }
                auto load = [&](const CUtensorMap* tm, int kv_tile, uint32_t tag) {
                    if (!ok) return;
                    const int s = prod % kFwdStages;
                    const uint32_t parity = ((prod / kFwdStages) & 1u) ^ 1u;
                    if (!mbar_wait(bar(kBarRingEmpty + s), parity, abort_flag)) {
                        report_timeout(p.status, 1, 9, prod, tag);
                        ok = false;
                        return;
                    }
                    mbar_expect_tx(bar(kBarRingFull + s), kTileBytes);
                    tma_load_3d(ring(s), tm, 0, kv_tile * 128, bhk, bar(kBarRingFull + s));
                    tma_load_3d(ring(s) + kPanelBytes, tm, 64, kv_tile * 128, bhk, bar(kBarRingFull + s));
                    ++prod;
                };
                const int ln[2] = {n0, shared_mode ? 0 : n1};
                const int nmax = ln[0] > ln[1] ? ln[0] : ln[1];
                for (int t = 0; t < 2; ++t)
                    if (ln[t] > 0) load(&tm_k, kv_tile_of(t, 0), 100 + t);
                for (int i = 0; i < nmax && ok; ++i) {
                    for (int t = 0; t < 2; ++t) {
                        if (i < ln[t]) {
                            load(&tm_v, kv_tile_of(t, i), 200 + t);
                            if (i + 1 < ln[t]) load(&tm_k, kv_tile_of(t, i + 1), 100 + t);
                        }
                    }
                }
            }
        } else if (warp == 8 || warp == 10) {
            // -------------------------------------------------------------- MMA issuers
            // One issuing warp per query tile (warp 8: tile A, warp 10: tile B): an issuing warp is blocked
            // while it polls barriers, and with one warp per tile those bubbles are filled by the other tile's
            // MMAs (one warp for both tiles, in the order S_A PV_A S_B PV_B: 2 % slower).
            // The warps stay converged (ptx.cuh says why): all-ones mask, S = 30720, 24 heads,
            // 10.6 ms with one issuing lane each, 9.1 ms with the whole warp.
            const int t = warp == 8 ? 0 : 1;
            const int nt = t ? n1 : n0;
            if (nt > 0) {
                bool ok = true;
                const uint32_t sQt = t ? sQ1 : sQ0;
                const uint32_t tS = tmem + kTmemS;
                const uint32_t tP = tmem + (t ? kTmemPB : kTmemPA);
                const uint32_t tO = tmem + kTmemO + static_cast<uint32_t>(t) * 128u;
                const int ln1 = shared_mode ? 0 : n1;   // what the loader streams for tile B
                // Position of an operand in the loader's global order -> ring slot and parity.
                auto wait_full = [&](uint32_t pos, uint32_t tag) -> int {
                    const int s = pos % kFwdStages;
                    if (!mbar_wait_warp(bar(kBarRingFull + s), (pos / kFwdStages) & 1u, abort_flag)) {
                        report_timeout(p.status, 1, static_cast<uint32_t>(warp), pos, tag);
                        ok = false;
                    }
                    return s;
                };
                // Every ring slot needs two releases per use: one from each tile's issuer when the
                // tiles share the stream, both from the only consumer otherwise.
                auto release = [&](int s) {
                    umma_commit(bar(kBarRingEmpty + s));
                    if (!shared_mode) umma_commit(bar(kBarRingEmpty + s));
                };
                // Loader order: K(A,0) K(B,0), then per step i: V(A,i) K(A,i+1) V(B,i) K(B,i+1).
                uint32_t g = (n0 > 0 ? 1u : 0u) + (ln1 > 0 ? 1u : 0u);   // loads before step 0
                const uint32_t pos_k0 = (t == 1 && !shared_mode) ? (n0 > 0 ? 1u : 0u) : 0u;
                if (!mbar_wait_warp(bar(kBarQFull + t), 0, abort_flag)) {
                    report_timeout(p.status, 1, static_cast<uint32_t>(warp), 0, 300 + t);
                    ok = false;
                }
                // Order of the scores in the shared S buffer: A(0) B(0) A(1) B(1) ..., the rest of the longer
                // list on its own.  Scores may be written once those before them are in registers.
                auto wait_s_free = [&](int i) {   // before S of this tile's step i
                    const int n_other = t ? n0 : n1;
                    const int other = t ? i : i - 1;
                    int who = -1, step = 0;
                    if (other >= 0 && other < n_other) {
                        who = t ^ 1;
                        step = other;
                    } else if (i > 0) {
                        who = t;
                        step = i - 1;
                    }
                    if (who >= 0 && !mbar_wait_warp(bar(kBarSLoaded + who), step & 1u, abort_flag)) {
                        report_timeout(p.status, 1, static_cast<uint32_t>(warp), i, 350 + t);
                        ok = false;
                    }
                };
                int slot_k = wait_full(pos_k0, 310 + t);
                if (ok) wait_s_free(0);
                if (ok) {
                    tc_fence_after();
                    mma_tile_kk(tS, sQt, ring(slot_k), false);
                    umma_commit(bar(kBarSFull + t));
                    release(slot_k);
                }
                for (int i = 0; i < nt && ok; ++i) {
                    const uint32_t a_v = (i < n0), a_k = (i + 1 < n0), b_v = (i < ln1), b_k = (i + 1 < ln1);
                    const bool own_a = t == 0 || shared_mode;
                    const uint32_t pos_v = own_a ? g : g + a_v + a_k;
                    const uint32_t pos_k = pos_v + 1;
                    g += a_v + a_k + b_v + b_k;
                    const bool more = i + 1 < nt;
                    const int slot_v = wait_full(pos_v, 330 + t);
                    if (!ok) break;
                    if (i < 64) FBA_TRACE_REC(p.status, 1024 + i * 8 + t * 4 + 0);
#pragma unroll
                    for (int q = 0; q < kFwdPieces; ++q) {
                        if (ok && q == kFwdScoresAt && more) {
                            slot_k = wait_full(pos_k, 340 + t);
                            if (ok) wait_s_free(i + 1);
                            if (ok) {
                                tc_fence_after();
                                mma_tile_kk(tS, sQt, ring(slot_k), false);
                                umma_commit(bar(kBarSFull + t));
                                release(slot_k);
                            }
                            if (i < 64) FBA_TRACE_REC(p.status, 1024 + i * 8 + t * 4 + 1);
                        }
                        if (ok && !mbar_wait_warp(bar(kBarP + 4 * t + q), i & 1u, abort_flag)) {
                            report_timeout(p.status, 1, static_cast<uint32_t>(warp), i, 320 + t);
                            ok = false;
                        }
                        if (ok) {
                            tc_fence_after();
                            mma_pv_piece(tO, tP, ring(slot_v), q, i > 0 || q > 0);
                        }
                    }
                    if (!ok) break;
                    umma_commit(bar(kBarPvDone + t));
                    release(slot_v);
                    if (i < 64) FBA_TRACE_REC(p.status, 1024 + i * 8 + t * 4 + 2);
                }
            }
        }
    } else {
        // ------------------------------------------------------------------ softmax + epilogue
        reg_inc<216>();
        const int t = warp >> 2;                       // 0: tile A, 1: tile B
        const int row = (warp & 3) * 32 + lane;        // row inside the tile == TMEM lane
        const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
        const uint32_t tS = tmem + lane_base + kTmemS;
        const uint32_t tP = tmem + lane_base + (t ? kTmemPB : kTmemPA);
        const uint32_t tO = tmem + lane_base + kTmemO + static_cast<uint32_t>(t) * 128u;
        const int mt = t ? mt1 : mt0;
        const int nt = t ? n1 : n0;
        const long long lrow = t ? lrow1 : lrow0;
        const uint32_t sQt = t ? sQ1 : sQ0;
        const bool tile_valid = mt < p.n_mtiles;
        const float c = p.scale_log2;
        const int g = row >> 4;
        const bool tracer = (warp & 3) == 0 && lane == 0;

        float off = 0.f;        // exponent offset (scaled-by-c row max the exponentials refer to)
        bool have_off = false;  // false until the row has seen a finite score
        float2 l2a = make_float2(0.f, 0.f), l2b = make_float2(0.f, 0.f);
        bool ok = true;

        for (int i = 0; i < nt && ok; ++i) {
            if (!mbar_wait(bar(kBarSFull + t), i & 1u, abort_flag)) {
                if (lane == 0) report_timeout(p.status, 1, static_cast<uint32_t>(warp), i, 400 + t);
                ok = false;
            }
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after();
            if (tracer && i < 64) FBA_TRACE_REC(p.status, i * 8 + t * 4 + 0);
            uint32_t u[128];
#pragma unroll
            for (int cc = 0; cc < 4; ++cc)
                tmem_ld32(tS + 32u * cc, reinterpret_cast<uint32_t(&)[32]>(u[32 * cc]));
            tmem_wait_ld();
            tc_fence_before();
            mbar_arrive(bar(kBarSLoaded + t));
            if (tracer && i < 64) FBA_TRACE_REC(p.status, i * 8 + t * 4 + 1);

            if (p.list.msk != nullptr) {
                const uint32_t w = p.list.msk[lrow * p.list.stride + i / sub];
                if (w != 0xffffu) {
                    const bool keep0 = (w >> g) & 1u, keep1 = (w >> (8 + g)) & 1u;
#pragma unroll
                    for (int j = 0; j < 64; ++j) {
                        if (!keep0) u[j] = 0xff800000u;
                        if (!keep1) u[64 + j] = 0xff800000u;
                    }
                }
            }
            // Row maximum: four independent chains of three-input maxima.
            float mm[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) mm[j] = fmaxf(__uint_as_float(u[j]), __uint_as_float(u[4 + j]));
#pragma unroll
            for (int j = 8; j < 128; j += 8)
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    mm[e] = max3(mm[e], __uint_as_float(u[j + e]), __uint_as_float(u[j + 4 + e]));
            const float mx = fmaxf(max3(mm[0], mm[1], mm[2]), mm[3]);
            if (tracer && i < 64) FBA_TRACE_REC(p.status, i * 8 + t * 4 + 2);

            float alpha = 1.f;
            const float cand = mx * c;
            if (!have_off) {
                if (mx > -INFINITY) {
                    off = cand;
                    have_off = true;
                }
            } else if (cand - off > 8.f) {
                alpha = ex2_approx(off - cand);
                off = cand;
            }
            if (i > 0) {
                // The previous step's P V must have read P before it is overwritten, and finished O
                // before that is rescaled; it was issued a softmax phase ago.
                if (!mbar_wait(bar(kBarPvDone + t), (i - 1) & 1u, abort_flag)) {
                    if (lane == 0) report_timeout(p.status, 1, static_cast<uint32_t>(warp), i, 410 + t);
                    ok = false;
                }
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                tc_fence_after();
            }
            if (i > 0 && __any_sync(0xffffffffu, alpha != 1.f)) {
                // Rescale this warp's 32 rows of O; the next P V waits for the P barriers.
#pragma unroll
                for (int cc = 0; cc < 4; ++cc) {
                    uint32_t v[32];
                    tmem_ld32(tO + 32u * cc, v);
                    tmem_wait_ld();
#pragma unroll
                    for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) * alpha);
                    tmem_st32(tO + 32u * cc, v);
                }
            }
            l2a.x *= alpha;
            l2a.y *= alpha;
            l2b.x *= alpha;
            l2b.y *= alpha;
            const float neg_off = have_off ? -off : 0.f;
            // P goes to TMEM in pieces (keys in ascending order); a piece is announced to the
            // issuer once its TMEM store has completed.
            uint32_t pk[64];
            const float2 c2 = make_float2(c, c), off2 = make_float2(neg_off, neg_off);
#pragma unroll
            for (int j = 0; j < 64; ++j) {
                // Packed pairs throughout: with scalar multiply-adds and sums the kernel takes 5 % more clocks.
                const float2 x = fma2(make_float2(__uint_as_float(u[2 * j]), __uint_as_float(u[2 * j + 1])), c2, off2);
                const float2 e = make_float2(ex2_approx(x.x), ex2_approx(x.y));
                if (j & 1) l2b = add2(l2b, e);
                else l2a = add2(l2a, e);
                pk[j] = pack_bf16x2(e.x, e.y);
                if (j % kFwdPiecePairs == kFwdPiecePairs - 1) {
                    const int q = j / kFwdPiecePairs;
                    tmem_st16(tP + 16u * q, reinterpret_cast<uint32_t(&)[16]>(pk[16 * q]));
                    tmem_wait_st();
                    tc_fence_before();
                    mbar_arrive(bar(kBarP + 4 * t + q));
                    if (q == 0 && tracer && i < 64) FBA_TRACE_REC(p.status, 3072 + i * 4 + t);
                }
            }
            if (tracer && i < 64) FBA_TRACE_REC(p.status, i * 8 + t * 4 + 3);
        }
        const float l = (l2a.x + l2a.y) + (l2b.x + l2b.y);

        // Epilogue: O / l -> bf16 -> swizzled staging in this tile's Q buffer -> TMA store.
        if (tile_valid) {
            if (nt > 0 && ok) {
                if (!mbar_wait(bar(kBarPvDone + t), (nt - 1) & 1u, abort_flag)) {
                    if (lane == 0) report_timeout(p.status, 1, static_cast<uint32_t>(warp), 0, 500 + t);
                    ok = false;
                }
                ok = __all_sync(0xffffffffu, ok);
            }
            if (ok) {
                tc_fence_after();
                const float inv_l = l > 0.f ? 1.f / l : 0.f;
                uint8_t* stage = base_ptr + kFwdSmemQ + static_cast<uint32_t>(t) * kTileBytes;
#pragma unroll
                for (int cc = 0; cc < 4; ++cc) {
                    uint32_t v[32];
                    if (nt > 0) {
                        tmem_ld32(tO + 32u * cc, v);
                        tmem_wait_ld();
                    } else {
#pragma unroll
                        for (int j = 0; j < 32; ++j) v[j] = 0u;
                    }
#pragma unroll
                    for (int q4 = 0; q4 < 4; ++q4) {
                        uint4 w;
                        w.x = pack_bf16x2(__uint_as_float(v[8 * q4 + 0]) * inv_l, __uint_as_float(v[8 * q4 + 1]) * inv_l);
                        w.y = pack_bf16x2(__uint_as_float(v[8 * q4 + 2]) * inv_l, __uint_as_float(v[8 * q4 + 3]) * inv_l);
                        w.z = pack_bf16x2(__uint_as_float(v[8 * q4 + 4]) * inv_l, __uint_as_float(v[8 * q4 + 5]) * inv_l);
                        w.w = pack_bf16x2(__uint_as_float(v[8 * q4 + 6]) * inv_l, __uint_as_float(v[8 * q4 + 7]) * inv_l);
                        const int chunk = cc * 4 + q4;  // 16-byte chunk 0..15 of the 256-byte row
                        const uint32_t o = static_cast<uint32_t>(chunk >> 3) * kPanelBytes +
                                           static_cast<uint32_t>(row) * 128u +
                                           (static_cast<uint32_t>((chunk & 7) ^ (row & 7)) << 4);
                        *reinterpret_cast<uint4*>(stage + o) = w;
                    }
                }
                const int grow = mt * 128 + row;
                if (p.lse != nullptr && grow < p.Sq)
                    p.lse[static_cast<long long>(bh) * p.Sq + grow] =
                        l > 0.f ? (off + lg2_approx(l)) * kLn2 : -INFINITY;
                fence_proxy_async_smem();
            }
            named_bar_sync(1 + t, 128);
            if (ok && (warp & 3) == 0 && lane == 0) {
                tma_store_3d(&tm_o, 0, mt * 128, bh, sQt);
                tma_store_3d(&tm_o, 64, mt * 128, bh, sQt + kPanelBytes);
                tma_commit_group();
                tma_wait_group0();
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 8) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

}  // namespace fba

using namespace fba;

static int check_list(const fba_list_t* l, const char* who) {
    if (!l || !l->idx || !l->cnt) return set_error(FBA_ERR_BAD_ARG, who);
    if (l->stride <= 0 || l->rows_per_bh <= 0 || l->rows_div <= 0 || l->sub <= 0 ||
        (l->bh_stride != 0 && l->bh_stride != l->rows_per_bh))
        return set_error(FBA_ERR_BAD_ARG, who);
    return FBA_OK;
}

static int fwd_impl(const void* q, const void* k, const void* v, void* o, float* lse, int B, int Hq,
                    int Hkv, int Sq, int Skv, const fba_list_t* q2k, float softmax_scale, uint32_t* status,
                    void* stream_) {
    ProfRange range("fba_fwd");
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (!q || !k || !v || !o || !status)
        return set_error(FBA_ERR_BAD_ARG, "fba_fwd: null pointer argument");
    if (!(softmax_scale > 0.f) || !(softmax_scale < INFINITY))
        return set_error(FBA_ERR_BAD_ARG, "fba_fwd: softmax_scale must be positive and finite");
    if (B <= 0 || Hq <= 0 || Hkv <= 0 || Sq <= 0 || Skv <= 0)
        return set_error(FBA_ERR_BAD_ARG, "fba_fwd: non-positive size");
    if (Hq % Hkv != 0) return set_error(FBA_ERR_BAD_ARG, "fba_fwd: Hq must be a multiple of Hkv");
    if (Sq < 128 || Skv < 128)
        return set_error(FBA_ERR_BAD_ARG, "fba_fwd: sequence lengths below 128 are not supported");
    int rc = check_list(q2k, "fba_fwd: malformed q2k list");
    if (rc != FBA_OK) return rc;
    const int n_mtiles = (Sq + 127) / 128;
    const int n_ntiles = (Skv + 127) / 128;
    if (static_cast<long long>(q2k->rows_per_bh) * q2k->rows_div < n_mtiles ||
        static_cast<long long>(q2k->stride) * q2k->sub < n_ntiles)
        return set_error(FBA_ERR_BAD_ARG, "fba_fwd: q2k list does not cover the sequences");
    // An entry stands for `sub` whole key tiles and a list row for `rows_div` whole query tiles: a
    // sequence that ends inside such a group would make the kernel touch tiles past its end.
    if (n_ntiles % q2k->sub != 0 || n_mtiles % q2k->rows_div != 0)
        return set_error(FBA_ERR_BAD_ARG,
                         "fba_fwd: ceil(Skv/128) must be a multiple of q2k->sub and ceil(Sq/128) of q2k->rows_div");
    if (static_cast<long long>(B) * Hq > 65535)
        return set_error(FBA_ERR_TOO_LARGE, "fba_fwd: B * Hq exceeds 65535");
    DeviceGuard guard;
    if ((rc = guard.bind(q)) != FBA_OK) return rc;

    CUtensorMap tm_q, tm_k, tm_v, tm_o;
    if ((rc = make_tmap_bf16(&tm_q, q, Sq, static_cast<long long>(B) * Hq, 128)) != FBA_OK) return rc;
    if ((rc = make_tmap_bf16(&tm_k, k, Skv, static_cast<long long>(B) * Hkv, 128)) != FBA_OK) return rc;
    if ((rc = make_tmap_bf16(&tm_v, v, Skv, static_cast<long long>(B) * Hkv, 128)) != FBA_OK) return rc;
    if ((rc = make_tmap_bf16(&tm_o, o, Sq, static_cast<long long>(B) * Hq, 128)) != FBA_OK) return rc;

    {
        cudaError_t e = cudaFuncSetAttribute(fba_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             static_cast<int>(kFwdSmemBytes));
        if (e != cudaSuccess) {
            cudaGetLastError();
            return set_error(FBA_ERR_LAUNCH, "fba_fwd: cannot raise the dynamic shared memory limit");
        }
    }
    FwdParams p;
    p.list = to_dev(*q2k);
    p.lse = lse;
    p.status = status;
    p.n_mtiles = n_mtiles;
    p.Sq = Sq;
    p.Hq = Hq;
    p.Hkv = Hkv;
    p.scale_log2 = softmax_scale * kLog2e;
    dim3 grid((n_mtiles + 1) / 2, B * Hq);
    timing_mark(1, true, stream);
    fba_fwd_kernel<<<grid, kFwdThreads, kFwdSmemBytes, stream>>>(tm_q, tm_k, tm_v, tm_o, p);
    rc = check_launch("fba_fwd_kernel");
    timing_mark(1, false, stream);
    return rc;
}

extern "C" int fba_fwd(const void* q, const void* k, const void* v, void* o, float* lse, int B, int Hq,
                       int Hkv, int Sq, int Skv, const fba_list_t* q2k, uint32_t* status, void* stream) {
    if (!lse) return set_error(FBA_ERR_BAD_ARG, "fba_fwd: null pointer argument");
    return fwd_impl(q, k, v, o, lse, B, Hq, Hkv, Sq, Skv, q2k, kSoftmaxScale, status, stream);
}

extern "C" int fba_fwd_scaled(const void* q, const void* k, const void* v, void* o, float* lse, int B,
                              int Hq, int Hkv, int Sq, int Skv, const fba_list_t* q2k,
                              float softmax_scale, uint32_t* status, void* stream) {
    return fwd_impl(q, k, v, o, lse, B, Hq, Hkv, Sq, Skv, q2k, softmax_scale, status, stream);
}
