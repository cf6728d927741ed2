// Distance GEMM on the 5th-generation tensor cores (tcgen05 + TMEM), operands
// staged by TMA, with the top-k selection fused into the epilogue so that the
// nq x nb score matrix is never written to HBM.
//
// Replaces the reference's simdgroup_gemm_* kernels (shaders/simdgroup_gemm.metal:26-481,
// shaders/simdgroup_gemm_bf16.metal:23-242, shaders/simdgroup_gemm_family9.metal:27-470),
// their host dispatch (src/MetalDistance.mm:225-323) and, through the fused
// epilogue, fused_l2_topk_* (shaders/fused_l2_topk.metal:19-444).
//
// Two shapes of one kernel (352 threads, one CTA per SM, persistent over work items):
//  * single CTA (up to 128 queries): tile 128 x 256, cta_group::1, two TMEM accumulators;
//  * CTA pair (more queries): a cluster of two CTAs computes a 256 x 512 tile with
//    cta_group::2 MMAs (M = 256); each CTA stages its own 128 query rows and half of the X
//    rows of every k-block, and holds two 256-column accumulators (all 512 TMEM columns).
// Roles of the warps:
//   warp 0      TMA producer: Q tile (128 x 64) and X tile per k-block, 128-byte swizzle,
//               4-stage mbarrier ring
//   warps 1,10  MMA issuers: tcgen05.mma kind::f16, N = 256, K = 16, fp32 accumulators in
//               TMEM; the pair shape has two chains of them (columns 0-255 and 256-511 of the
//               tile), one issuing warp each.
//   warps 2-9   epilogue: tcgen05.ld (thread t owns query row t of the tile, two warps per
//               TMEM lane quarter, half of an accumulator's columns each), one max per column (the
//               L2 bias -||x||^2/2 is part of the dot product: 8 extra K columns, see
//               rows.cu), filter against the row's bound, hits staged in shared memory and
//               worked off after the accumulator has been released.
// Epilogue modes:
//   top-k   a sorted list of up to 32 entries per (row, column range, column half) in the
//           thread's registers; every item yields partial lists, merged afterwards
//   filter  a fixed per-row threshold; every column under it is appended to the row's
//           candidate buffer in global memory
//   store   the keys are written out as a matrix (k beyond the list paths, pairwise distances)
//   minima  the smallest key of every four columns is (samples that thresholds are taken from)
// The mode is a template parameter (eight instantiations with the two shapes): only the top-k
// kernels carry list registers.  A work item is (query block, column range).
//
// Large launches draw the 1 kW power cap: 10,000 queries, 1 M fp16 rows of d = 768, run at 1.54 GHz, the
// tensor pipe busy for 12,300 of a tile's 16,000 cycles; 4,096 queries, 10 M bf16 rows of d = 1536, at 1.1 - 1.3 GHz, 25,100
// of 29,000.
//
// FP32 storage: both operands are split into three bf16 planes
// (x = x0 + x1 + x2 exactly to 24 bits) and six plane products
// (0,0) (0,1) (1,0) (0,2) (2,0) (1,1) are accumulated in the same fp32 TMEM
// accumulator; the dropped products are below 2^-24 relative.
//
// Every wait on an mbarrier is bounded: after ~1 s of clock the waiting thread
// records kDevErrBarrierWait in the status word, raises the CTA abort flag and
// all roles drain out, TMEM is released and the kernel returns.
#include <atomic>
#include <cstdlib>
#include <type_traits>

#include "gemm_common.cuh"

namespace b200f {

namespace {

constexpr int A_STAGE_BYTES = BM * BK * 2;  // 16 KiB
constexpr int KMAX = B200F_FUSED_MAX_K;
constexpr int MMA2_WARP = 2 + NUM_EPI_WARPS;   // second MMA issuer (pair shape): one thread per accumulator chain
constexpr int NUM_THREADS = 32 * (3 + NUM_EPI_WARPS);

// Two shapes of the same kernel:
//  PAIR = false  one CTA per tile: M = 128 queries, N = 256 rows of X, cta_group::1
//  PAIR = true   two CTAs of a cluster share a 256 x 256 tile (cta_group::2): each CTA stages
//                its own 128 query rows and HALF of the X rows of every k-block, so the
//                shared-memory fill per FLOP is halved; the MMA is issued by the even CTA.
template <bool PAIR>
struct Cfg {
    static constexpr int STAGES = 4;
    static constexpr int B_ROWS = PAIR ? 128 : 256;        // rows of X this CTA stages per sub-tile
    // The pair shape computes two 256-column sub-tiles at once (same query k-block, two X k-blocks,
    // both TMEM halves): 48 KiB of shared-memory fill a CTA and 1,024 cycles of MMAs, where a 256 x 256 tile takes 64
    // (with two such accumulators in turn and 32 KiB stages 1 M fp16 rows of d = 768 took 15,983 us, 14,484 this way).  The price
    // is that a chain's epilogue does not overlap its own next MMAs.  One thread and one chain of
    // MMAs fill the tensor pipe (128.5 cycles per 256 x 256 x 16), so one chain's MMAs cover the other's epilogue:
    // each has its own accumulator-full / accumulator-free barriers, and they are read one after the other.
    static constexpr int NSUB = PAIR ? 2 : 1;              // 256-column sub-tiles per tile
    static constexpr int TILE_N = NSUB * BN;               // columns of X per tile: 512 / 256
    static constexpr int ACC_BUFS = PAIR ? 1 : 2;          // TMEM accumulator buffers of TILE_N columns
    static constexpr int B_SUB_BYTES = B_ROWS * BK * 2;    // 16 / 32 KiB
    static constexpr int B_STAGE_BYTES = NSUB * B_SUB_BYTES;  // 32 KiB either way
    static constexpr int QB = PAIR ? 256 : 128;            // query rows per work item
    // shared memory map (bytes from the 1024-aligned dynamic base)
    static constexpr int SM_A = 0;
    static constexpr int SM_B = SM_A + STAGES * A_STAGE_BYTES;
    static constexpr int SM_LKEY = SM_B + STAGES * B_STAGE_BYTES;
    // store mode transposes 32 x 32 blocks per epilogue warp here (32 x 33 floats each)
    static constexpr int SM_BAR = SM_LKEY + ((NUM_EPI_WARPS * 32 * 33 * 4 + 127) / 128) * 128;
    // barriers: full[STAGES] empty[STAGES] tfull[2] tempty[2]
    static constexpr int SM_TMEMPTR = SM_BAR + (2 * STAGES + 4) * 8;
    static constexpr int SM_ABORT = SM_TMEMPTR + 4;
    static constexpr int SMEM_BYTES = SM_ABORT + 4 + 8;
};

// Per-row candidate list held in REGISTERS by the thread that owns the row: 32 (key, id)
// pairs sorted ascending by key, every index static so nothing spills.  Inserting s drops
// the largest element: slot j takes the old slot j-1 if that is greater than s, keeps its
// value if it is <= s, and takes s otherwise.  Elements equal to s stay in front of it
// (ids arrive ascending).  For k < 32 the first 32-k slots hold -INF sentinels, so the
// k-th best key is always slot 31.
__device__ __forceinline__ void reglist_insert(float (&lk)[KMAX], int32_t (&li)[KMAX], float s,
                                               int32_t id) {
    float pk = -CUDART_INF_F;
    int32_t pi = -1;
#pragma unroll
    for (int j = 0; j < KMAX; j++) {
        const float cur = lk[j];
        const int32_t ci = li[j];
        const bool shift = pk > s;
        const bool keep = cur <= s;
        lk[j] = shift ? pk : (keep ? cur : s);
        li[j] = shift ? pi : (keep ? ci : id);
        pk = cur;
        pi = ci;
    }
}

// Hits of the tile in flight are staged per thread (stage_columns) and worked off AFTER the accumulator has been handed
// back to the MMA issuers, so that list insertion runs beside the next tile's MMAs instead of in front of them.  Only a
// thread whose stage fills up inside one tile (list warm-up, massive ties) drains it on the spot.
__device__ __forceinline__ void drain_to_list(float (&lk)[KMAX], int32_t (&li)[KMAX], const float* sk,
                                              const int32_t* si, int n, float& thr, float& thr_eff) {
    for (int i = 0; i < n; i++) {
        const float sc = sk[i * STAGE_LD];
        if (sc < thr_eff) {  // the list may have tightened since the entry was staged
            reglist_insert(lk, li, sc, si[i * STAGE_LD]);
            thr = lk[KMAX - 1];
            thr_eff = fminf(thr_eff, thr);
        }
    }
}

// MODE is a template parameter: the filter and store instantiations carry no list registers.
template <bool PAIR, int MODE>
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_topk_kernel(const __grid_constant__ CUtensorMap tmap_a,
                 const __grid_constant__ CUtensorMap tmap_b, const GemmParams p) {
    using C = Cfg<PAIR>;
    constexpr int STAGES = C::STAGES;
    constexpr int B_STAGE_BYTES = C::B_STAGE_BYTES;
    constexpr int TILE_N = C::TILE_N;
    constexpr int SM_A = C::SM_A, SM_B = C::SM_B, SM_LKEY = C::SM_LKEY;
    constexpr int SM_BAR = C::SM_BAR, SM_TMEMPTR = C::SM_TMEMPTR, SM_ABORT = C::SM_ABORT;
    // pair: all epilogue warps on one accumulator after the other, or half of them on each (lists, whose first tiles insert
    // nearly every column: 1,000 queries, 12,000 rows, k = 2: 145 us, 201 in turn)
    constexpr bool IN_TURN = MODE != MODE_TOPK;
    extern __shared__ __align__(1024) uint8_t smem[];
    const uint32_t sbase = smem_u32(smem);
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);   // uniform
    const int lane = threadIdx.x & 31;
    const uint32_t cta_rank = PAIR ? cluster_ctarank() : 0u;   // 0 = MMA issuer of the pair
    const int64_t unit = PAIR ? (blockIdx.x >> 1) : blockIdx.x;  // work is dealt to CTAs / CTA pairs
    const int64_t nunits = PAIR ? (gridDim.x >> 1) : gridDim.x;

    volatile uint32_t* tmem_ptr = reinterpret_cast<volatile uint32_t*>(smem + SM_TMEMPTR);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + SM_ABORT);

    const uint32_t bar_full = sbase + SM_BAR;
    const uint32_t bar_empty = bar_full + STAGES * 8;
    const uint32_t bar_tfull = bar_empty + STAGES * 8;
    const uint32_t bar_tempty = bar_tfull + 2 * 8;

    pdl_wait();
    pdl_trigger();
    // A launch that redoes rows counted on the device usually finds none: leave before any
    // barrier or TMEM allocation (the value is the same for every thread of every CTA).
    if (p.nq_dev && *p.nq_dev <= 0) return;

    if ((sbase & 1023u) != 0) {  // swizzled tiles need a 1024-byte aligned base (same in both CTAs)
        if (threadIdx.x == 0 && p.status) atomicOr(p.status, kDevErrSmemAlign);
        return;
    }

    if (threadIdx.x == 0) {
        *abort_flag = 0;
        for (int s = 0; s < STAGES; s++) {
            mbar_init(bar_full + s * 8, 1);
            mbar_init(bar_empty + s * 8, PAIR ? 2 : 1);   // one commit per issuing thread
        }
        for (int s = 0; s < 2; s++) {
            // single CTA: barrier s = accumulator buffer s, all epilogue warps;
            // pair: barrier s = chain s, the epilogue warps of both CTAs
            mbar_init(bar_tfull + s * 8, 1);
            mbar_init(bar_tempty + s * 8, (PAIR && IN_TURN ? 2 : 1) * NUM_EPI_WARPS);
        }
        mbar_fence_init();
    }
    if (warp == 1) {
        if (PAIR) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                                 sbase + SM_TMEMPTR),
                         "r"(TMEM_COLS)
                         : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                                 sbase + SM_TMEMPTR),
                         "r"(TMEM_COLS)
                         : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
    }
    tc_fence_before();
    __syncthreads();
    if (PAIR) cluster_sync_all();  // the peer's barriers exist before anything arrives on them
    tc_fence_after();
    const uint32_t tmem_base = *tmem_ptr;

    // live query rows: known to the host, or left in device memory by an earlier kernel
    const int64_t nq_live = p.nq_dev ? min((int64_t)*p.nq_dev, p.nq) : p.nq;
    const int nqb = p.nq_dev ? (int)((nq_live + C::QB - 1) / C::QB) : p.nqb;
    const int64_t nitems = (int64_t)nqb * p.P;
    const int kb_total = p.kb_per_pass * (p.npass - 1) + p.kb_last_pass;

    if (warp == 0) {
        // ------------------------------ TMA producer ------------------------------
        if (lane == 0) {
            fence_proxy_async_global();   // the query operand
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int64_t item = unit; item < nitems && ok; item += nunits) {
                const int qb = (int)(item % nqb);
                const int64_t xr = item / nqb;
                const int64_t t0 = xr * p.tiles_per_range;
                const int64_t t1 = min(t0 + p.tiles_per_range, p.ntiles);
                for (int64_t t = t0; t < t1 && ok; t++) {
                    const int xrow = (int)(p.col0 + t * p.tile_stride * TILE_N);
                    for (int kb = 0; kb < kb_total; kb++) {
                        if (!mbar_wait(bar_empty + stage * 8, phase ^ 1, abort_flag, p.status)) {
                            ok = false;
                            break;
                        }
                        const int pass = min(kb / p.kb_per_pass, p.npass - 1);
                        const int kk = (kb - pass * p.kb_per_pass) * BK;
                        const int pa = (p.pass_a >> (4 * pass)) & 15;
                        const int pb = (p.pass_b >> (4 * pass)) & 15;
                        if (PAIR) {
                            // both CTAs' copies complete on the issuer's barrier
                            const uint32_t fb = map_to_cta(bar_full + stage * 8, 0);
                            if (cta_rank == 0)
                                mbar_arrive_expect_tx(bar_full + stage * 8,
                                                      2 * (A_STAGE_BYTES + B_STAGE_BYTES));
                            tma_load_3d_pair(sbase + SM_A + stage * A_STAGE_BYTES, &tmap_a, fb, kk,
                                             qb * C::QB + (int)cta_rank * BM, pa);
#pragma unroll
                            for (int sub = 0; sub < C::NSUB; sub++)
                                tma_load_3d_pair(sbase + SM_B + stage * B_STAGE_BYTES + sub * C::B_SUB_BYTES,
                                                 &tmap_b, fb, kk, xrow + sub * BN + (int)cta_rank * C::B_ROWS, pb);
                        } else {
                            mbar_arrive_expect_tx(bar_full + stage * 8, p.a_rows * BK * 2 + B_STAGE_BYTES);
                            tma_load_3d(sbase + SM_A + stage * A_STAGE_BYTES, &tmap_a,
                                        bar_full + stage * 8, kk, qb * BM, pa);
                            tma_load_3d(sbase + SM_B + stage * B_STAGE_BYTES, &tmap_b,
                                        bar_full + stage * 8, kk, xrow, pb);
                        }
                        if (++stage == STAGES) {
                            stage = 0;
                            phase ^= 1;
                        }
                    }
                }
            }
            // Let every copy this thread issued land before the CTA's shared memory goes
            // away: wait (bounded) until the consumer released, or the data arrived in,
            // each stage that is still in flight.
            if (!ok) {
                long long t0 = clock64();
                while (clock64() - t0 < 2000000LL) {
                }
            }
        }
    } else if (warp == 1 || warp == MMA2_WARP) {
        // ------------------------------ MMA issuer --------------------------------
        // The whole warp walks through the tiles and one lane issues, so that control flow and operands stay uniform: the tensor
        // pipe idles whenever no MMA is issued.  In the pair shape the two accumulator chains of a tile have a warp each (warp
        // 1: columns 0-255, warp MMA2_WARP: 256-511), so that neither waits for the other's accumulator.
        const int chain = (warp == 1) ? 0 : 1;
        if (cta_rank == 0 && (chain == 0 || PAIR)) {
            const bool leader = elect_one();
            int stage = 0;
            uint32_t phase = 0;
            int acc = 0;
            uint32_t acc_phase = 0;
            bool ok = true;
            const uint64_t da0 = make_smem_desc(sbase + SM_A);
            const uint64_t db0 = make_smem_desc(sbase + SM_B);
            // the last k-block of a plane product may hold fewer than 64 valid K elements
            // (TMA zero-fills the rest): skip the all-zero sub-steps
            const int nk4_pass = (p.k_extent - (p.kb_per_pass - 1) * BK + UMMA_K - 1) / UMMA_K;
            const int nk4_end = (p.k_extent_last - (p.kb_last_pass - 1) * BK + UMMA_K - 1) / UMMA_K;
            for (int64_t item = unit; item < nitems && ok; item += nunits) {
                const int64_t xr = item / nqb;
                const int64_t t0 = xr * p.tiles_per_range;
                const int64_t t1 = min(t0 + p.tiles_per_range, p.ntiles);
                for (int64_t t = t0; t < t1 && ok; t++) {
                    const int bi = PAIR ? chain : acc;  // barrier pair of this chain / buffer
                    ok = __all_sync(0xffffffffu, mbar_wait(bar_tempty + bi * 8, acc_phase ^ 1, abort_flag, p.status));
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t d_tmem = tmem_base + acc * TILE_N + chain * BN;
                    int kin = 0;
                    const int kb_early = kb_total - p.kb_last_pass;   // k-blocks of the products before the last
                    uint32_t accumulate = 0;
                    for (int kb = 0; kb < kb_total; kb++) {
                        ok = __all_sync(0xffffffffu, mbar_wait(bar_full + stage * 8, phase, abort_flag, p.status));
                        if (!ok) break;
                        const uint64_t da = da0 + (uint64_t)(stage * (A_STAGE_BYTES >> 4));
                        const uint64_t db = db0 + (uint64_t)(stage * (B_STAGE_BYTES >> 4) + chain * (C::B_SUB_BYTES >> 4));
                        int nk4 = BK / UMMA_K;
                        if (kb < kb_early) {
                            if (++kin == p.kb_per_pass) {
                                kin = 0;
                                nk4 = nk4_pass;
                            }
                        } else if (kb == kb_total - 1) {
                            nk4 = nk4_end;
                        }
#pragma unroll
                        for (int k4 = 0; k4 < BK / UMMA_K; k4++) {
                            // advance 32 bytes (16 elements) along K inside the swizzle row
                            if (k4 < nk4) {
                                tc_mma_f16_by<PAIR>(leader, d_tmem, da + (uint64_t)(k4 * 2), db + (uint64_t)(k4 * 2), p.idesc,
                                                    k4 > 0 ? 1 : accumulate);
                                accumulate = 1;
                            }
                        }
                        tc_commit_by<PAIR>(leader, bar_empty + stage * 8);   // frees the stage when the MMAs retire
                        if (++stage == STAGES) {
                            stage = 0;
                            phase ^= 1;
                        }
                    }
                    if (!ok) break;
                    tc_commit_by<PAIR>(leader, bar_tfull + bi * 8);   // this chain's accumulator complete
                    if (C::ACC_BUFS == 2) {
                        acc ^= 1;
                        if (acc == 0) acc_phase ^= 1;
                    } else {
                        acc_phase ^= 1;
                    }
                }
            }
            if (!ok) {   // let the MMAs in flight retire before tensor memory goes away
                const long long t0 = clock64();
                while (clock64() - t0 < 200000LL) {
                }
            }
        }
    } else if (warp >= 2 && warp < 2 + NUM_EPI_WARPS) {
        // ------------------------------ epilogue -----------------------------------
        const int ew = warp & 3;              // TMEM lane quarter this warp may read
        const int eh = (warp - 2) >> 2;       // which half of an accumulator's columns this warp scans
        constexpr int CH_PER_HALF = PAIR && !IN_TURN ? BN / 32 : BN / 64;
        const int warp_rows = PAIR ? 32 : p.warp_rows;
        const int row = ew * warp_rows + lane;   // row of the tile owned by this thread, if lane < warp_rows
        int acc = 0;
        uint32_t acc_phase = 0;
        bool ok = true;
        const int k = p.k;
        float lk[KMAX];     // this thread's row list (see reglist_insert)
        int32_t li[KMAX];
        // this thread's stage (see drain_to_list); the area serves the transposes in store mode
        float* const stage_key = reinterpret_cast<float*>(smem + SM_LKEY) + (threadIdx.x - 64);
        int32_t* const stage_idx =
                reinterpret_cast<int32_t*>(smem + SM_LKEY) + STAGE_N * STAGE_LD + (threadIdx.x - 64);
        int nstaged = 0;
        for (int64_t item = unit; item < nitems && ok; item += nunits) {
            const int qb = (int)(item % nqb);
            const int64_t xr = item / nqb;
            const int64_t t0 = xr * p.tiles_per_range;
            const int64_t t1 = min(t0 + p.tiles_per_range, p.ntiles);
            const int64_t grow = (int64_t)qb * C::QB + (int64_t)cta_rank * BM + row;
            const bool row_live = grow < nq_live && lane < warp_rows;
            // slot of the row's bound array this list publishes to
            uint32_t* const gslot = p.gthr ? p.gthr + grow * p.gslots + (int)((2 * xr + eh) % p.gslots) : nullptr;
            float ksc = p.kscale;          // this row's key scale
            // coherent loads: the kernel before a programmatic launch wrote the map
            if (p.rowscale && row_live) ksc *= __ldcg(p.rowscale + (p.rowscale_map ? (int64_t)__ldcg(p.rowscale_map + grow) : grow));
            float thr = CUDART_INF_F;      // worst key of this thread's list (k-th best of the range)
            float thr_eff = CUDART_INF_F;  // filter: min(thr, bound shared by all ranges of the row)
            float thr_pub = CUDART_INF_F;  // last value published to gthr
            float radd = 0.f;
            if (MODE == MODE_TOPK) {
#pragma unroll
                for (int j = 0; j < KMAX; j++) {
                    lk[j] = (j >= KMAX - k) ? CUDART_INF_F : -CUDART_INF_F;
                    li[j] = -1;
                }
            } else if (MODE == MODE_FILTER) {
                thr_eff = row_live ? filter_threshold(__ldcg(p.fthr + grow * p.fthr_stride + p.fthr_pos) / ksc) : -CUDART_INF_F;   // -INF passes nothing
            } else if (row_live && p.rowadd) {
                radd = p.rowadd[grow];
            }
            auto drain = [&]() {
                if (drain_stage(p.cand_cnt + grow, p.cand_key + grow * p.cand_cap, p.cand_idx + grow * p.cand_cap, p.cand_cap, ksc,
                                stage_key, stage_idx, nstaged))
                    thr_eff = -CUDART_INF_F;
                nstaged = 0;
            };
            for (int64_t t = t0; t < t1 && ok; t++) {
                // Pair: one accumulator after the other, all eight warps on each, so that the first is back with its
                // issuer, whose MMAs by themselves fill the pipe, while the second is read.  Half of the warps on each at the same
                // time left the pipe idle for all of it (10,000 queries, 1 M fp16 rows of d = 768: a fifth of a tile's 17,500 cycles).
#pragma unroll 1
                for (int sub = PAIR && !IN_TURN ? eh : 0; sub < (PAIR && !IN_TURN ? eh + 1 : C::NSUB); sub++) {
                const int buf = PAIR ? sub : acc;
                const int64_t c_tile = p.col0 + t * p.tile_stride * TILE_N + sub * BN;
                {
                    const bool w = mbar_wait(bar_tfull + buf * 8, acc_phase, abort_flag, p.status);
                    if (!__all_sync(0xffffffffu, w)) {  // keep the warp converged for tcgen05.ld
                        ok = false;
                        break;
                    }
                }
                tc_fence_after();
                if (MODE == MODE_TOPK && row_live) {
                    // A full list's worst key bounds the row's 32nd best from above; the largest
                    // of gslots such keys (distinct lists) bounds the (32 * gslots)-th best, which
                    // is at or beyond the k-th.  Publish ours, adopt the bound.  A key equal to
                    // the bound may still win a tie on the id, so the filter admits s <= bound.
                    if (thr < thr_pub) {
                        atomicMin(gslot, float_to_ordered(thr));
                        thr_pub = thr;
                    }
                    uint32_t g = 0;
                    for (int sidx = 0; sidx < p.gslots; sidx++)
                        g = max(g, __ldcg(p.gthr + grow * p.gslots + sidx));
                    const float gnext = (g >= 0xff800000u) ? CUDART_INF_F : ordered_to_float(g + 1u);
                    thr_eff = fminf(thr, gnext);
                }
                // The accumulator holds t = q.x (- ||x||^2/2 for L2): larger is better; the
                // lists keep s = -t (smaller is better).  Rows of X beyond the last valid
                // column are zero-filled by TMA (t = 0) and must be masked out.
                const bool partial = c_tile + BN > p.ncols_end;
                const uint32_t taddr = tmem_base + ((uint32_t)(ew * 32) << 16) + buf * BN;
                auto release = [&]() {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) {
                        if (PAIR) mbar_arrive_cluster(map_to_cta(bar_tempty + buf * 8, 0));
                        else mbar_arrive(bar_tempty + buf * 8);
                    }
                };
                // this warp's columns
                const int64_t chalf = c_tile + (PAIR && !IN_TURN ? 0 : eh * CH_PER_HALF * 32);
                const uint32_t thalf = taddr + (PAIR && !IN_TURN ? 0 : eh * CH_PER_HALF * 32);
                if constexpr (MODE == MODE_TOPK) {
#pragma unroll 1
                for (int ch = 0; ch < CH_PER_HALF; ch++) {
                    uint32_t r[32];
                    tc_ld32(thalf + ch * 32, r);
                    tc_wait_ld();
                    const int64_t cbase = chalf + ch * 32;
                    if (partial) mask_columns(r, cbase, p.ncols_end);
                    float gm[4];
                    group_maxima(r, gm);
                    // entered by the whole warp when any row has a candidate in this chunk
                    if (__any_sync(0xffffffffu, row_live && -fmaxf(max3(gm[0], gm[1], gm[2]), gm[3]) < thr_eff)) {
#pragma unroll
                        for (int g = 0; g < 4; g++) {
                            const bool hit = row_live && -gm[g] < thr_eff;
                            if (!__any_sync(0xffffffffu, hit)) continue;
                            if (hit) {
                                if (nstaged > STAGE_N - 8) {   // rare: list warm-up, massive ties
                                    drain_to_list(lk, li, stage_key, stage_idx, nstaged, thr, thr_eff);
                                    nstaged = 0;
                                }
#pragma unroll
                                for (int c = 0; c < 8; c++) {
                                    const float sc = -__uint_as_float(r[8 * g + c]);
                                    if (sc < thr_eff) {
                                        stage_key[nstaged * STAGE_LD] = sc;
                                        stage_idx[nstaged * STAGE_LD] = (int32_t)cbase + 8 * g + c;
                                        nstaged++;
                                    }
                                }
                            }
                        }
                        __syncwarp();
                    }
                }
                release();
                } else if constexpr (MODE == MODE_FILTER) {
                    auto stage = [&](uint32_t(&r)[32], int ch) {
                        stage_columns(r, chalf + ch * 32, p.ncols_end, partial, thr_eff, stage_key, stage_idx, nstaged, drain);
                    };
                    // reading ahead pays where hits hold most chunks up (300 queries, k = 1024, 1 M bf16 rows of d = 1024: 1,073 ->
                    // 965 us), not beside full query blocks with few (1,000 queries, k = 100: 1,760 against 1,888)
                    if (p.dense) scan_columns_ahead<CH_PER_HALF>(thalf, stage, release);
                    else scan_columns(thalf, CH_PER_HALF, stage, release);
                } else if constexpr (MODE == MODE_MINIMA) {
                    float* const out = p.out + grow * p.ld + (t * TILE_N + sub * BN + eh * CH_PER_HALF * 32) / MIN_GROUP;
                    scan_columns(
                            thalf, CH_PER_HALF,
                            [&](uint32_t(&r)[32], int ch) {
                                if (partial) mask_columns(r, chalf + ch * 32, p.ncols_end);
                                if (row_live) store_minima(r, ksc, out + ch * (32 / MIN_GROUP));
                            },
                            release);
                } else {
                    const bool whole = !partial && (p.ld & 7) == 0 && (reinterpret_cast<uintptr_t>(p.out) & 31) == 0;
                    // the list area is idle in this mode; tiles lie side by side in the output, whatever the stride
                    float* const tbuf = reinterpret_cast<float*>(smem + SM_LKEY) + (warp - 2) * (32 * 33);
                    const int64_t ohalf = t * TILE_N + sub * BN + eh * CH_PER_HALF * 32;
                    scan_columns(
                            thalf, CH_PER_HALF,
                            [&](uint32_t(&r)[32], int ch) {
                                store_keys(p, r, whole, grow, lane, warp_rows, nq_live, row_live, chalf + ch * 32, ohalf + ch * 32, ksc, radd, tbuf);
                            },
                            release);
                }
                }
                if (!ok) break;
                // the accumulators are back with the MMA issuers: now work off the staged hits
                if (MODE == MODE_TOPK && nstaged > 0) {
                    drain_to_list(lk, li, stage_key, stage_idx, nstaged, thr, thr_eff);
                    nstaged = 0;
                }
                if (MODE == MODE_FILTER && __any_sync(0xffffffffu, nstaged > STAGE_N / 2)) drain();
                __syncwarp();
                if (C::ACC_BUFS == 2) {
                    acc ^= 1;
                    if (acc == 0) acc_phase ^= 1;
                } else {
                    acc_phase ^= 1;
                }
            }
            if (MODE == MODE_FILTER && ok) drain();   // the next item has other rows
            if (MODE == MODE_TOPK && row_live && ok) {
                if (thr < thr_pub) atomicMin(gslot, float_to_ordered(thr));
                // two lists per (row, column range): one per column half
                float* okey = p.part_key + (grow * (2 * p.P) + 2 * xr + eh) * k - (KMAX - k);
                int32_t* oidx = p.part_idx + (grow * (2 * p.P) + 2 * xr + eh) * k - (KMAX - k);
#pragma unroll
                for (int j = 0; j < KMAX; j++) {
                    if (j >= KMAX - k) {
                        okey[j] = ksc * lk[j];  // INF stays INF for empty slots
                        oidx[j] = li[j];
                    }
                }
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (PAIR) cluster_sync_all();  // the peer may still read this CTA's tiles / signal its barriers
    if (warp == 1) {
        __syncwarp();
        if (PAIR)
            asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                         "r"(TMEM_COLS)
                         : "memory");
        else
            asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                         "r"(TMEM_COLS)
                         : "memory");
    }
}

// ---- host side -------------------------------------------------------------------------

int launch_common(const GemmOperands& op, const GemmPlan& plan, GemmParams& p, int64_t col0,
                  int64_t ncols, const Launch& ln) {
    if (op.nq <= 0 || ncols <= 0) return B200F_OK;
    if (col0 + ncols > op.nb || op.nb > 0x7fffffffLL) return B200F_ERR_BAD_ARG;
    CUtensorMap ma, mb;
    p.a_rows = plan.pair || op.nq >= BM ? BM : (int)round_up64(op.nq, 8);
    int rc = make_operand_map(&ma, op.a_planes, op.is_bf16, op.d_pad, op.nq, op.a_pitch, op.npl,
                              op.a_plane_stride, p.a_rows);
    if (rc != B200F_OK) return rc;
    rc = make_operand_map(&mb, op.b_planes, op.is_bf16, op.d_pad, op.nb, op.b_pitch, op.npl,
                          op.b_plane_stride, plan.pair ? Cfg<true>::B_ROWS : Cfg<false>::B_ROWS);
    if (rc != B200F_OK) return rc;

    p.nq = op.nq;
    p.nq_dev = op.nq_dev;
    if (p.tile_stride < 1) p.tile_stride = 1;
    p.col0 = col0;
    p.ncols_end = col0 + ncols;
    p.ntiles = plan.ntiles;
    p.tiles_per_range = plan.tiles_per_range;
    p.nqb = plan.nqb;
    p.P = plan.P;
    p.kb_per_pass = (int)ceil_div64(op.d_data, BK);
    p.k_extent = op.d_data;
    p.kb_last_pass = (int)ceil_div64(op.d_pad, BK);
    p.k_extent_last = op.d_pad;
    p.rowscale = op.rowscale;
    p.rowscale_map = op.rowscale_map;
    if (op.npl == 1) {
        p.npass = 1;
        p.pass_a = 0;
        p.pass_b = 0;
    } else if (op.npl == 2) {
        // two fp16 planes (22 bits): (1,0) (0,1) (0,0), smallest first; (1,1) is below 2^-22
        p.npass = 3;
        p.pass_a = 0x001u;
        p.pass_b = 0x010u;
    } else {
        // smallest products first: (1,1) (0,2) (2,0) (0,1) (1,0) (0,0)
        p.npass = 6;
        p.pass_a = 0x010201u;  // nibble i = plane of A in pass i (pass 0 is the lowest nibble)
        p.pass_b = 0x001021u;
    }
    // At most 64 queries are a tile of M = 64 (its rows lie in all four lane quarters, sixteen in each): half the operand reads and
    // products on rows that hold no query, which cost power where the memory is the bound.  Four batches of 24 queries in flight, 1,000,003
    // fp16 rows of d = 770: 1,380 -> 1,290 us at the power cap, 1.48 -> 1.61 GHz; 50 queries, k = 2048, 300,007 rows of d = 256,
    // below the cap: level.
    const int m = plan.pair ? 2 * BM : op.nq <= 64 ? 64 : BM;
    p.warp_rows = m == 64 ? 16 : 32;
    const uint32_t fmt = op.is_bf16 ? 1u : 0u;
    // fp32 accumulate, K-major operands, N = 256, M = 64 or 128 (one CTA) or 256 (CTA pair)
    p.idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(BN >> 3) << 17) |
              ((uint32_t)(m >> 4) << 24);

    typedef void (*KernelFn)(const CUtensorMap, const CUtensorMap, const GemmParams);
    static const KernelFn kernels[2][4] = {
            {gemm_topk_kernel<false, MODE_TOPK>, gemm_topk_kernel<false, MODE_STORE>,
             gemm_topk_kernel<false, MODE_FILTER>, gemm_topk_kernel<false, MODE_MINIMA>},
            {gemm_topk_kernel<true, MODE_TOPK>, gemm_topk_kernel<true, MODE_STORE>,
             gemm_topk_kernel<true, MODE_FILTER>, gemm_topk_kernel<true, MODE_MINIMA>}};
    static bool attr_set[kMaxDevices] = {false};   // the shared-memory opt-in is per device
    const int slot = device_slot();
    if (!attr_set[slot]) {
        for (int pr = 0; pr < 2; pr++)
            for (int m = 0; m < 4; m++)
                B200F_CUDA_TRY(cudaFuncSetAttribute(reinterpret_cast<const void*>(kernels[pr][m]),
                                                    cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                    pr ? Cfg<true>::SMEM_BYTES : Cfg<false>::SMEM_BYTES));
        attr_set[slot] = true;
    }
    if (p.mode < 0 || p.mode > 3) return B200F_ERR_BAD_ARG;
    const KernelFn kernel = kernels[plan.pair ? 1 : 0][p.mode];
    main_kernel_begin(ln);
    if (p.mode != MODE_TOPK && resident_fits(op, plan)) {
        rc = launch_resident(op, plan, p, ma, mb, ln);
        main_kernel_end(ln);
        if (rc != B200F_OK) return rc;
        count_launch();
        return B200F_OK;
    }
    if (plan.pair || ln.overlap) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)plan.grid, 1, 1);
        cfg.blockDim = dim3(NUM_THREADS, 1, 1);
        cfg.dynamicSmemBytes = plan.pair ? Cfg<true>::SMEM_BYTES : Cfg<false>::SMEM_BYTES;
        cfg.stream = ln.stream;
        cudaLaunchAttribute attr[2];
        cfg.attrs = attr;
        if (plan.pair) {
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = 2;
            attr[0].val.clusterDim.y = 1;
            attr[0].val.clusterDim.z = 1;
            cfg.numAttrs = 1;
        }
        if (ln.overlap) {
            attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            attr[cfg.numAttrs].val.programmaticStreamSerializationAllowed = 1;
            cfg.numAttrs++;
        }
        cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, ma, mb, p);
        if (e != cudaSuccess) {
            (void)cudaGetLastError();
            main_kernel_end(ln);
            return B200F_ERR_CUDA;
        }
    } else {
        kernel<<<plan.grid, NUM_THREADS, Cfg<false>::SMEM_BYTES, ln.stream>>>(ma, mb, p);
    }
    main_kernel_end(ln);
    count_launch();
    B200F_LAUNCH_CHECK();
    return B200F_OK;
}

}  // namespace

// Shape override (testing): b200f_set_gemm_shape, default from the environment variable
// B200F_GEMM_PAIR=0 / 1 read ONCE at the first plan.  -1 = choose by the number of queries.
static std::atomic<int> g_pair_override{-2};

static int pair_override() {
    int v = g_pair_override.load(std::memory_order_relaxed);
    if (v == -2) {
        const char* e = getenv("B200F_GEMM_PAIR");
        v = (e && (e[0] == '0' || e[0] == '1')) ? e[0] - '0' : -1;
        int expected = -2;
        if (!g_pair_override.compare_exchange_strong(expected, v)) v = expected;
    }
    return v;
}

// CTA pairs that can be resident at once (GPC boundaries may leave a few SMs unpaired).
static int max_active_pairs(int sm_count) {
    static int per_device[kMaxDevices] = {0};   // 0 = not asked yet on that device
    int& cached = per_device[device_slot()];
    if (cached <= 0) {
        cached = sm_count / 2;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)(sm_count / 2 * 2), 1, 1);
        cfg.blockDim = dim3(NUM_THREADS, 1, 1);
        cfg.dynamicSmemBytes = Cfg<true>::SMEM_BYTES;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 2;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaFuncSetAttribute(gemm_topk_kernel<true, MODE_TOPK>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 Cfg<true>::SMEM_BYTES) == cudaSuccess &&
            cudaOccupancyMaxActiveClusters(&n, gemm_topk_kernel<true, MODE_TOPK>, &cfg) == cudaSuccess && n > 0) {
            if (n < cached) cached = n;
        } else {
            (void)cudaGetLastError();
        }
    }
    return cached;
}

GemmPlan plan_gemm(int64_t nq, int64_t ncols, int sm_count) {
    GemmPlan g;
    const int ov = pair_override();
    g.pair = ov >= 0 ? ov : (nq > BM ? 1 : 0);       // a pair covers 256 query rows
    const int qb = g.pair ? 2 * BM : BM;
    const int units = g.pair ? max_active_pairs(sm_count) : sm_count;  // CTAs or CTA pairs that run at once
    g.units = units;
    g.nqb = (int)ceil_div64(nq, qb);
    g.tile_n = g.pair ? Cfg<true>::TILE_N : Cfg<false>::TILE_N;
    g.ntiles = ceil_div64(ncols, g.tile_n);
    if (g.nqb <= 0 || g.ntiles <= 0) {
        g.nqb = 0; g.ntiles = 0; g.P = 0; g.tiles_per_range = 0; g.grid = 0;
        return g;
    }
    // Number of column ranges: make nqb * P a multiple of the unit count when there is
    // enough work, keep at least ~32 tiles per range so list warm-up stays cheap.
    auto gcd = [](int64_t a, int64_t b) { while (b) { int64_t t = a % b; a = b; b = t; } return a; };
    int64_t P0 = units / gcd(units, g.nqb);
    int64_t P;
    if (P0 >= g.ntiles) {
        P = g.ntiles;
    } else {
        int64_t max_mult = g.ntiles / (P0 * 32);
        int64_t want_waves = 8;
        int64_t mult = (want_waves * units) / (P0 * g.nqb);
        if (mult < 1) mult = 1;
        if (max_mult < 1) max_mult = 1;
        if (mult > max_mult) mult = max_mult;
        P = P0 * mult;
    }
    if (P > 4096) P = 4096;
    g.tiles_per_range = ceil_div64(g.ntiles, P);
    g.P = (int)ceil_div64(g.ntiles, g.tiles_per_range);
    int64_t items = (int64_t)g.nqb * g.P;
    int64_t u = items < units ? items : units;
    g.grid = (int)(g.pair ? 2 * u : u);
    return g;
}

// Filter and store launches carry nothing from one tile of a range to the next: ranges as short as even
// out the last wave (1,000 queries, 100,000 rows: 784 tiles on 74 CTA pairs, 12 tile times with ranges of
// six, 11 with ranges of one), a tenth of a tile being what a range costs by itself.
static GemmPlan spread_plan(GemmPlan g) {
    double best = 0.0;
    const int64_t longest = g.tiles_per_range;
    for (int64_t tpr = 1; tpr <= longest; tpr = tpr < 8 ? tpr + 1 : tpr + tpr / 4) {
        const int64_t P = ceil_div64(g.ntiles, tpr);
        const double cost = (double)ceil_div64(P * g.nqb, g.units) * ((double)tpr + 0.1);
        if (tpr == 1 || cost < best) {
            best = cost;
            g.tiles_per_range = tpr;
            g.P = (int)P;
        }
    }
    if (longest > 0) {
        const int64_t items = (int64_t)g.nqb * g.P, u = items < g.units ? items : g.units;
        g.grid = (int)(g.pair ? 2 * u : u);
    }
    return g;
}

int launch_gemm_topk(const GemmOperands& op, const GemmPlan& plan, int64_t col0, int64_t ncols,
                     int64_t tile_stride, float kscale, int k, int gslots, float* part_key,
                     int32_t* part_idx, uint32_t* gthr, bool gthr_ready, int32_t* status,
                     const Launch& ln) {
    if (k <= 0 || k > KMAX || gslots < 1) return B200F_ERR_UNSUPPORTED;
    if (!gthr) return B200F_ERR_BAD_ARG;
    // all-ones is above every ordered float: no bound yet
    if (!gthr_ready) B200F_CUDA_TRY(cudaMemsetAsync(gthr, 0xff, (size_t)op.nq * gslots * sizeof(uint32_t), ln.stream));
    GemmParams p{};
    p.mode = MODE_TOPK;
    p.tile_stride = tile_stride;
    p.gslots = gslots;
    p.k = k;
    p.kscale = kscale;
    p.sign = 1.f;
    p.rowadd = nullptr;
    p.part_key = part_key;
    p.part_idx = part_idx;
    p.gthr = gthr;
    p.out = nullptr;
    p.ld = 0;
    p.status = status;
    return launch_common(op, plan, p, col0, ncols, ln);
}

int launch_gemm_filter(const GemmOperands& op, const GemmPlan& plan, float kscale, const float* thr,
                       int thr_stride, int thr_pos, float* cand_key, int32_t* cand_idx,
                       int32_t* cand_cnt, int cand_cap, int dense, int32_t* status,
                       const Launch& ln) {
    if (!thr || !cand_key || !cand_idx || !cand_cnt || cand_cap < 1) return B200F_ERR_BAD_ARG;
    GemmParams p{};
    p.mode = MODE_FILTER;
    p.kscale = kscale;
    p.sign = 1.f;
    p.fthr = thr;
    p.fthr_stride = thr_stride;
    p.fthr_pos = thr_pos;
    p.cand_key = cand_key;
    p.cand_idx = cand_idx;
    p.cand_cnt = cand_cnt;
    p.cand_cap = cand_cap;
    p.dense = dense;
    p.status = status;
    return launch_common(op, spread_plan(plan), p, 0, op.nb, ln);
}

int launch_gemm_store(const GemmOperands& op, const GemmPlan& plan, int64_t col0, int64_t ncols,
                      int64_t tile_stride, float kscale, float sign, const float* rowadd, float* out,
                      int64_t ld, int32_t* status, const Launch& ln) {
    GemmParams p{};
    p.mode = MODE_STORE;
    p.tile_stride = tile_stride;
    p.k = 0;
    p.kscale = kscale;
    p.sign = sign;
    p.rowadd = rowadd;
    p.part_key = nullptr;
    p.part_idx = nullptr;
    p.out = out;
    p.ld = ld;
    p.status = status;
    return launch_common(op, spread_plan(plan), p, col0, ncols, ln);
}

int launch_gemm_minima(const GemmOperands& op, const GemmPlan& plan, int64_t ncols, int64_t tile_stride, float kscale,
                       float* out, int64_t ld, int32_t* status, const Launch& ln) {
    if (!out || ld % 8 != 0 || (reinterpret_cast<uintptr_t>(out) & 31) != 0) return B200F_ERR_BAD_ARG;
    GemmParams p{};
    p.mode = MODE_MINIMA;
    p.tile_stride = tile_stride;
    p.kscale = kscale;
    p.sign = 1.f;
    p.out = out;
    p.ld = ld;
    p.status = status;
    return launch_common(op, spread_plan(plan), p, 0, ncols, ln);
}

}  // namespace b200f

extern "C" int b200f_set_gemm_shape(int shape) {
    if (shape < B200F_GEMM_SHAPE_AUTO || shape > B200F_GEMM_SHAPE_PAIR) return B200F_ERR_BAD_ARG;
    b200f::g_pair_override.store(shape, std::memory_order_relaxed);
    return B200F_OK;
}
