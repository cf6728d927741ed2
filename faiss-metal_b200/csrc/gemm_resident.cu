// Distance GEMM for narrow rows: the query block stays in shared memory, X alone is streamed.
//
// Serves the filter, store and minima launches of gemm_topk.cu (same operands, same outputs, bit for bit: every accumulator
// takes the same MMAs in the same order) where a query block and the k-blocks of one X tile fit shared memory
// together (resident_blocks): inner product on fp32 rows up to d = 192 and 16-bit rows up to d = 384, L2 with its eight norm
// columns up to 184 and 376; more than 128 queries.  A
// tile has so few MMAs there (36 at most) that reading its accumulator takes as long, and the pair shape of
// gemm_topk.cu, whose two accumulators fill the tensor memory, cannot do both at once.
//
// A cluster of two CTAs per 256 x 256 tile (cta_group::2, M = N = 256), persistent over work items (query block, every P-th
// X tile; neighbouring tiles in one item would leave the hits of rows that are near one another and stored side by side to a
// few CTAs: 100 of 1,000 queries near 15,000 equal rows in a row, 100,000 rows: 1,373 us a search, 866 so):
//   warp 0     producer: the CTA's half of the query block once per item, then its half (128 rows) of the X k-blocks,
//              16 KiB each, through a ring of barriers per block
//   warp 1     of the even CTA: MMAs of one tile after another into two accumulators of 256 columns.  The whole warp walks through
//              the tiles and one lane issues: by a lane alone an MMA took 190 cycles with the waits and commits around it, the
//              tensor pipe 128 (tile of 19 MMAs: 3,689 -> 2,920 cycles)
//   warps 2..  epilogue: a warp reads 32 rows and a part of the columns of one accumulator while the MMAs of the
//              next tile fill the other; twelve warps where hits are few, else eight
// X blocks that two plane products share (fp32 rows: plane 0 meets both query planes) are loaded once and used
// twice: 64 KiB a CTA and tile of d = 96 instead of 144 with the query blocks.
//
// Against the pair shape of gemm_topk.cu, at its introduction: 2,048 queries, k = 1024, 5 M fp32 rows of d = 96: 8.15 -> 6.08 ms a
// search; 1,000 queries, k = 10, 100,000 fp32 rows of d = 128: 189 -> 156 us; with twelve warps and the hits' queue the first takes
// 5.2 ms and draws the power cap (1.52 GHz).
#include "gemm_common.cuh"

namespace b200f {

namespace {

// Epilogue warps: three per TMEM lane quarter where hits are few (5,345 -> 5,170 us for the first search above), which their
// registers allow; else two.
template <int MODE>
constexpr int RES_EPI_WARPS = MODE == MODE_FILTER ? 12 : NUM_EPI_WARPS;
template <int MODE>
constexpr int RES_THREADS = 32 * (2 + RES_EPI_WARPS<MODE>);
constexpr int RES_BLOCK_BYTES = 128 * BK * 2;   // a k-block of 128 query rows or 128 rows of X
constexpr int RES_BLOCKS = 12;                  // query block and ring together
constexpr int RES_MAX_RING = 11;
constexpr int RES_SM_STAGE = RES_BLOCKS * RES_BLOCK_BYTES;
// barriers: full[ring] empty[ring] | query block full, empty | accumulators full[2] empty[2]
constexpr int RES_SM_BAR = RES_SM_STAGE + ((NUM_EPI_WARPS * 32 * 33 * 4 + 127) / 128) * 128;
constexpr int RES_SM_TMEMPTR = RES_SM_BAR + (2 * RES_MAX_RING + 6) * 8;
constexpr int RES_SM_ABORT = RES_SM_TMEMPTR + 4;
constexpr int RES_SMEM_BYTES = RES_SM_ABORT + 4 + 8;
constexpr int RES_TILE_N = 256;
static_assert(RES_EPI_WARPS<MODE_FILTER> * HITS_BYTES <= RES_SM_BAR - RES_SM_STAGE && HITS_BYTES % 16 == 0, "hits share the transposes' area");

struct ResidentParams {
    GemmParams g;        // ntiles and P count tiles of 256 columns; an item takes every P-th
    int nkd, nkl;        // k-blocks of a plane without and with the norm columns (plane 0 has them)
    int n_blocks;        // blocks of the query block, and of an X tile
    int ring;            // X blocks in shared memory, >= n_blocks
};

template <int MODE>
__global__ void __launch_bounds__(RES_THREADS<MODE>, 1)
gemm_resident_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                     const ResidentParams rp) {
    const GemmParams& p = rp.g;
    constexpr bool FILTER = MODE == MODE_FILTER || MODE == MODE_DENSE;
    extern __shared__ __align__(1024) uint8_t smem[];
    const uint32_t sbase = smem_u32(smem);
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);   // uniform
    const int lane = threadIdx.x & 31;
    const uint32_t cta_rank = cluster_ctarank();   // 0 = MMA issuer of the pair
    const int64_t unit = blockIdx.x >> 1, nunits = gridDim.x >> 1;

    volatile uint32_t* tmem_ptr = reinterpret_cast<volatile uint32_t*>(smem + RES_SM_TMEMPTR);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + RES_SM_ABORT);
    const uint32_t bar_full = sbase + RES_SM_BAR;
    const uint32_t bar_empty = bar_full + RES_MAX_RING * 8;
    const uint32_t bar_qfull = bar_empty + RES_MAX_RING * 8;
    const uint32_t bar_qempty = bar_qfull + 8;
    const uint32_t bar_tfull = bar_qempty + 8;
    const uint32_t bar_tempty = bar_tfull + 16;

    pdl_wait();
    pdl_trigger();
    // A launch that redoes rows counted on the device usually finds none: leave before any barrier or TMEM
    // allocation (the value is the same for every thread of every CTA).
    if (p.nq_dev && *p.nq_dev <= 0) return;
    if ((sbase & 1023u) != 0) {   // swizzled tiles need a 1024-byte aligned base (same in both CTAs)
        if (threadIdx.x == 0 && p.status) atomicOr(p.status, kDevErrSmemAlign);
        return;
    }
    if (threadIdx.x == 0) {
        *abort_flag = 0;
        for (int s = 0; s < rp.ring; s++) {
            mbar_init(bar_full + s * 8, 1);
            mbar_init(bar_empty + s * 8, 1);
        }
        mbar_init(bar_qfull, 1);
        mbar_init(bar_qempty, 1);
        for (int s = 0; s < 2; s++) {
            mbar_init(bar_tfull + s * 8, 1);
            mbar_init(bar_tempty + s * 8, 2 * RES_EPI_WARPS<MODE>);   // the epilogue warps of both CTAs
        }
        mbar_fence_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sbase + RES_SM_TMEMPTR),
                     "r"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();   // the peer's barriers exist before anything arrives on them
    tc_fence_after();
    const uint32_t tmem_base = *tmem_ptr;

    const int64_t nq_live = p.nq_dev ? min((int64_t)*p.nq_dev, p.nq) : p.nq;
    const int nqb = p.nq_dev ? (int)((nq_live + 255) / 256) : p.nqb;
    const int64_t nitems = (int64_t)nqb * p.P;
    const int nkd = rp.nkd, nkl = rp.nkl, nb = rp.n_blocks, ring = rp.ring;
    const bool two = p.npass > 1;   // two planes
    // first column of tile t: 512-column tiles, every tile_stride-th, in halves
    auto tile_col = [&](int64_t t) { return p.col0 + (t >> 1) * p.tile_stride * 512 + (t & 1) * RES_TILE_N; };

    if (warp == 0) {
        // ------------------------------ producer ------------------------------
        if (elect_one()) {
            fence_proxy_async_global();   // the query operand
            const uint32_t sb = sbase + nb * RES_BLOCK_BYTES;   // the ring
            const uint32_t full0 = map_to_cta(bar_full, 0), qfull0 = map_to_cta(bar_qfull, 0);
            int slot = 0, have_qb = -1;
            uint32_t phase = 0, qphase = 0;
            bool ok = true;
            for (int64_t item = unit; item < nitems && ok; item += nunits) {
                const int qb = (int)(item % nqb);
                if (qb != have_qb) {
                    if (!mbar_wait(bar_qempty, qphase ^ 1, abort_flag, p.status)) {
                        ok = false;
                        break;
                    }
                    if (cta_rank == 0) mbar_arrive_expect_tx(bar_qfull, 2 * nb * RES_BLOCK_BYTES);
                    // in the order of the products: the second plane's blocks first
                    for (int i = 0; i < nb; i++) {
                        const bool low = two && i < nkd;
                        tma_load_3d_pair(sbase + i * RES_BLOCK_BYTES, &tmap_a, qfull0, (two && !low ? i - nkd : i) * BK,
                                         qb * 256 + (int)cta_rank * BM, low ? 1 : 0);
                    }
                    qphase ^= 1;
                    have_qb = qb;
                }
                for (int64_t t = item / nqb; t < p.ntiles && ok; t += p.P) {
                    const int xrow = (int)tile_col(t) + (int)cta_rank * 128;
                    for (int i = 0; i < nb; i++) {
                        if (!mbar_wait(bar_empty + slot * 8, phase ^ 1, abort_flag, p.status)) {
                            ok = false;
                            break;
                        }
                        // order of first use: plane 0, plane 1, the norm columns' block of plane 0
                        const bool low = two && i >= nkd && i < 2 * nkd;
                        const int kb = !two || i < nkd ? i : i < 2 * nkd ? i - nkd : nkd;
                        // both CTAs' copies complete on the issuer's barrier
                        if (cta_rank == 0) mbar_arrive_expect_tx(bar_full + slot * 8, 2 * RES_BLOCK_BYTES);
                        tma_load_3d_pair(sb + slot * RES_BLOCK_BYTES, &tmap_b, full0 + slot * 8, kb * BK, xrow, low ? 1 : 0);
                        if (++slot == ring) {
                            slot = 0;
                            phase ^= 1;
                        }
                    }
                }
            }
            if (!ok) {   // let the copies in flight land before shared memory goes away
                const long long t0 = clock64();
                while (clock64() - t0 < 2000000LL) {
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ------------------------------ MMA issuer ------------------------------
        // The whole warp walks through the tiles and one lane issues.
        if (cta_rank == 0) {
            const bool leader = elect_one();
            const uint64_t da0 = make_smem_desc(sbase);
            const uint64_t db0 = make_smem_desc(sbase + nb * RES_BLOCK_BYTES);
            constexpr uint64_t BLOCK = RES_BLOCK_BYTES >> 4;
            // the last k-block of a product may hold fewer than 64 valid K elements (the rest is zero): skip those
            const int nk4_data = (p.k_extent - (nkd - 1) * BK + UMMA_K - 1) / UMMA_K;
            const int nk4_end = (p.k_extent_last - (nkl - 1) * BK + UMMA_K - 1) / UMMA_K;
            int base = 0;            // ring position of the tile's first block
            uint32_t phase = 0, qphase = 0, acc_phase = 0;
            int acc = 0, have_qb = -1;
            bool ok = true;
            uint32_t accumulate = 0;
            uint32_t d_tmem = 0;
            auto block = [&](uint64_t da, int s, int nk4) {   // a k-block of the query block and X block s of the ring
                const uint64_t db = db0 + (uint64_t)s * BLOCK;
                tc_mma_f16_by<true>(leader, d_tmem, da, db, p.idesc, accumulate);
                accumulate = 1;
                if (nk4 > 1) tc_mma_f16_by<true>(leader, d_tmem, da + 2, db + 2, p.idesc, 1);
                if (nk4 > 2) tc_mma_f16_by<true>(leader, d_tmem, da + 4, db + 4, p.idesc, 1);
                if (nk4 > 3) tc_mma_f16_by<true>(leader, d_tmem, da + 6, db + 6, p.idesc, 1);
            };
            auto full = [&](int s, uint32_t ph) {
                return mbar_try_wait(bar_full + s * 8, ph) || mbar_wait(bar_full + s * 8, ph, abort_flag, p.status);
            };
            for (int64_t item = unit; item < nitems && ok; item += nunits) {
                const int qb = (int)(item % nqb);
                if (qb != have_qb) {
                    ok = __all_sync(0xffffffffu, mbar_wait(bar_qfull, qphase, abort_flag, p.status));
                    if (!ok) break;
                    qphase ^= 1;
                    have_qb = qb;
                }
                for (int64_t t = item / nqb; t < p.ntiles && ok; t += p.P) {
                    ok = mbar_wait(bar_tempty + acc * 8, acc_phase ^ 1, abort_flag, p.status);
                    tc_fence_after();
                    d_tmem = tmem_base + acc * RES_TILE_N;
                    accumulate = 0;
                    int s = base;            // block by block through the ring
                    uint32_t ph = phase;
                    auto step = [&]() {
                        if (++s == ring) {
                            s = 0;
                            ph ^= 1;
                        }
                    };
                    uint64_t da = da0;
                    if (two) {
                        // query plane 1 with X plane 0, whose blocks stay
                        for (int kb = 0; kb < nkd; kb++, da += BLOCK, step()) {
                            ok = ok && full(s, ph);
                            block(da, s, kb < nkd - 1 ? 4 : nk4_data);
                        }
                        // query plane 0 with X plane 1
                        uint64_t da_low = da;
                        for (int kb = 0; kb < nkd; kb++, da_low += BLOCK, step()) {
                            ok = ok && full(s, ph);
                            block(da_low, s, kb < nkd - 1 ? 4 : nk4_data);
                            tc_commit_by<true>(leader, bar_empty + s * 8);   // its last use
                        }
                        // query plane 0 with X plane 0
                        int s0 = base;
                        for (int kb = 0; kb < nkd; kb++, da += BLOCK) {
                            block(da, s0, kb < nkl - 1 ? 4 : nk4_end);
                            tc_commit_by<true>(leader, bar_empty + s0 * 8);
                            if (++s0 == ring) s0 = 0;
                        }
                    }
                    // one plane: all its blocks; two: the norm columns' block, where they have one
                    for (int kb = two ? nkd : 0; kb < nkl; kb++, da += BLOCK, step()) {
                        ok = ok && full(s, ph);
                        block(da, s, kb < nkl - 1 ? 4 : nk4_end);
                        tc_commit_by<true>(leader, bar_empty + s * 8);
                    }
                    tc_commit_by<true>(leader, bar_tfull + acc * 8);
                    base = s;
                    phase = ph;
                    acc ^= 1;
                    if (acc == 0) acc_phase ^= 1;
                    ok = __all_sync(0xffffffffu, ok);   // a wait that ran out: the epilogues give up by themselves
                }
                const int64_t next = item + nunits;
                if (ok && next < nitems && (int)(next % nqb) != qb) tc_commit_by<true>(leader, bar_qempty);
            }
            if (!ok) {   // let the MMAs in flight retire before tensor memory goes away
                const long long t0 = clock64();
                while (clock64() - t0 < 200000LL) {
                }
            }
        }
        __syncwarp();
    } else {
        // ------------------------------ epilogue ------------------------------
        const int ew = warp & 3;            // TMEM lane quarter this warp may read
        // which chunks of 32 columns: three, three and two, or four and four
        const int part = (warp - 2) >> 2;
        constexpr int PER_WARP = MODE == MODE_FILTER ? 3 : 4;
        const int ch0 = part * PER_WARP, nch = min(PER_WARP, RES_TILE_N / 32 - ch0);
        const int row = ew * 32 + lane;
        float* const stage_key = reinterpret_cast<float*>(smem + RES_SM_STAGE) + (threadIdx.x - 64);
        int32_t* const stage_idx =
                reinterpret_cast<int32_t*>(smem + RES_SM_STAGE) + STAGE_N * STAGE_LD + (threadIdx.x - 64);
        const WarpHits hits = warp_hits(smem + RES_SM_STAGE + (warp - 2) * HITS_BYTES);
        const uint32_t tempty0 = map_to_cta(bar_tempty, 0);
        int acc = 0, nhits = 0, nstaged = 0;
        uint32_t acc_phase = 0;
        bool ok = true;
        for (int64_t item = unit; item < nitems && ok; item += nunits) {
            const int qb = (int)(item % nqb);
            const int64_t grow = (int64_t)qb * 256 + (int64_t)cta_rank * BM + row;
            const bool row_live = grow < nq_live;
            float ksc = p.kscale;
            // coherent loads: the kernel before a programmatic launch wrote the map
            if (p.rowscale && row_live) ksc *= __ldcg(p.rowscale + (p.rowscale_map ? (int64_t)__ldcg(p.rowscale_map + grow) : grow));
            float thr = -CUDART_INF_F, radd = 0.f;
            if (FILTER) {
                if (row_live) {
                    thr = filter_threshold(__ldcg(p.fthr + grow * p.fthr_stride + p.fthr_pos) / ksc);
                    if (__ldcg(p.cand_cnt + grow) > p.cand_cap) thr = -CUDART_INF_F;   // see drain_hits
                }
            } else if (row_live && p.rowadd) {
                radd = p.rowadd[grow];
            }
            auto drain = [&]() {   // the stage
                if (drain_stage(p.cand_cnt + grow, p.cand_key + grow * p.cand_cap, p.cand_idx + grow * p.cand_cap, p.cand_cap,
                                ksc, stage_key, stage_idx, nstaged))
                    thr = -CUDART_INF_F;
                nstaged = 0;
            };
            auto drain_queue = [&]() {
                const int64_t row0 = grow - lane;
                const unsigned over = drain_hits(p.cand_cnt + row0, p.cand_key + row0 * p.cand_cap, p.cand_idx + row0 * p.cand_cap,
                                                 p.cand_cap, ksc, hits.key, hits.col, hits.lane, nhits);
                if ((over >> lane) & 1u) thr = -CUDART_INF_F;
                nhits = 0;
            };
            for (int64_t t = item / nqb; t < p.ntiles; t += p.P) {
                const int64_t c_tile = tile_col(t);
                {
                    const bool w = mbar_wait(bar_tfull + acc * 8, acc_phase, abort_flag, p.status);
                    if (!__all_sync(0xffffffffu, w)) {   // keep the warp converged for tcgen05.ld
                        ok = false;
                        break;
                    }
                }
                tc_fence_after();
                const bool partial = c_tile + RES_TILE_N > p.ncols_end;
                const uint32_t taddr = tmem_base + ((uint32_t)(ew * 32) << 16) + acc * RES_TILE_N + ch0 * 32;
                const int64_t cbase = c_tile + ch0 * 32;
                auto release = [&]() {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_cluster(tempty0 + acc * 8);
                };
                if constexpr (MODE == MODE_FILTER) {
                    scan_columns(
                            taddr, nch,
                            [&](uint32_t(&r)[32], int ch) {
                                filter_columns(r, cbase + ch * 32, p.ncols_end, partial, thr, hits, nhits, drain_queue);
                            },
                            release);
                } else if constexpr (MODE == MODE_DENSE) {
                    scan_columns_ahead<PER_WARP>(
                            taddr,
                            [&](uint32_t(&r)[32], int ch) {
                                stage_columns(r, cbase + ch * 32, p.ncols_end, partial, thr, stage_key, stage_idx, nstaged, drain);
                            },
                            release);
                } else if constexpr (MODE == MODE_MINIMA) {
                    float* const out = p.out + grow * p.ld + (t * RES_TILE_N + ch0 * 32) / MIN_GROUP;
                    scan_columns(
                            taddr, PER_WARP,
                            [&](uint32_t(&r)[32], int ch) {
                                if (partial) mask_columns(r, cbase + ch * 32, p.ncols_end);
                                if (row_live) store_minima(r, ksc, out + ch * (32 / MIN_GROUP));
                            },
                            release);
                } else {
                    const bool whole = !partial && (p.ld & 7) == 0 && (reinterpret_cast<uintptr_t>(p.out) & 31) == 0;
                    float* const tbuf = reinterpret_cast<float*>(smem + RES_SM_STAGE) + (warp - 2) * (32 * 33);
                    const int64_t ocol = t * RES_TILE_N + ch0 * 32;
                    scan_columns(
                            taddr, nch,
                            [&](uint32_t(&r)[32], int ch) {
                                store_keys(p, r, whole, grow, lane, 32, nq_live, row_live, cbase + ch * 32, ocol + ch * 32, ksc, radd, tbuf);
                            },
                            release);
                }
                if (MODE == MODE_FILTER && nhits >= QUEUE_DRAIN) drain_queue();
                if (MODE == MODE_DENSE && __any_sync(0xffffffffu, nstaged > STAGE_N / 2)) drain();
                acc ^= 1;
                if (acc == 0) acc_phase ^= 1;
            }
            if (MODE == MODE_FILTER && ok) drain_queue();   // the next range may have other rows
            if (MODE == MODE_DENSE && ok) drain();
        }
    }

    tc_fence_before();
    __syncthreads();
    cluster_sync_all();   // the peer may still read this CTA's tiles / signal its barriers
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS)
                     : "memory");
    }
}

// Blocks of a query block, which are also those of an X tile; 0: no resident launch for these operands.
int resident_blocks(const GemmOperands& op) {
    const int nkd = (int)ceil_div64(op.d_data, BK), nkl = (int)ceil_div64(op.d_pad, BK);
    if (op.npl > 2) return 0;
    const int n = op.npl == 2 ? nkd + nkl : nkl;
    return 2 * n <= RES_BLOCKS ? n : 0;
}

}  // namespace

bool resident_fits(const GemmOperands& op, const GemmPlan& plan) { return plan.pair && resident_blocks(op) > 0; }

int launch_resident(const GemmOperands& op, const GemmPlan& plan, GemmParams& g, const CUtensorMap& ma,
                    const CUtensorMap& mb, const Launch& ln) {
    ResidentParams p{};
    p.n_blocks = resident_blocks(op);
    p.nkd = (int)ceil_div64(op.d_data, BK);
    p.nkl = (int)ceil_div64(op.d_pad, BK);
    p.ring = RES_BLOCKS - p.n_blocks < RES_MAX_RING ? RES_BLOCKS - p.n_blocks : RES_MAX_RING;
    // tiles of 256 columns; the second half of the last 512 may lie beyond the end
    int64_t ntiles = 2 * plan.ntiles;
    if (g.col0 + (plan.ntiles - 1) * g.tile_stride * 512 + RES_TILE_N >= g.ncols_end) ntiles--;
    // Items ("ranges", of tpr tiles at most) that leave the last wave full; a range costs the query block's way from L2, about one tile.  Of query blocks that are
    // counted on the device any number may be live, one above all: ranges for that one as well (100 of 2,048 queries redone over
    // 1 M fp16 rows of d = 256, k = 1000: 4,232 us with ranges for all eight blocks, 2,506 so).
    int64_t tpr_best = 1;
    double best = 0.0;
    for (int64_t tpr = 1; tpr <= ntiles && tpr <= 2048; tpr = tpr < 64 ? tpr + 1 : tpr + tpr / 32) {
        const int64_t P = ceil_div64(ntiles, tpr);
        auto waves = [&](int64_t blocks) { return (double)ceil_div64(P * blocks, plan.units); };
        const double cost = (g.nq_dev ? waves(1) + waves(plan.nqb) / plan.nqb : waves(plan.nqb)) * ((double)tpr + 1.0);
        if (tpr == 1 || cost < best) {
            best = cost;
            tpr_best = tpr;
        }
    }
    g.ntiles = ntiles;
    g.P = (int)ceil_div64(ntiles, tpr_best);
    p.g = g;
    const int64_t items = (int64_t)plan.nqb * g.P;
    const int grid = (int)(2 * (items < plan.units ? items : plan.units));

    typedef void (*KernelFn)(const CUtensorMap, const CUtensorMap, const ResidentParams);
    const KernelFn kernel = g.mode == MODE_FILTER   ? (g.dense ? gemm_resident_kernel<MODE_DENSE> : gemm_resident_kernel<MODE_FILTER>)
                            : g.mode == MODE_STORE ? gemm_resident_kernel<MODE_STORE>
                                                   : gemm_resident_kernel<MODE_MINIMA>;
    static bool attr_set[kMaxDevices] = {false};
    const int slot = device_slot();
    if (!attr_set[slot]) {
        for (KernelFn fn : {gemm_resident_kernel<MODE_FILTER>, gemm_resident_kernel<MODE_STORE>, gemm_resident_kernel<MODE_MINIMA>,
                            gemm_resident_kernel<MODE_DENSE>})
            B200F_CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, RES_SMEM_BYTES));
        attr_set[slot] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid, 1, 1);
    const int threads = g.mode == MODE_FILTER && !g.dense ? RES_THREADS<MODE_FILTER> : RES_THREADS<MODE_STORE>;
    cfg.blockDim = dim3((unsigned)threads, 1, 1);
    cfg.dynamicSmemBytes = RES_SMEM_BYTES;
    cfg.stream = ln.stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.numAttrs = 1;
    if (ln.overlap) {
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.numAttrs = 2;
    }
    cfg.attrs = attr;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, ma, mb, p);
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        return B200F_ERR_CUDA;
    }
    return B200F_OK;
}

}  // namespace b200f
