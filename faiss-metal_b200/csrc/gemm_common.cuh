// What the two distance GEMM kernels share: launch parameters, tcgen05 and TMA wrappers, the epilogue's work on
// accumulator columns, operand tensor maps.
#pragma once

#include <cuda.h>

#include "common.cuh"
#include "ptx.cuh"
#include "tensor_map.h"

namespace b200f {

constexpr int BM = 128;
constexpr int BN = 256;
constexpr int BK = 64;  // 16-bit elements: 128 bytes = one swizzle row
constexpr int UMMA_K = 16;
constexpr int NUM_EPI_WARPS = 8;   // two per TMEM lane quarter: each takes half of the tile's columns
constexpr int TMEM_COLS = 512;

enum { MODE_TOPK = 0, MODE_STORE = 1, MODE_FILTER = 2, MODE_MINIMA = 3, MODE_DENSE = 4 };

struct GemmParams {
    int64_t nq;
    int64_t col0;        // first global column (row of X) of this launch
    int64_t ncols_end;   // one past the last valid global column of this launch
    int64_t ntiles;      // column tiles in this launch
    int64_t tiles_per_range;
    int nqb;
    int P;
    // single CTA: rows of a query box, the live ones rounded up to 8.  Rows beyond the queries are never
    // fetched: zero-filling 104 of 128 rows held the ring back to one k-block per 1,900 cycles whatever
    // it cost to read X (24 queries, 1,000,003 fp16 rows of d = 770: 354 us a launch, 242 without).  What the
    // tile holds there instead reaches only accumulator rows that nobody reads.
    int a_rows;
    int warp_rows;       // single CTA: query rows in a TMEM lane quarter, 32 or (at most 64 queries) 16
    // k-blocks of 64 and valid K elements (multiple of 8) of a plane product.  The norm columns are zero in
    // every plane but the first, so only the last product, of the two first planes, takes them (d = 128,
    // three products: 25 MMAs a tile instead of 27, 7 k-blocks instead of 9).
    int kb_per_pass, kb_last_pass;
    int k_extent, k_extent_last;
    int npass;
    uint32_t pass_a;     // 4 bits per pass: plane index of A
    uint32_t pass_b;
    uint32_t idesc;
    int mode;
    int k;
    float kscale;        // key = -kscale * t  (2 for L2, 1 for inner product)
    // optional per-row factor on kscale (operands scaled per query row: fp16x2 planes); row j of
    // this launch is row rowscale_map[j] of the array when the map is set (redone rows)
    const float* rowscale;
    const int32_t* rowscale_map;
    float sign;
    const float* rowadd; // per query row, may be null (0)
    float* part_key;
    int32_t* part_idx;
    uint32_t* gthr;      // [nq][gslots] ordered-float 32nd-best keys published by the lists of a row
    int gslots;          // lists publish to slot (list number % gslots); the row's bound is the
                         // largest slot: gslots full lists hold 32 * gslots distinct candidates
    const int* nq_dev;   // when set: the number of live query rows is read from device memory
    int64_t tile_stride; // tile t of the launch is tile t * tile_stride of X (sampling passes)
    // MODE_FILTER: every column whose key is <= the row's threshold is appended to the row's
    // candidate buffer (position from an atomic counter; entries past cand_cap are only counted)
    const float* fthr;   // threshold of row q in scaled key units: fthr[q * fthr_stride + fthr_pos]
    int fthr_stride, fthr_pos;
    float* cand_key;     // [nq][cand_cap]
    int32_t* cand_idx;
    int32_t* cand_cnt;   // [nq]; hits of a row are counted until they no longer fit
    int cand_cap;
    int dense;           // MODE_FILTER: many hits expected
    float* out;
    int64_t ld;
    int32_t* status;
};

// ---- PTX wrappers (mbarrier and bounded-wait helpers come from ptx.cuh) -----------------

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag,
                                          int32_t* status) {
    return mbar_wait_bounded(bar, parity, abort_flag, status, kDevErrBarrierWait);
}

__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, uint32_t bar,
                                            int c0, int c1, int c2) {
    asm volatile(
            "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
            " [%0], [%1, {%3, %4, %5}], [%2];"
            ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
            : "memory");
}

__device__ __forceinline__ void tc_fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

// shared::cluster address of `addr` (a shared::cta address of this CTA) in CTA `rank`
__device__ __forceinline__ uint32_t map_to_cta(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}

__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// arrive on an mbarrier given by a shared::cluster address (own or peer CTA)
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}

// TMA load issued inside a CTA pair: the mbarrier may live in the peer CTA
__device__ __forceinline__ void tma_load_3d_pair(uint32_t dst, const CUtensorMap* map, uint32_t bar,
                                                 int c0, int c1, int c2) {
    asm volatile(
            "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
            " [%0], [%1, {%3, %4, %5}], [%2];"
            ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
            : "memory");
}

// Issued by the lane with `leader` of a whole converged warp: control flow and operands stay uniform.
template <bool PAIR>
__device__ __forceinline__ void tc_mma_f16_by(bool leader, uint32_t d_tmem, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                              uint32_t accumulate) {
    if (PAIR)
        asm volatile(
                "{\n\t"
                ".reg .pred p, q;\n\t"
                "setp.ne.b32 p, %4, 0;\n\t"
                "setp.ne.b32 q, %5, 0;\n\t"
                "@q tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t"
                "}\n" ::"r"(d_tmem),
                "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"((uint32_t)leader)
                : "memory");
    else
        asm volatile(
                "{\n\t"
                ".reg .pred p, q;\n\t"
                "setp.ne.b32 p, %4, 0;\n\t"
                "setp.ne.b32 q, %5, 0;\n\t"
                "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t"
                "}\n" ::"r"(d_tmem),
                "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"((uint32_t)leader)
                : "memory");
}
// Arrives on the barrier at `bar` (an address of this CTA), in a pair on both CTAs', when the MMAs issued so far retire.
template <bool PAIR>
__device__ __forceinline__ void tc_commit_by(bool leader, uint32_t bar) {
    if (PAIR)
        asm volatile(
                "{\n\t"
                ".reg .pred q;\n\t"
                "setp.ne.b32 q, %1, 0;\n\t"
                "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %2;\n\t"
                "}\n" ::"r"(bar),
                "r"((uint32_t)leader), "h"((uint16_t)3)
                : "memory");
    else
        asm volatile(
                "{\n\t"
                ".reg .pred q;\n\t"
                "setp.ne.b32 q, %1, 0;\n\t"
                "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t"
                "}\n" ::"r"(bar),
                "r"((uint32_t)leader)
                : "memory");
}

// 32 lanes x 32 consecutive fp32 columns -> 32 registers per thread
__device__ __forceinline__ void tc_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
            "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
            "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
              "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
              "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
              "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
              "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]),
              "=r"(r[31])
            : "r"(taddr)
            : "memory");
}
// The same wait, tied to the registers of one load: nothing that reads them moves in front of it.
__device__ __forceinline__ void tc_wait_ld32(uint32_t (&r)[32]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                   "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]),
                   "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]),
                   "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
                 :
                 : "memory");
}
// one 32-byte sector of a row
__device__ __forceinline__ void st_global_v8(float* dst, const float (&v)[8]) {
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst), "f"(v[0]), "f"(v[1]), "f"(v[2]),
                 "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
                 : "memory");
}
__device__ __forceinline__ void tc_wait_ld() {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// One thread of a converged warp, in a form the compiler knows to be one: what it issues stays uniform.
__device__ __forceinline__ bool elect_one() {
    uint32_t r;
    asm volatile(
            "{\n\t"
            ".reg .pred p;\n\t"
            "elect.sync _|p, 0xffffffff;\n\t"
            "selp.b32 %0, 1, 0, p;\n\t"
            "}\n"
            : "=r"(r));
    return r != 0;
}

// the largest of three in one instruction (fmaxf's treatment of NaN)
__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// K-major operand tile, 128-byte swizzle: rows of 128 bytes, 8-row groups 1024 bytes apart.
__device__ __forceinline__ uint64_t make_smem_desc(uint32_t saddr) {
    uint64_t desc = 0;
    desc |= (uint64_t)((saddr & 0x3FFFFu) >> 4);  // start address
    desc |= (uint64_t)1 << 16;                    // leading byte offset (unused with swizzle)
    desc |= (uint64_t)(1024 >> 4) << 32;          // stride byte offset between 8-row groups
    desc |= (uint64_t)1 << 46;                    // descriptor version (sm_100)
    desc |= (uint64_t)2 << 61;                    // SWIZZLE_128B
    return desc;
}

// Columns beyond the end were zero-filled: out of every comparison.
__device__ __forceinline__ void mask_columns(uint32_t (&r)[32], int64_t cbase, int64_t ncols_end) {
#pragma unroll
    for (int c = 0; c < 32; c++)
        if (cbase + c >= ncols_end) r[c] = 0xff800000u;   // -INF
}
// the largest of every group of eight columns
__device__ __forceinline__ void group_maxima(const uint32_t (&r)[32], float (&gm)[4]) {
#pragma unroll
    for (int g = 0; g < 4; g++) {
        const float a = max3(__uint_as_float(r[8 * g]), __uint_as_float(r[8 * g + 1]), __uint_as_float(r[8 * g + 2]));
        const float b = max3(__uint_as_float(r[8 * g + 3]), __uint_as_float(r[8 * g + 4]), __uint_as_float(r[8 * g + 5]));
        gm[g] = max3(fmaxf(__uint_as_float(r[8 * g + 6]), __uint_as_float(r[8 * g + 7])), a, b);
    }
}

// MODE_FILTER of the resident kernel, few hits.  The epilogue's code has to stay small: the hits' part runs for every second
// chunk of 32 columns at the usual thresholds, and unrolled comparisons of eight columns after the other cost 700 cycles a visit
// there.  So a row with a hit goes to shared memory whole, a loop looks at one such row at a time, a column per lane, and hits
// queue up there from tile to tile (2,048 queries, k = 1024, 5 M fp32 rows: 5,733 -> 5,256 us).
constexpr int HIT_ROWS = 8;     // rows of a chunk looked at together
constexpr int HIT_LD = 36;      // floats from one to the next
constexpr int QUEUE_N = 96;
constexpr int QUEUE_DRAIN = 64; // worked off between tiles from here on
constexpr int HITS_BYTES = HIT_ROWS * HIT_LD * 4 + HIT_ROWS * 4 + QUEUE_N * 12;
struct WarpHits {
    float* rows;      // [HIT_ROWS][HIT_LD]
    int* src;         // [HIT_ROWS] lanes they belong to
    float* key;       // [QUEUE_N] -accumulator
    int* col;
    int* lane;
};
__device__ __forceinline__ WarpHits warp_hits(uint8_t* area) {   // HITS_BYTES, 16-byte aligned
    WarpHits h;
    h.rows = reinterpret_cast<float*>(area);
    h.src = reinterpret_cast<int*>(h.rows + HIT_ROWS * HIT_LD);
    h.key = reinterpret_cast<float*>(h.src + HIT_ROWS);
    h.col = reinterpret_cast<int*>(h.key + QUEUE_N);
    h.lane = h.col + QUEUE_N;
    return h;
}

// n queued hits to the candidate buffers of the warp's 32 rows (cnt, ck, ci: those of its first).  One atomic takes the slots
// of a row's hits among 32; the counter also counts hits that no longer fit.  Returns the rows (a bit each) that have such: they
// are redone, and need no more of their hits.  All lanes call it, ksc is the lane's.
static __device__ __noinline__ unsigned drain_hits(int32_t* cnt, float* ck, int32_t* ci, int cap, float ksc, const float* key, const int* col,
                                        const int* lanes, int n) {
    const int lane = threadIdx.x & 31;
    unsigned over = 0;
    __syncwarp();
    for (int i0 = 0; i0 < n; i0 += 32) {
        const bool live = i0 + lane < n;
        const int row = live ? lanes[i0 + lane] : lane;
        const float k = __shfl_sync(0xffffffffu, ksc, row);
        const unsigned same = __match_any_sync(0xffffffffu, live ? row : 32);
        const int leader = __ffs(same) - 1;
        int base = 0;
        if (live && lane == leader) base = atomicAdd(cnt + row, __popc(same));
        const int pos = __shfl_sync(0xffffffffu, base, leader) + __popc(same & ((1u << lane) - 1u));
        if (live && pos < cap) {
            ck[(int64_t)row * cap + pos] = k * key[i0 + lane];
            ci[(int64_t)row * cap + pos] = col[i0 + lane];
        }
        over |= __reduce_or_sync(0xffffffffu, live && pos >= cap ? 1u << row : 0u);
    }
    __syncwarp();
    return over;
}

// 32 accumulator columns of the warp's rows: hits (-r < thr) to the queue, which holds n.  All lanes call it.  drain may lower
// thr.
template <typename Drain>
__device__ __forceinline__ void filter_columns(uint32_t (&r)[32], int64_t cbase, int64_t ncols_end, bool partial, const float& thr,
                                               const WarpHits& h, int& n, Drain drain) {
    if (partial) mask_columns(r, cbase, ncols_end);
    float gm[4];
    group_maxima(r, gm);
    unsigned rows = __ballot_sync(0xffffffffu, -fmaxf(max3(gm[0], gm[1], gm[2]), gm[3]) < thr);
    if (!rows) return;
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    do {
        const int rank = __popc(rows & below);
        const bool mine = ((rows >> lane) & 1u) && rank < HIT_ROWS;
        if (mine) {
            float4* dst = reinterpret_cast<float4*>(h.rows + rank * HIT_LD);
#pragma unroll
            for (int c = 0; c < 8; c++)
                dst[c] = make_float4(__uint_as_float(r[4 * c]), __uint_as_float(r[4 * c + 1]), __uint_as_float(r[4 * c + 2]),
                                     __uint_as_float(r[4 * c + 3]));
            h.src[rank] = lane;
        }
        const int take = min(__popc(rows), HIT_ROWS);
        rows &= ~__ballot_sync(0xffffffffu, mine);
        __syncwarp();
#pragma unroll 1
        for (int j = 0; j < take; j++) {
            const float key = -h.rows[j * HIT_LD + lane];
            const int src = h.src[j];
            const bool hit = key < __shfl_sync(0xffffffffu, thr, src);
            const unsigned b = __ballot_sync(0xffffffffu, hit);
            if (n > QUEUE_N - 32) drain();
            if (hit) {
                const int pos = n + __popc(b & below);
                h.key[pos] = key;
                h.col[pos] = (int)cbase + lane;
                h.lane[pos] = src;
            }
            n += __popc(b);
        }
        __syncwarp();
    } while (rows);
}

// Hits of gemm_topk.cu, and many of the resident kernel's, wait per thread in shared memory (entry i of a thread at [i * STAGE_LD]: raw key s = -t and column), found by groups of
// eight columns that hold one.  All lanes of the warp call it.
constexpr int STAGE_N = 16;
constexpr int STAGE_LD = 32 * NUM_EPI_WARPS;
template <typename Drain>
__device__ __forceinline__ void stage_columns(uint32_t (&r)[32], int64_t cbase, int64_t ncols_end, bool partial, float thr,
                                              float* stage_key, int32_t* stage_idx, int& nstaged, Drain drain) {
    if (partial) mask_columns(r, cbase, ncols_end);
    float gm[4];
    group_maxima(r, gm);
    if (!__any_sync(0xffffffffu, -fmaxf(max3(gm[0], gm[1], gm[2]), gm[3]) < thr)) return;
#pragma unroll
    for (int g = 0; g < 4; g++) {
        const bool hit = -gm[g] < thr;
        if (!__any_sync(0xffffffffu, hit)) continue;
        if (hit) {
            if (nstaged > STAGE_N - 8) drain();   // rare: massive ties
#pragma unroll
            for (int c = 0; c < 8; c++) {
                const float sc = -__uint_as_float(r[8 * g + c]);
                if (sc < thr) {
                    stage_key[nstaged * STAGE_LD] = sc;
                    stage_idx[nstaged * STAGE_LD] = (int32_t)cbase + 8 * g + c;
                    nstaged++;
                }
            }
        }
    }
    __syncwarp();
}
// A thread's n staged hits to its row's candidate buffer: one atomic takes their slots; the counter also counts entries
// that no longer fit.  True where there were such: the row is redone, and needs no more of its hits.
__device__ __forceinline__ bool drain_stage(int32_t* cnt, float* ck, int32_t* ci, int cap, float ksc, const float* sk,
                                            const int32_t* si, int n) {
    if (n <= 0) return false;
    const int base = atomicAdd(cnt, n);
    for (int i = 0; i < n; i++) {
        if (base + i < cap) {
            ck[base + i] = ksc * sk[i * STAGE_LD];
            ci[base + i] = si[i * STAGE_LD];
        }
    }
    return base + n > cap;
}

// NCH x 32 accumulator columns from taddr on, through `use(registers, chunk)`, a chunk while the next one is on its way;
// `release` is called once the last one has arrived.  For many hits, which hold a chunk up.
template <int NCH, typename Use, typename Release>
__device__ __forceinline__ void scan_columns_ahead(uint32_t taddr, Use use, Release release) {
    static_assert(NCH % 2 == 0, "chunks are taken in pairs");
    uint32_t a[32], b[32];
    tc_ld32(taddr, a);
#pragma unroll 1
    for (int ch = 0; ch < NCH; ch += 2) {
        tc_wait_ld32(a);
        tc_ld32(taddr + (ch + 1) * 32, b);
        use(a, ch);
        tc_wait_ld32(b);
        if (ch + 2 < NCH) tc_ld32(taddr + (ch + 2) * 32, a);
        else release();
        use(b, ch + 1);
    }
}

// nch x 32 accumulator columns from taddr on, through `use(registers, chunk)`; `release` is called once the last ones have
// arrived.  Reading 32 columns takes 40 cycles beside the other warps of the scheduler and MMAs, too few to read ahead.
template <typename Use, typename Release>
__device__ __forceinline__ void scan_columns(uint32_t taddr, int nch, Use use, Release release) {
    if (nch == 0) release();
#pragma unroll 1
    for (int ch = 0; ch < nch; ch++) {
        uint32_t r[32];
        tc_ld32(taddr + ch * 32, r);
        tc_wait_ld32(r);
        if (ch == nch - 1) release();
        use(r, ch);
    }
}

// MODE_MINIMA: of 32 columns of a thread's row the smallest key of every MIN_GROUP, one sector, to out.  Why groups of
// four: SAMPLE_GROUP (search.cu).
constexpr int MIN_GROUP = 4;
__device__ __forceinline__ void store_minima(const uint32_t (&r)[32], float ksc, float* out) {
    static_assert(32 / MIN_GROUP == 8, "a sector of minima");
    float v[8];
#pragma unroll
    for (int g = 0; g < 8; g++)
        v[g] = -ksc * fmaxf(max3(__uint_as_float(r[4 * g]), __uint_as_float(r[4 * g + 1]), __uint_as_float(r[4 * g + 2])),
                            __uint_as_float(r[4 * g + 3]));
    st_global_v8(out, v);
}

// Keys up to the threshold pass a filter whose comparison excludes its bound: the next float up (+INF, the
// threshold of a row whose sample was too small, stays).
__device__ __forceinline__ float filter_threshold(float t) {
    const uint32_t o = float_to_ordered(t);
    return (o >= 0xff800000u) ? t : ordered_to_float(o + 1u);
}

// MODE_STORE: 32 consecutive columns, from cbase, of the accumulator row a thread owns, to column ocol of the output.
// All lanes of a warp call it.  whole: whole sectors, straight from the registers; else (ragged or unaligned output,
// where that would touch 32 rows per instruction) the warp transposes the 32 x 32 block through tbuf
// [32][33] and writes one 128-byte row segment per instruction.
__device__ __forceinline__ void store_keys(const GemmParams& p, const uint32_t (&r)[32], bool whole, int64_t grow, int lane, int warp_rows,
                                           int64_t nq_live, bool row_live, int64_t cbase, int64_t ocol, float ksc,
                                           float radd, float* tbuf) {
    if (whole) {
        if (!row_live) return;
        float* o = p.out + grow * p.ld + ocol;
#pragma unroll
        for (int c = 0; c < 32; c += 8) {
            float v[8];
#pragma unroll
            for (int e = 0; e < 8; e++) v[e] = fmaf(p.sign, -ksc * __uint_as_float(r[c + e]), radd);
            st_global_v8(o + c, v);
        }
        return;
    }
#pragma unroll
    for (int c = 0; c < 32; c++) {
        const float key = -ksc * __uint_as_float(r[c]);
        tbuf[lane * 33 + c] = fmaf(p.sign, key, radd);
    }
    __syncwarp();
    const int64_t grow0 = grow - lane;   // first of this warp's rows
    const bool col_ok = cbase + lane < p.ncols_end;
    float* obase = p.out + ocol + lane;
#pragma unroll 8
    for (int rr = 0; rr < warp_rows; rr++) {
        const float v = tbuf[rr * 33 + lane];
        if (col_ok && grow0 + rr < nq_live) obase[(grow0 + rr) * p.ld] = v;
    }
    __syncwarp();
}

// ---- host side -------------------------------------------------------------------------

// 3-D map {k, row, plane} over a [planes][rows][pitch] 16-bit array; box {64, box_rows, 1}.
inline int make_operand_map(CUtensorMap* map, const uint16_t* base, int is_bf16, int64_t k_extent,
                     int64_t rows, int64_t pitch, int planes, int64_t plane_stride, int box_rows) {
    EncodeTiledFn fn = get_encode_fn();
    if (!fn) return B200F_ERR_CUDA;
    if ((reinterpret_cast<uintptr_t>(base) & 15) != 0 || (pitch % 8) != 0 ||
        (planes > 1 && (plane_stride % 8) != 0))
        return B200F_ERR_BAD_ARG;
    cuuint64_t dims[3] = {(cuuint64_t)k_extent, (cuuint64_t)rows, (cuuint64_t)planes};
    cuuint64_t pstride = (planes > 1) ? (cuuint64_t)plane_stride * 2 : (cuuint64_t)pitch * 2 * (cuuint64_t)(rows > 0 ? rows : 1);
    cuuint64_t strides[2] = {(cuuint64_t)pitch * 2, pstride};
    cuuint32_t box[3] = {(cuuint32_t)BK, (cuuint32_t)box_rows, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = fn(map, is_bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16,
                    3, const_cast<uint16_t*>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? B200F_OK : B200F_ERR_CUDA;
}

// gemm_resident.cu: the same filter and store launches with the query block kept in shared memory.  g: as for the
// general kernel; its ranges are chosen anew.
bool resident_fits(const GemmOperands& op, const GemmPlan& plan);
int launch_resident(const GemmOperands& op, const GemmPlan& plan, GemmParams& g, const CUtensorMap& ma,
                    const CUtensorMap& mb, const Launch& ln);

}  // namespace b200f
