// Selection by rank: radix threshold, sorting in registers, merging by binary search.
//
// Covers the same ground as block_select_min/max (shaders/block_select.metal:111-274) and the
// list merge of the fused kernels (shaders/fused_l2_topk.metal:88-131) for the two inputs that
// are small enough to need no streaming:
//
//  * row_select: the k best of a row's few hundred to few thousand (key, id) pairs in any order:
//    threshold-filtered candidates, or the partial lists the fused kernels leave.  See the kernel.
//  * rank_merge: P sorted result lists of k entries (other shards' answers), P k <= 8192.
//    The lists are runs already.  Only entries up to the largest of the lists' (k / P)-th keys
//    can belong to the result; each of those finds its position by binary search in the other
//    lists.  Final distances can tie where the keys a shard sorted by did not, so equal
//    distances need not come in label order inside a list: short runs of them are put in order
//    first, and a row that still is not strictly ordered is sorted outright in shared memory.
//
// Both write exactly what sort_select_kernel writes for the same input: ascending key, ties to the
// lower id / label.
#include <atomic>
#include <cfloat>
#include <cmath>

#include "common.cuh"
#include "ptx.cuh"

namespace b200f {

namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr uint64_t RS_EMPTY = ~0ull;
constexpr int RS_RUN = 512;    // most elements one warp sorts (16 per lane)

std::atomic<int> g_rank_select{1};

__device__ __forceinline__ uint64_t shfl_xor64(uint64_t v, int m) {
    const unsigned lo = __shfl_xor_sync(FULL, (unsigned)v, m);
    const unsigned hi = __shfl_xor_sync(FULL, (unsigned)(v >> 32), m);
    return ((uint64_t)hi << 32) | lo;
}

// Ascending sort of the 32 R words a warp holds; element e = lane * R + r sits in v[r] of lane.
template <int R>
__device__ __forceinline__ void warp_sort(uint64_t (&v)[R], int lane) {
#pragma unroll
    for (int size = 2; size <= 32 * R; size <<= 1) {
#pragma unroll
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            if (stride >= R) {
                const int ls = stride / R;
                const bool up = ((lane * R) & size) == 0;
                const bool keep_min = ((lane & ls) == 0) == up;
#pragma unroll
                for (int r = 0; r < R; r++) {
                    const uint64_t o = shfl_xor64(v[r], ls);
                    const bool less = v[r] < o;
                    v[r] = (less == keep_min) ? v[r] : o;
                }
            } else {
#pragma unroll
                for (int r = 0; r < R; r++) {
                    if ((r & stride) == 0) {
                        const bool up = (size < R) ? ((r & size) == 0) : (((lane * R) & size) == 0);
                        constexpr int RM = R - 1;   // no-op mask: keeps the index in range where the branch is dead
                        const uint64_t a = v[r], b = v[(r | stride) & RM];
                        const bool swap = (a > b) == up;
                        v[r] = swap ? b : a;
                        v[(r | stride) & RM] = swap ? a : b;
                    }
                }
            }
        }
    }
}

struct RowSelectParams {
    const float* keys;        // [nq][ld] keys, smaller is better
    const int32_t* ids;       // [nq][ld] row ids (-1 = empty); null: the id is the column, NaN keys are empty
    float last_key;           // ids null: keys beyond this one are empty too (+INF, or the largest finite one)
    const int32_t* cnt;       // candidates counted per row (may exceed ld: overflow); null: n
    int64_t ld;
    int64_t n;
    int64_t nb_total;         // rows in the shard (dirty)
    int64_t nq;
    const int* nq_dev;        // optional: live rows (<= nq), read on the device
    const int32_t* row_map;   // optional: row j belongs to query row_map[j]
    int32_t* redone;          // optional: receives *nq_dev unless that is zero
    int k;
    int bound;                // words of the staging area
    float out_sign;
    const float* qnorm;
    int clamp;
    float pad;
    int64_t label_base;
    float* out_dist;
    int64_t* out_labels;
    int32_t* dirty;           // optional: 1 when the result is not proven complete
    const float* thr;         // optional, [nq]: rows beyond this key may be missing from the input
    RedoRows redo;
};

__device__ __forceinline__ void rs_write(const RowSelectParams& p, int64_t qo, int rank, uint64_t w, int* s_beyond) {
    if (p.thr && rank == p.k - 1 && ordered_to_float((uint32_t)(w >> 32)) > p.thr[qo]) *s_beyond = 1;
    float dist = p.out_sign * ordered_to_float((uint32_t)(w >> 32)) + (p.qnorm ? p.qnorm[qo] : 0.f);
    if (p.clamp && dist < 0.f) dist = 0.f;
    p.out_dist[qo * p.k + rank] = dist;
    p.out_labels[qo * p.k + rank] = (int64_t)(uint32_t)w + p.label_base;
}

// Sort and place the c words staged in `runs` (all distinct); warp w takes words [w m, w m + m).
// The staging area becomes the sorted runs, 32 R words per warp.
template <int R>
__device__ __forceinline__ void rank_place(const RowSelectParams& p, int64_t qo, int c, int m,
                                           uint64_t* runs, int W, int* s_beyond) {
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    uint64_t v[R];
#pragma unroll
    for (int r = 0; r < R; r++) {
        const int t = r * 32 + lane;
        const int i = warp * m + t;
        v[r] = (t < m && i < c) ? runs[i] : RS_EMPTY;
    }
    __syncthreads();   // everybody holds their share: the area may be overwritten
    warp_sort<R>(v, lane);
    constexpr int N = 32 * R;
#pragma unroll
    for (int r = 0; r < R; r++) runs[warp * N + lane * R + r] = v[r];
    __syncthreads();
    int rank[R];
#pragma unroll
    for (int r = 0; r < R; r++) rank[r] = lane * R + r;
    for (int o = 0; o < W; o++) {
        if (o == warp) continue;
        // words are distinct: the lower bound is the count.  A fixed number of steps, so that the R
        // searches of a lane run side by side instead of one after the other.
        const uint64_t* run = runs + o * N;
        int lo[R];
#pragma unroll
        for (int r = 0; r < R; r++) lo[r] = 0;
#pragma unroll
        for (int step = N / 2; step > 0; step >>= 1) {
#pragma unroll
            for (int r = 0; r < R; r++) lo[r] += (run[lo[r] + step - 1] < v[r]) ? step : 0;
        }
#pragma unroll
        for (int r = 0; r < R; r++) rank[r] += lo[r] + (run[lo[r]] < v[r] ? 1 : 0);
    }
#pragma unroll
    for (int r = 0; r < R; r++)
        if (v[r] != RS_EMPTY && rank[r] < p.k) rs_write(p, qo, rank[r], v[r], s_beyond);
}

// The kk-th smallest x = key - mn of what `visit` enumerates (a callable that calls its argument with
// the ordered key of every live element of this thread), 8 bits a pass over `bits` significant
// bits, stopping when at most `slack` low bits are undecided: returns an upper bound of it that is
// exact for slack = 0; kk is left at how many elements equal to it are among the kk smallest.  All
// threads of the CTA call it; s_hist and s_sel are shared.
template <typename Visit>
__device__ __forceinline__ uint32_t radix_kth(Visit visit, uint32_t mn, int bits, int slack, int& kk,
                                              int* s_hist, int* s_sel) {
    const int tid = threadIdx.x, lane = tid & 31, T = blockDim.x;
    uint32_t prefix = 0;
    int hi = bits;
    while (hi > slack) {
        const int lo = hi > 8 ? hi - 8 : 0;
        const uint32_t mask = (1u << (hi - lo)) - 1u;
        for (int i = tid; i < 256; i += T) s_hist[i] = 0;
        __syncthreads();
        visit([&](uint32_t key) {
            const uint32_t x = key - mn;
            if ((uint32_t)((uint64_t)x >> hi) == prefix) atomicAdd(&s_hist[(x >> lo) & mask], 1);
        });
        __syncthreads();
        if (tid < 32) {
            int h[8], sum = 0;
#pragma unroll
            for (int i = 0; i < 8; i++) {
                h[i] = s_hist[lane * 8 + i];
                sum += h[i];
            }
            int incl = sum;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int up = __shfl_up_sync(FULL, incl, o);
                if (lane >= o) incl += up;
            }
            int below = incl - sum;
            if (below < kk && kk <= incl) {   // exactly one lane
                int digit = 0;
#pragma unroll
                for (int i = 0; i < 7; i++) {
                    if (digit == i && below + h[i] < kk) {
                        below += h[i];
                        digit = i + 1;
                    }
                }
                s_sel[0] = lane * 8 + digit;
                s_sel[1] = kk - below;
            }
        }
        __syncthreads();
        prefix = (prefix << (hi - lo)) | (uint32_t)s_sel[0];
        kk = s_sel[1];
        hi = lo;
    }
    return hi > 0 ? (uint32_t)((((uint64_t)prefix + 1) << hi) - 1) : prefix;
}

// Block-wide live count, smallest and largest key.
struct Spread {
    int live;
    uint32_t mn, mx;
};
__device__ __forceinline__ Spread block_spread(int live, uint32_t mn, uint32_t mx, int* s_live, uint32_t* s_min,
                                               uint32_t* s_max) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, W = blockDim.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        live += __shfl_xor_sync(FULL, live, o);
        mn = min(mn, __shfl_xor_sync(FULL, mn, o));
        mx = max(mx, __shfl_xor_sync(FULL, mx, o));
    }
    if (lane == 0) {
        s_live[warp] = live;
        s_min[warp] = mn;
        s_max[warp] = mx;
    }
    __syncthreads();
    live = lane < W ? s_live[lane] : 0;
    mn = lane < W ? s_min[lane] : 0xffffffffu;
    mx = lane < W ? s_max[lane] : 0u;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        live += __shfl_xor_sync(FULL, live, o);
        mn = min(mn, __shfl_xor_sync(FULL, mn, o));
        mx = max(mx, __shfl_xor_sync(FULL, mx, o));
    }
    return Spread{live, mn, mx};
}

constexpr int RS_COUNT_MAX = 256;   // so few words are placed by counting the smaller ones
constexpr int RS_BUCKETS = 2048;
constexpr int RS_BUCKET_MAX = 64;   // a fuller bucket: sorted runs instead

// The words' positions from 2,048 buckets of equal width in key: a word's rank is the number of words in the
// buckets before its own plus the smaller ones in it, one or two on average.  Sorted runs and binary
// searches in the other warps' took half of the 37 us that 2,900 candidates cost (k = 2048), now 18.5.  False, with nothing
// written, when the keys do not spread (equal keys, infinities).  All threads of the CTA call it.
__device__ bool bucket_place(const RowSelectParams& p, int64_t qo, int c, float lo, float hi, const uint64_t* words,
                             int* end, uint16_t* order, int* s_warp, int* s_beyond) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, T = blockDim.x;
    const float scale = (RS_BUCKETS - 1) / (hi - lo);
    if (!(scale > 0.f && scale < CUDART_INF_F && hi - lo < CUDART_INF_F)) return false;   // the same for every thread
    auto bucket = [&](uint64_t w) {   // ascending with the key; clamped against rounding
        return max(0, min((int)((ordered_to_float((uint32_t)(w >> 32)) - lo) * scale), RS_BUCKETS - 1));
    };
    for (int i = tid; i < RS_BUCKETS; i += T) end[i] = 0;
    __syncthreads();
    for (int i = tid; i < c; i += T) atomicAdd(&end[bucket(words[i])], 1);
    __syncthreads();
    // exclusive prefix sums in place: RS_BUCKETS / T consecutive buckets per thread (T >= 128)
    const int per = RS_BUCKETS / T;
    int sum = 0, most = 0;
    for (int i = 0; i < per; i++) {
        const int h = end[tid * per + i];
        sum += h;
        most = max(most, h);
    }
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int up = __shfl_up_sync(FULL, incl, o);
        if (lane >= o) incl += up;
    }
    if (lane == 31) s_warp[warp] = incl;
    if (__syncthreads_or(most > RS_BUCKET_MAX)) return false;
    int start = incl - sum;
    for (int w = 0; w < warp; w++) start += s_warp[w];
    for (int i = 0; i < per; i++) {
        const int h = end[tid * per + i];
        end[tid * per + i] = start;
        start += h;
    }
    __syncthreads();
    for (int i = tid; i < c; i += T) order[atomicAdd(&end[bucket(words[i])], 1)] = (uint16_t)i;
    __syncthreads();
    for (int i = tid; i < c; i += T) {
        const uint64_t w = words[i];
        const int b = bucket(w);
        const int first = b > 0 ? end[b - 1] : 0;
        int rank = first;
        for (int j = first; j < end[b]; j++) rank += words[order[j]] < w ? 1 : 0;
        if (rank < p.k) rs_write(p, qo, rank, w, s_beyond);
    }
    return true;
}

// The k best of a row that fits the CTA's registers, RS_REGS words a thread: read once, counted in buckets of equal
// width, and the buckets up to the one that holds the k-th word are scattered and ranked inside themselves.  Five
// barriers.  The buckets span [lo, hi]: hi is a key that k words are known to be up to (the largest of the warps'
// smallest keys where there are k warps, of the threads' where there are k threads, else the largest key), lo the second
// smallest of the warps' smallest keys, so that one row far nearer than the others (a query that is itself
// stored) does not stretch the buckets.  Four buckets a thread, 2,048 at most: clearing and summing 16 of them took
// longer than placing 130 candidates.  False, with nothing written, where the keys do not spread (ties, infinities).
// 50 rows of 3,900 candidates, k = 2048: 18 us with thread minima, radix digits and a second reading of the row;
// the search 116 -> 102.5 us.
// Ten words a thread, 64 registers (4 bytes of the longer way spilled): with eight 300 queries, k = 1024, on 300,000 rows take
// 201 us instead of 191, 100 queries on 10,000 rows 69.6 instead of 66.5; with twelve shorter rows take 1 - 2 % more (50 queries,
// k = 2048: 107.8 -> 109.3), 12,000 keys 59.0 instead of 62.8.
constexpr int RS_REGS = 10;
__device__ __forceinline__ bool register_select(const RowSelectParams& p, int64_t qo, const float* keys, const int32_t* ids, int n,
                                                uint64_t* words, int* end, int* s_live, uint32_t* s_min, uint32_t* s_max,
                                                uint32_t* s_maxmin, int* s_warp, int* s_cut, int& live, int& c, int* s_beyond) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, T = blockDim.x, W = T >> 5;
    // consecutive buckets belong to one thread, T words apart
    const int nbk = min(RS_BUCKETS, 4 * T), per = nbk / T, log_per = 31 - __clz(per);
    auto at = [&](int b) { return (b & (per - 1)) * T + (b >> log_per); };
    uint32_t key[RS_REGS];
    int32_t id[RS_REGS];
#pragma unroll
    for (int r = 0; r < RS_REGS; r++) {
        const int col = r * T + tid;
        id[r] = -1;
        key[r] = 0xffffffffu;
        if (col < n) {
            const float f = __ldca(keys + col) + 0.f;   // -0 becomes +0: the two tie
            id[r] = ids ? __ldca(ids + col) : (f <= p.last_key ? col : -1);
            key[r] = float_to_ordered(f);
        }
    }
    for (int i = tid; i < nbk; i += T) end[i] = 0;
    uint32_t tmin = 0xffffffffu, tmax = 0;
    int have = 0;
#pragma unroll
    for (int r = 0; r < RS_REGS; r++) {
        if (id[r] < 0) continue;
        tmin = min(tmin, key[r]);
        tmax = max(tmax, key[r]);
        have++;
    }
    {
        const uint32_t a = __reduce_min_sync(FULL, tmin), b = __reduce_max_sync(FULL, tmax), m = __reduce_max_sync(FULL, tmin);
        const int l = __reduce_add_sync(FULL, have);
        if (lane == 0) {
            s_min[warp] = a;
            s_max[warp] = b;
            s_maxmin[warp] = m;
            s_live[warp] = l;
        }
    }
    __syncthreads();
    const uint32_t wmin = lane < W ? s_min[lane] : 0xffffffffu;
    live = __reduce_add_sync(FULL, lane < W ? s_live[lane] : 0);
    const uint32_t mx = __reduce_max_sync(FULL, lane < W ? s_max[lane] : 0u);
    const uint32_t mn = __reduce_min_sync(FULL, wmin);
    const uint32_t mn_of_threads = __reduce_max_sync(FULL, lane < W ? s_maxmin[lane] : 0u);   // 0xffffffff: a thread without a word
    const uint32_t mn_of_warps = __reduce_max_sync(FULL, lane < W ? wmin : 0u);
    uint32_t hi_key = mx;
    if (p.k <= W && mn_of_warps != 0xffffffffu) hi_key = mn_of_warps;
    else if (p.k <= T && mn_of_threads != 0xffffffffu) hi_key = mn_of_threads;
    const int first = __ffs(__ballot_sync(FULL, wmin == mn)) - 1;
    uint32_t lo_key = __reduce_min_sync(FULL, lane == first ? 0xffffffffu : wmin);
    if (lo_key > hi_key) lo_key = mn;
    const float lo = ordered_to_float(lo_key), hi = ordered_to_float(hi_key);
    const float scale = (nbk - 1) / (hi - lo);
    if (live == 0 || !(scale > 0.f && scale < CUDART_INF_F && hi - lo < CUDART_INF_F)) return false;   // the same for every thread
    auto bucket = [&](uint32_t k) {   // ascending with the key
        return max(0, min((int)((ordered_to_float(k) - lo) * scale), nbk - 1));
    };
#pragma unroll
    for (int r = 0; r < RS_REGS; r++)
        if (id[r] >= 0 && key[r] <= hi_key) atomicAdd(&end[at(bucket(key[r]))], 1);
    __syncthreads();
    int sum = 0;
    for (int i = 0; i < per; i++) sum += end[i * T + tid];
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int up = __shfl_up_sync(FULL, incl, o);
        if (lane >= o) incl += up;
    }
    if (lane == 31) s_warp[warp] = incl;
    if (tid == 0) s_cut[0] = s_cut[1] = -1;
    __syncthreads();
    int start = incl - sum;
    for (int w = 0; w < warp; w++) start += s_warp[w];
    bool full = false;
    for (int i = 0; i < per; i++) {
        const int b = tid * per + i, h = end[i * T + tid];
        end[i * T + tid] = start;
        if (start < p.k && h > RS_BUCKET_MAX) full = true;
        if (start < p.k && start + h >= p.k) {   // one bucket of one thread
            s_cut[0] = b;
            s_cut[1] = start + h;
        }
        start += h;
    }
    if (tid == T - 1) s_cut[2] = start;   // words up to hi
    if (__syncthreads_or(full)) return false;
    // fewer than k up to hi: then hi is the largest key, and all of them count
    const int cut = s_cut[0] < 0 ? nbk - 1 : s_cut[0];
    c = s_cut[0] < 0 ? s_cut[2] : s_cut[1];
#pragma unroll
    for (int r = 0; r < RS_REGS; r++) {
        if (id[r] < 0 || key[r] > hi_key) continue;
        const int b = bucket(key[r]);
        if (b <= cut) words[atomicAdd(&end[at(b)], 1)] = ((uint64_t)key[r] << 32) | (uint32_t)id[r];
    }
    __syncthreads();
    for (int i = tid; i < c; i += T) {
        const uint64_t w = words[i];
        const int b = bucket((uint32_t)(w >> 32));
        const int from = b > 0 ? end[at(b - 1)] : 0, to = end[at(b)];
        int rank = from;
        for (int j = from; j < to; j++) rank += words[j] < w ? 1 : 0;
        if (rank < p.k) rs_write(p, qo, rank, w, s_beyond);
    }
    return true;
}

// One CTA per row, latency-bound (a row is a few KB in L1 / L2).  Rows of up to RS_REGS words a thread: register_select.
// Longer ones, and those whose keys do not spread: a pass over the keys leaves every
// thread with the M smallest keys of its share; with k <= M T / 2 the k-th smallest of those M T bounds the
// row's k-th key from above and admits little more than k keys (2 histogram passes over registers instead
// of 4 over the row: 10,000 rows of 20,000 keys, k = 1000: 2,415 us with M = 1, which leaves k > T / 2 to
// the passes over the row, 551 with M = 4).  Otherwise, or when that bound admits more than the
// staging area holds, the k-th key is found exactly by radix select over the row.  The words up to
// the bound are compacted and placed: by counting the smaller ones up to 256 of them, else from buckets of
// equal width, or sorted per warp and placed by binary search where the keys do not spread.  Where even the exact k-th key is shared by more than fit (hundreds
// of ties), a second radix select over the ids of those finds the ones that belong to the result.
template <int M>
__global__ void __launch_bounds__(1024) row_select_kernel(const RowSelectParams p) {
    extern __shared__ __align__(16) uint64_t rs_runs[];   // bound words, then the buckets of bucket_place
    __shared__ int s_hist[256];
    __shared__ uint32_t s_min[32], s_max[32];
    __shared__ int s_live[32];
    __shared__ int s_sel[4];
    __shared__ int s_count, s_have, s_beyond;
    pdl_wait();   // what the kernel before wrote is read with coherent loads
    pdl_trigger();
    const int W = blockDim.x >> 5;
    const int T = blockDim.x;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t nq_live = p.nq_dev ? min((int64_t)*p.nq_dev, p.nq) : p.nq;
    if (p.redone && p.nq_dev && nq_live > 0 && blockIdx.x == 0 && tid == 0) *p.redone = (int32_t)nq_live;
    for (int64_t q = blockIdx.x; q < nq_live; q += gridDim.x) {
        const int64_t cnt = p.cnt ? (int64_t)__ldcg(p.cnt + q) : p.n;
        const int n = (int)min(cnt, p.ld);
        const float* keys = p.keys + q * p.ld;
        const int32_t* ids = p.ids ? p.ids + q * p.ld : nullptr;
        const int64_t qo = p.row_map ? (int64_t)p.row_map[q] : q;
        int live = 0, c = 0;
        if (tid == 0) s_beyond = 0;   // behind several barriers before the first word is written
        if (n > RS_REGS * T || !register_select(p, qo, keys, ids, n, rs_runs, reinterpret_cast<int*>(rs_runs + p.bound), s_live,
                                                s_min, s_max, reinterpret_cast<uint32_t*>(s_hist), s_hist + 32, s_sel, live, c,
                                                &s_beyond)) {
            __syncthreads();
            // (ordered key, live) of column c; both loads are issued before either is used
            auto load = [&](int c, uint32_t& key, int32_t& id) {
                const float f = __ldca(keys + c) + 0.f;   // -0 becomes +0: the two tie
                id = ids ? __ldca(ids + c) : (f <= p.last_key ? c : -1);
                key = float_to_ordered(f);
            };
            live = 0;
            uint32_t mx = 0;
            uint32_t best[M];   // ascending
#pragma unroll
            for (int i = 0; i < M; i++) best[i] = 0xffffffffu;
#pragma unroll 8
            for (int col = tid; col < n; col += T) {
                uint32_t key;
                int32_t id;
                load(col, key, id);
                if (id >= 0) {
                    live++;
                    mx = max(mx, key);
#pragma unroll
                    for (int i = 0; i < M; i++) {
                        const uint32_t lo = min(best[i], key);
                        key = max(best[i], key);
                        best[i] = lo;
                    }
                }
            }
            uint32_t mn = best[0];
            const int my_have = min(live, M);
            if (tid == 0) s_count = s_have = 0;
            const Spread sp = block_spread(live, mn, mx, s_live, s_min, s_max);
            live = sp.live;
            mn = sp.mn;
            auto visit_all = [&](auto f) {
#pragma unroll 4
                for (int col = tid; col < n; col += T) {
                    uint32_t key;
                    int32_t id;
                    load(col, key, id);
                    if (id >= 0) f(key);
                }
            };
            const int bits = 32 - __clz(sp.mx - mn);   // significant bits of the spread (live > 0)
            uint32_t thr_x = live > 0 ? sp.mx - mn : 0;
            uint32_t tie_id = 0x7fffffffu;             // of the keys equal to thr_x: ids up to this one
            bool loose = false;
            if (live > p.k) {
                if (2 * p.k <= M * T) {
                    const int have = __reduce_add_sync(FULL, my_have);   // s_have was cleared before block_spread's barrier
                    if (lane == 0) atomicAdd(&s_have, have);
                    __syncthreads();
                    loose = s_have >= p.k;
                }
                if (loose) {
                    int kk = p.k;
                    thr_x = radix_kth(
                            [&](auto f) {
#pragma unroll
                                for (int i = 0; i < M; i++)
                                    if (i < my_have) f(best[i]);
                            },
                            mn, bits, bits > 16 ? bits - 16 : 0, kk,
                                      s_hist, s_sel);
                } else {
                    int kk = p.k;
                    thr_x = radix_kth(visit_all, mn, bits, 0, kk, s_hist, s_sel);
                }
            }
            // compaction of the candidates up to the threshold (k of them plus a few, or all)
            c = 0;
            for (int pass = 0; pass < 2; pass++) {
                for (int c0 = warp * 32; c0 < n; c0 += T) {
                    const int cc = c0 + lane;
                    bool keep = false;
                    uint64_t word = 0;
                    if (cc < n) {
                        uint32_t key;
                        int32_t id;
                        load(cc, key, id);
                        const uint32_t x = key - mn;           // live keys are >= mn
                        keep = id >= 0 && (x < thr_x || (x == thr_x && (uint32_t)id <= tie_id));
                        word = ((uint64_t)key << 32) | (uint32_t)id;
                    }
                    const unsigned b = __ballot_sync(FULL, keep);
                    int base = 0;
                    if (lane == 0 && b) base = atomicAdd(&s_count, __popc(b));
                    base = __shfl_sync(FULL, base, 0);
                    const int pos = base + __popc(b & ((1u << lane) - 1u));
                    if (keep && pos < p.bound) rs_runs[pos] = word;
                }
                __syncthreads();
                c = s_count;
                if (c <= p.bound || pass == 1) break;
                // more than fit: the exact k-th key, and of the keys equal to it the ids that are wanted
                // (exactly k words are kept the second time)
                __syncthreads();   // everybody has read the count
                if (tid == 0) s_count = 0;
                int kk = p.k;
                thr_x = radix_kth(visit_all, mn, bits, 0, kk, s_hist, s_sel);
                tie_id = radix_kth(
                        [&](auto f) {
                            for (int cc = tid; cc < n; cc += T) {
                                uint32_t key;
                                int32_t id;
                                load(cc, key, id);
                                if (id >= 0 && key - mn == thr_x) f((uint32_t)id);
                            }
                        },
                        0u, 31, 0, kk, s_hist, s_sel);
            }
            c = min(c, p.bound);   // ids are distinct: the second pass keeps k words
            if (c <= RS_COUNT_MAX) {
                for (int i = tid; i < c; i += T) {
                    const uint64_t w = rs_runs[i];
                    int rank = 0;
#pragma unroll 8
                    for (int j = 0; j < c; j++) rank += rs_runs[j] < w ? 1 : 0;
                    if (rank < p.k) rs_write(p, qo, rank, w, &s_beyond);
                }
            } else if (!bucket_place(p, qo, c, ordered_to_float(mn), ordered_to_float(mn + min(thr_x, sp.mx - mn)), rs_runs,
                                     reinterpret_cast<int*>(rs_runs + p.bound),
                                     reinterpret_cast<uint16_t*>(rs_runs + p.bound) + 2 * RS_BUCKETS, s_live, &s_beyond)) {
                const int m = (c + W - 1) / W;    // <= RS_RUN
                if (m <= 32) rank_place<1>(p, qo, c, m, rs_runs, W, &s_beyond);
                else if (m <= 64) rank_place<2>(p, qo, c, m, rs_runs, W, &s_beyond);
                else if (m <= 128) rank_place<4>(p, qo, c, m, rs_runs, W, &s_beyond);
                else if (m <= 256) rank_place<8>(p, qo, c, m, rs_runs, W, &s_beyond);
                else rank_place<16>(p, qo, c, m, rs_runs, W, &s_beyond);
            }
        }
        for (int j = c + tid; j < p.k; j += T) {
            p.out_dist[qo * p.k + j] = p.pad;
            p.out_labels[qo * p.k + j] = -1;
        }
        if (p.thr) __syncthreads();   // s_beyond is complete
        if (tid == 0 && p.dirty) {
            const bool bad = cnt > p.ld || (live < p.k && live < p.nb_total) || s_beyond;
            p.dirty[q] = bad ? 1 : 0;
            s_sel[0] = -1;
            if (bad && p.redo.count) {
                if (p.redo.all > 0) {
                    *p.redo.count = p.redo.all;
                } else {
                    const int j = atomicAdd(p.redo.count, 1);
                    p.redo.rows[j] = (int32_t)q;
                    s_sel[0] = j;
                }
            }
        }
        if (p.redo.out) {   // the query operand of a row to redo
            __syncthreads();
            const int j = s_sel[0];
            if (j >= 0) {
                const int vec_per_row = (int)(p.redo.pitch / 8);
                for (int v = tid; v < p.redo.npl * vec_per_row; v += T) {
                    const int pl = v / vec_per_row, c = v - pl * vec_per_row;
                    reinterpret_cast<uint4*>(p.redo.out + pl * p.redo.plane_stride + j * p.redo.pitch)[c] =
                            reinterpret_cast<const uint4*>(p.redo.a + pl * p.redo.plane_stride + q * p.redo.pitch)[c];
                }
            }
        }
        __syncthreads();   // the shared arrays are rewritten by the next row
    }
}

// Threshold of the filters: an upper bound of the r-th smallest of a row's n sample keys, the r-th
// smallest of the T thread minima (T several times r keeps it close; +INF where fewer than r threads
// have a key, which lets every row pass).  One CTA per row; out[q] may be exceeded by no key that
// belongs to the r smallest.
__global__ void __launch_bounds__(1024) row_bound_kernel(const float* keys, int64_t ld, int64_t n,
                                                         int group, int64_t nq, int r, float* __restrict__ out,
                                                         int32_t* __restrict__ bad, const float* __restrict__ qnorm,
                                                         float margin, float qnorm_max, int most) {
    __shared__ int s_hist[256];
    __shared__ uint32_t s_min[32], s_max[32];
    __shared__ int s_live[32];
    __shared__ int s_sel[2];
    extern __shared__ float rb_part[];   // [3][T], of minima
    const int tid = threadIdx.x, T = blockDim.x;   // a power of two
    pdl_wait();   // the sample's keys are read with coherent loads
    pdl_trigger();
    // four values a load: minima always, keys while that leaves every thread several
    const bool vec = (group > 1 || n >= 8 * T) && (ld & 3) == 0 && (reinterpret_cast<uintptr_t>(keys) & 15) == 0;
    for (int64_t q = blockIdx.x; q < nq; q += gridDim.x) {
        const float* row = keys + q * ld;
        float best = CUDART_INF_F;   // fminf drops NaN
        if (vec) {
            float m[4] = {CUDART_INF_F, CUDART_INF_F, CUDART_INF_F, CUDART_INF_F};
            constexpr int U = 4;   // loads on their way together
            for (int64_t c = (int64_t)tid * 4; c + 4 <= n; c += (int64_t)T * 4 * U) {
                float4 f[U];
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const int64_t cu = c + u * (int64_t)T * 4;
                    f[u] = cu + 4 <= n ? __ldcg(reinterpret_cast<const float4*>(row + cu))
                                       : make_float4(CUDART_INF_F, CUDART_INF_F, CUDART_INF_F, CUDART_INF_F);
                }
#pragma unroll
                for (int u = 0; u < U; u++) {
                    m[0] = fminf(m[0], f[u].x);
                    m[1] = fminf(m[1], f[u].y);
                    m[2] = fminf(m[2], f[u].z);
                    m[3] = fminf(m[3], f[u].w);
                }
            }
            if (tid < (n & 3)) m[0] = fminf(m[0], __ldcg(row + (n & ~(int64_t)3) + tid));
            if (group > 1) {
                // Each of a load's four goes to another thread, so that T minima in a row belong to T threads: near rows
                // side by side are as many of the minima that are ranked as they would be without groups.  One by one,
                // a coalesced load each, 1,000 rows of 1,664 took the search 3 us longer.
#pragma unroll
                for (int j = 1; j < 4; j++) rb_part[(j - 1) * T + tid] = m[j];
                __syncthreads();
#pragma unroll
                for (int j = 1; j < 4; j++) m[j] = rb_part[(j - 1) * T + ((tid + j * (T >> 2)) & (T - 1))];
            }
            best = fminf(fminf(m[0], m[1]), fminf(m[2], m[3]));
        } else {
#pragma unroll 4
            for (int64_t c = tid; c < n; c += T) best = fminf(best, __ldcg(row + c));
        }
        const bool have = best < CUDART_INF_F;
        const uint32_t key = float_to_ordered(best + 0.f);
        const Spread sp = block_spread(have ? 1 : 0, have ? key : 0xffffffffu, have ? key : 0u, s_live, s_min, s_max);
        float bound = CUDART_INF_F;
        if (sp.live >= r) {
            const int bits = 32 - __clz(sp.mx - sp.mn);
            int kk = r;
            // three digits: with keys of both signs the spread has 32 bits, and two would leave the bound
            // 2^-7 of the key loose
            const uint32_t x = radix_kth([&](auto f) { if (have) f(key); }, sp.mn, bits, bits > 24 ? bits - 24 : 0, kk,
                                         s_hist, s_sel);
            bound = ordered_to_float(sp.mn + min(x, sp.mx - sp.mn));
        }
        if (tid == 0) out[q] = bound;
        if (bad) {
            const float qn = __ldg(qnorm + q);
            const int under = __syncthreads_count(best <= bound + margin * qn);
            if (tid == 0 && (under > most || !(qn < qnorm_max))) atomicAdd(bad, 1);
        }
        __syncthreads();   // the shared arrays are rewritten by the next row
    }
}

// ---------------------------------------------------------------------------------------
// rank_merge
// ---------------------------------------------------------------------------------------
struct RankMergeParams {
    const float* dist;       // list l of query q at dist + l * stride_d + q * k
    const int64_t* labels;   // same layout with stride_l; -1 = empty slot
    int64_t stride_d, stride_l;
    int P;
    int64_t nq;
    int k;
    int Tp;                  // P k rounded up to a power of two (entries of the shared arrays)
    float key_sign;          // key = key_sign * dist, smaller is better
    float pad;
    float* out_dist;
    int64_t* out_labels;
};

constexpr int RM_MAX_LISTS = 256;   // P <= 8192 / 33

// (key, label) of a before (key, label) of b; an empty slot (label -1) is the largest label
__device__ __forceinline__ bool rm_before(uint32_t ka, uint64_t la, uint32_t kb, uint64_t lb) {
    return ka < kb || (ka == kb && la < lb);
}

__global__ void __launch_bounds__(512, 2) rank_merge_kernel(const RankMergeParams p) {
    extern __shared__ __align__(16) uint64_t rm_lab[];    // [Tp] labels, then [Tp] ordered keys
    __shared__ int s_live;
    __shared__ int s_start[RM_MAX_LISTS + 1];   // entries up to tau: list l holds [s_start[l], s_start[l+1]) of them
    const int T = p.P * p.k;
    uint32_t* rm_key = reinterpret_cast<uint32_t*>(rm_lab + p.Tp);
    const int tid = threadIdx.x;
    const int kp = (p.k + p.P - 1) / p.P;
    for (int64_t q = blockIdx.x; q < p.nq; q += gridDim.x) {
        __syncthreads();   // the previous row's readers are done
        if (tid == 0) s_live = 0;
        __syncthreads();
        // flat index over all lists: every thread's loads are in flight together
        int live = 0;
#pragma unroll 4
        for (int c = tid; c < p.Tp; c += blockDim.x) {
            uint64_t lab = RS_EMPTY;
            uint32_t key = 0xffffffffu;
            if (c < T) {
                const int l = c / p.k;
                const int64_t off = q * p.k + (c - l * p.k);
                const int64_t lb = __ldg(p.labels + (int64_t)l * p.stride_l + off);
                const float d = __ldg(p.dist + (int64_t)l * p.stride_d + off);
                if (lb >= 0) {
                    lab = (uint64_t)lb;
                    key = float_to_ordered(p.key_sign * d);
                    live++;
                }
            }
            rm_lab[c] = lab;
            rm_key[c] = key;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) live += __shfl_xor_sync(FULL, live, o);
        if ((tid & 31) == 0 && live) atomicAdd(&s_live, live);
        __syncthreads();
        // every list must ascend strictly in (key, label), empty slots last
        int bad = 0;
        for (int c = tid; c < T; c += blockDim.x) {
            if (c % p.k == 0) continue;
            const bool both_empty = rm_lab[c] == RS_EMPTY && rm_lab[c - 1] == RS_EMPTY;
            if (!both_empty && !rm_before(rm_key[c - 1], rm_lab[c - 1], rm_key[c], rm_lab[c])) bad = 1;
        }
        bad = __syncthreads_or(bad);
        if (bad) {
            // equal keys next to each other in label order: four odd-even rounds settle runs of
            // up to four (final distances that tie although the shard's keys did not)
            for (int phase = 0; phase < 4; phase++) {
                for (int l = 0; l < p.P; l++) {
                    for (int j = (phase & 1) + 2 * tid; j + 1 < p.k; j += 2 * blockDim.x) {
                        const int c = l * p.k + j;
                        if (rm_key[c] == rm_key[c + 1]) {
                            const uint64_t a = rm_lab[c], b = rm_lab[c + 1];
                            if (a > b) {
                                rm_lab[c] = b;
                                rm_lab[c + 1] = a;
                            }
                        }
                    }
                }
                __syncthreads();
            }
            bad = 0;
            for (int l = 0; l < p.P; l++) {
                for (int j = 1 + tid; j < p.k; j += blockDim.x) {
                    const int c = l * p.k + j;
                    const bool both_empty = rm_lab[c] == RS_EMPTY && rm_lab[c - 1] == RS_EMPTY;
                    if (!both_empty && !rm_before(rm_key[c - 1], rm_lab[c - 1], rm_key[c], rm_lab[c])) bad = 1;
                }
            }
            bad = __syncthreads_or(bad);
        }
        if (!bad) {
            // at least P * kp >= k entries have a key up to tau: nothing beyond it is in the result
            uint32_t tau = 0;
            for (int l = 0; l < p.P; l++) tau = max(tau, rm_key[l * p.k + kp - 1]);
            for (int l = tid; l < p.P; l += blockDim.x) {
                const uint32_t* run = rm_key + l * p.k;
                int lo = 0, hi = p.k;
                while (lo < hi) {
                    const int mid = (lo + hi) >> 1;
                    if (run[mid] <= tau) lo = mid + 1; else hi = mid;
                }
                s_start[l + 1] = lo;   // a count for now
            }
            __syncthreads();
            if (tid == 0) {
                s_start[0] = 0;
                for (int l = 0; l < p.P; l++) s_start[l + 1] += s_start[l];
            }
            __syncthreads();
            const int S = s_start[p.P];
            for (int e = tid; e < S; e += blockDim.x) {
                int l = 0;
                while (s_start[l + 1] <= e) l++;
                const int j = e - s_start[l];
                const uint64_t lab = rm_lab[l * p.k + j];
                const uint32_t key = rm_key[l * p.k + j];
                if (lab == RS_EMPTY) continue;
                int rank = j;
                for (int o = 0; o < p.P && rank < p.k; o++) {
                    if (o == l) continue;
                    // entries of list o that come first: an equal (key, label) in a lower list does
                    const int base = o * p.k;
                    int lo = 0, hi = s_start[o + 1] - s_start[o];
                    while (lo < hi) {
                        const int mid = (lo + hi) >> 1;
                        const uint32_t km = rm_key[base + mid];
                        bool first = km < key;
                        if (km == key) {
                            const uint64_t lm = rm_lab[base + mid];
                            first = lm < lab || (lm == lab && o < l);
                        }
                        if (first) lo = mid + 1; else hi = mid;
                    }
                    rank += lo;
                }
                if (rank < p.k) {
                    p.out_dist[q * p.k + rank] = p.key_sign * ordered_to_float(key);
                    p.out_labels[q * p.k + rank] = (int64_t)lab;
                }
            }
        } else {
            // any order at all: bitonic sort of the (key, label) records
            for (int size = 2; size <= p.Tp; size <<= 1) {
                for (int stride = size >> 1; stride > 0; stride >>= 1) {
                    for (int i = tid; i < (p.Tp >> 1); i += blockDim.x) {
                        const int pos = 2 * i - (i & (stride - 1));
                        const uint32_t ka = rm_key[pos], kb = rm_key[pos + stride];
                        const uint64_t la = rm_lab[pos], lb = rm_lab[pos + stride];
                        const bool up = (pos & size) == 0;
                        if (rm_before(kb, lb, ka, la) == up && !(ka == kb && la == lb)) {
                            rm_key[pos] = kb;
                            rm_key[pos + stride] = ka;
                            rm_lab[pos] = lb;
                            rm_lab[pos + stride] = la;
                        }
                    }
                    __syncthreads();
                }
            }
            for (int j = tid; j < p.k; j += blockDim.x) {
                const uint64_t lab = rm_lab[j];
                if (lab != RS_EMPTY) {
                    p.out_dist[q * p.k + j] = p.key_sign * ordered_to_float(rm_key[j]);
                    p.out_labels[q * p.k + j] = (int64_t)lab;
                }
            }
        }
        const int total = s_live;
        for (int j = total + tid; j < p.k; j += blockDim.x) {
            p.out_dist[q * p.k + j] = p.pad;
            p.out_labels[q * p.k + j] = -1;
        }
    }
}

}  // namespace

bool rank_select_enabled() { return g_rank_select.load(std::memory_order_relaxed) != 0; }

namespace {

// Threads per row: few for many rows of few candidates, many for few long rows.  The staging area
// holds 4 k words and at least 1024, 8192 at most: W warps sort at most RS_RUN words each.
int launch_row_select(RowSelectParams& p, int64_t n_typical, const Launch& ln) {
    if (p.nq <= 0) return B200F_OK;
    if (p.k < 1 || p.k > B200F_MAX_K) return B200F_ERR_UNSUPPORTED;
    const int64_t sm = cached_sm_count();
    int bound = 1024;
    while (bound < 4 * p.k && bound < 8192) bound <<= 1;
    int T = 128;
    while (T < 1024 && (T * RS_RUN < 32 * bound ||                         // the area must be sortable
                        (p.nq * T < sm * 512 && T * 4 < n_typical)))        // rows alone do not fill the SMs
        T <<= 1;
    if (p.k > 64 && T < 256) T = 256;
    // long rows: enough minima (four a thread beyond k = T / 2) to bound the k-th key without histogram
    // passes over the row
    while (T < 1024 && 4 * T < 2 * p.k && 16 * (int64_t)T < n_typical) T <<= 1;
    const bool four = 2 * p.k > T;
    p.bound = bound;
    const int smem = bound * 8 + RS_BUCKETS * 4 + bound * 2;   // words, buckets, order
    static bool attr_set[kMaxDevices] = {false};
    const int slot = device_slot();
    if (!attr_set[slot]) {
        for (auto* fn : {row_select_kernel<1>, row_select_kernel<4>})
            B200F_CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                8192 * 10 + RS_BUCKETS * 4));
        attr_set[slot] = true;
    }
    int64_t g = p.nq;
    const int64_t gcap = sm * (2048 / T);
    if (g > gcap) g = gcap;
    // rows counted on the device are usually few or none: idle CTAs leave at once
    if (p.nq_dev && g > sm) g = sm;
    // Launched before the distance kernel's SMs are idle the CTAs would keep its division of them, nearly all shared memory.
    // That matters where a row of keys is read several times and fits the L1 of an SM with one CTA: on most SMs (the matrix of
    // 148 queries on 32,000 rows, k = 10: 90 us a search, 79 launched plainly; 20 queries 62 and 65, 300 129 and 123 - 129), and
    // in a redo, where every SM has one, if it is of many rows (1,000 queries on 100,000 rows ordered by cluster, k = 40: 1,600 and
    // 1,330 us).  With nothing to redo the plain launch takes 2 us, and fewer than 600 queries are under 120.
    const bool several = !p.ids && n_typical > RS_REGS * T;
    const bool plain = several && (p.nq_dev ? p.nq >= 4 * sm : 2 * g > sm && g <= sm);
    B200F_CUDA_TRY(launch_kernel(four ? row_select_kernel<4> : row_select_kernel<1>, dim3((unsigned)g), T, smem,
                                 plain ? Launch(ln.stream) : ln, p));
    count_launch();
    B200F_LAUNCH_CHECK();
    return B200F_OK;
}

void set_output(RowSelectParams& p, int metric, const float* qnorm, int64_t label_base, float* out_dist,
                int64_t* out_labels) {
    const bool l2 = metric == B200F_METRIC_L2;
    p.out_sign = l2 ? 1.f : -1.f;
    p.qnorm = l2 ? qnorm : nullptr;
    p.clamp = l2 ? 1 : 0;
    p.pad = l2 ? kHostInf : -kHostInf;
    p.label_base = label_base;
    p.out_dist = out_dist;
    p.out_labels = out_labels;
}

}  // namespace

int row_bound_threads(int64_t nq, int64_t n, int r) {
    const int64_t sm = cached_sm_count();
    int T = 128;
    while (T < 1024 && (T < 8 * r || (nq < sm * 512 / T && T * 8 < n))) T <<= 1;
    return T;
}

int row_bound_most(int64_t nq, int64_t n, int r, double most) {
    const int T = row_bound_threads(nq, n, r);
    return (int)(T * (1.0 - std::exp(-most / T)));
}

int launch_row_bound(const float* keys, int64_t nq, int64_t n, int64_t ld, int group, int r, float* out, int32_t* bad,
                     const float* qnorm, float margin, float qnorm_max, double most, const Launch& ln) {
    if (r < 1 || r > 512 || n < 0 || ld < n || group < 1 || !keys || !out) return B200F_ERR_BAD_ARG;
    if (nq <= 0) return B200F_OK;
    const int64_t sm = cached_sm_count();
    const int T = row_bound_threads(nq, n * group, r);   // as many as the keys themselves would have
    int64_t g = nq;
    const int64_t gcap = sm * (2048 / T);
    if (g > gcap) g = gcap;
    const int most_minima = row_bound_most(nq, n, r, most);
    const size_t smem = group > 1 ? 3 * T * sizeof(float) : 0;
    B200F_CUDA_TRY(launch_kernel(row_bound_kernel, dim3((unsigned)g), T, smem, ln, keys, ld, n, group, nq, r, out, bad, qnorm,
                                 margin, qnorm_max, most_minima));
    count_launch();
    B200F_LAUNCH_CHECK();
    return B200F_OK;
}

int launch_rank_select(const float* cand_key, const int32_t* cand_idx, const int32_t* cand_cnt, int cap,
                       int64_t nb, int64_t nq, int k, int metric, const float* qnorm, int64_t label_base,
                       float* out_dist, int64_t* out_labels, int32_t* dirty, const float* thr,
                       const RedoRows& redo, const Launch& ln) {
    if (cap < 1 || !cand_cnt || !dirty) return B200F_ERR_BAD_ARG;
    RowSelectParams p{};
    p.keys = cand_key;
    p.ids = cand_idx;
    p.cnt = cand_cnt;
    p.ld = cap;
    p.nb_total = nb;
    p.nq = nq;
    p.k = k;
    p.dirty = dirty;
    p.thr = thr;
    p.redo = redo;
    set_output(p, metric, qnorm, label_base, out_dist, out_labels);
    return launch_row_select(p, cap / 4, ln);
}

int launch_merge_partials(const float* part_key, const int32_t* part_idx, int P, int64_t nq, int k,
                          int metric, const float* qnorm, int64_t label_base, float* out_dist,
                          int64_t* out_labels, const int* nq_dev, const int32_t* row_map, int32_t* redone,
                          int64_t nb, int32_t* dirty, const RedoRows& redo, const Launch& ln) {
    if (nq <= 0) return B200F_OK;
    if (k < 1 || k > 32 || P < 1) return B200F_ERR_UNSUPPORTED;
    RowSelectParams p{};
    p.keys = part_key;
    p.ids = part_idx;
    p.ld = (int64_t)P * k;
    p.n = (int64_t)P * k;
    p.nb_total = nb;
    p.dirty = dirty;
    p.redo = redo;
    p.nq = nq;
    p.nq_dev = nq_dev;
    p.row_map = row_map;
    p.redone = redone;
    p.k = k;
    set_output(p, metric, qnorm, label_base, out_dist, out_labels);
    return launch_row_select(p, p.n, ln);
}

int launch_matrix_select(const float* keys, int64_t nq, int64_t n, int64_t ld, int k, bool inf_empty, int metric,
                         const float* qnorm, int64_t label_base, float* out_dist, int64_t* out_labels,
                         const int* nq_dev, const int32_t* row_map, int32_t* redone, const Launch& ln) {
    if (n < 0 || n > 0x7fffffffLL || ld < n) return B200F_ERR_BAD_ARG;
    RowSelectParams p{};
    p.keys = keys;
    p.ld = ld;
    p.n = n;
    p.last_key = inf_empty ? FLT_MAX : kHostInf;
    p.nq = nq;
    p.nq_dev = nq_dev;
    p.row_map = row_map;
    p.redone = redone;
    p.k = k;
    set_output(p, metric, qnorm, label_base, out_dist, out_labels);
    return launch_row_select(p, n, ln);
}

bool rank_merge_fits(int P, int k) { return k > 32 && P >= 1 && (int64_t)P * k <= 8192; }

int launch_rank_merge(const float* dist, const int64_t* labels, int64_t stride_d, int64_t stride_l, int P,
                      int64_t nq, int k, int metric, float* out_dist, int64_t* out_labels,
                      cudaStream_t stream) {
    if (!rank_merge_fits(P, k)) return B200F_ERR_BAD_ARG;
    if (nq <= 0) return B200F_OK;
    const bool l2 = metric == B200F_METRIC_L2;
    RankMergeParams p{};
    p.dist = dist;
    p.labels = labels;
    p.stride_d = stride_d;
    p.stride_l = stride_l;
    p.P = P;
    p.nq = nq;
    p.k = k;
    p.key_sign = l2 ? 1.f : -1.f;
    p.pad = l2 ? kHostInf : -kHostInf;
    p.out_dist = out_dist;
    p.out_labels = out_labels;
    const int T = P * k;
    int Tp = 64;
    while (Tp < T) Tp <<= 1;
    p.Tp = Tp;
    const int smem = Tp * 12;
    static bool attr_set[kMaxDevices] = {false};
    const int slot = device_slot();
    if (!attr_set[slot]) {
        B200F_CUDA_TRY(cudaFuncSetAttribute(rank_merge_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            8192 * 12));
        attr_set[slot] = true;
    }
    const int threads = T > 4096 ? 512 : T > 1024 ? 256 : 128;
    int64_t g = nq;
    const int64_t gcap = (int64_t)cached_sm_count() * (threads == 128 ? 16 : 8);
    if (g > gcap) g = gcap;
    rank_merge_kernel<<<(int)g, threads, smem, stream>>>(p);
    count_launch();
    B200F_LAUNCH_CHECK();
    return B200F_OK;
}

}  // namespace b200f

extern "C" int b200f_set_rank_select(int on) {
    b200f::g_rank_select.store(on ? 1 : 0, std::memory_order_relaxed);
    return B200F_OK;
}
