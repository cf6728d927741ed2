// Row-wise kernels: squared norms, append-time conversion, reconstruction,
// query preparation and the synthetic-data generator.
//
// Replaces l2_norm / l2_norm_large / l2_norm_f16 / l2_norm_f16_large
// (shaders/l2_norm.metal:7-66, shaders/l2_norm_f16.metal:10-67), their dispatch
// (src/MetalL2Norm.mm:42-89) and the host conversion loops of MetalIndexFlat::add
// (src/MetalIndexFlat.mm:224-255).  One warp owns one row; lanes read 128-bit
// vectors and reduce with shuffles.  Squares are formed in fp32 (the reference's
// "f16" norm kernels square in half precision, which is not reproduced).
#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "ptx.cuh"

namespace b200f {

namespace {

constexpr int ROW_THREADS = 256;  // 8 warps = 8 rows per CTA pass

__device__ __forceinline__ float bf16_bits_to_float(uint16_t b) {
    return __uint_as_float((uint32_t)b << 16);
}
// fp32 -> bf16 bits, round to nearest even (src/MetalIndexFlat.mm:231-234)
__device__ __forceinline__ uint16_t float_to_bf16_bits(float f) {
    return __bfloat16_as_ushort(__float2bfloat16_rn(f));
}
__device__ __forceinline__ uint16_t float_to_fp16_bits(float f) {
    return __half_as_ushort(__float2half_rn(f));
}
__device__ __forceinline__ float fp16_bits_to_float(uint16_t b) {
    return __half2float(__ushort_as_half(b));
}

template <int STORAGE>
__device__ __forceinline__ float load_elem(const void* rows, int64_t off) {
    if (STORAGE == B200F_STORAGE_F32) return reinterpret_cast<const float*>(rows)[off];
    uint16_t b = reinterpret_cast<const uint16_t*>(rows)[off];
    return STORAGE == B200F_STORAGE_F16 ? fp16_bits_to_float(b) : bf16_bits_to_float(b);
}

// ---- norms -----------------------------------------------------------------------------
template <int STORAGE>
__global__ void row_norms_kernel(const void* __restrict__ rows, int64_t n, int d, int64_t pitch,
                                 float* __restrict__ out) {
    const int lane = threadIdx.x & 31;
    const int64_t warps_total = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t r = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); r < n;
         r += warps_total) {
        float s = 0.f;
        if (STORAGE == B200F_STORAGE_F32) {
            const float* row = reinterpret_cast<const float*>(rows) + r * pitch;
            if ((pitch & 3) == 0 && ((uintptr_t)rows & 15) == 0) {
                const int d4 = d >> 2;
                const float4* row4 = reinterpret_cast<const float4*>(row);
                for (int j = lane; j < d4; j += 32) {
                    float4 v = __ldg(row4 + j);
                    s = fmaf(v.x, v.x, s);
                    s = fmaf(v.y, v.y, s);
                    s = fmaf(v.z, v.z, s);
                    s = fmaf(v.w, v.w, s);
                }
                for (int j = (d4 << 2) + lane; j < d; j += 32) s = fmaf(row[j], row[j], s);
            } else {
                for (int j = lane; j < d; j += 32) s = fmaf(row[j], row[j], s);
            }
        } else {
            const uint16_t* row = reinterpret_cast<const uint16_t*>(rows) + r * pitch;
            if ((pitch & 7) == 0 && ((uintptr_t)rows & 15) == 0) {
                const int d8 = d >> 3;
                const uint4* row8 = reinterpret_cast<const uint4*>(row);
                for (int j = lane; j < d8; j += 32) {
                    uint4 v = __ldg(row8 + j);
                    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                    for (int t = 0; t < 4; t++) {
                        float a, b;
                        if (STORAGE == B200F_STORAGE_F16) {
                            a = fp16_bits_to_float((uint16_t)(w[t] & 0xffffu));
                            b = fp16_bits_to_float((uint16_t)(w[t] >> 16));
                        } else {
                            a = __uint_as_float(w[t] << 16);
                            b = __uint_as_float(w[t] & 0xffff0000u);
                        }
                        s = fmaf(a, a, s);
                        s = fmaf(b, b, s);
                    }
                }
                for (int j = (d8 << 3) + lane; j < d; j += 32) {
                    float a = load_elem<STORAGE>(row, j);
                    s = fmaf(a, a, s);
                }
            } else {
                for (int j = lane; j < d; j += 32) {
                    float a = load_elem<STORAGE>(row, j);
                    s = fmaf(a, a, s);
                }
            }
        }
        s = warp_sum(s);
        if (lane == 0) out[r] = s;
    }
}

// ---- norm columns ------------------------------------------------------------------------
// The tensor path and the 16-bit scan get "||x||^2" out of the same dot product as q.x: a
// stored row carries 8 extra columns [d8, d8+8) holding -||x||^2/2 split into 16-bit pieces
// c_i, the query row carries the matching scales S_i there, so that
//     q_ext . x_ext = q.x - ||x||^2/2      (L2 key = -2 * that, + ||q||^2 at the end).
// bf16 has the exponent range of fp32: three pieces at scale 1.  fp16 does not: four
// pieces at scales 2^12, 2^1, 2^-10, 2^-21 (each an exact fp16 value) cover
// ||x||^2/2 up to 2.7e8 with at least 22 significant bits.
__device__ __forceinline__ float norm_scale(int storage, int slot) {
    if (storage == B200F_STORAGE_F16) {
        return slot == 0 ? 4096.f : slot == 1 ? 2.f : slot == 2 ? 9.765625e-4f : slot == 3 ? 4.76837158203125e-7f : 0.f;
    }
    return slot < 3 ? 1.f : 0.f;
}

// pieces of v for the 8 norm columns (16-bit patterns), format = fp16 or bf16
__device__ __forceinline__ void norm_pieces(float v, int storage, uint16_t (&out)[8]) {
    float r = v;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const float S = norm_scale(storage, i);
        uint16_t bits = 0;
        if (S != 0.f) {
            const float c = r / S;
            float back;
            if (storage == B200F_STORAGE_F16) {
                bits = float_to_fp16_bits(c);
                back = fp16_bits_to_float(bits);
            } else {
                bits = float_to_bf16_bits(c);
                back = bf16_bits_to_float(bits);
            }
            r = fmaf(-S, back, r);
        }
        out[i] = bits;
    }
}

// ---- append-time conversion -----------------------------------------------------------
// Writes the stored row (pad columns zeroed), the squared norm of
// the stored values, for fp32 storage the split planes, and (norm_cols) the
// 8 norm columns after the d8 = round_up(d, 8) data columns of the 16-bit row / plane 0.
// FP32 storage keeps, beside the fp32 rows, split planes for the tensor path, in one of two formats:
//   kPlanesBf16x3  x = b0 + b1 + b2, three bf16 planes (24 bits, fp32's exponent range): six plane
//                  products reproduce the fp32 product to 2^-24
//   kPlanesFp16x2  x * s = h0 + h1, two fp16 planes (22 bits) of the row scaled by a power of two s
//                  chosen for the index (largest element of a sample of its first rows near 2^6): three
//                  plane products, half the tensor work and two thirds of the plane bytes.  fp16 has a narrow exponent
//                  range, so the format only holds while every stored row fits it.  `range_flag` is
//                  raised, and the index takes another scale or re-splits itself into bf16x3, by
//                    an element at or beyond 2^15 after scaling;
//                    a row whose largest element falls below 2^-4 (1/1024 of the scale target: its
//                    low plane would go subnormal and lose bits);
//                    with norm columns, a row whose ||s x||^2 / 2 is beyond what their four pieces
//                    hold (kNormPiecesMax): the first would be -inf and the row's keys NaN, on no
//                    result list even for a query equal to it.  Long before the first bound: d = 128
//                    from elements of 2,100 on.
constexpr int kPlanesBf16x3 = 0;
constexpr int kPlanesFp16x2 = 1;
constexpr float kNormPiecesMax = 4096.f * 65504.f;   // largest scale times the largest fp16 value

// V consecutive elements of a row per lane and access: 4 (or 8, load_rows_kernel) where the row
// length and every pitch and base allow it, else 2 or 1.
template <int V>
struct alignas(V * 4) FloatVec {
    float v[V];
};
template <int V>
struct alignas(V * 2) HalfVec {
    uint16_t v[V];
};
template <int V>
__device__ __forceinline__ void store_bits(uint16_t* p, const uint16_t (&b)[V]) {
    HalfVec<V> h;
#pragma unroll
    for (int e = 0; e < V; e++) h.v[e] = b[e];
    *reinterpret_cast<HalfVec<V>*>(p) = h;
}

// HBM-bound: 4 d bytes read and (fp32 rows, two fp16 planes) 8 d written per row.  A row belongs to
// lpr lanes of a warp, as many as leave each lane up to U vectors of it: they are loaded together, the row
// is read ONCE, and squares, conversions and the plane split all come from the same registers.
// 1,000,003 rows of d = 384, fp32 with fp16 planes: 720 us (6.5 TB/s); element by element with a second
// read of the row for the planes it took 940 us.  One vector per lane (a whole warp on a row of 128) kept
// too few loads in flight and a single lane busy with the norm pieces: add() of 1 GiB to an fp16 index of
// d = 128 took 0.63 ms (element by element 0.50), now 0.29 ms (5.7 TB/s read and written).
template <int STORAGE, int V>
__global__ void __launch_bounds__(ROW_THREADS)
store_rows_kernel(const float* __restrict__ src, int64_t src_pitch, int64_t n, int d, int lpr,
                  void* __restrict__ dst, int64_t dst_pitch, uint16_t* __restrict__ planes, int64_t plane_pitch,
                  int64_t plane_stride, int plane_format, float plane_scale, int32_t* __restrict__ range_flag,
                  float* __restrict__ norms, int norm_cols) {
    constexpr int U = V == 4 ? 4 : 8;
    const int lane = threadIdx.x & 31;
    const int sub = lane / lpr, cl = lane & (lpr - 1);
    const int d8 = (d + 7) & ~7;
    const int64_t rows_per_step = 32 / lpr;
    const int64_t warps_total = (int64_t)gridDim.x * (blockDim.x >> 5);
    // columns written: the stored row and the plane rows, pads included
    const int64_t width = (planes && plane_pitch > dst_pitch) ? plane_pitch : dst_pitch;
    for (int64_t r0 = ((int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * rows_per_step; r0 < n;
         r0 += warps_total * rows_per_step) {
        const int64_t r = r0 + sub;
        const bool live = r < n;
        const float* row = src + r * src_pitch;
        float* const outf = reinterpret_cast<float*>(dst) + r * dst_pitch;
        uint16_t* const outh = reinterpret_cast<uint16_t*>(dst) + r * dst_pitch;
        uint16_t* const p0 = planes + r * plane_pitch;
        const bool copy_row = STORAGE != B200F_STORAGE_F32 || outf != row;   // a re-split reads the stored rows themselves
        float s = 0.f, amax = 0.f;
        for (int64_t base = 0; base < d; base += (int64_t)lpr * V * U) {
            FloatVec<V> x[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int64_t j = base + ((int64_t)u * lpr + cl) * V;
#pragma unroll
                for (int e = 0; e < V; e++) x[u].v[e] = 0.f;
                if (live && j < d) x[u] = *reinterpret_cast<const FloatVec<V>*>(row + j);
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int64_t j = base + ((int64_t)u * lpr + cl) * V;
                if (!live || j >= d) continue;
                if (STORAGE == B200F_STORAGE_F32) {
#pragma unroll
                    for (int e = 0; e < V; e++) s = fmaf(x[u].v[e], x[u].v[e], s);
                    if (copy_row) *reinterpret_cast<FloatVec<V>*>(outf + j) = x[u];
                    if (!planes) continue;
                    uint16_t h0[V], h1[V], h2[V];
                    if (plane_format == kPlanesFp16x2) {
#pragma unroll
                        for (int e = 0; e < V; e++) {
                            const float v = x[u].v[e] * plane_scale;
                            amax = fmaxf(amax, fabsf(v));
                            h0[e] = float_to_fp16_bits(v);
                            h1[e] = float_to_fp16_bits(v - fp16_bits_to_float(h0[e]));   // the difference is exact
                        }
                    } else {
#pragma unroll
                        for (int e = 0; e < V; e++) {
                            h0[e] = float_to_bf16_bits(x[u].v[e]);
                            const float r1 = x[u].v[e] - bf16_bits_to_float(h0[e]);
                            h1[e] = float_to_bf16_bits(r1);
                            h2[e] = float_to_bf16_bits(r1 - bf16_bits_to_float(h1[e]));
                        }
                        store_bits<V>(p0 + 2 * plane_stride + j, h2);
                    }
                    store_bits<V>(p0 + j, h0);
                    store_bits<V>(p0 + plane_stride + j, h1);
                } else {
                    uint16_t h[V];
#pragma unroll
                    for (int e = 0; e < V; e++) {
                        float back;
                        if (STORAGE == B200F_STORAGE_F16) {
                            h[e] = float_to_fp16_bits(x[u].v[e]);
                            back = fp16_bits_to_float(h[e]);
                        } else {
                            h[e] = float_to_bf16_bits(x[u].v[e]);
                            back = bf16_bits_to_float(h[e]);
                        }
                        s = fmaf(back, back, s);
                    }
                    store_bits<V>(outh + j, h);
                }
            }
        }
        // pads behind the row's elements (a few columns), except the norm columns, which are written below
        for (int64_t j = d + (int64_t)cl * V; live && j < width; j += (int64_t)lpr * V) {
            const uint16_t z[V] = {};
            const bool ncol = norm_cols && j >= d8 && j < d8 + 8;
            if (STORAGE == B200F_STORAGE_F32) {
                if (copy_row && j < dst_pitch) *reinterpret_cast<FloatVec<V>*>(outf + j) = FloatVec<V>{};
                if (!planes || j >= plane_pitch) continue;
                if (!ncol) store_bits<V>(p0 + j, z);
                store_bits<V>(p0 + plane_stride + j, z);
                if (plane_format != kPlanesFp16x2) store_bits<V>(p0 + 2 * plane_stride + j, z);
            } else if (!ncol) {
                store_bits<V>(outh + j, z);
            }
        }
        for (int o = lpr >> 1; o > 0; o >>= 1) {
            s += __shfl_xor_sync(0xffffffffu, s, o);
            amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
        }
        if (!live || cl != 0) continue;
        if (range_flag && planes && plane_format == kPlanesFp16x2) {
            if (amax > 0.f && amax < 0.0625f) atomicOr(range_flag, 3);
            else if (amax >= 32768.f || (norm_cols && 0.5f * s * plane_scale * plane_scale > kNormPiecesMax))
                atomicOr(range_flag, 1);
        }
        if (norms) norms[r] = s;
        if (norm_cols) {
            uint16_t pc[8];
            if (STORAGE == B200F_STORAGE_F32 && plane_format == kPlanesFp16x2)
                // in the scaled units of the planes: (s x).(s x) / 2, fp16 pieces
                norm_pieces(-0.5f * s * plane_scale * plane_scale, B200F_STORAGE_F16, pc);
            else
                norm_pieces(-0.5f * s, STORAGE == B200F_STORAGE_F32 ? B200F_STORAGE_BF16 : STORAGE, pc);
            uint16_t* o = (STORAGE == B200F_STORAGE_F32) ? (planes ? p0 + d8 : nullptr) : outh + d8;
            if (o && (reinterpret_cast<uintptr_t>(o) & 15) == 0) {
                store_bits<8>(o, pc);
            } else if (o) {
#pragma unroll
                for (int i = 0; i < 8; i++) o[i] = pc[i];
            }
        }
    }
}

// Largest |element| of a block of fp32 rows (as the bit pattern of a non-negative float, which
// orders like an unsigned integer): what the index derives the fp16x2 plane scale from.
__global__ void rows_absmax_kernel(const float* __restrict__ src, int64_t pitch, int64_t n, int d,
                                   uint32_t* __restrict__ out_max_bits) {
    const int lane = threadIdx.x & 31;
    const int64_t warps_total = (int64_t)gridDim.x * (blockDim.x >> 5);
    float amax = 0.f;
    for (int64_t r = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); r < n; r += warps_total) {
        const float* row = src + r * pitch;
        for (int j = lane; j < d; j += 32) {
            const float v = fabsf(row[j]);
            if (v < CUDART_INF_F) amax = fmaxf(amax, v);   // NaN and INF do not set the scale
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    if (lane == 0 && amax > 0.f) atomicMax(out_max_bits, __float_as_uint(amax));
}

// Stored rows back to fp32, HBM-bound; lanes and vectors as in store_rows_kernel (fp32, 1,000,003 rows
// of d = 384: 480 us, 6.4 TB/s; one element per thread with a 64-bit division each: 935 us).
template <int STORAGE, int V>
__global__ void __launch_bounds__(ROW_THREADS)
load_rows_kernel(const void* __restrict__ rows, int64_t n, int d, int lpr, int64_t pitch, float* __restrict__ dst) {
    constexpr int U = 4;
    const int lane = threadIdx.x & 31;
    const int sub = lane / lpr, cl = lane & (lpr - 1);
    const int64_t rows_per_step = 32 / lpr;
    const int64_t warps_total = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t r0 = ((int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * rows_per_step; r0 < n;
         r0 += warps_total * rows_per_step) {
        const int64_t r = r0 + sub;
        if (r >= n) continue;
        float* const out = dst + r * (int64_t)d;
        for (int base = 0; base < d; base += lpr * V * U) {
            if constexpr (STORAGE == B200F_STORAGE_F32) {
                const float* row = reinterpret_cast<const float*>(rows) + r * pitch;
                FloatVec<V> x[U];
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const int j = base + (u * lpr + cl) * V;
                    if (j < d) x[u] = *reinterpret_cast<const FloatVec<V>*>(row + j);
                }
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const int j = base + (u * lpr + cl) * V;
                    if (j < d) *reinterpret_cast<FloatVec<V>*>(out + j) = x[u];
                }
            } else {
                const uint16_t* row = reinterpret_cast<const uint16_t*>(rows) + r * pitch;
                HalfVec<V> h[U];
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const int j = base + (u * lpr + cl) * V;
                    if (j < d) h[u] = *reinterpret_cast<const HalfVec<V>*>(row + j);
                }
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const int j = base + (u * lpr + cl) * V;
                    if (j >= d) continue;
                    FloatVec<V> x;
#pragma unroll
                    for (int e = 0; e < V; e++)
                        x.v[e] = STORAGE == B200F_STORAGE_F16 ? fp16_bits_to_float(h[u].v[e]) : bf16_bits_to_float(h[u].v[e]);
                    *reinterpret_cast<FloatVec<V>*>(out + j) = x;
                }
            }
        }
    }
}

// ---- query preparation -------------------------------------------------------------------
// fp32 queries -> operand planes of the tensor path (+ exact fp32 squared norms).
// One plane in the storage format (fp16 / bf16) or three bf16 split planes (fp32 storage).
// With norm_cols the 8 columns after d8 of plane 0 receive the norm scales (see above).
// A warp takes a row, or (WIDE) a whole CTA: a warp's chain of loads and conversions over a row of 770 took 18 us
// for 24 queries, whose launch every search waits for (now under 5).
template <bool WIDE>
__global__ void __launch_bounds__(ROW_THREADS) prepare_queries_kernel(const float* __restrict__ q, int64_t nq, int d, int storage,
                                       uint16_t* __restrict__ a, int64_t a_pitch,
                                       int64_t a_plane_stride, float* __restrict__ qnorm,
                                       int norm_cols, int plane_format, int x_scale_log2,
                                       float* __restrict__ rowscale, const SearchInit init) {
    pdl_trigger();   // never launched programmatically itself: everything before it has completed
    if (blockIdx.x == 0) {
        if (init.status && threadIdx.x < 4) init.status[threadIdx.x] = 0;
        if (init.count && threadIdx.x < 2) init.count[16 * threadIdx.x] = 0;
    }
    __shared__ float s_part[2][ROW_THREADS / 32];
    const int lane = WIDE ? threadIdx.x : threadIdx.x & 31;   // position among the threads of a row
    constexpr int LANES = WIDE ? ROW_THREADS : 32;
    const int d8 = (d + 7) & ~7;
    const int fmt = storage == B200F_STORAGE_F16 ? B200F_STORAGE_F16 : B200F_STORAGE_BF16;
    const bool fp16x2 = storage == B200F_STORAGE_F32 && plane_format == kPlanesFp16x2;
    const int64_t teams = (int64_t)gridDim.x * (ROW_THREADS / LANES);
    for (int64_t r = (int64_t)blockIdx.x * (ROW_THREADS / LANES) + (WIDE ? 0 : threadIdx.x >> 5); r < nq; r += teams) {
        const float* row = q + r * (int64_t)d;
        if (init.cand_cnt && lane == 0) init.cand_cnt[r] = 0;
        if (init.gthr)
            for (int j = lane; j < init.gslots; j += LANES) init.gthr[r * init.gslots + j] = 0xffffffffu;
        // fp16x2 planes: every query row gets its own power-of-two scale (largest element near
        // 2^6, as the stored rows), kept at most 2^3 above the rows' scale so that the norm-column
        // scales below stay inside fp16.  The kernel's accumulator is then (sq * sx) * t, and
        // rowscale[r] = 1 / (sq * sx) brings a key back to its units.
        float sq = 1.f, ratio = 1.f;
        if (fp16x2 && a) {
            float amax = 0.f;
            for (int j = lane; j < d; j += LANES) {
                const float v = fabsf(row[j]);
                if (v < CUDART_INF_F) amax = fmaxf(amax, v);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
            if (WIDE) {
                if ((threadIdx.x & 31) == 0) s_part[0][threadIdx.x >> 5] = amax;
                __syncthreads();
                for (int w = 0; w < ROW_THREADS / 32; w++) amax = fmaxf(amax, s_part[0][w]);
            }
            int e = 0;
            if (amax > 0.f) (void)frexpf(amax, &e);   // amax = m * 2^e, m in [0.5, 1)
            int lq = amax > 0.f ? 7 - e : x_scale_log2;
            if (lq > x_scale_log2 + 3) lq = x_scale_log2 + 3;
            if (lq > 126) lq = 126;
            if (lq < -126) lq = -126;
            sq = ldexpf(1.f, lq);
            ratio = ldexpf(1.f, lq - x_scale_log2);            // sq / sx
            if (rowscale && lane == 0) rowscale[r] = ldexpf(1.f, -(lq + x_scale_log2));
        }
        float s = 0.f;
        for (int j = lane; j < a_pitch || j < d; j += LANES) {
            float v = (j < d) ? row[j] : 0.f;
            s = fmaf(v, v, s);
            if (a && j < a_pitch) {
                uint16_t* p0 = a + r * a_pitch + j;
                const bool ncol = norm_cols && j >= d8 && j < d8 + 8;
                if (fp16x2) {
                    // norm columns: the stored side holds (sx x).(sx x) / 2 in fp16 pieces
                    const float w = ncol ? norm_scale(B200F_STORAGE_F16, j - d8) * ratio : v * sq;
                    const uint16_t h0 = float_to_fp16_bits(w);
                    p0[0] = h0;
                    p0[a_plane_stride] = ncol ? (uint16_t)0 : float_to_fp16_bits(w - fp16_bits_to_float(h0));
                    continue;
                }
                if (ncol) v = norm_scale(fmt, j - d8);
                if (storage == B200F_STORAGE_F16) {
                    *p0 = float_to_fp16_bits(v);
                } else if (storage == B200F_STORAGE_BF16) {
                    *p0 = float_to_bf16_bits(v);
                } else {
                    uint16_t b0 = float_to_bf16_bits(v);
                    float r1 = v - bf16_bits_to_float(b0);
                    uint16_t b1 = float_to_bf16_bits(r1);
                    float r2 = r1 - bf16_bits_to_float(b1);
                    p0[0] = b0;
                    p0[a_plane_stride] = b1;
                    p0[2 * a_plane_stride] = float_to_bf16_bits(r2);
                }
            }
        }
        if (qnorm) {
            s = warp_sum(s);
            if (WIDE) {
                if ((threadIdx.x & 31) == 0) s_part[1][threadIdx.x >> 5] = s;
                __syncthreads();
                s = 0.f;
                for (int w = 0; w < ROW_THREADS / 32; w++) s += s_part[1][w];
            }
            if (lane == 0) qnorm[r] = s;
        }
        if (WIDE) __syncthreads();   // the shared partials are rewritten by the next row
    }
}

// ---- synthetic generator -------------------------------------------------------------------
__device__ __forceinline__ uint64_t mix64(uint64_t z) {
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ULL;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebULL;
    return z ^ (z >> 31);
}

__device__ __forceinline__ float synth_value(uint64_t seed, int64_t row, int col, int dist) {
    uint64_t h = mix64(seed * 0x9e3779b97f4a7c15ULL + (uint64_t)row * 0xd1342543de82ef95ULL +
                       (uint64_t)col + 1);
    h = mix64(h);
    const float u1 = ((uint32_t)(h >> 40) + 0.5f) * (1.0f / 16777216.0f);  // (0,1)
    if (dist == 0) return ((uint32_t)(h >> 40)) * (1.0f / 16777216.0f);   // [0,1)
    const float u2 = ((uint32_t)(h & 0xffffffu)) * (1.0f / 16777216.0f);
    return sqrtf(-2.f * logf(u1)) * cospif(2.f * u2);
}

__global__ void fill_synthetic_kernel(float* __restrict__ dst, int64_t n, int d, int64_t row0,
                                      uint64_t seed, int dist, float scale) {
    const int lane = threadIdx.x & 31;
    const int64_t warps_total = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t r = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); r < n;
         r += warps_total) {
        float* row = dst + r * (int64_t)d;
        if (dist == 2) {
            float s = 0.f;
            for (int j = lane; j < d; j += 32) {
                float v = synth_value(seed, row0 + r, j, 1);
                s = fmaf(v, v, s);
            }
            s = warp_sum(s);
            const float inv = s > 0.f ? rsqrtf(s) : 0.f;
            for (int j = lane; j < d; j += 32) row[j] = synth_value(seed, row0 + r, j, 1) * inv;
        } else if (dist == 3) {
            // mixture of 1,000 gaussians: the centres (uniform in [-1,1]^d) are the same for
            // every seed, so that rows and queries of different seeds share them
            const uint64_t c = mix64(seed * 0x9e3779b97f4a7c15ULL + (uint64_t)(row0 + r) * 0xd1342543de82ef95ULL) % 1000u;
            for (int j = lane; j < d; j += 32)
                row[j] = 2.f * synth_value(0x6d697874ULL, (int64_t)c, j, 0) - 1.f +
                         scale * synth_value(seed, row0 + r, j, 1);
        } else {
            for (int j = lane; j < d; j += 32)
                row[j] = synth_value(seed, row0 + r, j, dist) * (dist == 1 ? scale : 1.f);
        }
    }
}

// Lanes that share a row of d elements read V at a time.
int lanes_for_row(int d, int v) {
    int lpr = 1;
    while (lpr < 32 && lpr * v < d) lpr <<= 1;
    return lpr;
}

// True when every offset (in elements) and the base (in elements of `bytes` bytes) are multiples of v.
bool vec_ok(const void* base, int bytes, int v, int64_t a, int64_t b = 0) {
    return (reinterpret_cast<uintptr_t>(base) % (size_t)(bytes * v)) == 0 && a % v == 0 && b % v == 0;
}

int grid_for_rows(int64_t n) {
    int64_t g = ceil_div64(n, ROW_THREADS / 32);
    int64_t cap = (int64_t)cached_sm_count() * 16;
    if (g > cap) g = cap;
    if (g < 1) g = 1;
    return (int)g;
}

}  // namespace

int device_slot() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        (void)cudaGetLastError();
        return 0;
    }
    return (dev >= 0 && dev < kMaxDevices) ? dev : kMaxDevices - 1;
}

// SM count of the CURRENT device (a process may drive several GPUs: one value per device).
int cached_sm_count() {
    static int sm[kMaxDevices] = {0};
    const int slot = device_slot();
    if (sm[slot] == 0) {
        int dev = 0, n = 0;
        if (cudaGetDevice(&dev) != cudaSuccess ||
            cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) {
            (void)cudaGetLastError();
            return kNumSMsDefault;
        }
        sm[slot] = n;
    }
    return sm[slot];
}

int launch_prepare_queries(const float* q, int64_t nq, int d, int storage, uint16_t* a_planes,
                           int64_t a_pitch, int64_t a_plane_stride, float* qnorm, int norm_cols,
                           int plane_format, int x_scale_log2, float* rowscale, const SearchInit& init,
                           cudaStream_t stream) {
    if (nq <= 0) return B200F_OK;
    // a CTA per row while that leaves no SM with more than a few
    const bool wide = d >= 128 && nq <= 8 * (int64_t)cached_sm_count();
    auto* kernel = wide ? prepare_queries_kernel<true> : prepare_queries_kernel<false>;
    kernel<<<wide ? (int)nq : grid_for_rows(nq), ROW_THREADS, 0, stream>>>(
            q, nq, d, storage, a_planes, a_pitch, a_plane_stride, qnorm, norm_cols, plane_format, x_scale_log2,
            rowscale, init);
    count_launch();
    B200F_LAUNCH_CHECK();
    return B200F_OK;
}

}  // namespace b200f

using namespace b200f;

extern "C" int b200f_row_norms(const void* rows, int storage, int64_t n, int d, int64_t pitch_elems,
                               float* out, void* stream) {
    if (n < 0 || d <= 0 || pitch_elems < d || (n > 0 && (!rows || !out))) return B200F_ERR_BAD_ARG;
    if (n == 0) return B200F_OK;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int g = grid_for_rows(n);
    switch (storage) {
        case B200F_STORAGE_F32:
            row_norms_kernel<B200F_STORAGE_F32><<<g, ROW_THREADS, 0, st>>>(rows, n, d, pitch_elems, out);
            break;
        case B200F_STORAGE_F16:
            row_norms_kernel<B200F_STORAGE_F16><<<g, ROW_THREADS, 0, st>>>(rows, n, d, pitch_elems, out);
            break;
        case B200F_STORAGE_BF16:
            row_norms_kernel<B200F_STORAGE_BF16><<<g, ROW_THREADS, 0, st>>>(rows, n, d, pitch_elems, out);
            break;
        default:
            return B200F_ERR_BAD_ARG;
    }
    count_launch();
    B200F_LAUNCH_CHECK();
    return B200F_OK;
}

namespace {
int store_rows_impl(const float* src, int64_t src_pitch, int64_t n, int d, int storage, void* dst_rows,
                    int64_t dst_pitch, uint16_t* planes, int64_t plane_pitch, int64_t plane_stride,
                    int plane_format, int plane_scale_log2, int32_t* range_flag, float* norms_or_null,
                    int norm_cols, void* stream) {
    if (n < 0 || d <= 0 || dst_pitch < d || src_pitch < d || (n > 0 && (!src || !dst_rows))) return B200F_ERR_BAD_ARG;
    if (planes && (plane_pitch < d || plane_stride < plane_pitch)) return B200F_ERR_BAD_ARG;
    if (plane_format != B200F_PLANES_BF16X3 && plane_format != B200F_PLANES_FP16X2) return B200F_ERR_BAD_ARG;
    if (plane_scale_log2 < -126 || plane_scale_log2 > 126) return B200F_ERR_BAD_ARG;
    if (norm_cols) {
        const int64_t need = ((d + 7) & ~7) + 8;
        if (storage == B200F_STORAGE_F32 ? (planes && plane_pitch < need) : dst_pitch < need)
            return B200F_ERR_BAD_ARG;
    }
    if (n == 0) return B200F_OK;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const float scale = std::ldexp(1.f, plane_scale_log2);
    const bool fp32 = storage == B200F_STORAGE_F32;
    if (!fp32) {
        planes = nullptr;
        plane_pitch = plane_stride = 0;
    }
    int v = 4;
    while (v > 1 && !(d % v == 0 && vec_ok(src, 4, v, src_pitch) && vec_ok(dst_rows, fp32 ? 4 : 2, v, dst_pitch) &&
                      (!planes || vec_ok(planes, 2, v, plane_pitch, plane_stride))))
        v >>= 1;
    // four vectors per lane, at least four lanes on rows that have as many (whole 32-byte sectors of
    // 16-bit elements per store)
    const int lpr = v == 4 ? std::max(lanes_for_row(d, 16), std::min(4, lanes_for_row(d, 4))) : lanes_for_row(d, 2 * v);
    const int g = grid_for_rows(ceil_div64(n, 32 / lpr));
    // macro: the kernel is a template over (storage, elements per access)
#define B200F_STORE_ROWS(ST, V)                                                                          \
    store_rows_kernel<ST, V><<<g, ROW_THREADS, 0, st>>>(src, src_pitch, n, d, lpr, dst_rows, dst_pitch,   \
                                                        planes, plane_pitch, plane_stride, plane_format, \
                                                        scale, range_flag, norms_or_null, norm_cols)
#define B200F_STORE_ROWS_V(ST)                    \
    do {                                          \
        if (v == 4) B200F_STORE_ROWS(ST, 4);      \
        else if (v == 2) B200F_STORE_ROWS(ST, 2); \
        else B200F_STORE_ROWS(ST, 1);             \
    } while (0)
    switch (storage) {
        case B200F_STORAGE_F32: B200F_STORE_ROWS_V(B200F_STORAGE_F32); break;
        case B200F_STORAGE_F16: B200F_STORE_ROWS_V(B200F_STORAGE_F16); break;
        case B200F_STORAGE_BF16: B200F_STORE_ROWS_V(B200F_STORAGE_BF16); break;
        default: return B200F_ERR_BAD_ARG;
    }
#undef B200F_STORE_ROWS_V
#undef B200F_STORE_ROWS
    count_launch();
    B200F_LAUNCH_CHECK();
    return B200F_OK;
}
}  // namespace

extern "C" int b200f_store_rows(const float* src, int64_t n, int d, int storage, void* dst_rows,
                                int64_t dst_pitch, uint16_t* planes, int64_t plane_pitch,
                                int64_t plane_stride, float* norms_or_null, int norm_cols,
                                void* stream) {
    return store_rows_impl(src, d, n, d, storage, dst_rows, dst_pitch, planes, plane_pitch, plane_stride,
                           B200F_PLANES_BF16X3, 0, nullptr, norms_or_null, norm_cols, stream);
}

extern "C" int b200f_store_rows_fp32(const float* src, int64_t src_pitch, int64_t n, int d, float* dst_rows,
                                     int64_t dst_pitch, uint16_t* planes, int64_t plane_pitch,
                                     int64_t plane_stride, int plane_format, int plane_scale_log2,
                                     int32_t* range_flag, float* norms_or_null, int norm_cols, void* stream) {
    return store_rows_impl(src, src_pitch, n, d, B200F_STORAGE_F32, dst_rows, dst_pitch, planes, plane_pitch,
                           plane_stride, plane_format, plane_scale_log2, range_flag, norms_or_null, norm_cols, stream);
}

extern "C" int b200f_rows_absmax(const float* rows, int64_t n, int d, int64_t pitch_elems, uint32_t* max_bits,
                                 void* stream) {
    if (n < 0 || d <= 0 || pitch_elems < d || !max_bits || (n > 0 && !rows)) return B200F_ERR_BAD_ARG;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    B200F_CUDA_TRY(cudaMemsetAsync(max_bits, 0, sizeof(uint32_t), st));
    if (n == 0) return B200F_OK;
    rows_absmax_kernel<<<grid_for_rows(n), ROW_THREADS, 0, st>>>(rows, pitch_elems, n, d, max_bits);
    count_launch();
    B200F_LAUNCH_CHECK();
    return B200F_OK;
}

extern "C" int b200f_load_rows(const void* rows, int storage, int64_t n, int d, int64_t pitch_elems,
                               float* dst, void* stream) {
    if (n < 0 || d <= 0 || pitch_elems < d || (n > 0 && (!rows || !dst))) return B200F_ERR_BAD_ARG;
    if (n == 0) return B200F_OK;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const bool fp32 = storage == B200F_STORAGE_F32;
    int v = fp32 ? 4 : 8;
    while (v > 1 && !(d % v == 0 && vec_ok(rows, fp32 ? 4 : 2, v, pitch_elems) && vec_ok(dst, 4, v, 0))) v >>= 1;
    const int lpr = lanes_for_row(d, v);
    const int g = grid_for_rows(ceil_div64(n, 32 / lpr));
#define B200F_LOAD_ROWS(ST, V) load_rows_kernel<ST, V><<<g, ROW_THREADS, 0, st>>>(rows, n, d, lpr, pitch_elems, dst)
    switch (storage) {
        case B200F_STORAGE_F32:
            if (v == 4) B200F_LOAD_ROWS(B200F_STORAGE_F32, 4);
            else if (v == 2) B200F_LOAD_ROWS(B200F_STORAGE_F32, 2);
            else B200F_LOAD_ROWS(B200F_STORAGE_F32, 1);
            break;
        case B200F_STORAGE_F16:
            if (v == 8) B200F_LOAD_ROWS(B200F_STORAGE_F16, 8);
            else if (v >= 2) B200F_LOAD_ROWS(B200F_STORAGE_F16, 2);
            else B200F_LOAD_ROWS(B200F_STORAGE_F16, 1);
            break;
        case B200F_STORAGE_BF16:
            if (v == 8) B200F_LOAD_ROWS(B200F_STORAGE_BF16, 8);
            else if (v >= 2) B200F_LOAD_ROWS(B200F_STORAGE_BF16, 2);
            else B200F_LOAD_ROWS(B200F_STORAGE_BF16, 1);
            break;
        default:
            return B200F_ERR_BAD_ARG;
    }
#undef B200F_LOAD_ROWS
    count_launch();
    B200F_LAUNCH_CHECK();
    return B200F_OK;
}

extern "C" int b200f_fill_synthetic(float* dst, int64_t n, int d, int64_t row0, uint64_t seed,
                                    int dist, float scale, void* stream) {
    if (n < 0 || d <= 0 || dist < 0 || dist > 3 || (n > 0 && !dst)) return B200F_ERR_BAD_ARG;
    if (n == 0) return B200F_OK;
    fill_synthetic_kernel<<<grid_for_rows(n), ROW_THREADS, 0, static_cast<cudaStream_t>(stream)>>>(
            dst, n, d, row0, seed, dist, scale);
    count_launch();
    B200F_LAUNCH_CHECK();
    return B200F_OK;
}
