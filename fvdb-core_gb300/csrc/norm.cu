// Group normalisation of jagged voxel features, forward and backward (fvdb.nn.GroupNorm,
// reference fvdb/nn/modules.py:408-432): each (grid, channel group) is normalised over its voxels
// and the group's channels.
//
//   forward   chunk statistics -> (grid, group) mean and 1/sqrt(var + eps) -> y = (x - mean) r w + b
//   backward  chunk sums of dy and dy xhat per channel -> per (grid, channel) -> per (grid, group)
//             -> dx = r (dy w - A1 - xhat A2);  dw = sum dy xhat, db = sum dy
//
// Bound by HBM: forward reads x twice and writes y, backward reads x and dy twice and writes dx.
// 1.31M voxels x 64 channels in four grids, BF16, forward and backward together (GB300): 184 ms as
// torch segment sums (their backward adds every row into one of four gradient rows), 0.37 ms here:
// statistics 61 us, normalisation 48, gradient sums 66, dx 69, the merges 31.
//
// A CTA owns a chunk of consecutive rows; every thread keeps one vector column (V channels of one
// group) and kRowsPerThread rows of it in registers, so the chunk's variance is taken about the
// chunk's own mean from registers, without a second read.  Rows of several grids in a chunk are
// handled one segment at a time.  Segment s of the (chunk, grid) pairs is stored at slot
// chunk + grid: both indices only grow from row to row, so no two pairs share a slot.  Chunks are
// merged in FP64 in a fixed order (pairwise mean / M2 update): results are reproducible.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <type_traits>

#include "common.cuh"

namespace fvgb {
namespace {

constexpr int kNT = 256;
constexpr int kRowsPerThread = 8;  // forward: one operand
constexpr int kRowsBackward = 4;   // backward: two operands in as many registers
constexpr int kSumIters = 4;       // row groups a CTA adds up before it folds its thread rows

template <typename T>
struct NNum;
template <>
struct NNum<float> {
    using A = float;
    __device__ static float to(float v) { return v; }
    __device__ static float from(float v) { return v; }
};
template <>
struct NNum<double> {
    using A = double;
    __device__ static double to(double v) { return v; }
    __device__ static double from(double v) { return v; }
};
template <>
struct NNum<__nv_bfloat16> {
    using A = float;
    __device__ static float to(__nv_bfloat16 v) { return __bfloat162float(v); }
    __device__ static __nv_bfloat16 from(float v) { return __float2bfloat16_rn(v); }
};
template <>
struct NNum<__half> {
    using A = float;
    __device__ static float to(__half v) { return __half2float(v); }
    __device__ static __half from(float v) { return __float2half_rn(v); }
};

struct NormArgs {
    const int64_t *joff;  // [B + 1]
    int32_t B;
    int64_t n;
    int32_t C, G, cpg;  // channels, groups, channels per group
    int32_t Q, QB;      // vector columns per row; columns per CTA (blockIdx.y slabs)
    int32_t rpi;        // rows a CTA covers per thread row (kNT / QB)
    int64_t chunk_rows; // rpi * kRowsPerThread
};

// Rows [lo, hi) of grid b, clamped to [0, n].
__device__ __forceinline__ void grid_rows(const NormArgs &a, int32_t b, int64_t &lo, int64_t &hi) {
    lo = min(max(a.joff[b], (int64_t)0), a.n);
    hi = min(max(a.joff[b + 1], lo), a.n);
}

// Sum over the thread rows rr of the CTA for each column qq, returned by every thread of the column.
// sm: kNT entries.  Columns that divide a warp fold its thread rows by shuffles first.
template <typename A>
__device__ __forceinline__ A column_sum(A v, A *sm, int rr, int qq, int QB, int rpi, int half) {
    __syncthreads();
    if (QB <= 32 && (QB & (QB - 1)) == 0) {
        for (int o = QB; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        const int lane = threadIdx.x & 31;
        if (lane < QB) sm[(threadIdx.x >> 5) * QB + lane] = v;
        __syncthreads();
        A t = 0;
#pragma unroll
        for (int w = 0; w < kNT / 32; ++w) t += sm[w * QB + qq];
        return t;
    }
    if (rr < rpi) sm[rr * QB + qq] = v;
    for (int s = half; s > 0; s >>= 1) {
        __syncthreads();
        if (rr < s && rr + s < rpi) sm[rr * QB + qq] += sm[(rr + s) * QB + qq];
    }
    __syncthreads();
    return sm[qq];
}

// stat[slot][q] = {mean, M2} of the slot's rows in vector column q
template <typename T, int V>
__global__ void __launch_bounds__(kNT, 4) gn_stats_kernel(NormArgs a, const T *__restrict__ x,
                                                       typename NNum<T>::A *__restrict__ stat) {
    using A = typename NNum<T>::A;
    __shared__ A sm[kNT];
    const int tid = threadIdx.x, qq = tid % a.QB, rr = tid / a.QB;
    const int q = blockIdx.y * a.QB + qq;
    const bool col = rr < a.rpi && q < a.Q;
    int half = 1;
    while (half * 2 < a.rpi) half *= 2;
    const int64_t r0 = (int64_t)blockIdx.x * a.chunk_rows, r1 = min(a.n, r0 + a.chunk_rows);
    const int32_t b0 = batch_of_warp(a.joff, a.B, r0), b1 = batch_of_warp(a.joff, a.B, r1 - 1);
    Raw<T, V> p[kRowsPerThread];
#pragma unroll
    for (int i = 0; i < kRowsPerThread; ++i) {
        const int64_t r = r0 + rr + (int64_t)i * a.rpi;
        if (col && r < r1) p[i] = ld_raw<T, V>(x + r * a.C + (int64_t)q * V);
    }
    for (int32_t b = b0; b <= b1; ++b) {
        int64_t lo, hi;
        grid_rows(a, b, lo, hi);
        lo = max(lo, r0);
        hi = min(hi, r1);
        if (lo >= hi) continue;  // the same for every thread
        A s = 0;
#pragma unroll
        for (int i = 0; i < kRowsPerThread; ++i) {
            const int64_t r = r0 + rr + (int64_t)i * a.rpi;
            if (col && r >= lo && r < hi) {
                const Elems<T, V> x_ = unpack<T, V>(p[i]);
#pragma unroll
                for (int e = 0; e < V; ++e) s += NNum<T>::to(x_.v[e]);
            }
        }
        const A mean = column_sum<A>(s, sm, rr, qq, a.QB, a.rpi, half) / (A)((hi - lo) * V);
        A m2 = 0;
#pragma unroll
        for (int i = 0; i < kRowsPerThread; ++i) {
            const int64_t r = r0 + rr + (int64_t)i * a.rpi;
            if (col && r >= lo && r < hi) {
                const Elems<T, V> x_ = unpack<T, V>(p[i]);
#pragma unroll
                for (int e = 0; e < V; ++e) {
                    const A d = NNum<T>::to(x_.v[e]) - mean;
                    m2 += d * d;
                }
            }
        }
        m2 = column_sum<A>(m2, sm, rr, qq, a.QB, a.rpi, half);
        if (col && rr == 0) {
            A *dst = stat + (((int64_t)blockIdx.x + b) * a.Q + q) * 2;
            dst[0] = mean;
            dst[1] = m2;
        }
    }
}

// Slots of grid b: chunks first..last (last < first for an empty grid).
__device__ __forceinline__ void grid_chunks(const NormArgs &a, int32_t b, int64_t &lo, int64_t &hi, int64_t &first,
                                            int64_t &last) {
    grid_rows(a, b, lo, hi);
    first = lo / a.chunk_rows;
    last = lo < hi ? (hi - 1) / a.chunk_rows : first - 1;
}

__device__ __forceinline__ double block_sum(double v, double *sm) {
    __syncthreads();
    sm[threadIdx.x] = v;
    for (int s = kNT / 2; s > 0; s >>= 1) {
        __syncthreads();
        if (threadIdx.x < (unsigned)s) sm[threadIdx.x] += sm[threadIdx.x + s];
    }
    __syncthreads();
    return sm[0];
}

// CTA per (grid, group): mean and 1 / sqrt(var + eps), merged over the group's columns of the
// grid's slots in FP64 (total mean first, then M2 about it)
template <typename A>
__global__ void __launch_bounds__(kNT) gn_merge_kernel(NormArgs a, int32_t V, const A *__restrict__ stat, double eps,
                                                       A *__restrict__ mean_out, A *__restrict__ rstd_out) {
    __shared__ double sm[kNT];
    const int32_t b = blockIdx.x, g = blockIdx.y;
    int64_t lo, hi, first, last;
    grid_chunks(a, b, lo, hi, first, last);
    const int32_t cols = a.cpg / V, q0 = g * cols;
    const int64_t items = (last - first + 1) * cols;
    auto rows_of = [&](int64_t c) {
        return min(hi, (c + 1) * a.chunk_rows) - max(lo, c * a.chunk_rows);
    };
    double s = 0;
    for (int64_t i = threadIdx.x; i < items; i += kNT) {
        const int64_t c = first + i / cols;
        s += (double)stat[((c + b) * a.Q + q0 + i % cols) * 2] * (double)(rows_of(c) * V);
    }
    const double count = (double)(hi - lo) * a.cpg;
    const double mean = count > 0 ? block_sum(s, sm) / count : 0.0;
    double m2 = 0;
    for (int64_t i = threadIdx.x; i < items; i += kNT) {
        const int64_t c = first + i / cols;
        const A *p = stat + ((c + b) * a.Q + q0 + i % cols) * 2;
        const double d = (double)p[0] - mean;
        m2 += (double)p[1] + (double)(rows_of(c) * V) * d * d;
    }
    m2 = block_sum(m2, sm);
    if (threadIdx.x == 0) {
        mean_out[(int64_t)b * a.G + g] = (A)mean;
        rstd_out[(int64_t)b * a.G + g] = (A)(1.0 / sqrt((count > 0 ? m2 / count : 0.0) + eps));
    }
}

template <typename T, int V>
__global__ void __launch_bounds__(kNT, 4) gn_apply_kernel(NormArgs a, const T *__restrict__ x,
                                                       const typename NNum<T>::A *__restrict__ mean,
                                                       const typename NNum<T>::A *__restrict__ rstd,
                                                       const typename NNum<T>::A *__restrict__ w,
                                                       const typename NNum<T>::A *__restrict__ bias,
                                                       T *__restrict__ y) {
    using A = typename NNum<T>::A;
    const int tid = threadIdx.x, qq = tid % a.QB, rr = tid / a.QB;
    const int q = blockIdx.y * a.QB + qq;
    const int64_t r0 = (int64_t)blockIdx.x * a.chunk_rows, r1 = min(a.n, r0 + a.chunk_rows);
    const int32_t b0 = batch_of_warp(a.joff, a.B, r0), b1 = batch_of_warp(a.joff, a.B, r1 - 1);
    if (rr >= a.rpi || q >= a.Q) return;
    Raw<T, V> p[kRowsPerThread];
#pragma unroll
    for (int i = 0; i < kRowsPerThread; ++i) {
        const int64_t r = r0 + rr + (int64_t)i * a.rpi;
        if (r < r1) p[i] = ld_raw<T, V>(x + r * a.C + (int64_t)q * V);
    }
    const int32_t g = q * V / a.cpg;
    A wv[V], bv[V];
#pragma unroll
    for (int e = 0; e < V; ++e) {
        wv[e] = w ? w[q * V + e] : (A)1;
        bv[e] = bias ? bias[q * V + e] : (A)0;
    }
#pragma unroll
    for (int i = 0; i < kRowsPerThread; ++i) {
        const int64_t r = r0 + rr + (int64_t)i * a.rpi;
        if (r >= r1) continue;
        const int64_t k = (int64_t)(b0 == b1 ? b0 : batch_of(a.joff, a.B, r)) * a.G + g;
        const A m = mean[k], s = rstd[k];
        const Elems<T, V> x_ = unpack<T, V>(p[i]);
        Elems<T, V> o;
#pragma unroll
        for (int e = 0; e < V; ++e) o.v[e] = NNum<T>::from((NNum<T>::to(x_.v[e]) - m) * s * wv[e] + bv[e]);
        st_vec<T, V>(y + r * a.C + (int64_t)q * V, o);
    }
}

// part[slot][0][c] = sum of dy, part[slot][1][c] = sum of dy * xhat over the slot's rows
template <typename T, int V>
__global__ void __launch_bounds__(kNT, 4) gn_grad_sums_kernel(NormArgs a, const T *__restrict__ x,
                                                           const T *__restrict__ dy,
                                                           const typename NNum<T>::A *__restrict__ mean,
                                                           const typename NNum<T>::A *__restrict__ rstd,
                                                           typename NNum<T>::A *__restrict__ part) {
    using A = typename NNum<T>::A;
    __shared__ A sm[2 * V * kNT];
    const int tid = threadIdx.x, qq = tid % a.QB, rr = tid / a.QB;
    const int q = blockIdx.y * a.QB + qq;
    const bool col = rr < a.rpi && q < a.Q;
    int half = 1;
    while (half * 2 < a.rpi) half *= 2;
    const int64_t r0 = (int64_t)blockIdx.x * a.chunk_rows, r1 = min(a.n, r0 + a.chunk_rows);
    const int32_t b0 = batch_of_warp(a.joff, a.B, r0), b1 = batch_of_warp(a.joff, a.B, r1 - 1);
    for (int32_t b = b0; b <= b1; ++b) {
        int64_t lo, hi;
        grid_rows(a, b, lo, hi);
        lo = max(lo, r0);
        hi = min(hi, r1);
        if (lo >= hi) continue;
        A s1[V], s2[V];
#pragma unroll
        for (int e = 0; e < V; ++e) s1[e] = s2[e] = 0;
        if (col) {
            const int64_t k = (int64_t)b * a.G + q * V / a.cpg;
            const A m = mean[k], rs = rstd[k];
            const int64_t group = (int64_t)a.rpi * kRowsBackward;
            for (int64_t g0 = r0 + (lo - r0) / group * group; g0 < hi; g0 += group) {
                Raw<T, V> p[kRowsBackward], d[kRowsBackward];
#pragma unroll
                for (int i = 0; i < kRowsBackward; ++i) {
                    const int64_t r = g0 + rr + (int64_t)i * a.rpi;
                    if (r < lo || r >= hi) continue;
                    p[i] = ld_raw<T, V>(x + r * a.C + (int64_t)q * V);
                    d[i] = ld_raw<T, V>(dy + r * a.C + (int64_t)q * V);
                }
#pragma unroll
                for (int i = 0; i < kRowsBackward; ++i) {
                    const int64_t r = g0 + rr + (int64_t)i * a.rpi;
                    if (r < lo || r >= hi) continue;
                    const Elems<T, V> x_ = unpack<T, V>(p[i]), g_ = unpack<T, V>(d[i]);
#pragma unroll
                    for (int e = 0; e < V; ++e) {
                        const A g = NNum<T>::to(g_.v[e]);
                        s1[e] += g;
                        s2[e] += g * ((NNum<T>::to(x_.v[e]) - m) * rs);
                    }
                }
            }
        }
        if (a.QB <= 32 && (a.QB & (a.QB - 1)) == 0) {
            // columns that divide a warp: fold its thread rows by shuffles, then the warps' sums
#pragma unroll
            for (int e = 0; e < V; ++e)
                for (int o = a.QB; o < 32; o <<= 1) {
                    s1[e] += __shfl_xor_sync(0xffffffffu, s1[e], o);
                    s2[e] += __shfl_xor_sync(0xffffffffu, s2[e], o);
                }
            __syncthreads();
            const int lane = tid & 31;
            if (lane < a.QB)
#pragma unroll
                for (int e = 0; e < V; ++e) {
                    sm[e * kNT + (tid >> 5) * a.QB + lane] = s1[e];
                    sm[(V + e) * kNT + (tid >> 5) * a.QB + lane] = s2[e];
                }
            __syncthreads();
            // one thread per (sum, column): 2 V x QB of them, strided over the CTA
            for (int i = tid; i < 2 * V * a.QB; i += kNT) {
                const int j = i / a.QB, c = i % a.QB;
                const int64_t qc = (int64_t)blockIdx.y * a.QB + c;
                if (qc >= a.Q) continue;
                A t = 0;
#pragma unroll
                for (int w = 0; w < kNT / 32; ++w) t += sm[j * kNT + w * a.QB + c];
                part[((int64_t)blockIdx.x + b) * 2 * a.C + (j / V) * a.C + qc * V + j % V] = t;
            }
            continue;
        }
        // fold the thread rows together: entry j of thread t at sm[j * kNT + t]
        __syncthreads();
#pragma unroll
        for (int e = 0; e < V; ++e) {
            sm[e * kNT + tid] = s1[e];
            sm[(V + e) * kNT + tid] = s2[e];
        }
        for (int s = half; s > 0; s >>= 1) {
            __syncthreads();
            if (rr < s && rr + s < a.rpi)
#pragma unroll
                for (int j = 0; j < 2 * V; ++j) sm[j * kNT + tid] += sm[j * kNT + tid + s * a.QB];
        }
        __syncthreads();
        if (col && rr == 0) {
            A *dst = part + ((int64_t)blockIdx.x + b) * 2 * a.C + (int64_t)q * V;
#pragma unroll
            for (int e = 0; e < V; ++e) {
                dst[e] = sm[e * kNT + tid];
                dst[a.C + e] = sm[(V + e) * kNT + tid];
            }
        }
    }
}

// CTA per (grid, 32 of the 2C sums, one of kSlices interleaved shares of the grid's slots):
// sums[z][b][j] in FP64 (fixed order)
constexpr int kSumWarps = 32;
constexpr int kSlices = 8;
template <typename A>
__global__ void __launch_bounds__(32 * kSumWarps) gn_grad_merge_kernel(NormArgs a, const A *__restrict__ part,
                                                                       double *__restrict__ sums) {
    __shared__ double sm[kSumWarps][33];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int32_t b = blockIdx.x;
    const int64_t j = (int64_t)blockIdx.y * 32 + lane;
    int64_t lo, hi, first, last;
    grid_chunks(a, b, lo, hi, first, last);
    double s = 0;
    if (j < 2 * a.C)
#pragma unroll 4
        for (int64_t c = first + blockIdx.z * kSumWarps + warp; c <= last; c += kSumWarps * kSlices)
            s += (double)part[(c + b) * 2 * a.C + j];
    sm[warp][lane] = s;
    __syncthreads();
    if (warp == 0 && j < 2 * a.C) {
        double t = 0;
#pragma unroll
        for (int w = 0; w < kSumWarps; ++w) t += sm[w][lane];
        sums[((int64_t)blockIdx.z * a.B + b) * 2 * a.C + j] = t;
    }
}

// thread i < B*G: A1, A2 of (grid, group); thread i >= B*G: dw, db of channel i - B*G
template <typename A>
__global__ void gn_coef_kernel(NormArgs a, const double *__restrict__ sums, const A *__restrict__ w,
                               A *__restrict__ coef, A *__restrict__ dw, A *__restrict__ db) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t bg = (int64_t)a.B * a.G;
    auto sum_of = [&](int32_t b, int32_t j) {
        double t = 0;
#pragma unroll
        for (int z = 0; z < kSlices; ++z) t += sums[((int64_t)z * a.B + b) * 2 * a.C + j];
        return t;
    };
    if (i < bg) {
        const int32_t b = (int32_t)(i / a.G), g = (int32_t)(i % a.G);
        int64_t lo, hi;
        grid_rows(a, b, lo, hi);
        const double count = (double)(hi - lo) * a.cpg;
        double s1 = 0, s2 = 0;
        for (int32_t c = g * a.cpg; c < (g + 1) * a.cpg; ++c) {
            const double wc = w ? (double)w[c] : 1.0;
            s1 += wc * sum_of(b, c);
            s2 += wc * sum_of(b, a.C + c);
        }
        coef[2 * i] = (A)(count > 0 ? s1 / count : 0.0);
        coef[2 * i + 1] = (A)(count > 0 ? s2 / count : 0.0);
    } else if (i < bg + a.C) {
        const int32_t c = (int32_t)(i - bg);
        double s1 = 0, s2 = 0;
        for (int32_t b = 0; b < a.B; ++b) {
            s1 += sum_of(b, c);
            s2 += sum_of(b, a.C + c);
        }
        if (db) db[c] = (A)s1;
        if (dw) dw[c] = (A)s2;
    }
}

template <typename T, int V>
__global__ void __launch_bounds__(kNT, 4) gn_dx_kernel(NormArgs a, const T *__restrict__ x, const T *__restrict__ dy,
                                                    const typename NNum<T>::A *__restrict__ mean,
                                                    const typename NNum<T>::A *__restrict__ rstd,
                                                    const typename NNum<T>::A *__restrict__ w,
                                                    const typename NNum<T>::A *__restrict__ coef,
                                                    T *__restrict__ dx) {
    using A = typename NNum<T>::A;
    const int tid = threadIdx.x, qq = tid % a.QB, rr = tid / a.QB;
    const int q = blockIdx.y * a.QB + qq;
    const int64_t r0 = (int64_t)blockIdx.x * a.chunk_rows, r1 = min(a.n, r0 + a.chunk_rows);
    const int32_t b0 = batch_of_warp(a.joff, a.B, r0), b1 = batch_of_warp(a.joff, a.B, r1 - 1);
    if (rr >= a.rpi || q >= a.Q) return;
    Raw<T, V> p[kRowsBackward], d[kRowsBackward];
#pragma unroll
    for (int i = 0; i < kRowsBackward; ++i) {
        const int64_t r = r0 + rr + (int64_t)i * a.rpi;
        if (r < r1) {
            p[i] = ld_raw<T, V>(x + r * a.C + (int64_t)q * V);
            d[i] = ld_raw<T, V>(dy + r * a.C + (int64_t)q * V);
        }
    }
    const int32_t g = q * V / a.cpg;
    A wv[V];
#pragma unroll
    for (int e = 0; e < V; ++e) wv[e] = w ? w[q * V + e] : (A)1;
#pragma unroll
    for (int i = 0; i < kRowsBackward; ++i) {
        const int64_t r = r0 + rr + (int64_t)i * a.rpi;
        if (r >= r1) continue;
        const int64_t k = (int64_t)(b0 == b1 ? b0 : batch_of(a.joff, a.B, r)) * a.G + g;
        const A m = mean[k], s = rstd[k], c1 = coef[2 * k], c2 = coef[2 * k + 1];
        const Elems<T, V> x_ = unpack<T, V>(p[i]), g_ = unpack<T, V>(d[i]);
        Elems<T, V> o;
#pragma unroll
        for (int e = 0; e < V; ++e) {
            const A xhat = (NNum<T>::to(x_.v[e]) - m) * s;
            o.v[e] = NNum<T>::from(s * (NNum<T>::to(g_.v[e]) * wv[e] - c1 - xhat * c2));
        }
        st_vec<T, V>(dx + r * a.C + (int64_t)q * V, o);
    }
}

// Widest vector (<= 16 bytes) that stays inside one channel group and keeps every address aligned.
int pick_vec(int32_t cpg, int elem, const void *const *ptrs, int n_ptrs) {
    int v = 16 / elem;
    while (v > 1) {
        bool ok = cpg % v == 0;
        for (int i = 0; i < n_ptrs; ++i) ok = ok && ((uintptr_t)ptrs[i] % (uintptr_t)(v * elem)) == 0;
        if (ok) break;
        v >>= 1;
    }
    return v;
}

NormArgs norm_args(const int64_t *joff, int32_t B, int64_t n, int32_t C, int32_t G, int V, int rows) {
    NormArgs a;
    a.joff = joff;
    a.B = B;
    a.n = n;
    a.C = C;
    a.G = G;
    a.cpg = C / G;
    a.Q = C / V;
    a.QB = a.Q < kNT ? a.Q : kNT;
    a.rpi = kNT / a.QB;
    a.chunk_rows = (int64_t)a.rpi * rows;
    return a;
}

// Bytes of one call's scratch for the finest chunking any vector width can give.
size_t norm_ws(int64_t n, int32_t B, int32_t C, int32_t G, size_t acc, bool backward) {
    // chunks are shortest at V = 1 (most vector columns); slots = chunks + grids
    size_t need = 0;
    for (int V = 1; V <= 8; V *= 2) {
        if ((C / G) % V) break;
        const NormArgs a = norm_args(nullptr, B, n, C, G, V, backward ? kRowsBackward * kSumIters : kRowsPerThread);
        const size_t slots = (size_t)ceil_div(n > 0 ? n : 1, a.chunk_rows) + (size_t)B;
        const size_t s = backward ? slots * 2 * (size_t)C * acc : slots * (size_t)a.Q * 2 * acc;
        if (s > need) need = s;
    }
    need = (need + 255) & ~(size_t)255;
    if (backward) need += (((size_t)kSlices * B * 2 * C * 8 + 255) & ~(size_t)255) + (((size_t)B * G * 2 * acc + 255) & ~(size_t)255);
    return need + 256;
}

template <typename T, int V>
void run_forward(const NormArgs &a, const void *x, const void *w, const void *b, double eps, void *y, void *mean,
                 void *rstd, void *ws, cudaStream_t s) {
    using A = typename NNum<T>::A;
    const dim3 grid((unsigned)ceil_div(a.n, a.chunk_rows), (unsigned)ceil_div(a.Q, a.QB));
    gn_stats_kernel<T, V><<<grid, kNT, 0, s>>>(a, (const T *)x, (A *)ws);
    gn_merge_kernel<A><<<dim3((unsigned)a.B, (unsigned)a.G), kNT, 0, s>>>(a, V, (const A *)ws, eps, (A *)mean, (A *)rstd);
    gn_apply_kernel<T, V><<<grid, kNT, 0, s>>>(a, (const T *)x, (const A *)mean, (const A *)rstd, (const A *)w,
                                               (const A *)b, (T *)y);
}

template <typename T, int V>
void run_backward(const NormArgs &a, const void *x, const void *dy, const void *w, const void *mean, const void *rstd,
                  void *dx, void *dw, void *db, void *ws, cudaStream_t s) {
    using A = typename NNum<T>::A;
    const int64_t chunks = ceil_div(a.n, a.chunk_rows);
    uint8_t *p = (uint8_t *)ws;
    A *part = (A *)p;
    p += ((size_t)(chunks + a.B) * 2 * a.C * sizeof(A) + 255) & ~(size_t)255;
    double *sums = (double *)p;
    p += ((size_t)kSlices * a.B * 2 * a.C * 8 + 255) & ~(size_t)255;
    A *coef = (A *)p;
    const dim3 grid((unsigned)chunks, (unsigned)ceil_div(a.Q, a.QB));
    gn_grad_sums_kernel<T, V><<<grid, kNT, 0, s>>>(a, (const T *)x, (const T *)dy, (const A *)mean, (const A *)rstd, part);
    gn_grad_merge_kernel<A><<<dim3((unsigned)a.B, (unsigned)ceil_div(2 * a.C, 32), kSlices), 32 * kSumWarps, 0, s>>>(a, part, sums);
    gn_coef_kernel<A><<<(unsigned)ceil_div((int64_t)a.B * a.G + a.C, 128), 128, 0, s>>>(a, sums, (const A *)w, coef,
                                                                                       (A *)dw, (A *)db);
    NormArgs ax = a;  // dx: one row group per CTA
    ax.chunk_rows = (int64_t)a.rpi * kRowsBackward;
    const dim3 grid_dx((unsigned)ceil_div(a.n, ax.chunk_rows), grid.y);
    if (dx)
        gn_dx_kernel<T, V><<<grid_dx, kNT, 0, s>>>(ax, (const T *)x, (const T *)dy, (const A *)mean, (const A *)rstd,
                                                (const A *)w, coef, (T *)dx);
}

template <typename T, typename F>
void by_vec(int V, F &&f) {
    switch (V) {
        case 1: f(std::integral_constant<int, 1>()); break;
        case 2: f(std::integral_constant<int, 2>()); break;
        case 4:
            if constexpr (sizeof(T) <= 4) f(std::integral_constant<int, 4>());
            break;
        default:
            if constexpr (sizeof(T) <= 2) f(std::integral_constant<int, 8>());
    }
}

template <typename F>
int by_dtype(int32_t dtype, F &&f) {
    switch (dtype) {
        case FVGB_F32: f((float *)nullptr); break;
        case FVGB_F64: f((double *)nullptr); break;
        case FVGB_BF16: f((__nv_bfloat16 *)nullptr); break;
        case FVGB_F16: f((__half *)nullptr); break;
        default: return FVGB_ETYPE;
    }
    return FVGB_OK;
}

int elem_size(int32_t dtype) { return dtype == FVGB_F64 ? 8 : (dtype == FVGB_F32 ? 4 : 2); }

// dtype and sizes one launch can take (grid.y limits the grids' and groups' product axes)
int norm_check(int32_t dtype, int64_t n, int32_t C, int32_t G, int32_t B) {
    if (dtype != FVGB_F32 && dtype != FVGB_F64 && dtype != FVGB_BF16 && dtype != FVGB_F16) return FVGB_ETYPE;
    if (n < 0 || C < 1 || G < 1 || B < 1 || C % G != 0 || G > 65535 || C > 65535) return FVGB_EINVAL;
    if (n / kRowsBackward > INT32_MAX - 1) return FVGB_EINVAL;
    return FVGB_OK;
}

}  // namespace
}  // namespace fvgb

using namespace fvgb;

extern "C" int fvgb_group_norm_workspace(int32_t dtype, int64_t n, int32_t channels, int32_t groups, int32_t num_grids,
                                         int32_t backward, size_t *bytes) {
    const int st = norm_check(dtype, n, channels, groups, num_grids);
    if (st || !bytes) return st ? st : FVGB_EINVAL;
    *bytes = norm_ws(n, num_grids, channels, groups, dtype == FVGB_F64 ? 8 : 4, backward != 0);
    return FVGB_OK;
}

extern "C" int fvgb_group_norm_forward(int32_t dtype, const void *x, int64_t n, int32_t channels, int32_t groups,
                                       const int64_t *joffsets, int32_t num_grids, const void *weight,
                                       const void *bias, double eps, void *y, void *mean, void *rstd, void *workspace,
                                       size_t workspace_bytes, fvgb_stream_t stream) {
    size_t need = 0;
    int st = fvgb_group_norm_workspace(dtype, n, channels, groups, num_grids, 0, &need);
    if (st) return st;
    if (n == 0) return FVGB_OK;
    if (!x || !y || !mean || !rstd || !joffsets) return FVGB_EINVAL;
    if (!workspace || workspace_bytes < need) return FVGB_ENOSPACE;
    const void *ptrs[2] = {x, y};
    const int V = pick_vec(channels / groups, elem_size(dtype), ptrs, 2);
    const NormArgs a = norm_args(joffsets, num_grids, n, channels, groups, V, kRowsPerThread);
    void *ws = reinterpret_cast<void *>(((uintptr_t)workspace + 255) & ~(uintptr_t)255);
    st = by_dtype(dtype, [&](auto *t) {
        using T = std::remove_pointer_t<decltype(t)>;
        by_vec<T>(V, [&](auto v) {
            run_forward<T, decltype(v)::value>(a, x, weight, bias, eps, y, mean, rstd, ws, as_stream(stream));
        });
    });
    if (st) return st;
    count_launches(3);
    return launch_status();
}

extern "C" int fvgb_group_norm_backward(int32_t dtype, const void *x, const void *dy, int64_t n, int32_t channels,
                                        int32_t groups, const int64_t *joffsets, int32_t num_grids, const void *weight,
                                        const void *mean, const void *rstd, void *dx, void *dweight, void *dbias,
                                        void *workspace, size_t workspace_bytes, fvgb_stream_t stream) {
    size_t need = 0;
    int st = fvgb_group_norm_workspace(dtype, n, channels, groups, num_grids, 1, &need);
    if (st) return st;
    if (n == 0) return FVGB_OK;
    if (!x || !dy || !mean || !rstd || !joffsets) return FVGB_EINVAL;
    if (!workspace || workspace_bytes < need) return FVGB_ENOSPACE;
    const void *ptrs[3] = {x, dy, dx};
    const int V = pick_vec(channels / groups, elem_size(dtype), ptrs, 3);
    const NormArgs a = norm_args(joffsets, num_grids, n, channels, groups, V, kRowsBackward * kSumIters);
    void *ws = reinterpret_cast<void *>(((uintptr_t)workspace + 255) & ~(uintptr_t)255);
    st = by_dtype(dtype, [&](auto *t) {
        using T = std::remove_pointer_t<decltype(t)>;
        by_vec<T>(V, [&](auto v) {
            run_backward<T, decltype(v)::value>(a, x, dy, weight, mean, rstd, dx, dweight, dbias, ws, as_stream(stream));
        });
    });
    if (st) return st;
    count_launches(dx ? 4 : 3);
    return launch_status();
}
