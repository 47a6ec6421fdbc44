// Gradient of a convolution's fused bias and ReLU: masks the output gradient where the layer's
// output is not positive and sums the bias gradient in the same pass.
//
// Bound by HBM: reads dy (and y), writes the masked dy.  Two layers of 1.27M x 64 BF16, one with a
// ReLU: a comparison, a mixed-type product and two column sums took 538 us, 124 us here.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <type_traits>

#include "common.cuh"

namespace fvgb {
namespace {

constexpr int kNT = 256;
constexpr int kRows = 4;  // rows a thread has in flight

template <typename T>
struct PNum {
    using A = float;
};
template <>
struct PNum<double> {
    using A = double;
};
__device__ __forceinline__ float up(float v) { return v; }
__device__ __forceinline__ double up(double v) { return v; }
__device__ __forceinline__ float up(__nv_bfloat16 v) { return __bfloat162float(v); }
__device__ __forceinline__ float up(__half v) { return __half2float(v); }
__device__ __forceinline__ void down(float v, float &o) { o = v; }
__device__ __forceinline__ void down(double v, double &o) { o = v; }
__device__ __forceinline__ void down(float v, __nv_bfloat16 &o) { o = __float2bfloat16_rn(v); }
__device__ __forceinline__ void down(float v, __half &o) { o = __float2half_rn(v); }

// A thread keeps one vector column and walks rows; CTA b takes row blocks b, b + gridDim.x, ...
// part[b][c] = the CTA's column sums (part null: no bias gradient; y null: no ReLU).  The mask is a
// product with 0 or 1, as the layer's backward is: a NaN or infinity in dy stays a NaN.
template <typename T, int V>
__global__ void __launch_bounds__(kNT, 4) bias_relu_bwd_kernel(const T *__restrict__ dy, const T *__restrict__ y,
                                                            int64_t n, int32_t C, int32_t QB, T *__restrict__ out,
                                                            typename PNum<T>::A *__restrict__ part) {
    using A = typename PNum<T>::A;
    __shared__ A sm[V * kNT];
    const int tid = threadIdx.x, qq = tid % QB, rr = tid / QB, rpi = kNT / QB;
    const int64_t q = (int64_t)blockIdx.y * QB + qq;
    const bool col = rr < rpi && q * V < C;
    A s[V];
#pragma unroll
    for (int e = 0; e < V; ++e) s[e] = 0;
    const int64_t step = (int64_t)gridDim.x * rpi * kRows;
    if (col)
        for (int64_t r0 = (int64_t)blockIdx.x * rpi * kRows + rr; r0 < n; r0 += step) {
            Raw<T, V> g[kRows], p[kRows];
#pragma unroll
            for (int i = 0; i < kRows; ++i) {
                const int64_t r = r0 + (int64_t)i * rpi;
                if (r >= n) continue;
                g[i] = ld_raw<T, V>(dy + r * C + q * V);
                if (y) p[i] = ld_raw<T, V>(y + r * C + q * V);
            }
#pragma unroll
            for (int i = 0; i < kRows; ++i) {
                const int64_t r = r0 + (int64_t)i * rpi;
                if (r >= n) continue;
                Elems<T, V> o = unpack<T, V>(g[i]);
                if (y) {
                    const Elems<T, V> f = unpack<T, V>(p[i]);
#pragma unroll
                    for (int e = 0; e < V; ++e) down(up(o.v[e]) * (up(f.v[e]) > (A)0 ? (A)1 : (A)0), o.v[e]);
                    st_vec<T, V>(out + r * C + q * V, o);
                }
#pragma unroll
                for (int e = 0; e < V; ++e) s[e] += up(o.v[e]);
            }
        }
    if (!part) return;
#pragma unroll
    for (int e = 0; e < V; ++e) sm[e * kNT + tid] = s[e];
    int half = 1;
    while (half * 2 < rpi) half *= 2;
    for (; half > 0; half >>= 1) {
        __syncthreads();
        if (rr < half && rr + half < rpi)
#pragma unroll
            for (int e = 0; e < V; ++e) sm[e * kNT + tid] += sm[e * kNT + tid + half * QB];
    }
    if (col && rr == 0)
#pragma unroll
        for (int e = 0; e < V; ++e) part[(int64_t)blockIdx.x * C + q * V + e] = sm[e * kNT + tid];
}

// db[c] = sum of the CTAs' partial sums, FP64 in a fixed order.  A CTA takes kMergeCols columns: FP64 runs
// at a few lanes per SM and clock, so 32 columns per CTA left the work of 64 channels to two SMs (608
// partial rows: 13.7 us; 3.8 us over sixteen).
constexpr int kMergeCols = 4, kMergeThreads = 256;
template <typename A>
__global__ void __launch_bounds__(kMergeThreads) column_merge_kernel(const A *__restrict__ part, int64_t parts, int32_t C,
                                                                     A *__restrict__ db) {
    __shared__ double sm[kMergeThreads / 32][kMergeCols];
    const int col = threadIdx.x % kMergeCols, row = threadIdx.x / kMergeCols;
    const int64_t c = (int64_t)blockIdx.x * kMergeCols + col;
    double s = 0;
    if (c < C)
#pragma unroll 4
        for (int64_t p = row; p < parts; p += kMergeThreads / kMergeCols) s += (double)part[p * C + c];
#pragma unroll
    for (int o = kMergeCols; o < 32; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) < kMergeCols) sm[threadIdx.x >> 5][col] = s;
    __syncthreads();
    if (threadIdx.x < kMergeCols && c < C) {
        double t = 0;
#pragma unroll
        for (int w = 0; w < kMergeThreads / 32; ++w) t += sm[w][col];
        db[c] = (A)t;
    }
}

// s = rsqrt(var + eps) * weight, t = -mean * s + bias: an inference-mode batch norm as
// x -> x s + t, in FP32 with one rounding per operation; every parameter of one type, weight and bias
// optional.
template <typename T>
__global__ void fold_batch_norm_kernel(const T *__restrict__ mean, const T *__restrict__ var, const T *__restrict__ weight,
                                       const T *__restrict__ bias, int32_t c, float eps, float *__restrict__ s,
                                       float *__restrict__ t) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c) return;
    float a = rsqrtf(__fadd_rn((float)up(var[i]), eps));
    if (weight) a = __fmul_rn(a, (float)up(weight[i]));
    float b = __fmul_rn(-(float)up(mean[i]), a);
    if (bias) b = __fadd_rn(b, (float)up(bias[i]));
    s[i] = a;
    t[i] = b;
}

// shift = bias * s + t (FP32)
template <typename T>
__global__ void fold_bias_kernel(const T *__restrict__ bias, const float *__restrict__ s, const float *__restrict__ t,
                                 int32_t c, float *__restrict__ shift) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < c) shift[i] = __fadd_rn(__fmul_rn((float)up(bias[i]), s[i]), t[i]);
}

template <typename F>
int by_type(int32_t dtype, F &&f) {
    switch (dtype) {
        case FVGB_F32: f((float *)nullptr); break;
        case FVGB_F64: f((double *)nullptr); break;
        case FVGB_BF16: f((__nv_bfloat16 *)nullptr); break;
        case FVGB_F16: f((__half *)nullptr); break;
        default: return FVGB_ETYPE;
    }
    count_launches(1);
    return launch_status();
}

int64_t part_ctas(int64_t n) { return std::min<int64_t>(std::max<int64_t>(ceil_div(n, 64), 1), (int64_t)device_sm_count() * 4); }

template <typename T, int V>
void launch(const void *dy, const void *y, int64_t n, int32_t C, void *out, void *db, void *ws, cudaStream_t s) {
    using A = typename PNum<T>::A;
    const int32_t Q = C / V, QB = Q < kNT ? Q : kNT;
    const int64_t ctas = part_ctas(n);
    bias_relu_bwd_kernel<T, V><<<dim3((unsigned)ctas, (unsigned)ceil_div(Q, QB)), kNT, 0, s>>>(
        (const T *)dy, (const T *)y, n, C, QB, (T *)out, db ? (A *)ws : nullptr);
    if (db) column_merge_kernel<A><<<(unsigned)ceil_div(C, kMergeCols), kMergeThreads, 0, s>>>((const A *)ws, ctas, C, (A *)db);
}

template <typename T>
void by_width(bool vec, const void *dy, const void *y, int64_t n, int32_t C, void *out, void *db, void *ws,
              cudaStream_t s) {
    if (vec) launch<T, 16 / sizeof(T)>(dy, y, n, C, out, db, ws, s);
    else launch<T, 1>(dy, y, n, C, out, db, ws, s);
}

}  // namespace
}  // namespace fvgb

using namespace fvgb;

extern "C" int fvgb_bias_relu_backward_workspace(int32_t dtype, int64_t n, int32_t c, size_t *bytes) {
    if (!bytes || n < 0 || c < 1) return FVGB_EINVAL;
    *bytes = (size_t)part_ctas(n) * c * (dtype == FVGB_F64 ? 8 : 4) + 256;
    return FVGB_OK;
}

extern "C" int fvgb_bias_relu_backward(int32_t dtype, const void *dy, const void *y, int64_t n, int32_t c, void *out,
                                       void *dbias, void *workspace, size_t workspace_bytes, fvgb_stream_t stream) {
    size_t need = 0;
    const int st = fvgb_bias_relu_backward_workspace(dtype, n, c, &need);
    if (st) return st;
    if (dtype != FVGB_F32 && dtype != FVGB_F64 && dtype != FVGB_BF16 && dtype != FVGB_F16) return FVGB_ETYPE;
    if (c > 256 * 65535) return FVGB_EINVAL;
    if (n > 0 && (!dy || (y && !out))) return FVGB_EINVAL;
    if (dbias && (!workspace || workspace_bytes < need)) return FVGB_ENOSPACE;
    const int elem = dtype == FVGB_F64 ? 8 : (dtype == FVGB_F32 ? 4 : 2);
    const bool vec = (c * elem) % 16 == 0 && (((uintptr_t)dy | (uintptr_t)y | (uintptr_t)out) & 15) == 0;
    void *ws = reinterpret_cast<void *>(((uintptr_t)workspace + 255) & ~(uintptr_t)255);
    cudaStream_t s = as_stream(stream);
    switch (dtype) {
        case FVGB_F32: by_width<float>(vec, dy, y, n, c, out, dbias, ws, s); break;
        case FVGB_F64: by_width<double>(vec, dy, y, n, c, out, dbias, ws, s); break;
        case FVGB_BF16: by_width<__nv_bfloat16>(vec, dy, y, n, c, out, dbias, ws, s); break;
        default: by_width<__half>(vec, dy, y, n, c, out, dbias, ws, s);
    }
    count_launches(dbias ? 2 : 1);
    return launch_status();
}

extern "C" int fvgb_fold_batch_norm(int32_t dtype, const void *mean, const void *var, const void *weight,
                                    const void *bias, int32_t c, float eps, float *scale, float *shift,
                                    fvgb_stream_t stream) {
    if (c < 1 || !mean || !var || !scale || !shift) return FVGB_EINVAL;
    return by_type(dtype, [&](auto *p) {
        using T = std::remove_pointer_t<decltype(p)>;
        fold_batch_norm_kernel<T><<<(unsigned)ceil_div(c, 128), 128, 0, as_stream(stream)>>>(
            (const T *)mean, (const T *)var, (const T *)weight, (const T *)bias, c, eps, scale, shift);
    });
}

extern "C" int fvgb_fold_bias(int32_t dtype, const void *bias, const float *s, const float *t, int32_t c, float *shift,
                              fvgb_stream_t stream) {
    if (c < 1 || !bias || !s || !t || !shift) return FVGB_EINVAL;
    return by_type(dtype, [&](auto *p) {
        using T = std::remove_pointer_t<decltype(p)>;
        fold_bias_kernel<T><<<(unsigned)ceil_div(c, 128), 128, 0, as_stream(stream)>>>((const T *)bias, s, t, c, shift);
    });
}
