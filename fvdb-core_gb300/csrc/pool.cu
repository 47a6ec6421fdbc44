// Pooling between a fine and a coarse grid and nearest-neighbour upsampling (the neighbours of
// sparse convolutions in a sparse UNet: fvdb.nn.MaxPool / AvgPool / UpsamplingNearest).
//
// Semantics follow the reference kernels:
//   * pooling: coarse voxel c reads the window of fine voxels c*stride + (i, j, k), i < p0, j < p1,
//     k < p2 (axis a of the window <-> ijk axis a), visited i-outer / k-inner; max starts at -inf
//     (an empty window stays -inf), average = (sum of the window's active voxels in the
//     accumulation type, rounded to the data type) * (1 / (p0 p1 p2) rounded to the data type)
//     (src/fvdb/detail/ops/DownsampleGridMaxPool.cu:19-69, DownsampleGridAvgPool.cu:19-64,144);
//   * max-pool gradient: each window's gradient goes to its first strict maximum;
//     average gradient: fine voxel f gets grad(c) * (1 / (p0 p1 p2)) from the window c holding it
//     (DownsampleGridMaxPool.cu:71-126, DownsampleGridAvgPool.cu:68-112);
//   * upsampling: fine voxel f copies coarse voxel floor(f / factor); its gradient sums the
//     children (src/fvdb/detail/ops/UpsampleGridNearest.cu:19-110).
// Differences, each on inputs where the reference's result is undefined or racy: the coarse
// coordinate of upsampling is an exact integer floor (the reference divides in the data type,
// inexact for 16-bit data beyond |ijk| = 256), a fine voxel without a coarse parent reads zero
// (the reference reads the row before its grid's first), and gradients of overlapping windows
// (stride < pool factor) add up (the reference's concurrent assignments keep one of them).
//
// A group of G lanes owns one output voxel and each lane moves one 16-byte vector of its row (G = the
// power of two >= vectors per row, so a 64-channel BF16 row takes 8 lanes and a warp works on four
// voxels).  The window's rows come from a window map (fvgb_window_map, built leaf by leaf with one
// hash probe per source leaf) or, without one, from one leaf-hash lookup per window position, which
// the group's lanes share.  Bound by HBM with a map, by the lookups' latency without.  1.31M fine and
// 0.36M coarse voxels, 64 BF16 channels, factor 2 (GB300), one warp per voxel and one element per
// lane before: max 190 us, its gradient 235 + 115 for the FP32 buffer, upsampling 464, its gradient
// 192; here 59, 113 + 43 for zeroing, 46 and 59, and 18 for each window map.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <initializer_list>
#include <type_traits>

#include "common.cuh"

namespace fvgb {
namespace {

constexpr int kPoolWarps = 8;
constexpr int kMaxWindow = 512;  // pool factor / upsampling factor volume (8x8x8)

__device__ __forceinline__ int64_t voxel_at(const FvgbGrid &g, int32_t b, int32_t x, int32_t y, int32_t z) {
    const int32_t lid = find_leaf(g, b, x >> 3, y >> 3, z >> 3);
    if (lid < 0) return -1;
    return leaf_voxel_index(g.leaves[lid], leaf_bit(x, y, z));
}

template <typename T>
struct Num;
template <>
struct Num<float> {
    using Acc = float;
    __device__ static float to(float v) { return v; }
    __device__ static float from(float v) { return v; }
};
template <>
struct Num<double> {
    using Acc = double;
    __device__ static double to(double v) { return v; }
    __device__ static double from(double v) { return v; }
};
template <>
struct Num<__half> {
    using Acc = float;
    __device__ static float to(__half v) { return __half2float(v); }
    __device__ static __half from(float v) { return __float2half_rn(v); }
};
template <>
struct Num<__nv_bfloat16> {
    using Acc = float;
    __device__ static float to(__nv_bfloat16 v) { return __bfloat162float(v); }
    __device__ static __nv_bfloat16 from(float v) { return __float2bfloat16_rn(v); }
};

// x * y in the data type's arithmetic: both rounded to T, multiplied in the accumulation type,
// the product rounded to T (c10::Half / BFloat16 multiply through float).
template <typename T>
__device__ __forceinline__ T mul_in(T a, double b) {
    using A = typename Num<T>::Acc;
    return Num<T>::from(Num<T>::to(a) * Num<T>::to(Num<T>::from((A)b)));
}

// Lane groups of a CTA: G = 1 << gs lanes per output voxel, and the shared window indices of each.
struct Groups {
    int gs;     // log2 lanes per group
    int W;      // window entries stored per group
    size_t smem;
};

constexpr int kGroupThreads = 256;
constexpr int kGroupSmem = 32 * 1024;

// lookups: the group's lanes also share one leaf-hash lookup per window entry, so a narrow row gets lanes
// for those (0.02M voxels, one channel, 4^3 windows: 89 us a call with one lane per voxel).
Groups groups_for(int32_t vecs, int W, bool lookups = false) {
    Groups g;
    g.gs = 0;
    const int lanes = lookups && W > vecs ? W : vecs;
    while ((1 << g.gs) < lanes && g.gs < 5) ++g.gs;
    while (g.gs < 5 && (size_t)(kGroupThreads >> g.gs) * W * 4 > kGroupSmem) ++g.gs;
    g.W = W;
    g.smem = (size_t)(kGroupThreads >> g.gs) * W * 4;
    return g;
}

// Window indices of one output voxel into the group's shared array (window order i-outer, k-inner):
// lane l of the group fills positions l, l + G, ...  Every lane of the warp calls it (groups whose
// voxel is past the end with an empty window).
__device__ __forceinline__ void window_indices(const FvgbGrid &g, int32_t b, int3 base, int3 ext, int32_t *idx, int lane,
                                               int G) {
    const int W = ext.x * ext.y * ext.z;
    for (int w = lane; w < W; w += G) {
        const int i = w / (ext.y * ext.z), j = (w / ext.z) % ext.y, k = w % ext.z;
        const int64_t v = voxel_at(g, b, base.x + i, base.y + j, base.z + k);
        idx[w] = (int32_t)v;
    }
    __syncwarp();
}

// The same from a window map.
__device__ __forceinline__ void map_indices(const int32_t *map, int64_t c, bool on, int W, int32_t *idx, int lane, int G) {
    if (on)
        for (int w = lane; w < W; w += G) idx[w] = __ldg(map + c * W + w);
    __syncwarp();
}

constexpr int kAhead = 8;    // window rows a lane has in flight, 16 bytes each
constexpr int kUpAhead = 4;  // rows of the upsampling copy, which its stores pace (eight: 67 us for 46)

// Reduction over the window rows of every coarse voxel: maximum (MAX), or the sum, rounded and times
// `avg` where SCALE.  Serves pooling and the upsampling gradient.  Over `map` where given (the grids
// are then not read), else by lookups.
template <typename T, int V, bool MAX, bool SCALE>
__global__ void __launch_bounds__(kGroupThreads, 4) window_reduce_kernel(FvgbGrid fine, FvgbGrid coarse, int3 pf, int3 st,
                                                                      const int32_t *__restrict__ map, int64_t n_coarse,
                                                                      Groups gr, const T *__restrict__ x, int64_t ldx,
                                                                      int32_t C, T *__restrict__ y, int64_t ldy,
                                                                      double avg) {
    using A = typename Num<T>::Acc;
    extern __shared__ int32_t widx[];
    const int G = 1 << gr.gs, group = threadIdx.x >> gr.gs, lane = threadIdx.x & (G - 1);
    const int W = gr.W;
    int32_t *idx = widx + group * W;
    const int64_t c = (int64_t)blockIdx.x * (kGroupThreads >> gr.gs) + group;
    const bool on = c < n_coarse;
    if (map) {
        map_indices(map, c, on, W, idx, lane, G);
    } else {
        int32_t b = 0;
        int3 base = make_int3(0, 0, 0), ext = make_int3(0, 0, 0);
        if (on) {
            b = batch_of(coarse.voxel_offsets, coarse.num_grids, c);
            base = make_int3(coarse.ijk[3 * c] * st.x, coarse.ijk[3 * c + 1] * st.y, coarse.ijk[3 * c + 2] * st.z);
            ext = pf;
        }
        window_indices(fine, b, base, ext, idx, lane, G);
    }
    if (!on) return;
    for (int32_t ch = lane * V; ch < C; ch += G * V) {
        A acc[V];
#pragma unroll
        for (int e = 0; e < V; ++e) acc[e] = MAX ? (A)(-INFINITY) : (A)0;
        for (int w0 = 0; w0 < W; w0 += kAhead) {
            Raw<T, V> p[kAhead];
            int32_t f[kAhead];
#pragma unroll
            for (int u = 0; u < kAhead; ++u) {
                f[u] = w0 + u < W ? idx[w0 + u] : -1;
                if (f[u] >= 0) p[u] = ld_raw<T, V>(x + (int64_t)f[u] * ldx + ch);
            }
#pragma unroll
            for (int u = 0; u < kAhead; ++u) {
                if (f[u] < 0) continue;
                const Elems<T, V> row = unpack<T, V>(p[u]);
#pragma unroll
                for (int e = 0; e < V; ++e) {
                    const A v = Num<T>::to(row.v[e]);
                    if constexpr (MAX) {
                        if constexpr (sizeof(A) == 8) acc[e] = fmax(v, acc[e]);
                        else acc[e] = fmaxf(v, acc[e]);
                    } else {
                        acc[e] = acc[e] + v;
                    }
                }
            }
        }
        Elems<T, V> o;
#pragma unroll
        for (int e = 0; e < V; ++e) o.v[e] = SCALE ? mul_in<T>(Num<T>::from(acc[e]), avg) : Num<T>::from(acc[e]);
        st_vec<T, V>(y + c * ldy + ch, o);
    }
}

// The same by lookups for windows of more than kGroupWindow positions: a warp per coarse voxel, a lookup
// per lane, then a channel per lane.  The lookups set the pace here, and 32 registers let the SM hold twice
// the warps of window_reduce_kernel (1.19M surface voxels, 3^3 windows at stride 3, 32 FP32 channels: 188
// us with that kernel, 112 with this; 2^3 windows, 0.35M coarse: 78 with that, 145 with this).
constexpr int kGroupWindow = 8;
template <typename T, bool MAX, bool SCALE>
__global__ void __launch_bounds__(kPoolWarps * 32) window_lookup_kernel(FvgbGrid fine, FvgbGrid coarse, int3 pf, int3 st,
                                                                        const T *__restrict__ x, int64_t ldx, int32_t C,
                                                                        T *__restrict__ y, int64_t ldy, double avg) {
    using A = typename Num<T>::Acc;
    __shared__ int32_t widx[kPoolWarps][kMaxWindow];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int W = pf.x * pf.y * pf.z;
    for (int64_t c = (int64_t)blockIdx.x * kPoolWarps + warp; c < coarse.num_voxels; c += (int64_t)gridDim.x * kPoolWarps) {
        const int32_t b = batch_of(coarse.voxel_offsets, coarse.num_grids, c);
        const int3 base = make_int3(coarse.ijk[3 * c] * st.x, coarse.ijk[3 * c + 1] * st.y, coarse.ijk[3 * c + 2] * st.z);
        window_indices(fine, b, base, pf, widx[warp], lane, 32);
        for (int ch = lane; ch < C; ch += 32) {
            A acc = MAX ? (A)(-INFINITY) : (A)0;
            for (int w = 0; w < W; ++w) {
                const int32_t f = widx[warp][w];
                if (f < 0) continue;
                const A v = Num<T>::to(x[(int64_t)f * ldx + ch]);
                if constexpr (!MAX) acc = acc + v;
                else if constexpr (sizeof(A) == 8) acc = fmax(v, acc);
                else acc = fmaxf(v, acc);
            }
            y[c * ldy + ch] = SCALE ? mul_in<T>(Num<T>::from(acc), avg) : Num<T>::from(acc);
        }
        __syncwarp();
    }
}

// Max-pool gradient where no two windows overlap (stride >= window on every axis): each fine voxel
// belongs to one window at most, so its row is written once -- the gradient where it holds the
// window's first strict maximum, zero elsewhere -- without a buffer to add into.  Rows of voxels in
// no window stay as the caller zeroed them.
template <typename T, int V>
__global__ void __launch_bounds__(kGroupThreads, 4) maxpool_bwd_disjoint_kernel(const int32_t *__restrict__ map,
                                                                             int64_t n_coarse, Groups gr,
                                                                             const T *__restrict__ x, int64_t ldx,
                                                                             int32_t C, const T *__restrict__ dy,
                                                                             int64_t lddy, T *__restrict__ dx) {
    using A = typename Num<T>::Acc;
    extern __shared__ int32_t widx[];
    const int G = 1 << gr.gs, group = threadIdx.x >> gr.gs, lane = threadIdx.x & (G - 1);
    const int W = gr.W;
    int32_t *idx = widx + group * W;
    const int64_t c = (int64_t)blockIdx.x * (kGroupThreads >> gr.gs) + group;
    const bool on = c < n_coarse;
    map_indices(map, c, on, W, idx, lane, G);
    if (!on) return;
    for (int32_t ch = lane * V; ch < C; ch += G * V) {
        const Elems<T, V> g = unpack<T, V>(ld_raw<T, V>(dy + c * lddy + ch));
        A best[V];
        int32_t arg[V];
#pragma unroll
        for (int e = 0; e < V; ++e) best[e] = (A)(-INFINITY), arg[e] = -1;
        for (int w0 = 0; w0 < W; w0 += kAhead) {
            Raw<T, V> p[kAhead];
            int32_t f[kAhead];
#pragma unroll
            for (int u = 0; u < kAhead; ++u) {
                f[u] = w0 + u < W ? idx[w0 + u] : -1;
                if (f[u] >= 0) p[u] = ld_raw<T, V>(x + (int64_t)f[u] * ldx + ch);
            }
#pragma unroll
            for (int u = 0; u < kAhead; ++u) {
                if (f[u] < 0) continue;
                const Elems<T, V> row = unpack<T, V>(p[u]);
#pragma unroll
                for (int e = 0; e < V; ++e) {
                    const A v = Num<T>::to(row.v[e]);
                    if (v > best[e]) best[e] = v, arg[e] = f[u];
                }
            }
        }
        for (int w = 0; w < W; ++w) {
            const int32_t f = idx[w];
            if (f < 0) continue;
            Elems<T, V> o;
#pragma unroll
            for (int e = 0; e < V; ++e) o.v[e] = arg[e] == f ? g.v[e] : Num<T>::from((A)0);
            st_vec<T, V>(dx + (int64_t)f * C + ch, o);
        }
    }
}

// Max-pool gradient of overlapping windows: per window and channel, grad to the first strict
// maximum, added into the accumulation buffer dx (zero-initialised by the caller).
template <typename T>
__global__ void __launch_bounds__(kPoolWarps * 32) maxpool_bwd_kernel(FvgbGrid fine, FvgbGrid coarse, int3 pf, int3 st,
                                                                      const T *__restrict__ x, int64_t ldx, int32_t C,
                                                                      const T *__restrict__ dy, int64_t lddy,
                                                                      typename Num<T>::Acc *__restrict__ dx) {
    using A = typename Num<T>::Acc;
    __shared__ int32_t widx[kPoolWarps][kMaxWindow];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int W = pf.x * pf.y * pf.z;
    for (int64_t c = (int64_t)blockIdx.x * kPoolWarps + warp; c < coarse.num_voxels;
         c += (int64_t)gridDim.x * kPoolWarps) {
        const int32_t b = batch_of(coarse.voxel_offsets, coarse.num_grids, c);
        const int3 base = make_int3(coarse.ijk[3 * c] * st.x, coarse.ijk[3 * c + 1] * st.y, coarse.ijk[3 * c + 2] * st.z);
        window_indices(fine, b, base, pf, widx[warp], lane, 32);
        for (int ch = lane; ch < C; ch += 32) {
            A best = (A)(-INFINITY);
            int32_t arg = -1;
            for (int w = 0; w < W; ++w) {
                const int32_t f = widx[warp][w];
                if (f < 0) continue;
                const A v = Num<T>::to(x[(int64_t)f * ldx + ch]);
                if (v > best) {
                    best = v;
                    arg = f;
                }
            }
            if (arg >= 0) atomicAdd(dx + (int64_t)arg * C + ch, Num<T>::to(dy[c * lddy + ch]));
        }
        __syncwarp();
    }
}

// Average-pool gradient, gathered per fine voxel: the coarse voxels whose window holds fine
// voxel f are c with c*s <= f < c*s + p per axis.
template <typename T, int V>
__global__ void __launch_bounds__(kGroupThreads, 4) avgpool_bwd_kernel(FvgbGrid fine, FvgbGrid coarse, int3 pf, int3 st,
                                                                    Groups gr, int32_t C, const T *__restrict__ dy,
                                                                    int64_t lddy, T *__restrict__ dx, int64_t lddx,
                                                                    double avg) {
    using A = typename Num<T>::Acc;
    extern __shared__ int32_t widx[];
    const int G = 1 << gr.gs, group = threadIdx.x >> gr.gs, lane = threadIdx.x & (G - 1);
    int32_t *idx = widx + group * gr.W;
    auto fdiv = [](int32_t a, int32_t b) { return a >= 0 ? a / b : -((-a + b - 1) / b); };
    const int64_t f = (int64_t)blockIdx.x * (kGroupThreads >> gr.gs) + group;
    const bool on = f < fine.num_voxels;
    int32_t b = 0;
    int3 lo = make_int3(0, 0, 0), ext = make_int3(0, 0, 0);
    if (on) {
        b = batch_of(fine.voxel_offsets, fine.num_grids, f);
        const int32_t fx = fine.ijk[3 * f], fy = fine.ijk[3 * f + 1], fz = fine.ijk[3 * f + 2];
        // candidate coarse range per axis: [ceil((f - p + 1) / s), floor(f / s)]
        lo = make_int3(-fdiv(-(fx - pf.x + 1), st.x), -fdiv(-(fy - pf.y + 1), st.y), -fdiv(-(fz - pf.z + 1), st.z));
        const int3 hi = make_int3(fdiv(fx, st.x), fdiv(fy, st.y), fdiv(fz, st.z));
        ext = make_int3(max(hi.x - lo.x + 1, 0), max(hi.y - lo.y + 1, 0), max(hi.z - lo.z + 1, 0));
    }
    const int W = ext.x * ext.y * ext.z;  // <= gr.W
    window_indices(coarse, b, lo, ext, idx, lane, G);
    if (!on) return;
    for (int32_t ch = lane * V; ch < C; ch += G * V) {
        bool any = false;
        A acc[V];
#pragma unroll
        for (int e = 0; e < V; ++e) acc[e] = (A)0;
        for (int w = 0; w < W; ++w) {
            const int32_t c = idx[w];
            if (c < 0) continue;
            const Elems<T, V> p = unpack<T, V>(ld_raw<T, V>(dy + (int64_t)c * lddy + ch));
#pragma unroll
            for (int e = 0; e < V; ++e) {
                const A g = Num<T>::to(mul_in<T>(p.v[e], avg));
                acc[e] = any ? acc[e] + g : g;
            }
            any = true;
        }
        Elems<T, V> o;
#pragma unroll
        for (int e = 0; e < V; ++e) o.v[e] = Num<T>::from(acc[e]);
        st_vec<T, V>(dx + f * lddx + ch, o);
    }
}

// Nearest upsampling: fine voxel f copies coarse voxel floor(f / factor) (zero without one).  A warp
// takes 32 consecutive fine voxels: each lane looks up one parent, then the warp's lane groups copy
// the rows.
template <typename T, int V>
__global__ void __launch_bounds__(kGroupThreads, 4) upsample_fwd_kernel(FvgbGrid coarse, FvgbGrid fine, int3 fac, int gs,
                                                                     const T *__restrict__ x, int64_t ldx, int32_t C,
                                                                     T *__restrict__ y, int64_t ldy) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int G = 1 << gs, sub = lane >> gs, gl = lane & (G - 1), per = 32 >> gs;
    auto fdiv = [](int32_t a, int32_t b) { return a >= 0 ? a / b : -((-a + b - 1) / b); };
    const int64_t f0 = ((int64_t)blockIdx.x * (kGroupThreads / 32) + warp) * 32;
    if (f0 >= fine.num_voxels) return;  // warp-uniform
    int32_t c = -1;
    const int64_t fl = f0 + lane;
    if (fl < fine.num_voxels) {
        const int32_t b = batch_of(fine.voxel_offsets, fine.num_grids, fl);
        c = (int32_t)voxel_at(coarse, b, fdiv(fine.ijk[3 * fl], fac.x), fdiv(fine.ijk[3 * fl + 1], fac.y),
                              fdiv(fine.ijk[3 * fl + 2], fac.z));
    }
    for (int i0 = 0; i0 < G; i0 += kUpAhead) {  // G = 32 / per rounds of `per` voxels, kUpAhead at a time
        int32_t p[kUpAhead];
#pragma unroll
        for (int u = 0; u < kUpAhead; ++u) p[u] = __shfl_sync(0xffffffffu, c, ((i0 + u) * per + sub) & 31);
        for (int32_t ch = gl * V; ch < C; ch += G * V) {
            Raw<T, V> o[kUpAhead];  // copied as bytes; zero is all zero bits in every type
#pragma unroll
            for (int u = 0; u < kUpAhead; ++u) {
                o[u] = Raw<T, V>{};
                if (p[u] >= 0 && i0 + u < G) o[u] = ld_raw<T, V>(x + (int64_t)p[u] * ldx + ch);
            }
#pragma unroll
            for (int u = 0; u < kUpAhead; ++u) {
                const int64_t f = f0 + (i0 + u) * per + sub;
                if (i0 + u < G && f < fine.num_voxels) *reinterpret_cast<Raw<T, V> *>(y + f * ldy + ch) = o[u];
            }
        }
    }
}

// Candidates of the subdivided grid: coarse voxel c (where mask[c] != 0, or every voxel without a
// mask) yields c*factor + (i, j, k); out_valid marks the kept ones.
__global__ void subdivide_candidates_kernel(FvgbGrid coarse, int3 fac, const uint8_t *__restrict__ mask,
                                            int32_t *__restrict__ out, uint8_t *__restrict__ valid) {
    const int W = fac.x * fac.y * fac.z;
    const int64_t total = coarse.num_voxels * W;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t c = e / W;
        const int w = (int)(e % W);
        const int i = w / (fac.y * fac.z), j = (w / fac.z) % fac.y, k = w % fac.z;
        out[3 * e] = coarse.ijk[3 * c] * fac.x + i;
        out[3 * e + 1] = coarse.ijk[3 * c + 1] * fac.y + j;
        out[3 * e + 2] = coarse.ijk[3 * c + 2] * fac.z + k;
        valid[e] = mask ? (uint8_t)(mask[c] != 0) : (uint8_t)1;
    }
}

unsigned pool_blocks(int64_t items) {
    const int64_t b = ceil_div(items, kPoolWarps);
    return (unsigned)std::min<int64_t>(std::max<int64_t>(b, 1), 65535 * 16);
}

bool vec_ok(const int32_t *v, int max_volume) {
    if (!v || v[0] < 1 || v[1] < 1 || v[2] < 1) return false;
    return (int64_t)v[0] * v[1] * v[2] <= max_volume;
}

template <template <typename> class F, typename... Args>
int dispatch_dtype(int32_t dtype, Args &&...args) {
    switch (dtype) {
        case FVGB_F32: F<float>::run(args...); break;
        case FVGB_F64: F<double>::run(args...); break;
        case FVGB_F16: F<__half>::run(args...); break;
        case FVGB_BF16: F<__nv_bfloat16>::run(args...); break;
        default: return FVGB_ETYPE;
    }
    count_launches(1);
    return launch_status();
}

// The vector width of rows of C channels at the given addresses and strides: 16 bytes where every
// row is whole 16-byte pieces, else one element.
template <typename T>
bool whole_vectors(int32_t C, std::initializer_list<const void *> ptrs, std::initializer_list<int64_t> lds) {
    constexpr int V = 16 / sizeof(T);
    bool ok = C % V == 0;
    for (const void *p : ptrs) ok = ok && ((uintptr_t)p & 15) == 0;
    for (int64_t ld : lds) ok = ok && ld % V == 0;
    return ok;
}
template <int V>
using Width = std::integral_constant<int, V>;
template <typename T, typename F>
void by_width(bool vec, F &&f) {
    if (vec) f(Width<16 / sizeof(T)>());
    else f(Width<1>());
}
unsigned group_blocks(int64_t items, const Groups &g) { return (unsigned)ceil_div(items, (int64_t)(kGroupThreads >> g.gs)); }

constexpr int kPoolSum = 2;  // mode of the window sum (upsampling gradient)

// Windows over a map, or by lookups between two grids (map null).
struct Windows {
    FvgbGrid fine, coarse;
    int3 pf, st;
    const int32_t *map;
    int64_t n_coarse;
    int W;
};

template <typename T>
struct PoolFwd {
    static void run(int mode, const Windows &w, const void *x, int64_t ldx, int32_t C, void *y, int64_t ldy,
                    cudaStream_t s) {
        const double avg = 1.0 / (double)w.W;
        if (!w.map && w.W > kGroupWindow) {
            const unsigned blocks = pool_blocks(w.n_coarse);
            if (mode == FVGB_POOL_MAX)
                window_lookup_kernel<T, true, false><<<blocks, kPoolWarps * 32, 0, s>>>(w.fine, w.coarse, w.pf, w.st, (const T *)x,
                                                                                     ldx, C, (T *)y, ldy, avg);
            else if (mode == FVGB_POOL_AVG)
                window_lookup_kernel<T, false, true><<<blocks, kPoolWarps * 32, 0, s>>>(w.fine, w.coarse, w.pf, w.st, (const T *)x,
                                                                                     ldx, C, (T *)y, ldy, avg);
            else
                window_lookup_kernel<T, false, false><<<blocks, kPoolWarps * 32, 0, s>>>(w.fine, w.coarse, w.pf, w.st, (const T *)x,
                                                                                      ldx, C, (T *)y, ldy, avg);
            return;
        }
        by_width<T>(whole_vectors<T>(C, {x, y}, {ldx, ldy}), [&](auto v) {
            constexpr int V = decltype(v)::value;
            const Groups g = groups_for(C / V, w.W, !w.map);
            const unsigned blocks = group_blocks(w.n_coarse, g);
            if (mode == FVGB_POOL_MAX)
                window_reduce_kernel<T, V, true, false><<<blocks, kGroupThreads, g.smem, s>>>(
                    w.fine, w.coarse, w.pf, w.st, w.map, w.n_coarse, g, (const T *)x, ldx, C, (T *)y, ldy, avg);
            else if (mode == FVGB_POOL_AVG)
                window_reduce_kernel<T, V, false, true><<<blocks, kGroupThreads, g.smem, s>>>(
                    w.fine, w.coarse, w.pf, w.st, w.map, w.n_coarse, g, (const T *)x, ldx, C, (T *)y, ldy, avg);
            else
                window_reduce_kernel<T, V, false, false><<<blocks, kGroupThreads, g.smem, s>>>(
                    w.fine, w.coarse, w.pf, w.st, w.map, w.n_coarse, g, (const T *)x, ldx, C, (T *)y, ldy, avg);
        });
    }
};
template <typename T>
struct MaxPoolBwd {
    static void run(const FvgbGrid &f, const FvgbGrid &c, int3 pf, int3 st, const void *x, int64_t ldx, int32_t C,
                    const void *dy, int64_t lddy, void *dx_acc, cudaStream_t s) {
        maxpool_bwd_kernel<T><<<pool_blocks(c.num_voxels), kPoolWarps * 32, 0, s>>>(
            f, c, pf, st, (const T *)x, ldx, C, (const T *)dy, lddy, (typename Num<T>::Acc *)dx_acc);
    }
};
template <typename T>
struct MaxPoolBwdDisjoint {
    static void run(const int32_t *map, int64_t n_coarse, int W, const void *x, int64_t ldx, int32_t C, const void *dy,
                    int64_t lddy, void *dx, cudaStream_t s) {
        by_width<T>(whole_vectors<T>(C, {x, dy, dx}, {ldx, lddy}), [&](auto v) {
            constexpr int V = decltype(v)::value;
            const Groups g = groups_for(C / V, W);
            maxpool_bwd_disjoint_kernel<T, V><<<group_blocks(n_coarse, g), kGroupThreads, g.smem, s>>>(
                map, n_coarse, g, (const T *)x, ldx, C, (const T *)dy, lddy, (T *)dx);
        });
    }
};
template <typename T>
struct AvgPoolBwd {
    static void run(const FvgbGrid &f, const FvgbGrid &c, int3 pf, int3 st, int32_t C, const void *dy, int64_t lddy,
                    void *dx, int64_t lddx, cudaStream_t s) {
        const double avg = 1.0 / ((double)pf.x * pf.y * pf.z);
        // coarse voxels per axis whose window can hold one fine voxel
        const int W = (int)(ceil_div(pf.x, st.x) * ceil_div(pf.y, st.y) * ceil_div(pf.z, st.z));
        by_width<T>(whole_vectors<T>(C, {dy, dx}, {lddy, lddx}), [&](auto w) {
            constexpr int V = decltype(w)::value;
            const Groups g = groups_for(C / V, W, true);
            avgpool_bwd_kernel<T, V><<<group_blocks(f.num_voxels, g), kGroupThreads, g.smem, s>>>(
                f, c, pf, st, g, C, (const T *)dy, lddy, (T *)dx, lddx, avg);
        });
    }
};
template <typename T>
struct UpFwd {
    static void run(const FvgbGrid &c, const FvgbGrid &f, int3 fac, const void *x, int64_t ldx, int32_t C, void *y,
                    int64_t ldy, cudaStream_t s) {
        by_width<T>(whole_vectors<T>(C, {x, y}, {ldx, ldy}), [&](auto w) {
            constexpr int V = decltype(w)::value;
            const Groups g = groups_for(C / V, 1);
            upsample_fwd_kernel<T, V><<<(unsigned)ceil_div(f.num_voxels, kGroupThreads), kGroupThreads, 0, s>>>(
                c, f, fac, g.gs, (const T *)x, ldx, C, (T *)y, ldy);
        });
    }
};
bool grids_ok(const FvgbGrid *a, const FvgbGrid *b) {
    return a && b && a->num_grids == b->num_grids && a->num_voxels >= 0 && b->num_voxels >= 0;
}

}  // namespace
}  // namespace fvgb

using namespace fvgb;

extern "C" int fvgb_pool_forward(int32_t mode, int32_t dtype, const FvgbGrid *fine, const FvgbGrid *coarse,
                                 const int32_t pool[3], const int32_t stride[3], const void *x, int64_t ldx,
                                 int32_t C, void *y, int64_t ldy, fvgb_stream_t stream) {
    if ((mode != FVGB_POOL_MAX && mode != FVGB_POOL_AVG) || !grids_ok(fine, coarse) || !vec_ok(pool, kMaxWindow) ||
        !vec_ok(stride, 1 << 30) || C < 1 || ldx < C || ldy < C)
        return FVGB_EINVAL;
    if (coarse->num_voxels == 0) return FVGB_OK;
    if (!y || (fine->num_voxels > 0 && !x)) return FVGB_EINVAL;
    const Windows w{*fine,   *coarse, make_int3(pool[0], pool[1], pool[2]), make_int3(stride[0], stride[1], stride[2]),
                    nullptr, coarse->num_voxels, pool[0] * pool[1] * pool[2]};
    return dispatch_dtype<PoolFwd>(dtype, mode, w, x, ldx, C, y, ldy, as_stream(stream));
}

extern "C" int fvgb_maxpool_backward(int32_t dtype, const FvgbGrid *fine, const FvgbGrid *coarse, const int32_t pool[3],
                                     const int32_t stride[3], const void *x, int64_t ldx, int32_t C, const void *dy,
                                     int64_t lddy, void *dx_acc, fvgb_stream_t stream) {
    if (!grids_ok(fine, coarse) || !vec_ok(pool, kMaxWindow) || !vec_ok(stride, 1 << 30) || C < 1 || ldx < C ||
        lddy < C)
        return FVGB_EINVAL;
    if (coarse->num_voxels == 0 || fine->num_voxels == 0) return FVGB_OK;
    if (!x || !dy || !dx_acc) return FVGB_EINVAL;
    return dispatch_dtype<MaxPoolBwd>(dtype, *fine, *coarse, make_int3(pool[0], pool[1], pool[2]),
                                      make_int3(stride[0], stride[1], stride[2]), x, ldx, C, dy, lddy, dx_acc,
                                      as_stream(stream));
}

extern "C" int fvgb_pool_forward_map(int32_t mode, int32_t dtype, const int32_t *map, int64_t n_coarse, int32_t window,
                                     const void *x, int64_t ldx, int32_t C, void *y, int64_t ldy,
                                     fvgb_stream_t stream) {
    if ((mode != FVGB_POOL_MAX && mode != FVGB_POOL_AVG && mode != kPoolSum) || n_coarse < 0 || window < 1 ||
        window > kMaxWindow || C < 1 || ldx < C || ldy < C)
        return FVGB_EINVAL;
    if (n_coarse == 0) return FVGB_OK;
    if (!map || !y) return FVGB_EINVAL;
    Windows w{};
    w.map = map;
    w.n_coarse = n_coarse;
    w.W = window;
    return dispatch_dtype<PoolFwd>(dtype, mode, w, x, ldx, C, y, ldy, as_stream(stream));
}

extern "C" int fvgb_maxpool_backward_map(int32_t dtype, const int32_t *map, int64_t n_coarse, int32_t window,
                                         const void *x, int64_t ldx, int32_t C, const void *dy, int64_t lddy, void *dx,
                                         fvgb_stream_t stream) {
    if (n_coarse < 0 || window < 1 || window > kMaxWindow || C < 1 || ldx < C || lddy < C) return FVGB_EINVAL;
    if (n_coarse == 0) return FVGB_OK;
    if (!map || !x || !dy || !dx) return FVGB_EINVAL;
    return dispatch_dtype<MaxPoolBwdDisjoint>(dtype, map, n_coarse, window, x, ldx, C, dy, lddy, dx, as_stream(stream));
}

extern "C" int fvgb_avgpool_backward(int32_t dtype, const FvgbGrid *fine, const FvgbGrid *coarse, const int32_t pool[3],
                                     const int32_t stride[3], int32_t C, const void *dy, int64_t lddy, void *dx,
                                     int64_t lddx, fvgb_stream_t stream) {
    if (!grids_ok(fine, coarse) || !vec_ok(pool, kMaxWindow) || !vec_ok(stride, 1 << 30) || C < 1 || lddy < C ||
        lddx < C)
        return FVGB_EINVAL;
    if (fine->num_voxels == 0) return FVGB_OK;
    if (!dx || (coarse->num_voxels > 0 && !dy)) return FVGB_EINVAL;
    return dispatch_dtype<AvgPoolBwd>(dtype, *fine, *coarse, make_int3(pool[0], pool[1], pool[2]),
                                      make_int3(stride[0], stride[1], stride[2]), C, dy, lddy, dx, lddx,
                                      as_stream(stream));
}

extern "C" int fvgb_upsample_forward(int32_t dtype, const FvgbGrid *coarse, const FvgbGrid *fine, const int32_t factor[3],
                                     const void *x, int64_t ldx, int32_t C, void *y, int64_t ldy,
                                     fvgb_stream_t stream) {
    if (!grids_ok(fine, coarse) || !vec_ok(factor, kMaxWindow) || C < 1 || ldx < C || ldy < C) return FVGB_EINVAL;
    if (fine->num_voxels == 0) return FVGB_OK;
    if (!y || (coarse->num_voxels > 0 && !x)) return FVGB_EINVAL;
    return dispatch_dtype<UpFwd>(dtype, *coarse, *fine, make_int3(factor[0], factor[1], factor[2]), x, ldx, C, y, ldy,
                                 as_stream(stream));
}

extern "C" int fvgb_upsample_backward(int32_t dtype, const FvgbGrid *coarse, const FvgbGrid *fine,
                                      const int32_t factor[3], const void *dy, int64_t lddy, int32_t C, void *dx,
                                      int64_t lddx, fvgb_stream_t stream) {
    if (!grids_ok(fine, coarse) || !vec_ok(factor, kMaxWindow) || C < 1 || lddy < C || lddx < C) return FVGB_EINVAL;
    if (coarse->num_voxels == 0) return FVGB_OK;
    if (!dx || (fine->num_voxels > 0 && !dy)) return FVGB_EINVAL;
    const int3 f = make_int3(factor[0], factor[1], factor[2]);
    const Windows w{*fine, *coarse, f, f, nullptr, coarse->num_voxels, factor[0] * factor[1] * factor[2]};
    return dispatch_dtype<PoolFwd>(dtype, kPoolSum, w, dy, lddy, C, dx, lddx, as_stream(stream));
}

extern "C" int fvgb_subdivide_candidates(const FvgbGrid *coarse, const int32_t factor[3], const uint8_t *mask,
                                         int32_t *out_ijk, uint8_t *out_valid, fvgb_stream_t stream) {
    if (!coarse || !vec_ok(factor, kMaxWindow)) return FVGB_EINVAL;
    const int64_t total = coarse->num_voxels * factor[0] * factor[1] * factor[2];
    if (total == 0) return FVGB_OK;
    if (!out_ijk || !out_valid) return FVGB_EINVAL;
    const unsigned blocks = (unsigned)std::min<int64_t>(ceil_div(total, 256), 65535 * 16);
    subdivide_candidates_kernel<<<blocks, 256, 0, as_stream(stream)>>>(*coarse, make_int3(factor[0], factor[1], factor[2]),
                                                                      mask, out_ijk, out_valid);
    count_launches(1);
    return launch_status();
}
