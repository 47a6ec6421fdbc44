// Device grid builder: jagged ijk -> sorted unique voxels in NanoVDB order -> leaf table
// + leaf hash.  No host synchronisation inside any entry point; sizes that the caller
// must allocate from (unique count, leaf count) are left in device memory.
//
// Reference behaviour replaced: dispatchCreateNanoGridFromIJK<kCUDA>
// (src/fvdb/detail/ops/BuildGridFromIjk.cu:26-83), which loops over the grids on the
// host and calls nanovdb::tools::cuda::voxelsToGrid per grid.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <cub/cub.cuh>
#include <type_traits>

#include "common.cuh"

namespace fvgb {
namespace {

struct SortWs {
    uint64_t *keys_a, *keys_b;
    int32_t *bidx_a, *bidx_b;
    int32_t *flags;  // n+1
    void *cub_tmp;
    size_t cub_bytes;
};

inline size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

size_t cub_sort_bytes(int64_t n) {
    size_t a = 0, b = 0, c = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, a, (uint64_t *)nullptr, (uint64_t *)nullptr,
                                    (int32_t *)nullptr, (int32_t *)nullptr, n, 0, 63);
    cub::DeviceRadixSort::SortPairs(nullptr, b, (int32_t *)nullptr, (int32_t *)nullptr,
                                    (uint64_t *)nullptr, (uint64_t *)nullptr, n, 0, 32);
    cub::DeviceScan::ExclusiveSum(nullptr, c, (int32_t *)nullptr, (int32_t *)nullptr, n + 1);
    size_t m = a > b ? a : b;
    return m > c ? m : c;
}

size_t sort_ws_layout(int64_t n, SortWs *ws, char *base) {
    size_t off = 0;
    const size_t nn = (size_t)(n > 0 ? n : 1);
    auto take = [&](size_t bytes) {
        char *p = base ? base + off : nullptr;
        off = align_up(off + bytes, 256);
        return p;
    };
    SortWs w;
    w.keys_a = (uint64_t *)take(nn * 8);
    w.keys_b = (uint64_t *)take(nn * 8);
    w.bidx_a = (int32_t *)take(nn * 4);
    w.bidx_b = (int32_t *)take(nn * 4);
    w.flags = (int32_t *)take((nn + 1) * 4);
    w.cub_bytes = cub_sort_bytes(n);
    w.cub_tmp = take(w.cub_bytes);
    if (ws) *ws = w;
    return off;
}

// box_lo/box_hi: bounds every coordinate must lie in (the whole coordinate range when the
// caller promises none); a coordinate outside raises FVGB_ERANGE.
// fold > 0: every key agrees above bit `fold` (coordinates inside a box), so the grid index
// replaces those bits and one radix sort orders by (grid, key).
__global__ void keys_kernel(const int32_t *__restrict__ ijk, const int64_t *__restrict__ joff,
                            int32_t B, int64_t n, int3 box_lo, int3 box_hi, int32_t fold,
                            uint64_t *__restrict__ keys, int32_t *__restrict__ bidx, int32_t *__restrict__ err) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int32_t x = ijk[3 * i], y = ijk[3 * i + 1], z = ijk[3 * i + 2];
    if (!coord_in_range(x) || !coord_in_range(y) || !coord_in_range(z) || x < box_lo.x || x > box_hi.x ||
        y < box_lo.y || y > box_hi.y || z < box_lo.z || z > box_hi.z)
        atomicExch(err, FVGB_ERANGE);
    const int32_t b = batch_of(joff, B, i);
    uint64_t k = order_key(x, y, z);
    if (fold > 0) k = (k & ((1ull << fold) - 1ull)) | ((uint64_t)b << fold);
    keys[i] = k;
    bidx[i] = b;
}

// One past the highest order_key bit that can differ between coordinates in [lo, hi] (per
// axis): coordinate bits above the highest bit where lo and hi differ are shared by the whole
// box.  Coordinate bit c of x lands on key bit 6+c (leaf), 14+c (lower node), 24+c (upper node)
// or 42+c (root); y sits 3, 4, 5 or 9 positions below x in those fields and z twice as far.
// Within an axis a higher coordinate bit always maps to a higher key bit, so all keys of the
// box agree above the returned bit and sorting only the bits below it orders them exactly as a
// full 63-bit sort.
int order_key_end_bit(const int32_t lo[3], const int32_t hi[3]) {
    static const int kBase[3] = {6, 3, 0};  // x, y, z offset of the leaf field
    int end = 1;
    for (int a = 0; a < 3; ++a) {
        if (lo[a] > hi[a]) continue;
        const uint32_t d = (uint32_t)lo[a] ^ (uint32_t)hi[a];
        if (!d) continue;
        int h = 31;
        while (!((d >> h) & 1u)) --h;
        int kb;
        if (h < 3)
            kb = kBase[a] + h;                    // leaf: bits 0..8
        else if (h < 7)
            kb = 9 + 4 * (2 - a) + (h - 3);       // lower node: x 17..20, y 13..16, z 9..12
        else if (h < 12)
            kb = 21 + 5 * (2 - a) + (h - 7);      // upper node: x 31..35, y 26..30, z 21..25
        else if (h < 21)
            kb = 36 + 9 * (2 - a) + (h - 12);     // root: x 54..62, y 45..53, z 36..44
        else
            return 63;
        if (kb + 1 > end) end = kb + 1;
    }
    return end;
}

__global__ void unique_flags_kernel(const uint64_t *__restrict__ keys,
                                    const int32_t *__restrict__ bidx, int64_t n,
                                    int32_t *__restrict__ flags) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i > n) return;
    if (i == n) { flags[i] = 0; return; }
    flags[i] = (i == 0 || keys[i] != keys[i - 1] || bidx[i] != bidx[i - 1]) ? 1 : 0;
}

// low_mask / high: a folded key keeps the order key's bits under low_mask; the bits above are
// `high` for every voxel (no folding: low_mask all ones, high zero).
__global__ void unique_write_kernel(const uint64_t *__restrict__ keys,
                                    const int32_t *__restrict__ bidx,
                                    const int32_t *__restrict__ pos, int64_t n, uint64_t low_mask,
                                    uint64_t high, int32_t *__restrict__ out_ijk) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const bool first = (i == 0 || keys[i] != keys[i - 1] || bidx[i] != bidx[i - 1]);
    if (!first) return;
    int32_t x, y, z;
    key_to_coord((keys[i] & low_mask) | high, x, y, z);
    const int64_t p = pos[i];
    out_ijk[3 * p] = x;
    out_ijk[3 * p + 1] = y;
    out_ijk[3 * p + 2] = z;
}

// out_joff[b] = number of unique voxels in grids < b  (bidx sorted ascending)
__global__ void offsets_kernel(const int32_t *__restrict__ bidx, const int32_t *__restrict__ pos,
                               int64_t n, int32_t B, int64_t *__restrict__ out_joff) {
    const int32_t b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b > B) return;
    int64_t lo = 0, hi = n;  // first i with bidx[i] >= b
    while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        if (bidx[mid] < b) lo = mid + 1; else hi = mid;
    }
    out_joff[b] = pos[lo];  // pos has n+1 entries; pos[n] = total
}

__global__ void leaf_flags_kernel(const int32_t *__restrict__ ijk, const int64_t *__restrict__ joff,
                                  int32_t B, int64_t n, int32_t *__restrict__ flags) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (i >= joff[B]) {  // n is a capacity; the voxel count lives on the device
        flags[i] = 0;
        return;
    }
    int32_t f = 1;
    if (i > 0) {
        const int32_t b0 = batch_of(joff, B, i - 1), b1 = batch_of(joff, B, i);
        f = (b0 != b1 || (ijk[3 * i] >> 3) != (ijk[3 * i - 3] >> 3) ||
             (ijk[3 * i + 1] >> 3) != (ijk[3 * i - 2] >> 3) ||
             (ijk[3 * i + 2] >> 3) != (ijk[3 * i - 1] >> 3)) ? 1 : 0;
    }
    flags[i] = f;
}

__global__ void leaf_count_kernel(const int32_t *__restrict__ ids, const int64_t *__restrict__ joff, int32_t B,
                                  int64_t *__restrict__ out) {
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    const int64_t n = joff[B];
    out[0] = n > 0 ? (int64_t)ids[n - 1] : 0;  // inclusive scan
    out[1] = n;
}

__global__ void leaf_fill_kernel(const int32_t *__restrict__ ijk, const int64_t *__restrict__ joff,
                                 int32_t B, int64_t n, const int32_t *__restrict__ leaf_ids,
                                 FvgbLeaf *__restrict__ leaves) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int32_t id = leaf_ids[i] - 1;  // inclusive scan
    const int32_t x = ijk[3 * i], y = ijk[3 * i + 1], z = ijk[3 * i + 2];
    FvgbLeaf &L = leaves[id];
    const bool first = (i == 0) || leaf_ids[i - 1] != leaf_ids[i];
    if (first) {
        L.origin[0] = x & ~7;
        L.origin[1] = y & ~7;
        L.origin[2] = z & ~7;
        L.batch = batch_of(joff, B, i);
        L.base = i;
    }
    const uint32_t bit = leaf_bit(x, y, z);
    atomicOr(reinterpret_cast<unsigned long long *>(&L.mask[bit >> 6]), 1ull << (bit & 63));
}

__global__ void leaf_finish_kernel(FvgbLeaf *__restrict__ leaves, int64_t L, int32_t *__restrict__ slots,
                                   int64_t cap) {
    const int64_t id = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= L) return;
    FvgbLeaf &lf = leaves[id];
    uint32_t run = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
        lf.prefix[w] = (uint16_t)run;
        run += __popcll(lf.mask[w]);
    }
    const uint64_t cap_mask = (uint64_t)cap - 1;
    uint64_t h = leaf_hash(lf.batch, lf.origin[0] >> 3, lf.origin[1] >> 3, lf.origin[2] >> 3) & cap_mask;
    for (int64_t probe = 0; probe < cap; ++probe) {
        const int32_t prev = atomicCAS(slots + h, -1, (int32_t)id);
        if (prev == -1) break;
        h = (h + 1) & cap_mask;
    }
}

// One coordinate of VoxelCoordTransform(1/w, -o/w).apply(p).round() in the arithmetic type T
// that the reference uses for the points' dtype (opmath: double for FP64 points, float for
// FP32/FP16/BF16): scale and translation are the double quotients rounded once to T, the
// transform is one fused multiply-add in T, and round() is floor(v + 1/2) in T
// (src/fvdb/detail/VoxelCoordTransform.h:86-110,230-330, BuildGridFromPoints.cu:27-43).
__device__ __forceinline__ int32_t voxelise(float p, float s, float t) {
    return (int32_t)floorf(__fadd_rn(__fmaf_rn(p, s, t), 0.5f));
}
__device__ __forceinline__ int32_t voxelise(double p, double s, double t) {
    return (int32_t)floor(__dadd_rn(__fma_rn(p, s, t), 0.5));
}

template <typename P>
__device__ __forceinline__ float point_as_float(P v) { return (float)v; }
template <>
__device__ __forceinline__ float point_as_float<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <>
__device__ __forceinline__ float point_as_float<__half>(__half v) { return __half2float(v); }

// P: storage type of the points; T: arithmetic type (double for FP64 points, else float).
template <typename T, typename P>
__device__ __forceinline__ T point_value(P v) {
    if constexpr (sizeof(T) == 8) return (T)v;
    else return point_as_float<P>(v);
}

// The scale and translation of the block's first grid are divided out once per block (FP64
// divisions: per point and axis they took 1.18 ms for 7.9M points, 30 times what the bytes take).
// A block that spans several grids divides for each row of the others.
constexpr int kPointRows = 8;  // points per thread

template <typename P, typename T>
__global__ void __launch_bounds__(256) points_kernel(const P *__restrict__ pts, const int64_t *__restrict__ joff,
                                                     int32_t B, int64_t n, const double *__restrict__ vs,
                                                     const double *__restrict__ org, int32_t *__restrict__ out) {
    __shared__ T fac[6];
    __shared__ int32_t sb[2];
    const int64_t base = (int64_t)blockIdx.x * 256 * kPointRows;
    const int64_t last = min(n, base + 256 * kPointRows) - 1;
    if (threadIdx.x < 2) sb[threadIdx.x] = batch_of(joff, B, threadIdx.x == 0 ? base : last);
    __syncthreads();
    if (threadIdx.x < 3) {
        const double w = vs[3 * sb[0] + threadIdx.x], o = org[3 * sb[0] + threadIdx.x];
        fac[threadIdx.x] = (T)(1.0 / w);
        fac[3 + threadIdx.x] = (T)(-o / w);
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kPointRows; ++q) {
        const int64_t i = base + q * 256 + threadIdx.x;
        if (i > last) return;
        const int32_t b = sb[0] == sb[1] ? sb[0] : batch_of(joff, B, i);
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            T s = fac[a], t = fac[3 + a];
            if (b != sb[0]) {
                const double w = vs[3 * b + a], o = org[3 * b + a];
                s = (T)(1.0 / w);
                t = (T)(-o / w);
            }
            out[3 * i + a] = voxelise(point_value<T>(pts[3 * i + a]), s, t);
        }
    }
}

__global__ void conv_candidates_kernel(FvgbGrid g, int3 ks, int3 st, int coarse, int32_t kc,
                                       int32_t *__restrict__ out, uint8_t *__restrict__ valid) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= g.num_voxels) return;
    const int32_t x = g.ijk[3 * i], y = g.ijk[3 * i + 1], z = g.ijk[3 * i + 2];
    if (coarse) {
        // floor(ijk / stride) with the stride Coord applied x<->s0 (CoarseIjkForFineGrid.cu:34-35),
        // in integer arithmetic (exact for int32 inputs; avoids FP64 on the device)
        auto fdiv = [](int32_t a, int32_t b) { return a >= 0 ? a / b : -((-a + b - 1) / b); };
        out[3 * i] = fdiv(x, st.x);
        out[3 * i + 1] = fdiv(y, st.y);
        out[3 * i + 2] = fdiv(z, st.z);
        valid[i] = 1;
        return;
    }
    const int lo0 = (ks.x % 2 == 0) ? 0 : -(ks.x - 1) / 2, hi0 = (ks.x % 2 == 0) ? ks.x - 1 : (ks.x - 1) / 2;
    const int lo1 = (ks.y % 2 == 0) ? 0 : -(ks.y - 1) / 2, hi1 = (ks.y % 2 == 0) ? ks.y - 1 : (ks.y - 1) / 2;
    const int lo2 = (ks.z % 2 == 0) ? 0 : -(ks.z - 1) / 2, hi2 = (ks.z % 2 == 0) ? ks.z - 1 : (ks.z - 1) / 2;
    int64_t c = i * kc;
    // BuildGridForConv.cu:99-121: di over k0 moves z, dk over k2 moves x; C remainder
    for (int di = lo0; di <= hi0; ++di)
        for (int dj = lo1; dj <= hi1; ++dj)
            for (int dk = lo2; dk <= hi2; ++dk, ++c) {
                const int32_t dx = x + dk, dy = y + dj, dz = z + di;
                const bool ok = (dx % st.z == 0) && (dy % st.y == 0) && (dz % st.x == 0);
                valid[c] = ok ? 1 : 0;
                out[3 * c] = ok ? dx / st.z : 0;
                out[3 * c + 1] = ok ? dy / st.y : 0;
                out[3 * c + 2] = ok ? dz / st.x : 0;
            }
}

__global__ void compact_flags_kernel(const uint8_t *__restrict__ valid, int64_t n, int32_t *__restrict__ f) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i > n) return;
    f[i] = (i < n && valid[i]) ? 1 : 0;
}

__global__ void compact_write_kernel(const int32_t *__restrict__ ijk, const uint8_t *__restrict__ valid,
                                     const int32_t *__restrict__ pos, int64_t n, int32_t *__restrict__ out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || !valid[i]) return;
    const int64_t p = pos[i];
    out[3 * p] = ijk[3 * i];
    out[3 * p + 1] = ijk[3 * i + 1];
    out[3 * p + 2] = ijk[3 * i + 2];
}

__global__ void compact_offsets_kernel(const int64_t *__restrict__ src_joff, int32_t B, int64_t per,
                                       const int32_t *__restrict__ pos, int64_t *__restrict__ out) {
    const int32_t b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b > B) return;
    out[b] = pos[src_joff[b] * per];
}

// Writes leaf p of the index order (its grid b, origin and first voxel; `word` = mask word lane / 4 of a
// converged warp): its voxels in bit order, its table entry and its hash slot.
__device__ __forceinline__ void emit_leaf(uint64_t word, int32_t ox, int32_t oy, int32_t oz, int32_t b, int32_t base,
                                          int64_t p, int lane, int32_t *out_ijk, FvgbLeaf *leaves, int32_t *slots,
                                          int64_t cap) {
    const int w = lane >> 2, sub = (lane & 3) * 16;
    // exclusive prefix of the words' populations, the same for the four lanes of a word
    int pre = 0;
#pragma unroll
    for (int v = 0; v < 7; ++v) {
        const int c = __popcll(__shfl_sync(0xffffffffu, word, v * 4));
        if (v < w) pre += c;
    }
    FvgbLeaf &lf = leaves[p];
    if ((lane & 3) == 0) {
        lf.mask[w] = word;
        lf.prefix[w] = (uint16_t)pre;
    }
    if (lane < 3) {
        lf.origin[lane] = lane == 0 ? ox : (lane == 1 ? oy : oz);
        lf.pad[lane] = 0;
    }
    if (lane == 0) {
        lf.batch = b;
        lf.base = base;
        const uint64_t cap_mask = (uint64_t)cap - 1;
        uint64_t s = leaf_hash(b, ox >> 3, oy >> 3, oz >> 3) & cap_mask;
        for (int64_t probe = 0; probe < cap; ++probe) {
            if (atomicCAS(slots + s, -1, (int32_t)p) == -1) break;
            s = (s + 1) & cap_mask;
        }
    }
    int64_t r = (int64_t)base + pre + __popcll(sub ? (word & ((1ull << sub) - 1ull)) : 0ull);
    uint32_t bits = (uint32_t)(word >> sub) & 0xffffu;
    while (bits) {
        const int i = w * 64 + sub + __ffs(bits) - 1;
        bits &= bits - 1;
        out_ijk[3 * r] = ox + (i >> 6);
        out_ijk[3 * r + 1] = oy + ((i >> 3) & 7);
        out_ijk[3 * r + 2] = oz + (i & 7);
        ++r;
    }
}

constexpr int kThreads = 256;
inline unsigned blocks_for(int64_t n) { return (unsigned)ceil_div(n > 0 ? n : 1, kThreads); }

}  // namespace
}  // namespace fvgb

using namespace fvgb;

extern "C" int fvgb_ijk_sort_unique_workspace(int64_t n, int32_t num_grids, size_t *bytes) {
    if (!bytes || n < 0 || num_grids < 1) return FVGB_EINVAL;
    *bytes = sort_ws_layout(n, nullptr, nullptr) + 256;
    return FVGB_OK;
}

namespace fvgb {
namespace {
int sort_unique(const int32_t *ijk, const int64_t *joffsets, int32_t num_grids, int64_t n, const int32_t *box_lo,
                const int32_t *box_hi, int32_t *out_ijk, int64_t *out_joffsets, int32_t *err_dev, void *workspace,
                size_t workspace_bytes, fvgb_stream_t stream) {
    if (n < 0 || num_grids < 1 || !joffsets || !out_joffsets || !err_dev) return FVGB_EINVAL;
    if (n > 0 && (!ijk || !out_ijk)) return FVGB_EINVAL;
    if (n >= (int64_t)INT32_MAX) return FVGB_EINVAL;
    cudaStream_t s = as_stream(stream);
    char *base = reinterpret_cast<char *>(((uintptr_t)workspace + 255) & ~(uintptr_t)255);
    SortWs w;
    const size_t need = sort_ws_layout(n, &w, base);
    if (!workspace || need + 256 > workspace_bytes) return FVGB_ENOSPACE;
    if (n == 0) {
        if (cudaMemsetAsync(out_joffsets, 0, sizeof(int64_t) * (num_grids + 1), s) != cudaSuccess)
            return launch_status();
        return launch_status();
    }
    int3 lo = make_int3(INT32_MIN, INT32_MIN, INT32_MIN), hi = make_int3(INT32_MAX, INT32_MAX, INT32_MAX);
    int end_bit = 63;
    if (box_lo && box_hi) {
        for (int a = 0; a < 3; ++a)
            if (box_lo[a] > box_hi[a]) return FVGB_EINVAL;
        lo = make_int3(box_lo[0], box_lo[1], box_lo[2]);
        hi = make_int3(box_hi[0], box_hi[1], box_hi[2]);
        end_bit = order_key_end_bit(box_lo, box_hi);
    }
    int grid_bits = 0;
    while ((1ll << grid_bits) < num_grids) ++grid_bits;
    // inside a box the keys agree above end_bit: the grid index takes those bits (one sort)
    const int fold = (box_lo && box_hi && num_grids > 1 && end_bit + grid_bits <= 63) ? end_bit : 0;
    uint64_t low_mask = ~0ull, high = 0;
    if (fold) {
        low_mask = (1ull << fold) - 1ull;
        high = order_key(box_lo[0], box_lo[1], box_lo[2]) & ~low_mask;
    }
    keys_kernel<<<blocks_for(n), kThreads, 0, s>>>(ijk, joffsets, num_grids, n, lo, hi, fold, w.keys_a, w.bidx_a,
                                                   err_dev);
    size_t tb = w.cub_bytes;
    // 1) sort by voxel key (stable radix, only the bits that can differ), 2) stable sort by grid
    //    index -- or one sort when the grid index is folded into the key: grids stay contiguous
    //    and every grid's voxels stay in key order.
    cub::DeviceRadixSort::SortPairs(w.cub_tmp, tb, w.keys_a, w.keys_b, w.bidx_a, w.bidx_b, n, 0,
                                    fold ? fold + grid_bits : end_bit, s);
    const uint64_t *keys = w.keys_b;
    const int32_t *bidx = w.bidx_b;
    if (num_grids > 1 && !fold) {
        tb = w.cub_bytes;
        cub::DeviceRadixSort::SortPairs(w.cub_tmp, tb, w.bidx_b, w.bidx_a, w.keys_b, w.keys_a, n, 0, grid_bits, s);
        keys = w.keys_a;
        bidx = w.bidx_a;
    }
    unique_flags_kernel<<<blocks_for(n + 1), kThreads, 0, s>>>(keys, bidx, n, w.flags);
    tb = w.cub_bytes;
    // exclusive scan in place over n+1 flags: pos[n] = unique count
    int32_t *pos = reinterpret_cast<int32_t *>(w.keys_a == keys ? (void *)w.keys_b : (void *)w.keys_a);
    cub::DeviceScan::ExclusiveSum(w.cub_tmp, tb, w.flags, pos, n + 1, s);
    unique_write_kernel<<<blocks_for(n), kThreads, 0, s>>>(keys, bidx, pos, n, low_mask, high, out_ijk);
    offsets_kernel<<<(unsigned)ceil_div(num_grids + 1, kThreads), kThreads, 0, s>>>(bidx, pos, n, num_grids,
                                                                                    out_joffsets);
    count_launches(4);
    return launch_status();
}
}  // namespace
}  // namespace fvgb

extern "C" int fvgb_ijk_sort_unique(const int32_t *ijk, const int64_t *joffsets, int32_t num_grids,
                                    int64_t n, int32_t *out_ijk, int64_t *out_joffsets,
                                    int32_t *err_dev, void *workspace, size_t workspace_bytes,
                                    fvgb_stream_t stream) {
    return fvgb::sort_unique(ijk, joffsets, num_grids, n, nullptr, nullptr, out_ijk, out_joffsets, err_dev,
                             workspace, workspace_bytes, stream);
}

extern "C" int fvgb_ijk_sort_unique_in_box(const int32_t *ijk, const int64_t *joffsets, int32_t num_grids,
                                           int64_t n, const int32_t *box_lo, const int32_t *box_hi,
                                           int32_t *out_ijk, int64_t *out_joffsets, int32_t *err_dev,
                                           void *workspace, size_t workspace_bytes, fvgb_stream_t stream) {
    if (!box_lo || !box_hi) return FVGB_EINVAL;
    return fvgb::sort_unique(ijk, joffsets, num_grids, n, box_lo, box_hi, out_ijk, out_joffsets, err_dev,
                             workspace, workspace_bytes, stream);
}

extern "C" int fvgb_scan_workspace(int64_t n, size_t *bytes) {
    if (!bytes || n < 0) return FVGB_EINVAL;
    size_t c = 0;
    cub::DeviceScan::InclusiveSum(nullptr, c, (int32_t *)nullptr, (int32_t *)nullptr, n + 1);
    size_t c2 = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, c2, (int32_t *)nullptr, (int32_t *)nullptr, n + 1);
    if (c2 > c) c = c2;
    *bytes = c + (size_t)(n + 2) * 4 + 512;
    return FVGB_OK;
}

extern "C" int fvgb_grid_leaf_scan(const int32_t *ijk, const int64_t *joffsets, int32_t num_grids,
                                   int64_t n, int32_t *leaf_ids, int64_t *num_leaves_dev,
                                   void *workspace, size_t workspace_bytes, fvgb_stream_t stream) {
    if (n < 0 || num_grids < 1 || !num_leaves_dev || (n > 0 && (!ijk || !leaf_ids))) return FVGB_EINVAL;
    size_t need = 0;
    fvgb_scan_workspace(n, &need);
    if (!workspace || workspace_bytes < need) return FVGB_ENOSPACE;
    cudaStream_t s = as_stream(stream);
    char *base = reinterpret_cast<char *>(((uintptr_t)workspace + 255) & ~(uintptr_t)255);
    int32_t *flags = reinterpret_cast<int32_t *>(base);
    void *tmp = base + ((size_t)(n + 2) * 4 + 255) / 256 * 256;
    size_t tb = need - ((size_t)(n + 2) * 4 + 255) / 256 * 256 - 256;
    if (n > 0) {
        leaf_flags_kernel<<<blocks_for(n), kThreads, 0, s>>>(ijk, joffsets, num_grids, n, flags);
        cub::DeviceScan::InclusiveSum(tmp, tb, flags, leaf_ids, n, s);
    }
    leaf_count_kernel<<<1, 32, 0, s>>>(leaf_ids, joffsets, num_grids, num_leaves_dev);
    count_launches(n > 0 ? 2 : 1);
    return launch_status();
}

extern "C" int fvgb_grid_index_build(const FvgbGrid *g, const int32_t *leaf_ids, fvgb_stream_t stream) {
    if (!g || g->num_voxels < 0 || g->num_leaves < 0) return FVGB_EINVAL;
    if (g->hash_capacity < 2 * g->num_leaves || (g->hash_capacity & (g->hash_capacity - 1)) != 0)
        return FVGB_EINVAL;
    cudaStream_t s = as_stream(stream);
    FvgbLeaf *leaves = const_cast<FvgbLeaf *>(g->leaves);
    int32_t *slots = const_cast<int32_t *>(g->hash_slots);
    if (g->hash_capacity > 0 && cudaMemsetAsync(slots, 0xff, sizeof(int32_t) * g->hash_capacity, s) != cudaSuccess)
        return launch_status();
    if (g->num_leaves > 0 && cudaMemsetAsync(leaves, 0, sizeof(FvgbLeaf) * g->num_leaves, s) != cudaSuccess)
        return launch_status();
    if (g->num_voxels > 0) {
        leaf_fill_kernel<<<blocks_for(g->num_voxels), kThreads, 0, s>>>(g->ijk, g->voxel_offsets, g->num_grids,
                                                                       g->num_voxels, leaf_ids, leaves);
        leaf_finish_kernel<<<blocks_for(g->num_leaves), kThreads, 0, s>>>(leaves, g->num_leaves, slots,
                                                                         g->hash_capacity);
        count_launches(2);
    }
    return launch_status();
}

extern "C" int fvgb_points_to_ijk(int32_t dtype, const void *points, const int64_t *joffsets, int32_t num_grids,
                                  int64_t n, const double *voxel_sizes, const double *origins,
                                  int32_t *out_ijk, fvgb_stream_t stream) {
    if (dtype != FVGB_F32 && dtype != FVGB_F64 && dtype != FVGB_F16 && dtype != FVGB_BF16) return FVGB_ETYPE;
    if (n < 0 || num_grids < 1 || (n > 0 && (!points || !out_ijk || !voxel_sizes || !origins || !joffsets)))
        return FVGB_EINVAL;
    if (n == 0) return FVGB_OK;
    cudaStream_t s = as_stream(stream);
    const unsigned blocks = (unsigned)ceil_div(n, (int64_t)kThreads * kPointRows);
    switch (dtype) {
        case FVGB_F64:
            points_kernel<double, double><<<blocks, kThreads, 0, s>>>((const double *)points, joffsets, num_grids, n,
                                                                      voxel_sizes, origins, out_ijk);
            break;
        case FVGB_F16:
            points_kernel<__half, float><<<blocks, kThreads, 0, s>>>((const __half *)points, joffsets, num_grids, n,
                                                                     voxel_sizes, origins, out_ijk);
            break;
        case FVGB_BF16:
            points_kernel<__nv_bfloat16, float><<<blocks, kThreads, 0, s>>>(
                (const __nv_bfloat16 *)points, joffsets, num_grids, n, voxel_sizes, origins, out_ijk);
            break;
        default:
            points_kernel<float, float><<<blocks, kThreads, 0, s>>>((const float *)points, joffsets, num_grids, n,
                                                                    voxel_sizes, origins, out_ijk);
    }
    count_launches(1);
    return launch_status();
}

extern "C" int fvgb_conv_grid_candidates(const FvgbGrid *g, const int32_t ksize[3], const int32_t stride[3],
                                         int32_t *out_ijk, uint8_t *out_valid, fvgb_stream_t stream) {
    if (!g || !ksize || !stride) return FVGB_EINVAL;
    for (int a = 0; a < 3; ++a)
        if (ksize[a] < 1 || stride[a] < 1) return FVGB_EINVAL;
    if (g->num_voxels == 0) return FVGB_OK;
    const int coarse = (stride[0] == 1 && stride[1] == 1 && stride[2] == 1) ||
                       (stride[0] == ksize[0] && stride[1] == ksize[1] && stride[2] == ksize[2]);
    const int32_t kc = coarse ? 1 : ksize[0] * ksize[1] * ksize[2];
    conv_candidates_kernel<<<blocks_for(g->num_voxels), kThreads, 0, as_stream(stream)>>>(
        *g, make_int3(ksize[0], ksize[1], ksize[2]), make_int3(stride[0], stride[1], stride[2]), coarse, kc,
        out_ijk, out_valid);
    count_launches(1);
    return launch_status();
}

extern "C" int fvgb_compact_ijk(const int32_t *ijk, const uint8_t *valid, const int64_t *src_joffsets,
                                int32_t num_grids, int64_t per_voxel, int64_t n, int32_t *out_ijk,
                                int64_t *out_joffsets, void *workspace, size_t workspace_bytes,
                                fvgb_stream_t stream) {
    if (n < 0 || num_grids < 1 || per_voxel < 1 || !src_joffsets || !out_joffsets) return FVGB_EINVAL;
    size_t need = 0;
    fvgb_scan_workspace(n, &need);
    if (!workspace || workspace_bytes < need) return FVGB_ENOSPACE;
    cudaStream_t s = as_stream(stream);
    char *base = reinterpret_cast<char *>(((uintptr_t)workspace + 255) & ~(uintptr_t)255);
    int32_t *flags = reinterpret_cast<int32_t *>(base);
    const size_t head = ((size_t)(n + 2) * 4 + 255) / 256 * 256;
    void *tmp = base + head;
    size_t tb = need - head - 256;
    compact_flags_kernel<<<blocks_for(n + 1), kThreads, 0, s>>>(valid, n, flags);
    cub::DeviceScan::ExclusiveSum(tmp, tb, flags, flags, n + 1, s);  // in place: flags -> positions
    compact_write_kernel<<<blocks_for(n), kThreads, 0, s>>>(ijk, valid, flags, n, out_ijk);
    compact_offsets_kernel<<<(unsigned)ceil_div(num_grids + 1, kThreads), kThreads, 0, s>>>(
        src_joffsets, num_grids, per_voxel, flags, out_joffsets);
    count_launches(3);
    return launch_status();
}

namespace fvgb {
namespace {
__global__ void ijk_to_index_kernel(FvgbGrid g, const int32_t *__restrict__ q, const int64_t *__restrict__ qoff,
                                    int64_t n, int32_t cumulative, int64_t *__restrict__ out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int32_t b = batch_of(qoff, g.num_grids, i);
    const int32_t x = q[3 * i], y = q[3 * i + 1], z = q[3 * i + 2];
    int64_t idx = -1;
    const int32_t id = find_leaf(g, b, x >> 3, y >> 3, z >> 3);
    if (id >= 0) idx = leaf_voxel_index(g.leaves[id], leaf_bit(x, y, z));
    if (idx >= 0 && !cumulative) idx -= g.voxel_offsets[b];
    out[i] = idx;
}
}  // namespace
}  // namespace fvgb

extern "C" int fvgb_ijk_to_index(const FvgbGrid *grid, const int32_t *ijk, const int64_t *joffsets, int64_t n,
                                 int32_t cumulative, int64_t *out, fvgb_stream_t stream) {
    if (!grid || n < 0 || !joffsets || (n > 0 && (!ijk || !out))) return FVGB_EINVAL;
    if (n == 0) return FVGB_OK;
    ijk_to_index_kernel<<<blocks_for(n), kThreads, 0, as_stream(stream)>>>(*grid, ijk, joffsets, n, cumulative, out);
    count_launches(1);
    return launch_status();
}

// ---------------------------------------------------------------------------------------------
// Coarse grid of floor(ijk / f) built leaf by leaf, for power-of-two factors f <= 8 per axis: a
// fine leaf (8^3 voxels) falls inside one coarse leaf, so the fine leaves are grouped by coarse
// leaf (a radix sort of one key per fine leaf, not per voxel), each coarse leaf's occupancy mask
// is the OR of its fine leaves' voxels mapped down, and the coarse voxels are written leaf by
// leaf in bit order.  Coarse leaves sorted by (grid, order key) and voxels by bit within a leaf
// is the NanoVDB index order: the result is identical to sorting floor(ijk / f) voxel by voxel.
namespace fvgb {
namespace {

constexpr int kCoarseMaxGrids = 1024;  // the grid index takes the key's top 10 bits

struct CoarseWs {
    uint64_t *keys_a, *keys_b, *cmask;
    int32_t *vals_a, *vals_b, *cid, *count, *base;
    int4 *corig;
    void *cub_tmp;
    size_t cub_bytes;
};

size_t coarse_ws_layout(int64_t nl, CoarseWs *w, char *base) {
    size_t cub_bytes = 0, c = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, c, (uint64_t *)nullptr, (uint64_t *)nullptr, (int32_t *)nullptr,
                                    (int32_t *)nullptr, (int)nl, 0, 64);
    cub_bytes = c;
    cub::DeviceRadixSort::SortPairs(nullptr, c, (uint32_t *)nullptr, (uint32_t *)nullptr, (int32_t *)nullptr,
                                    (int32_t *)nullptr, (int)nl, 0, 32);
    if (c > cub_bytes) cub_bytes = c;
    cub::DeviceScan::InclusiveSum(nullptr, c, (int32_t *)nullptr, (int32_t *)nullptr, (int)nl);
    if (c > cub_bytes) cub_bytes = c;
    cub::DeviceScan::ExclusiveSum(nullptr, c, (int32_t *)nullptr, (int32_t *)nullptr, (int)nl + 1);
    if (c > cub_bytes) cub_bytes = c;
    size_t off = 0;
    auto take = [&](size_t bytes) {
        char *p = base ? base + off : nullptr;
        off += (bytes + 255) & ~(size_t)255;
        return p;
    };
    const size_t n = (size_t)nl;
    char *ka = take(n * 8), *kb = take(n * 8), *cm = take(n * 64), *va = take(n * 4), *vb = take(n * 4),
         *ci = take((n + 1) * 4), *co = take((n + 1) * 4), *ba = take((n + 1) * 4), *og = take(n * 16),
         *tmp = take(cub_bytes);
    if (w) {
        w->keys_a = (uint64_t *)ka, w->keys_b = (uint64_t *)kb, w->cmask = (uint64_t *)cm;
        w->vals_a = (int32_t *)va, w->vals_b = (int32_t *)vb, w->cid = (int32_t *)ci, w->count = (int32_t *)co;
        w->base = (int32_t *)ba, w->corig = (int4 *)og, w->cub_tmp = tmp, w->cub_bytes = cub_bytes;
    }
    return off;
}

// key of fine leaf l: (grid << vb) | ((order key of its coarse leaf's origin & low_mask) >> 9); the
// bits above low_mask agree for every coarse voxel of the bounding box, so dropping them keeps the
// order and shortens the sort
__global__ void coarse_keys_kernel(const FvgbLeaf *__restrict__ leaves, int64_t nl, int3 sh, uint64_t low_mask,
                                   int vb, uint64_t *__restrict__ keys, int32_t *__restrict__ vals) {
    const int64_t l = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (l >= nl) return;
    const FvgbLeaf &lf = leaves[l];
    const int32_t cx = (lf.origin[0] >> (sh.x + 3)) << 3, cy = (lf.origin[1] >> (sh.y + 3)) << 3,
                  cz = (lf.origin[2] >> (sh.z + 3)) << 3;
    keys[l] = ((uint64_t)lf.batch << vb) | ((order_key(cx, cy, cz) & low_mask) >> 9);
    vals[l] = (int32_t)l;
}

template <typename Key>
__global__ void coarse_flags_kernel(const Key *__restrict__ keys, int64_t nl, int32_t *__restrict__ flags) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= nl) return;
    flags[p] = (p == 0 || keys[p] != keys[p - 1]) ? 1 : 0;
}

// keys that fit 32 bits, narrowed for a sort with half the traffic and a smaller footprint
__global__ void narrow_keys_kernel(const uint64_t *__restrict__ k64, int64_t nl, uint32_t *__restrict__ k32) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p < nl) k32[p] = (uint32_t)k64[p];
}

// warp per sorted fine leaf: OR its voxels, mapped down, into its coarse leaf's mask
__global__ void coarse_mask_kernel(const FvgbLeaf *__restrict__ leaves, int64_t nl, int3 sh,
                                   const int32_t *__restrict__ vals, const int32_t *__restrict__ cid,
                                   uint64_t *__restrict__ cmask, int4 *__restrict__ corig) {
    __shared__ unsigned long long wm[8][8];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t p = (int64_t)blockIdx.x * 8 + warp;
    if (p >= nl) return;  // whole warps leave together
    const FvgbLeaf &lf = leaves[vals[p]];
    const int32_t c = cid[p] - 1;
    if (lane < 8) wm[warp][lane] = 0ull;
    __syncwarp();
    const uint64_t word = lf.mask[lane >> 2];
    const int sub = (lane & 3) * 16;
    for (int i = 0; i < 16; ++i) {
        if (!((word >> (sub + i)) & 1ull)) continue;
        const int b = (lane >> 2) * 64 + sub + i;
        const int32_t gx = lf.origin[0] + (b >> 6), gy = lf.origin[1] + ((b >> 3) & 7), gz = lf.origin[2] + (b & 7);
        const uint32_t cb = leaf_bit(gx >> sh.x, gy >> sh.y, gz >> sh.z);
        atomicOr(&wm[warp][cb >> 6], 1ull << (cb & 63));
    }
    __syncwarp();
    if (lane < 8) {
        const unsigned long long m = wm[warp][lane];
        if (m) atomicOr(reinterpret_cast<unsigned long long *>(cmask) + (int64_t)c * 8 + lane, m);
    }
    if (lane == 0)  // every fine leaf of coarse leaf c writes the same origin
        corig[c] = make_int4((lf.origin[0] >> (sh.x + 3)) << 3, (lf.origin[1] >> (sh.y + 3)) << 3,
                             (lf.origin[2] >> (sh.z + 3)) << 3, lf.batch);
}

// voxels per coarse leaf (zero past the coarse-leaf count, for the exclusive scan over nl + 1)
__global__ void coarse_count_kernel(const uint64_t *__restrict__ cmask, const int32_t *__restrict__ cid, int64_t nl,
                                    int32_t *__restrict__ count) {
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c > nl) return;
    const int64_t lc = cid[nl - 1];
    int32_t n = 0;
    if (c < lc)
#pragma unroll
        for (int w = 0; w < 8; ++w) n += __popcll(cmask[c * 8 + w]);
    count[c] = n;
}

// warp per coarse leaf: its voxels in bit order, and their leaf ids (1-based)
__global__ void coarse_emit_kernel(const uint64_t *__restrict__ cmask, const int4 *__restrict__ corig,
                                   const int32_t *__restrict__ cid, const int32_t *__restrict__ base, int64_t nl,
                                   int32_t *__restrict__ out_ijk, int32_t *__restrict__ leaf_ids) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t c = (int64_t)blockIdx.x * 8 + warp;
    if (c >= nl || c >= cid[nl - 1]) return;
    const int w = lane >> 2, sub = (lane & 3) * 16;
    int32_t rank = base[c];
    for (int v = 0; v < w; ++v) rank += __popcll(cmask[c * 8 + v]);
    const uint64_t word = cmask[c * 8 + w];
    rank += __popcll(sub ? (word & ((1ull << sub) - 1ull)) : 0ull);
    const int4 o = corig[c];
    for (int i = 0; i < 16; ++i) {
        if (!((word >> (sub + i)) & 1ull)) continue;
        const int b = w * 64 + sub + i;
        out_ijk[3 * (int64_t)rank] = o.x + (b >> 6);
        out_ijk[3 * (int64_t)rank + 1] = o.y + ((b >> 3) & 7);
        out_ijk[3 * (int64_t)rank + 2] = o.z + (b & 7);
        leaf_ids[rank] = (int32_t)c + 1;
        ++rank;
    }
}

// meta[b] = first voxel of grid b (b <= B), meta[B+1] = coarse leaves, meta[B+2] = voxels
__global__ void coarse_offsets_kernel(const int4 *__restrict__ corig, const int32_t *__restrict__ cid,
                                      const int32_t *__restrict__ base, int64_t nl, int32_t B,
                                      int64_t *__restrict__ meta) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b > B) return;
    const int64_t lc = cid[nl - 1];
    int64_t lo = 0, hi = lc;  // first coarse leaf with grid >= b
    while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        if (corig[mid].w < b) lo = mid + 1; else hi = mid;
    }
    meta[b] = base[lo];
    if (b == 0) {
        meta[B + 1] = lc;
        meta[B + 2] = base[lc];
    }
}

// Up to kHashLeaves fine leaves the coarse leaves are found through a hash table and put in order by
// counting, for each, the keys below its own: five launches with little shared memory instead of
// seventeen.  The build runs beside convolutions whose CTAs leave about 30 KB of shared memory per SM;
// the radix sort's passes waited for those CTAs to end, and the host, which waits for the counts,
// waited with them (inference step, 1.31M voxels in 21.7k fine leaves: 763 us a step with the sort, 646 us
// with this; pooling over the same grid, nothing beside it: 652 -> 575 us).  Counting is quadratic in the
// coarse leaves (a quarter of the fine ones on surfaces), which at kHashLeaves coarse leaves is about the
// sort's time.
constexpr int64_t kHashLeaves = 49152;
constexpr int kRankThreads = 256, kRankSplit = 8, kScanThreads = 1024;

// Workspace of the hashed build.
struct CoarseHash {
    uint64_t *table;   // [cap] keys, all ones where free
    int32_t *slot_id;  // [cap] coarse leaf of a taken slot, in insertion order
    uint64_t *key;     // [nl]
    int32_t *slot;     // [nl] slot of each fine leaf
    int32_t *order;    // [nl] coarse leaf at each place of the index order
    int32_t *count;    // [nl] voxels of the coarse leaf at each place
    int32_t *grid;     // [nl] grid of the coarse leaf at each place
    int32_t *base;     // [nl + 1] first voxel of each place
    int32_t *found;    // [1] coarse leaves - 1 (cleared to all ones together with the table before it)
    uint64_t *cmask;   // [nl][8]
    int4 *corig;       // [nl]
    int64_t cap;
};

__global__ void coarse_insert_kernel(const FvgbLeaf *__restrict__ leaves, int64_t nl, int3 sh, uint64_t low_mask, int vb,
                                     CoarseHash h) {
    const int64_t l = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (l >= nl) return;
    const FvgbLeaf &lf = leaves[l];
    const int32_t cx = (lf.origin[0] >> (sh.x + 3)) << 3, cy = (lf.origin[1] >> (sh.y + 3)) << 3,
                  cz = (lf.origin[2] >> (sh.z + 3)) << 3;
    const uint64_t key = ((uint64_t)lf.batch << vb) | ((order_key(cx, cy, cz) & low_mask) >> 9);
    const uint64_t cap_mask = (uint64_t)h.cap - 1;
    uint64_t m = key * 0x9E3779B97F4A7C15ull;
    m ^= m >> 32;
    uint64_t s = m & cap_mask;
    for (int64_t probe = 0; probe < h.cap; ++probe) {  // at most half full: a free slot is found
        const uint64_t k = atomicCAS(reinterpret_cast<unsigned long long *>(h.table + s), ~0ull, key);
        if (k == ~0ull) {
            const int32_t id = atomicAdd(h.found, 1) + 1;
            h.slot_id[s] = id;
            h.key[id] = key;
            h.corig[id] = make_int4(cx, cy, cz, lf.batch);
#pragma unroll
            for (int w = 0; w < 8; ++w) h.cmask[(int64_t)id * 8 + w] = 0;
            break;
        }
        if (k == key) break;
        s = (s + 1) & cap_mask;
    }
    h.slot[l] = (int32_t)s;
}

// warp per fine leaf: OR its voxels, mapped down, into its coarse leaf's mask.  A lane folds its two
// rows of eight z positions as bytes, so it costs two shared-memory updates however full the leaf is
// (21.7k leaves: 15.6 us voxel by voxel, 4.6 us).
__global__ void __launch_bounds__(256) coarse_or_kernel(const FvgbLeaf *__restrict__ leaves, int64_t nl, int3 sh,
                                                        CoarseHash h, int32_t *__restrict__ slots, int64_t cap) {
    __shared__ uint32_t wm[8][16];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t l = (int64_t)blockIdx.x * 8 + warp;
    // the leaf hash that coarse_place_kernel fills starts out free
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < cap; i += (int64_t)gridDim.x * 256) slots[i] = -1;
    if (l >= nl) return;  // whole warps leave together
    const FvgbLeaf &lf = leaves[l];
    const int64_t c = h.slot_id[h.slot[l]];
    if (lane < 16) wm[warp][lane] = 0u;
    __syncwarp();
    const uint32_t two = (uint32_t)(lf.mask[lane >> 2] >> ((lane & 3) * 16)) & 0xffffu;
    // leaf origins are multiples of 8: row (x, y) goes to row (ox + (x >> shift), oy + (y >> shift)),
    // its first z position to oz
    const int ox = (lf.origin[0] >> sh.x) & 7, oy = (lf.origin[1] >> sh.y) & 7, oz = (lf.origin[2] >> sh.z) & 7;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        uint32_t r = (two >> (8 * e)) & 0xffu;
        if (!r) continue;
        if (sh.z >= 1) {  // OR of neighbours, then every second bit
            r = (r | (r >> 1)) & 0x55u;
            r = (r | (r >> 1)) & 0x33u;
            r = (r | (r >> 2)) & 0x0fu;
        }
        if (sh.z >= 2) r = ((r | (r >> 1)) & 1u) | (((r >> 2) | (r >> 3)) & 1u) << 1;
        if (sh.z >= 3) r = (r | (r >> 1)) & 1u;
        const int row = (ox + ((lane >> 2) >> sh.x)) * 8 + oy + (((lane & 3) * 2 + e) >> sh.y);
        atomicOr(&wm[warp][row >> 2], (r << oz) << ((row & 3) * 8));
    }
    __syncwarp();
    if (lane < 16) {
        const uint32_t m = wm[warp][lane];
        if (m) atomicOr(reinterpret_cast<uint32_t *>(h.cmask) + c * 16 + lane, m);
    }
}

// Place of coarse leaf i in the index order = keys below its own (keys are distinct): kRankSplit threads
// per leaf share the counting, so that a few thousand leaves fill the SMs and each thread's chain is
// short (5.9k leaves: 35 us with a thread per leaf, 9.3 us).
template <typename Key>
__global__ void __launch_bounds__(kRankThreads) coarse_rank_kernel(CoarseHash h) {
    __shared__ Key keys[kRankThreads];
    constexpr int kOwn = kRankThreads / kRankSplit;  // leaves per CTA
    const int32_t n = *h.found + 1;
    if ((int64_t)blockIdx.x * kOwn >= n) return;
    const int part = threadIdx.x % kRankSplit;
    const int32_t i = blockIdx.x * kOwn + threadIdx.x / kRankSplit;
    const Key mine = i < n ? (Key)h.key[i] : (Key)0;
    int32_t rank = 0;
    Key next = threadIdx.x < n ? (Key)h.key[threadIdx.x] : (Key)~(Key)0;  // never below a key
    for (int32_t j0 = 0; j0 < n; j0 += kRankThreads) {
        __syncthreads();
        keys[threadIdx.x] = next;
        __syncthreads();
        const int32_t j = j0 + kRankThreads + threadIdx.x;
        next = j < n ? (Key)h.key[j] : (Key)~(Key)0;
#pragma unroll
        for (int t = 0; t < kRankThreads / kRankSplit; ++t) rank += keys[t * kRankSplit + part] < mine ? 1 : 0;
    }
#pragma unroll
    for (int o = kRankSplit / 2; o; o >>= 1) rank += __shfl_xor_sync(0xffffffffu, rank, o);
    // the leaf's mask words, one per thread
    static_assert(kRankSplit == 8, "a mask word per thread");
    int32_t c = i < n ? __popcll(h.cmask[(int64_t)i * 8 + part]) : 0;
#pragma unroll
    for (int o = kRankSplit / 2; o; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if (i >= n || part != 0) return;
    h.order[rank] = i;
    h.count[rank] = c;
    h.grid[rank] = h.corig[i].w;
}

// One CTA: first voxel of every place (count and grid of each of n > 0 places given, base [n + 1]) and
// first voxel of every grid, offsets [B + 1]; returns the voxels.
__device__ __forceinline__ int32_t scan_places(int32_t n, const int32_t *__restrict__ count,
                                               const int32_t *__restrict__ grid, int32_t B, int32_t *__restrict__ base,
                                               int64_t *__restrict__ offsets) {
    using Scan = cub::BlockScan<int32_t, kScanThreads>;
    __shared__ typename Scan::TempStorage tmp;
    int32_t run = 0;
    constexpr int kItems = 8;
    for (int32_t p0 = 0; p0 < n; p0 += kScanThreads * kItems) {
        int32_t v[kItems], g[kItems + 1], total;
        const int32_t q = p0 + threadIdx.x * kItems;
        const bool whole = q + kItems <= n;  // 16-byte accesses: the arrays start on 256 bytes
        g[0] = q > 0 && q < n ? grid[q - 1] : -1;
        if (whole) {
#pragma unroll
            for (int i = 0; i < kItems; i += 4) {
                const int4 a = *reinterpret_cast<const int4 *>(count + q + i);
                const int4 b = *reinterpret_cast<const int4 *>(grid + q + i);
                v[i] = a.x, v[i + 1] = a.y, v[i + 2] = a.z, v[i + 3] = a.w;
                g[i + 1] = b.x, g[i + 2] = b.y, g[i + 3] = b.z, g[i + 4] = b.w;
            }
        } else {
#pragma unroll
            for (int i = 0; i < kItems; ++i) {
                v[i] = q + i < n ? count[q + i] : 0;
                g[i + 1] = q + i < n ? grid[q + i] : -1;
            }
        }
        __syncthreads();
        Scan(tmp).ExclusiveSum(v, v, total);
        if (whole) {
#pragma unroll
            for (int i = 0; i < kItems; i += 4)
                *reinterpret_cast<int4 *>(base + q + i) =
                    make_int4(run + v[i], run + v[i + 1], run + v[i + 2], run + v[i + 3]);
        }
#pragma unroll
        for (int i = 0; i < kItems; ++i) {
            const int32_t p = q + i;
            if (p >= n) break;
            if (!whole) base[p] = run + v[i];
            for (int32_t b = g[i] + 1; b <= g[i + 1]; ++b) offsets[b] = run + v[i];  // grids that begin here
            if (p == n - 1)
                for (int32_t b = g[i + 1] + 1; b <= B; ++b) offsets[b] = run + total;  // and those after the last
        }
        run += total;
    }
    if (threadIdx.x == 0) base[n] = run;
    return run;
}

// meta[b] = first voxel of grid b, meta[B+1] = coarse leaves, meta[B+2] = voxels
__global__ void __launch_bounds__(kScanThreads) coarse_scan_kernel(CoarseHash h, int32_t B, int64_t *meta) {
    const int32_t n = *h.found + 1;
    const int32_t voxels = scan_places(n, h.count, h.grid, B, h.base, meta);
    if (threadIdx.x == 0) {
        meta[B + 1] = n;
        meta[B + 2] = voxels;
        meta[B + 3] = 0;
    }
}

// warp per place: its voxels in bit order, its leaf table entry and its hash slot
__global__ void __launch_bounds__(256) coarse_place_kernel(CoarseHash h, int32_t *__restrict__ out_ijk,
                                                           FvgbLeaf *__restrict__ leaves, int32_t *__restrict__ slots,
                                                           int64_t cap) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t p = (int64_t)blockIdx.x * 8 + warp;
    if (p > *h.found) return;
    const int64_t c = h.order[p];
    const int4 o = h.corig[c];
    emit_leaf(h.cmask[c * 8 + (lane >> 2)], o.x, o.y, o.z, o.w, h.base[p], p, lane, out_ijk, leaves, slots, cap);
}

// 8 + 4 bytes per slot (2 to 4 slots per fine leaf) and 108 per fine leaf
size_t coarse_hash_layout(int64_t nl, CoarseHash *w, char *base) {
    CoarseHash h;
    h.cap = 64;
    while (h.cap < 2 * nl) h.cap <<= 1;
    size_t off = 0;
    auto take = [&](size_t bytes) {
        char *p = base ? base + off : nullptr;
        off += (bytes + 255) & ~(size_t)255;
        return p;
    };
    const size_t n = (size_t)nl;
    h.table = (uint64_t *)take((size_t)h.cap * 8);
    h.found = (int32_t *)take(4);
    h.slot_id = (int32_t *)take((size_t)h.cap * 4);
    h.key = (uint64_t *)take(n * 8);
    h.slot = (int32_t *)take(n * 4);
    h.order = (int32_t *)take(n * 4);
    h.count = (int32_t *)take(n * 4);
    h.grid = (int32_t *)take(n * 4);
    h.base = (int32_t *)take((n + 1) * 4);
    h.cmask = (uint64_t *)take(n * 64);
    h.corig = (int4 *)take(n * 16);
    if (w) *w = h;
    return off;
}

}  // namespace
}  // namespace fvgb

extern "C" int fvgb_coarse_grid_workspace(int64_t num_fine_leaves, size_t *bytes) {
    if (!bytes || num_fine_leaves < 0 || num_fine_leaves >= INT32_MAX) return FVGB_EINVAL;
    *bytes = fvgb::coarse_ws_layout(std::max<int64_t>(num_fine_leaves, 1), nullptr, nullptr) + 256;
    return FVGB_OK;
}

extern "C" int fvgb_coarse_grid_build(const FvgbGrid *fine, const int32_t factor[3], const int32_t *box_lo,
                                      const int32_t *box_hi, int32_t *out_ijk, int64_t *meta, int32_t *leaf_ids,
                                      void *workspace, size_t workspace_bytes, fvgb_stream_t stream) {
    if (!fine || !factor || !meta) return FVGB_EINVAL;
    if (fine->num_grids < 1 || fine->num_grids > kCoarseMaxGrids) return FVGB_EINVAL;
    int sh[3];
    for (int a = 0; a < 3; ++a) {
        const int f = factor[a];
        if (f != 1 && f != 2 && f != 4 && f != 8) return FVGB_EINVAL;
        sh[a] = f == 1 ? 0 : (f == 2 ? 1 : (f == 4 ? 2 : 3));
    }
    const int64_t nl = fine->num_leaves;
    if (nl == 0) return FVGB_EINVAL;  // callers handle empty grids themselves
    if (!out_ijk || !leaf_ids || !fine->leaves) return FVGB_EINVAL;
    size_t need = 0;
    int st = fvgb_coarse_grid_workspace(nl, &need);
    if (st) return st;
    if (!workspace || workspace_bytes < need) return FVGB_ENOSPACE;
    cudaStream_t s = as_stream(stream);
    char *base = reinterpret_cast<char *>(((uintptr_t)workspace + 255) & ~(uintptr_t)255);
    CoarseWs w;
    coarse_ws_layout(nl, &w, base);
    const int3 shv = make_int3(sh[0], sh[1], sh[2]);
    // key bits: the order-key bits that vary inside the coarse bounding box (all 63 without one),
    // less the 9 leaf bits, under the grid index
    int end_bit = 63;
    if (box_lo && box_hi) {
        for (int a = 0; a < 3; ++a)
            if (box_lo[a] > box_hi[a]) return FVGB_EINVAL;
        end_bit = order_key_end_bit(box_lo, box_hi);
    }
    const int vb = end_bit > 9 ? end_bit - 9 : 0;
    const uint64_t low_mask = end_bit >= 63 ? ~0ull : ((1ull << end_bit) - 1ull);
    int grid_bits = 0;
    while ((1 << grid_bits) < fine->num_grids) ++grid_bits;
    const int sort_bits = std::max(1, vb + grid_bits);
    if (cudaMemsetAsync(w.cmask, 0, (size_t)nl * 64, s) != cudaSuccess) return launch_status();
    coarse_keys_kernel<<<blocks_for(nl), kThreads, 0, s>>>(fine->leaves, nl, shv, low_mask, vb, w.keys_a, w.vals_a);
    size_t tb = w.cub_bytes;
    int launched = 6;  // keys, flags, mask, count, emit, offsets (+ narrow)
    if (sort_bits <= 32) {
        // 32-bit keys: the sort's kernels need less shared memory, so they also fit on SMs that a
        // running convolution kernel occupies
        uint32_t *k32a = reinterpret_cast<uint32_t *>(w.keys_b);  // the narrowed keys
        uint32_t *k32b = reinterpret_cast<uint32_t *>(w.keys_a);  // sorted: keys_a is free once narrowed
        narrow_keys_kernel<<<blocks_for(nl), kThreads, 0, s>>>(w.keys_a, nl, k32a);
        cub::DeviceRadixSort::SortPairs(w.cub_tmp, tb, k32a, k32b, w.vals_a, w.vals_b, (int)nl, 0, sort_bits, s);
        coarse_flags_kernel<uint32_t><<<blocks_for(nl), kThreads, 0, s>>>(k32b, nl, w.count);
        ++launched;
    } else {
        cub::DeviceRadixSort::SortPairs(w.cub_tmp, tb, w.keys_a, w.keys_b, w.vals_a, w.vals_b, (int)nl, 0, sort_bits,
                                        s);
        coarse_flags_kernel<uint64_t><<<blocks_for(nl), kThreads, 0, s>>>(w.keys_b, nl, w.count);
    }
    tb = w.cub_bytes;
    cub::DeviceScan::InclusiveSum(w.cub_tmp, tb, w.count, w.cid, (int)nl, s);
    coarse_mask_kernel<<<(unsigned)ceil_div(nl, 8), 256, 0, s>>>(fine->leaves, nl, shv, w.vals_b, w.cid, w.cmask,
                                                                w.corig);
    coarse_count_kernel<<<blocks_for(nl + 1), kThreads, 0, s>>>(w.cmask, w.cid, nl, w.count);
    tb = w.cub_bytes;
    cub::DeviceScan::ExclusiveSum(w.cub_tmp, tb, w.count, w.base, (int)nl + 1, s);
    coarse_emit_kernel<<<(unsigned)ceil_div(nl, 8), 256, 0, s>>>(w.cmask, w.corig, w.cid, w.base, nl, out_ijk,
                                                                leaf_ids);
    coarse_offsets_kernel<<<(unsigned)ceil_div(fine->num_grids + 1, kThreads), kThreads, 0, s>>>(
        w.corig, w.cid, w.base, nl, fine->num_grids, meta);
    count_launches(launched);  // CUB's own launches are not counted
    return launch_status();
}

// ---------------------------------------------------------------------------------------------
// Grid build through a leaf hash, for inputs with many rows per leaf: the rows of ijk (or points)
// are never sorted.  One pass inserts every row's leaf into an open-addressing table, ORs the row's
// voxel into the slot's 512-bit mask and counts the voxels that were new, so one read tells the host
// every size; then only the leaves are sorted and the voxels are written leaf by leaf in bit order,
// with the leaf table and the leaf hash in the same kernel.  Leaves sorted by (grid, order key) and
// voxels by bit is the order of the voxel sort, so the grid is identical to fvgb_ijk_sort_unique's.
// 7.9M points, 1.31M voxels, 22k leaves in four grids: voxelise, sort, unique and index took 1.9 ms,
// 0.21 ms here, bound by the random reads of the table and the masks.  The table has room for
// rows / 8 leaves at three quarters full; an input with more (fewer than eight rows per leaf) raises
// `overflow` and is left to the sort, which takes the bounding box from here (the rows' own: it is
// complete whatever the table's state) in place of a pass and a host read of its own.
namespace fvgb {
namespace {

constexpr uint64_t kEmptyLeaf = ~0ull;
constexpr int kHashRows = 4;      // rows per thread (more cost occupancy: 169 us with 8, 151 with 2, 132 with 4, before slots were counted; now 139)
constexpr int kHashProbes = 512;  // a full neighbourhood of the table counts as overflow
constexpr int kTakenCounters = 64;  // CTAs count the slots they take on a line of their share of these
constexpr int kHashMaxGrids = 1023;  // the grid index takes the key's top 10 bits (all ones: the empty slot)

struct LeafHash {
    uint64_t *table;    // [cap] leaf keys, kEmptyLeaf where free
    uint64_t *mask;     // [cap][8] voxels of the slot's leaf, cleared with the pass
    int32_t *taken;     // [kTakenCounters][32] slots taken, cleared with the masks before them
    uint64_t *keys;     // [max_leaves] key of each leaf, in insertion order
    uint32_t *leaf_slot;  // [max_leaves] its slot
    uint32_t cap;
    int32_t max_leaves;
};

size_t leaf_hash_layout(int64_t n, LeafHash *w, char *base) {
    size_t off = 0;
    auto take = [&](size_t bytes) {
        char *p = base ? base + off : nullptr;
        off = align_up(off + bytes, 256);
        return p;
    };
    LeafHash h;
    h.max_leaves = (int32_t)std::max<int64_t>(512, ceil_div(n, (int64_t)8));
    h.cap = (uint32_t)((int64_t)h.max_leaves / 3 * 4 + 4);
    h.table = (uint64_t *)take((size_t)h.cap * 8);
    h.mask = (uint64_t *)take((size_t)h.cap * 64);
    h.taken = (int32_t *)take((size_t)kTakenCounters * 32 * 4);
    h.keys = (uint64_t *)take((size_t)h.max_leaves * 8);
    h.leaf_slot = (uint32_t *)take((size_t)h.max_leaves * 4);
    if (w) *w = h;
    return off;
}

// first slot tried for a leaf: the key's hash scaled to the table (its size is no power of two)
__device__ __forceinline__ uint32_t leaf_home(const LeafHash &h, uint64_t key) {
    uint64_t m = key * 0x9E3779B97F4A7C15ull;
    m ^= m >> 32;
    m *= 0xD6E8FEB86659FD93ull;
    return __umulhi((uint32_t)(m >> 32), h.cap);
}

// The slot of a leaf, from slot s on, or kNoSlot where the table is too full for the input, with kMade set
// where this thread took it.  stat: [0] leaves, [1] error word, [2] overflow, [3..5] largest -x, -y, -z, [6..8]
// largest x, y, z, [9..] voxels of each grid.
// An input with too many leaves fills the table in the first wave of CTAs, before any of them ends and
// adds up its leaves, and probes of a full table are as long as they may be (1.05M scattered rows: 1.6 ms).
// So the CTAs count slots as they take them, each on one of kTakenCounters lines; whoever brings a line
// past its share of max_leaves, and every 1/16 of that further, adds them all up.  Lines that are all
// below that leave the table below 80 % full.  The others look at the overflow word after each leaf that they
// bring and in long probes.
constexpr uint64_t kNoSlot = 0xffffffffu, kMade = 1ull << 32;
__device__ __forceinline__ uint64_t insert_leaf(uint64_t *table, int32_t *taken, uint32_t cap, int32_t max_leaves, uint64_t key,
                                             uint32_t s, int32_t *stat) {
    for (int probe = 1; probe <= kHashProbes; ++probe) {
        uint64_t k = *reinterpret_cast<volatile uint64_t *>(table + s);
        if (k == kEmptyLeaf) {
            k = atomicCAS(reinterpret_cast<unsigned long long *>(table + s), kEmptyLeaf, key);
            if (k == kEmptyLeaf) {  // this thread's leaf
                const int32_t share = max_leaves / kTakenCounters, step = (share + 15) / 16;
                const int32_t past = atomicAdd(taken + (blockIdx.x % kTakenCounters) * 32, 1) - share;
                if (past >= 0 && past % step == 0) {
                    int32_t n = 0;
                    for (int c = 0; c < kTakenCounters; ++c) n += *reinterpret_cast<volatile int32_t *>(taken + c * 32);
                    if (n > max_leaves) stat[2] = 1;
                }
                return s | kMade;
            }
        }
        if (k == key) return s;
        s = s + 1 < cap ? s + 1 : 0;
        if (probe % 16 == 0 && *reinterpret_cast<volatile int32_t *>(stat + 2)) return kNoSlot;
    }
    stat[2] = 1;
    return kNoSlot;
}

__global__ void stat_init_kernel(int32_t *stat, int32_t n) {
    const int32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) stat[i] = i >= 3 && i < 9 ? INT32_MIN : 0;
}

// The pass over ijk rows (P = int32_t) or points (P = the points' type, voxelised in T).
template <typename P, typename T>
__global__ void __launch_bounds__(256, 5) leaf_insert_kernel(const P *__restrict__ in, const int64_t *__restrict__ joff,
                                                          int32_t B, int64_t n, const double *__restrict__ vs,
                                                          const double *__restrict__ org, LeafHash h,
                                                          int32_t *__restrict__ stat) {
    constexpr bool kPoints = !std::is_same<P, int32_t>::value;
    __shared__ T fac[6];
    __shared__ int32_t sb[2], full, made, first_id, box[7][8];
    __shared__ uint32_t made_slot[256 * kHashRows];  // slots that the CTA took
    const int64_t base = (int64_t)blockIdx.x * 256 * kHashRows;
    const int64_t last = min(n, base + 256 * kHashRows) - 1;
    if (threadIdx.x < 2) sb[threadIdx.x] = batch_of(joff, B, threadIdx.x == 0 ? base : last);
    if (threadIdx.x == 2) {
        full = *reinterpret_cast<volatile int32_t *>(stat + 2);
        made = 0;
    }
    __syncthreads();
    if (kPoints) {
        if (threadIdx.x < 3) {
            const double w = vs[3 * sb[0] + threadIdx.x], o = org[3 * sb[0] + threadIdx.x];
            fac[threadIdx.x] = (T)(1.0 / w);
            fac[3 + threadIdx.x] = (T)(-o / w);
        }
        __syncthreads();
    }
    int32_t c[kHashRows][3];
    bool range = true;
    int32_t lim[6];
#pragma unroll
    for (int e = 0; e < 6; ++e) lim[e] = INT32_MIN;
#pragma unroll
    for (int q = 0; q < kHashRows; ++q) {
        const int64_t i = min(base + q * 256 + threadIdx.x, last);  // past the end: the last row again
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            if constexpr (kPoints) {
                T s = fac[a], t = fac[3 + a];
                if (sb[0] != sb[1]) {
                    const int32_t b = batch_of(joff, B, i);
                    if (b != sb[0]) {
                        const double w = vs[3 * b + a], o = org[3 * b + a];
                        s = (T)(1.0 / w);
                        t = (T)(-o / w);
                    }
                }
                c[q][a] = voxelise(point_value<T>(in[3 * i + a]), s, t);
            } else {
                c[q][a] = in[3 * i + a];
            }
            range = range && coord_in_range(c[q][a]);
            lim[a] = max(lim[a], -c[q][a]);
            lim[3 + a] = max(lim[3 + a], c[q][a]);
        }
    }
    int32_t fresh = 0;  // voxels this thread set
    uint64_t key[kHashRows], word[kHashRows];
    uint32_t slot[kHashRows], bit[kHashRows];
    if (!full) {  // else the input is left to the sort, which wants the bounding box alone
        // Every step's accesses for all rows go out together: the first probe, which finds most leaves, the
        // mask words, and the updates, whose results are looked at last (one after another each update's
        // wait added up: 200 us for 7.9M points, 132 us).
#pragma unroll
        for (int q = 0; q < kHashRows; ++q) {
            const int64_t i = min(base + q * 256 + threadIdx.x, last);
            const int32_t b = sb[0] == sb[1] ? sb[0] : batch_of(joff, B, i);
            const uint64_t k = order_key(c[q][0], c[q][1], c[q][2]);
            bit[q] = (uint32_t)(k & 511);
            key[q] = ((uint64_t)b << 54) | (k >> 9);
            slot[q] = leaf_home(h, key[q]);
            word[q] = __ldcg(h.table + slot[q]);
        }
    }
    if (!range) stat[1] = FVGB_ERANGE;
#pragma unroll
    for (int e = 0; e < 6; ++e) {
        const int32_t v = __reduce_max_sync(0xffffffffu, lim[e]);
        if ((threadIdx.x & 31) == 0) box[e][threadIdx.x >> 5] = v;
    }
    if (!full) {
        bool lost = false, took = false;
#pragma unroll
        for (int q = 0; q < kHashRows; ++q) {
            if (word[q] == key[q] || lost) continue;
            // who brings one leaf after another may be in an input of too many (a look per row, all at one
            // address, took 30 us of 7.9M points' first wave)
            if (took && *reinterpret_cast<volatile int32_t *>(stat + 2)) {
                lost = true;
                continue;
            }
            const uint64_t at = insert_leaf(h.table, h.taken, h.cap, h.max_leaves, key[q], slot[q], stat);
            slot[q] = (uint32_t)at;
            took = at & kMade;
            if (took) made_slot[atomicAdd(&made, 1)] = (uint32_t)at;
            lost = at == kNoSlot;
        }
#pragma unroll
        for (int q = 0; q < kHashRows; ++q) {
            if (lost) slot[q] = 0;  // the masks no longer matter
            word[q] = __ldcg(h.mask + (size_t)slot[q] * 8 + (bit[q] >> 6));
        }
#pragma unroll
        for (int q = 0; q < kHashRows; ++q) {
            const uint64_t m = 1ull << (bit[q] & 63);
            if (!(word[q] & m))  // most rows of a dense cloud have nothing to set
                word[q] = atomicOr(reinterpret_cast<unsigned long long *>(h.mask + (size_t)slot[q] * 8 + (bit[q] >> 6)), m);
        }
#pragma unroll
        for (int q = 0; q < kHashRows; ++q) {
            if (word[q] >> (bit[q] & 63) & 1) continue;
            if (sb[0] == sb[1]) ++fresh;
            else atomicAdd(stat + 9 + (int32_t)(key[q] >> 54), 1);
        }
    }
    fresh = __reduce_add_sync(0xffffffffu, fresh);
    if ((threadIdx.x & 31) == 0) box[6][threadIdx.x >> 5] = fresh;
    __syncthreads();
    // leaves are numbered by the CTA: one update of the count for all of its own (one per leaf, all on one
    // address, took 5 ns each: 0.9 ms for 175k leaves)
    const int32_t n_made = made;
    if (n_made) {
        if (threadIdx.x == 0) first_id = atomicAdd(stat, n_made);
        __syncthreads();
        for (int32_t i = threadIdx.x; i < n_made; i += 256) {
            const int32_t id = first_id + i;
            if (id < h.max_leaves) {
                h.keys[id] = __ldcg(h.table + made_slot[i]);
                h.leaf_slot[id] = made_slot[i];
            } else {
                stat[2] = 1;
            }
        }
    }
    // the bounding box, once per CTA: every update reads one address (a read per warp, 31k warps on
    // 7.9M points, set the kernel's pace: 170 us against 102), and the new voxels of the CTA's grid
    if (threadIdx.x < 6) {
        int32_t v = box[threadIdx.x][0];
#pragma unroll
        for (int w = 1; w < 8; ++w) v = max(v, box[threadIdx.x][w]);
        if (v > *reinterpret_cast<volatile int32_t *>(stat + 3 + threadIdx.x)) atomicMax(stat + 3 + threadIdx.x, v);
    } else if (threadIdx.x == 32) {
        int32_t v = 0;
#pragma unroll
        for (int w = 0; w < 8; ++w) v += box[6][w];
        if (v) atomicAdd(stat + 9 + sb[0], v);
    }
}

// sort key of leaf i: (grid << vb) | the order-key bits that vary inside the bounding box
template <typename Key>
__global__ void leaf_sort_keys_kernel(LeafHash h, int64_t L, uint64_t low, int vb, Key *__restrict__ keys,
                                      int32_t *__restrict__ vals) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= L) return;
    const uint64_t k = h.keys[i];
    keys[i] = (Key)(((k >> 54) << vb) | (k & low));
    vals[i] = (int32_t)i;
}

__global__ void leaf_counts_kernel(LeafHash h, int64_t L, const int32_t *__restrict__ vals, int32_t *__restrict__ count) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p > L) return;
    int32_t c = 0;
    if (p < L) {
        const uint64_t *m = h.mask + (size_t)h.leaf_slot[vals[p]] * 8;
#pragma unroll
        for (int w = 0; w < 8; ++w) c += __popcll(m[w]);
    }
    count[p] = c;  // zero past the last leaf, for the exclusive scan over L + 1
}

// Up to kTileLeaves leaves are sorted by two kernels: tiles of kSortTile leaves each in shared memory
// (place = keys of the tile below its own), then every leaf finds by binary search the keys below its
// own in the other tiles: a CTA takes 32 leaves next to each other in a tile, whose searches read the
// same entries, and its eight warps share the tiles.  The second kernel also counts the leaf's voxels,
// and one CTA scans them (leaf_scan_kernel).  Four launches against the radix sort's and scan's
// nineteen (22k leaves: 71 us of small kernels, 27 us here).  A leaf searches every tile, so the
// cost grows with the square: at kTileLeaves it is about the radix sort's.
constexpr int kSortTile = 512;
constexpr int64_t kTileLeaves = 65536;

template <typename Key>
__global__ void __launch_bounds__(kSortTile) leaf_tile_kernel(LeafHash h, int64_t L, uint64_t low, int vb,
                                                              Key *__restrict__ keys, int32_t *__restrict__ vals,
                                                              int32_t *__restrict__ slots, int64_t cap) {
    __shared__ __align__(16) Key tile[kSortTile];
    const int64_t base = (int64_t)blockIdx.x * kSortTile, i = base + threadIdx.x;
    // the leaf hash that leaf_emit_kernel fills starts out free
    for (int64_t j = i; j < cap; j += (int64_t)gridDim.x * kSortTile) slots[j] = -1;
    Key mine = ~(Key)0;  // past the last leaf: never below a key
    if (i < L) {
        const uint64_t k = h.keys[i];
        mine = (Key)(((k >> 54) << vb) | (k & low));
    }
    tile[threadIdx.x] = mine;
    __syncthreads();
    if (i >= L) return;
    int32_t place = 0;
#pragma unroll 16
    for (int t = 0; t < kSortTile; ++t) place += tile[t] < mine ? 1 : 0;
    keys[base + place] = mine;
    vals[base + place] = (int32_t)i;
}

template <typename Key>
__global__ void __launch_bounds__(256) leaf_rank_kernel(LeafHash h, int32_t L, const Key *__restrict__ keys,
                                                        const int32_t *__restrict__ vals, int32_t *__restrict__ order,
                                                        int32_t *__restrict__ count, int32_t *__restrict__ grid) {
    __shared__ int32_t part[8][32], voxels[8][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int32_t p = min(blockIdx.x * 32 + lane, L - 1), own = p / kSortTile;
    const Key mine = keys[p];
    const int32_t id = vals[p];
    voxels[warp][lane] = __popcll(h.mask[(size_t)h.leaf_slot[id] * 8 + warp]);  // a mask word per warp
    int32_t below = 0;
    for (int32_t t = warp; t * kSortTile < L; t += 8) {
        const int32_t first = t * kSortTile;
        if (t == own) {
            below += p - first;
            continue;
        }
        int32_t lo = first, hi = min(L, first + kSortTile);
        while (lo < hi) {
            const int32_t mid = (lo + hi) >> 1;
            if (__ldg(keys + mid) < mine) lo = mid + 1; else hi = mid;
        }
        below += lo - first;
    }
    part[warp][lane] = below;
    __syncthreads();
    if (warp != 0 || blockIdx.x * 32 + lane >= L) return;
    int32_t rank = 0, c = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) rank += part[w][lane], c += voxels[w][lane];
    order[rank] = id;
    count[rank] = c;
    grid[rank] = (int32_t)(h.keys[id] >> 54);
}

__global__ void __launch_bounds__(kScanThreads) leaf_scan_kernel(int32_t L, const int32_t *__restrict__ count,
                                                                 const int32_t *__restrict__ grid, int32_t B,
                                                                 int32_t *__restrict__ first,
                                                                 int64_t *__restrict__ offsets) {
    scan_places(L, count, grid, B, first, offsets);
}

// warp per leaf in index order
__global__ void __launch_bounds__(256) leaf_emit_kernel(LeafHash h, int64_t L, const int32_t *__restrict__ vals,
                                                        const int32_t *__restrict__ first,
                                                        int32_t *__restrict__ out_ijk, FvgbLeaf *__restrict__ leaves,
                                                        int32_t *__restrict__ slots, int64_t cap) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t p = (int64_t)blockIdx.x * 8 + warp;
    if (p >= L) return;
    const int32_t id = vals[p];
    const uint64_t key = h.keys[id];
    int32_t ox, oy, oz;
    key_to_coord((key & ((1ull << 54) - 1ull)) << 9, ox, oy, oz);
    emit_leaf(h.mask[(size_t)h.leaf_slot[id] * 8 + (lane >> 2)], ox, oy, oz, (int32_t)(key >> 54), first[p], p, lane, out_ijk, leaves,
              slots, cap);
}

// meta[b] = first voxel of grid b (b <= B)
__global__ void leaf_offsets_kernel(const FvgbLeaf *__restrict__ leaves, const int32_t *__restrict__ first, int64_t L,
                                    int32_t B, int64_t *__restrict__ meta) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b > B) return;
    int64_t lo = 0, hi = L;
    while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        if (leaves[mid].batch < b) lo = mid + 1; else hi = mid;
    }
    meta[b] = first[lo];
}

struct LeafSortWs {
    uint64_t *keys_a, *keys_b;
    int32_t *vals_a, *vals_b, *count, *first, *grid;
    void *cub_tmp;
    size_t cub_bytes;
};

size_t leaf_sort_layout(int64_t L, LeafSortWs *w, char *base) {
    size_t cub_bytes = 0, c = 0;
    if (L > kTileLeaves) {
        cub::DeviceRadixSort::SortPairs(nullptr, cub_bytes, (uint64_t *)nullptr, (uint64_t *)nullptr, (int32_t *)nullptr,
                                        (int32_t *)nullptr, (int)L, 0, 64);
        cub::DeviceRadixSort::SortPairs(nullptr, c, (uint32_t *)nullptr, (uint32_t *)nullptr, (int32_t *)nullptr,
                                        (int32_t *)nullptr, (int)L, 0, 32);
        cub_bytes = c > cub_bytes ? c : cub_bytes;
        cub::DeviceScan::ExclusiveSum(nullptr, c, (int32_t *)nullptr, (int32_t *)nullptr, (int)L + 1);
        cub_bytes = c > cub_bytes ? c : cub_bytes;
    }
    size_t off = 0;
    auto take = [&](size_t bytes) {
        char *p = base ? base + off : nullptr;
        off = align_up(off + bytes, 256);
        return p;
    };
    LeafSortWs s;
    s.keys_a = (uint64_t *)take((size_t)L * 8);
    s.keys_b = (uint64_t *)take((size_t)L * 8);
    s.vals_a = (int32_t *)take((size_t)L * 4);
    s.vals_b = (int32_t *)take((size_t)L * 4);
    s.count = (int32_t *)take((size_t)(L + 1) * 4);
    s.first = (int32_t *)take((size_t)(L + 1) * 4);
    s.grid = (int32_t *)s.keys_b;  // the tile sort leaves the second key buffer free
    s.cub_bytes = cub_bytes;
    s.cub_tmp = take(cub_bytes);
    if (w) *w = s;
    return off;
}

char *align_ws(void *p) { return reinterpret_cast<char *>(((uintptr_t)p + 255) & ~(uintptr_t)255); }

template <typename P, typename T>
void launch_insert(const void *in, const int64_t *joff, int32_t B, int64_t n, const double *vs, const double *org,
                   const LeafHash &h, int32_t *stat, cudaStream_t s) {
    const unsigned blocks = (unsigned)ceil_div(n, (int64_t)256 * kHashRows);
    leaf_insert_kernel<P, T><<<blocks, 256, 0, s>>>((const P *)in, joff, B, n, vs, org, h, stat);
}

}  // namespace
}  // namespace fvgb

extern "C" int fvgb_leaf_hash_workspace(int64_t n, size_t *bytes) {
    if (!bytes || n < 1 || n >= (int64_t)INT32_MAX) return FVGB_EINVAL;
    *bytes = leaf_hash_layout(n, nullptr, nullptr) + 256;
    return FVGB_OK;
}

extern "C" int fvgb_leaf_hash_insert(int32_t dtype, const void *rows, const int64_t *joffsets, int32_t num_grids,
                                     int64_t n, const double *voxel_sizes, const double *origins, int32_t *stat,
                                     void *workspace, size_t workspace_bytes, fvgb_stream_t stream) {
    size_t need = 0;
    const int st = fvgb_leaf_hash_workspace(n, &need);
    if (st) return st;
    if (num_grids < 1 || num_grids > kHashMaxGrids || !rows || !joffsets || !stat) return FVGB_EINVAL;
    if (dtype >= 0 && (!voxel_sizes || !origins)) return FVGB_EINVAL;
    if (dtype >= 0 && dtype != FVGB_F32 && dtype != FVGB_F64 && dtype != FVGB_F16 && dtype != FVGB_BF16)
        return FVGB_ETYPE;
    if (!workspace || workspace_bytes < need) return FVGB_ENOSPACE;
    cudaStream_t s = as_stream(stream);
    LeafHash h;
    leaf_hash_layout(n, &h, align_ws(workspace));
    if (cudaMemsetAsync(h.table, 0xff, (size_t)h.cap * 8, s) != cudaSuccess ||
        cudaMemsetAsync(h.mask, 0, (size_t)(reinterpret_cast<char *>(h.taken + kTakenCounters * 32) - reinterpret_cast<char *>(h.mask)),
                        s) != cudaSuccess)
        return launch_status();
    stat_init_kernel<<<(unsigned)ceil_div(num_grids + 9, 256), 256, 0, s>>>(stat, num_grids + 9);
    if (dtype < 0) launch_insert<int32_t, float>(rows, joffsets, num_grids, n, nullptr, nullptr, h, stat, s);
    else if (dtype == FVGB_F64) launch_insert<double, double>(rows, joffsets, num_grids, n, voxel_sizes, origins, h, stat, s);
    else if (dtype == FVGB_F16) launch_insert<__half, float>(rows, joffsets, num_grids, n, voxel_sizes, origins, h, stat, s);
    else if (dtype == FVGB_BF16)
        launch_insert<__nv_bfloat16, float>(rows, joffsets, num_grids, n, voxel_sizes, origins, h, stat, s);
    else launch_insert<float, float>(rows, joffsets, num_grids, n, voxel_sizes, origins, h, stat, s);
    count_launches(1);
    return launch_status();
}

extern "C" int fvgb_leaf_hash_finish_workspace(int64_t num_leaves, size_t *bytes) {
    if (!bytes || num_leaves < 1 || num_leaves >= INT32_MAX) return FVGB_EINVAL;
    *bytes = leaf_sort_layout(num_leaves, nullptr, nullptr) + 256;
    return FVGB_OK;
}

extern "C" int fvgb_leaf_hash_finish(int64_t n, int32_t num_grids, int64_t num_leaves, const int32_t box_lo[3],
                                     const int32_t box_hi[3], void *insert_workspace, size_t insert_bytes,
                                     int32_t *out_ijk, int64_t *out_joffsets, FvgbLeaf *leaves, int32_t *hash_slots,
                                     int64_t hash_capacity, void *workspace, size_t workspace_bytes,
                                     fvgb_stream_t stream) {
    size_t need = 0, need_insert = 0;
    int st = fvgb_leaf_hash_finish_workspace(num_leaves, &need);
    if (!st) st = fvgb_leaf_hash_workspace(n, &need_insert);
    if (st) return st;
    if (num_grids < 1 || num_grids > kHashMaxGrids || !out_ijk || !out_joffsets || !leaves || !hash_slots || !box_lo ||
        !box_hi || hash_capacity < 2 * num_leaves || (hash_capacity & (hash_capacity - 1)))
        return FVGB_EINVAL;
    for (int a = 0; a < 3; ++a)
        if (box_lo[a] > box_hi[a]) return FVGB_EINVAL;
    if (!insert_workspace || insert_bytes < need_insert || !workspace || workspace_bytes < need) return FVGB_ENOSPACE;
    cudaStream_t s = as_stream(stream);
    LeafHash h;
    leaf_hash_layout(n, &h, align_ws(insert_workspace));
    if (num_leaves > h.max_leaves) return FVGB_EINVAL;
    LeafSortWs w;
    leaf_sort_layout(num_leaves, &w, align_ws(workspace));
    const int64_t L = num_leaves;
    const int end_bit = order_key_end_bit(box_lo, box_hi);
    const int vb = end_bit > 9 ? end_bit - 9 : 0;
    const uint64_t low = (1ull << vb) - 1ull;
    int grid_bits = 0;
    while ((1 << grid_bits) < num_grids) ++grid_bits;
    const int bits = std::max(1, vb + grid_bits);
    uint32_t *ka = reinterpret_cast<uint32_t *>(w.keys_a), *kb = reinterpret_cast<uint32_t *>(w.keys_b);
    const unsigned warps = (unsigned)ceil_div(L, 8), ranks = (unsigned)ceil_div(L, 32);
    if (L <= kTileLeaves) {
        const unsigned tiles = (unsigned)ceil_div(L, (int64_t)kSortTile);
        if (bits <= 32) {
            leaf_tile_kernel<uint32_t><<<tiles, kSortTile, 0, s>>>(h, L, low, vb, ka, w.vals_a, hash_slots, hash_capacity);
            leaf_rank_kernel<uint32_t><<<ranks, 256, 0, s>>>(h, (int32_t)L, ka, w.vals_a, w.vals_b, w.count, w.grid);
        } else {
            leaf_tile_kernel<uint64_t><<<tiles, kSortTile, 0, s>>>(h, L, low, vb, w.keys_a, w.vals_a, hash_slots,
                                                                  hash_capacity);
            leaf_rank_kernel<uint64_t><<<ranks, 256, 0, s>>>(h, (int32_t)L, w.keys_a, w.vals_a, w.vals_b, w.count, w.grid);
        }
        leaf_scan_kernel<<<1, kScanThreads, 0, s>>>((int32_t)L, w.count, w.grid, num_grids, w.first, out_joffsets);
        leaf_emit_kernel<<<warps, 256, 0, s>>>(h, L, w.vals_b, w.first, out_ijk, leaves, hash_slots, hash_capacity);
        count_launches(4);
        return launch_status();
    }
    if (cudaMemsetAsync(hash_slots, 0xff, sizeof(int32_t) * hash_capacity, s) != cudaSuccess) return launch_status();
    size_t tb = w.cub_bytes;
    if (bits <= 32) {
        leaf_sort_keys_kernel<uint32_t><<<blocks_for(L), kThreads, 0, s>>>(h, L, low, vb, ka, w.vals_a);
        cub::DeviceRadixSort::SortPairs(w.cub_tmp, tb, ka, kb, w.vals_a, w.vals_b, (int)L, 0, bits, s);
    } else {
        leaf_sort_keys_kernel<uint64_t><<<blocks_for(L), kThreads, 0, s>>>(h, L, low, vb, w.keys_a, w.vals_a);
        cub::DeviceRadixSort::SortPairs(w.cub_tmp, tb, w.keys_a, w.keys_b, w.vals_a, w.vals_b, (int)L, 0, bits, s);
    }
    leaf_counts_kernel<<<blocks_for(L + 1), kThreads, 0, s>>>(h, L, w.vals_b, w.count);
    tb = w.cub_bytes;
    cub::DeviceScan::ExclusiveSum(w.cub_tmp, tb, w.count, w.first, (int)L + 1, s);
    leaf_emit_kernel<<<warps, 256, 0, s>>>(h, L, w.vals_b, w.first, out_ijk, leaves, hash_slots, hash_capacity);
    leaf_offsets_kernel<<<(unsigned)ceil_div(num_grids + 1, kThreads), kThreads, 0, s>>>(leaves, w.first, L, num_grids,
                                                                                         out_joffsets);
    count_launches(4);
    return launch_status();
}

extern "C" int fvgb_coarse_grid_index_workspace(int64_t num_fine_leaves, size_t *bytes) {
    if (!bytes || num_fine_leaves < 1 || num_fine_leaves > fvgb::kHashLeaves) return FVGB_EINVAL;
    *bytes = fvgb::coarse_hash_layout(num_fine_leaves, nullptr, nullptr) + 256;
    return FVGB_OK;
}

extern "C" int fvgb_coarse_grid_index(const FvgbGrid *fine, const int32_t factor[3], const int32_t box_lo[3],
                                      const int32_t box_hi[3], int32_t *out_ijk, int64_t *meta, FvgbLeaf *leaves,
                                      int32_t *hash_slots, int64_t hash_capacity, void *workspace,
                                      size_t workspace_bytes, fvgb_stream_t stream) {
    if (!fine || !factor || !meta || !out_ijk || !leaves || !hash_slots || !box_lo || !box_hi) return FVGB_EINVAL;
    if (fine->num_grids < 1 || fine->num_grids > kCoarseMaxGrids || !fine->leaves) return FVGB_EINVAL;
    size_t need = 0;
    const int64_t nl = fine->num_leaves;
    const int st = fvgb_coarse_grid_index_workspace(nl, &need);
    if (st) return st;
    if (hash_capacity < 2 * nl || (hash_capacity & (hash_capacity - 1))) return FVGB_EINVAL;
    if (!workspace || workspace_bytes < need) return FVGB_ENOSPACE;
    int sh[3];
    for (int a = 0; a < 3; ++a) {
        const int f = factor[a];
        if ((f != 1 && f != 2 && f != 4 && f != 8) || box_lo[a] > box_hi[a]) return FVGB_EINVAL;
        sh[a] = f == 1 ? 0 : (f == 2 ? 1 : (f == 4 ? 2 : 3));
    }
    const int3 shv = make_int3(sh[0], sh[1], sh[2]);
    const int end_bit = order_key_end_bit(box_lo, box_hi);
    const int vb = end_bit > 9 ? end_bit - 9 : 0;
    const uint64_t low_mask = end_bit >= 63 ? ~0ull : ((1ull << end_bit) - 1ull);
    int grid_bits = 0;
    while ((1 << grid_bits) < fine->num_grids) ++grid_bits;
    const int bits = vb + grid_bits;
    if (bits >= 64) return FVGB_ERANGE;  // a key of all ones is the table's free slot
    cudaStream_t s = as_stream(stream);
    CoarseHash h;
    coarse_hash_layout(nl, &h, align_ws(workspace));
    if (cudaMemsetAsync(h.table, 0xff, (size_t)(reinterpret_cast<char *>(h.found + 1) - reinterpret_cast<char *>(h.table)),
                        s) != cudaSuccess)
        return launch_status();
    coarse_insert_kernel<<<blocks_for(nl), kThreads, 0, s>>>(fine->leaves, nl, shv, low_mask, vb, h);
    coarse_or_kernel<<<(unsigned)ceil_div(nl, 8), 256, 0, s>>>(fine->leaves, nl, shv, h, hash_slots, hash_capacity);
    const unsigned ranks = (unsigned)ceil_div(nl, (int64_t)(kRankThreads / kRankSplit));
    if (bits <= 32) coarse_rank_kernel<uint32_t><<<ranks, kRankThreads, 0, s>>>(h);
    else coarse_rank_kernel<uint64_t><<<ranks, kRankThreads, 0, s>>>(h);
    coarse_scan_kernel<<<1, kScanThreads, 0, s>>>(h, fine->num_grids, meta);
    coarse_place_kernel<<<(unsigned)ceil_div(nl, 8), 256, 0, s>>>(h, out_ijk, leaves, hash_slots, hash_capacity);
    count_launches(5);
    return launch_status();
}
