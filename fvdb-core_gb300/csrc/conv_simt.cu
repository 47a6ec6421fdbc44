// CUDA-core contractions: the plain FP32 form (no TF32) and the FP64 form.
//
// Forward:  y[m,:] (+)= sum_k x[map[m,k],:] . W[k]   (one CTA owns a 128x64 output tile; every
//           output element is written exactly once, no atomics).  Offsets whose 128 map entries
//           are all -1 are skipped.  With the transposed map and W^T strides the same kernel is
//           the data gradient.
// Wgrad:    dW[k,ci,co] = sum_m x[map[m,k],ci] * dy[m,co] with per-CTA partials and a
//           fixed-order FP64 reduction across CTAs.
//
// Replaces the gather -> torch::mm_out -> scatter loop of
// src/fvdb/detail/ops/convolution/backend/SparseConvolutionKernelMap.cu:116-415.
#include "common.cuh"

namespace fvgb {
namespace {

constexpr int NT = 256;

template <typename T>
struct Vec4;
template <>
struct Vec4<float> {
    __device__ static void load(const float *p, float (&v)[4]) {
        const float4 q = *reinterpret_cast<const float4 *>(p);
        v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
    }
};
template <>
struct Vec4<double> {
    __device__ static void load(const double *p, double (&v)[4]) {
        const double2 a = *reinterpret_cast<const double2 *>(p), b = *reinterpret_cast<const double2 *>(p + 2);
        v[0] = a.x, v[1] = a.y, v[2] = b.x, v[3] = b.y;
    }
};

// One 16-byte vector from p (zeros for null)
__device__ __forceinline__ void ldvec(const float *p, float *v) {
    const float4 q = p ? __ldg(reinterpret_cast<const float4 *>(p)) : make_float4(0.f, 0.f, 0.f, 0.f);
    v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
}
__device__ __forceinline__ void ldvec(const double *p, double *v) {
    const double2 q = p ? __ldg(reinterpret_cast<const double2 *>(p)) : make_double2(0.0, 0.0);
    v[0] = q.x, v[1] = q.y;
}

// One CTA per FM-row x FN-channel output tile, a thread per 8 rows x 4 channels: 128 x 64, or 128 x 32
// where the last 64 channels would be at most half used (64->32 FP32, 0.11M voxels: 438 us with
// 64-wide tiles, 334 us with 256 x 32, whose 427 CTAs left the second wave half empty, 280 us with 128 x 32).  Per
// offset with any present row and per 16-channel slice (8 for FP64), the gathered rows (transposed, so a
// thread's 8 rows are two vector loads) and the weight slice go through shared memory; the
// slice after is loaded into registers while this one is multiplied, so one barrier per slice
// separates the two shared-memory buffers.  VEC (whole 16-byte pieces in x rows and W columns,
// W's output channels contiguous): operands are fetched 16 bytes at a time; with one element per
// load the fetches and their bounds checks took a third of the issue slots (0.11M voxels, row
// order, the 32->64->32 FP32 training step's four contractions: 1.69 ms element by element, 1.34 ms
// in vectors).
constexpr int kStageK = 32;  // offsets up to which a tile's map rows are staged in shared memory

// What an output value gets on its way out: the channel's bias, then the ReLU -- the additions and
// comparisons of separate passes over y, without the passes (0.11M x 64 FP32: 12 us each, and a launch).
template <typename T>
struct Finish {
    const T *bias;  // [cout], null: none
    int32_t relu;
    __device__ __forceinline__ T operator()(T v, int32_t n) const {
        if (bias) v = v + __ldg(bias + n);
        return relu && v < T(0) ? T(0) : v;  // NaN stays
    }
};

template <typename T, bool VEC, int FM, int FN>
__global__ void __launch_bounds__((FM / 8) * (FN / 4)) conv_fwd_simt_kernel(const T *__restrict__ x, int64_t n_x, int32_t cin,
                                                           int64_t ldx, const int32_t *__restrict__ map,
                                                           int64_t n_out, int32_t K, int64_t ldm,
                                                           const T *__restrict__ w, int64_t wsk, int64_t wsci,
                                                           int64_t wsco, T *__restrict__ y, int32_t cout,
                                                           int64_t ldy, int32_t accumulate,
                                                           const int32_t *__restrict__ out_rows, Finish<T> fin) {
    // map row m (m < n_out) computes output row out_rows[m] (m itself when out_rows is null)
    constexpr int NT = (FM / 8) * (FN / 4);  // threads: 8 rows x 4 channels each
    constexpr int FK = sizeof(T) == 8 ? 8 : 16;  // channels per slice (static shared memory < 48 KB)
    constexpr int QA = FM * FK / NT, QB = FK * FN / NT;
    // the tile's map rows, all offsets, where they were staged (K <= kStageK): one coalesced read, and
    // the offsets no row has are known at once; else one offset's column at a time
    extern __shared__ __align__(16) int32_t tile_map[];
    __shared__ int32_t rows[2][FM];
    __shared__ uint32_t wmask[NT / 32];
    __shared__ __align__(16) T As[2][FK][FM + 4];
    __shared__ __align__(16) T Bs[2][FK][FN + 4];
    const int tid = threadIdx.x, tx = tid % (FN / 4), ty = tid / (FN / 4);
    const int64_t m0 = (int64_t)blockIdx.x * FM;
    const int32_t n0 = blockIdx.y * FN;
    T acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = T(0);

    const bool staged = K <= kStageK;
    uint32_t offsets = 0;  // staged: the offsets some row of the tile has
    if (staged) {
        const int64_t n_here = n_out - m0 < FM ? n_out - m0 : FM;
        const int32_t words = (int32_t)n_here * K;
        uint32_t mine = 0;
        // kBatch entries in flight per thread (one at a time a tile waited fourteen times for its map: 1.05M
        // scattered rows in row order, one offset per tile, 32->33 FP32: 484 us)
        constexpr int kBatch = 8;
        const int step = NT % K;  // of an entry's offset from one entry of a thread to its next
        int k = tid % K;
        for (int e0 = tid; e0 < FM * K; e0 += kBatch * NT) {
            int32_t v[kBatch];
#pragma unroll
            for (int i = 0; i < kBatch; ++i) {
                const int e = e0 + i * NT;
                v[i] = e >= words ? -1 : ldm == K ? __ldg(map + m0 * K + e) : __ldg(map + (m0 + e / K) * ldm + e % K);
            }
#pragma unroll
            for (int i = 0; i < kBatch; ++i) {
                const int e = e0 + i * NT;
                if (e < FM * K) {
                    tile_map[e] = v[i] < n_x ? v[i] : -1;
                    if (v[i] >= 0 && v[i] < n_x) mine |= 1u << k;
                }
                k += step;
                if (k >= K) k -= K;
            }
        }
        mine = __reduce_or_sync(0xffffffffu, mine);
        if ((tid & 31) == 0) wmask[tid >> 5] = mine;
        __syncthreads();
#pragma unroll
        for (int i = 0; i < NT / 32; ++i) offsets |= wmask[i];
    }
    // rows of offset k into rows[rb]; true if any is present (a CTA-wide vote)
    auto load_rows = [&](int32_t k, int rb) -> bool {
        if (staged) return (offsets >> k) & 1u;
        int valid = 0;
        for (int t = tid; t < FM; t += NT) {
            const int64_t r = m0 + t;
            int32_t v = r < n_out ? map[r * ldm + k] : -1;
            if (v >= n_x) v = -1;
            rows[rb][t] = v;
            valid |= v >= 0;
        }
        return __syncthreads_or(valid) != 0;
    };
    // per thread: A elements e = tid + 256 q (q < QA) -> (row e / FK, channel e % FK); B elements
    // e = tid + 256 q (q < QB) -> (channel e / 64, column e % 64)
    // VEC: the same slices in 16-byte vectors of VW elements
    constexpr int VW = 16 / sizeof(T), VA = QA / VW, VB = (QB + VW - 1) / VW;
    T ra[QA], rb4[VB * VW];
    auto fetch = [&](int32_t k, int32_t c0, int rbuf) {
        if constexpr (VEC) {
#pragma unroll
            for (int q = 0; q < VA; ++q) {
                const int e = tid + q * NT, r = e / (FK / VW), c = (e % (FK / VW)) * VW;
                const int32_t src = staged ? tile_map[r * K + k] : rows[rbuf][r];
                const bool on = src >= 0 && c0 + c < cin;
                ldvec(on ? x + (int64_t)src * ldx + c0 + c : nullptr, &ra[q * VW]);
            }
#pragma unroll
            for (int q = 0; q < VB; ++q) {
                const int e = tid + q * NT, c = e / (FN / VW), n = (e % (FN / VW)) * VW;
                const bool on = c < FK && c0 + c < cin && n0 + n < cout;
                ldvec(on ? w + k * wsk + (int64_t)(c0 + c) * wsci + n0 + n : nullptr, &rb4[q * VW]);
            }
        } else {
#pragma unroll
            for (int q = 0; q < QA; ++q) {
                const int e = tid + q * NT, r = e / FK, c = e % FK;
                const int32_t src = staged ? tile_map[r * K + k] : rows[rbuf][r];
                ra[q] = (src >= 0 && c0 + c < cin) ? x[(int64_t)src * ldx + c0 + c] : T(0);
            }
#pragma unroll
            for (int q = 0; q < QB; ++q) {
                const int e = tid + q * NT, c = e / FN, n = e % FN;
                rb4[q] = (c0 + c < cin && n0 + n < cout)
                             ? w[k * wsk + (int64_t)(c0 + c) * wsci + (int64_t)(n0 + n) * wsco]
                             : T(0);
            }
        }
    };
    auto store = [&](int buf) {
        if constexpr (VEC) {
#pragma unroll
            for (int q = 0; q < VA; ++q) {
                const int e = tid + q * NT, r = e / (FK / VW), c = (e % (FK / VW)) * VW;
#pragma unroll
                for (int v = 0; v < VW; ++v) As[buf][c + v][r] = ra[q * VW + v];
            }
#pragma unroll
            for (int q = 0; q < VB; ++q) {
                const int e = tid + q * NT, c = e / (FN / VW), n = (e % (FN / VW)) * VW;
                if (c < FK)
#pragma unroll
                    for (int v = 0; v < VW; ++v) Bs[buf][c][n + v] = rb4[q * VW + v];
            }
        } else {
#pragma unroll
            for (int q = 0; q < QA; ++q) {
                const int e = tid + q * NT;
                As[buf][e % FK][e / FK] = ra[q];
            }
#pragma unroll
            for (int q = 0; q < QB; ++q) {
                const int e = tid + q * NT;
                Bs[buf][e / FN][e % FN] = rb4[q];
            }
        }
    };

    // walk (offset, channel slice) pairs, skipping offsets with no present row
    int32_t k = 0;
    int rbuf = 0;
    while (k < K && !load_rows(k, rbuf)) ++k;
    if (k < K) {
        int32_t c0 = 0;
        fetch(k, c0, rbuf);
        store(0);
        __syncthreads();
        int buf = 0;
        while (true) {
            // the next (offset, slice)
            int32_t kn = k, cn = c0 + FK;
            int rn = rbuf;
            if (cn >= cin) {
                cn = 0;
                rn = rbuf ^ 1;
                ++kn;
                while (kn < K && !load_rows(kn, rn)) ++kn;
            }
            const bool more = kn < K;
            if (more) fetch(kn, cn, rn);
#pragma unroll
            for (int c = 0; c < FK; ++c) {
                T a[8], b[4];
                T a0[4], a1[4];
                Vec4<T>::load(&As[buf][c][ty * 8], a0);
                Vec4<T>::load(&As[buf][c][ty * 8 + 4], a1);
#pragma unroll
                for (int i = 0; i < 4; ++i) a[i] = a0[i], a[i + 4] = a1[i];
                Vec4<T>::load(&Bs[buf][c][tx * 4], b);
#pragma unroll
                for (int i = 0; i < 8; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc[i][j] = fma(a[i], b[j], acc[i][j]);
            }
            if (!more) break;
            store(buf ^ 1);
            __syncthreads();
            buf ^= 1;
            k = kn, c0 = cn, rbuf = rn;
        }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int64_t t = m0 + ty * 8 + i;
        if (t >= n_out) continue;
        const int64_t r = out_rows ? (int64_t)out_rows[t] : t;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int32_t n = n0 + tx * 4 + j;
            if (n >= cout) continue;
            T *dst = y + r * ldy + n;
            *dst = fin(accumulate ? (T)(*dst + acc[i][j]) : acc[i][j], n);
        }
    }
}

// Short rows: few output channels, or few rows.  A lane group of
// cout / 4 lanes owns one output row and walks that row's present entries only -- the tiles above
// multiply an offset for all of their rows as soon as one row has it -- with the whole weight tensor
// in shared memory.  Sums run over offsets, then channels, as in the tiles: the same results.
// 20,000 scattered voxels (2.9 of 27 offsets present per row), 16->16: 55 us in 128 x 64 tiles,
// 13 us here, bound by the latency of one row's dependent loads.
constexpr int kShortSmem = 96 * 1024;

template <typename T>
__global__ void __launch_bounds__(NT) conv_fwd_short_kernel(const T *__restrict__ x, int64_t n_x, int32_t cin, int64_t ldx,
                                                            const int32_t *__restrict__ map, int64_t n_out, int32_t K,
                                                            int64_t ldm, const T *__restrict__ w, int64_t wsk,
                                                            int64_t wsci, T *__restrict__ y, int32_t cout, int64_t ldy,
                                                            int32_t accumulate, const int32_t *__restrict__ out_rows,
                                                            int gs, Finish<T> fin) {
    constexpr int VW = 16 / sizeof(T);
    extern __shared__ __align__(16) uint8_t short_smem[];
    T *ws = reinterpret_cast<T *>(short_smem);  // [K][cin][cout]
    const int lane = threadIdx.x & 31;
    const int G = 1 << gs, gl = lane & (G - 1);
    const int64_t m = ((int64_t)blockIdx.x * NT + threadIdx.x) >> gs;
    // the row's occupancy, entries shared over the group's lanes
    uint32_t present = 0;
    if (m < n_out)
        for (int k = gl; k < K; k += G) {
            const int32_t v = __ldg(map + m * ldm + k);
            if (v >= 0 && v < n_x) present |= 1u << k;
        }
    for (int o = 1; o < G; o <<= 1) present |= __shfl_xor_sync(0xffffffffu, present, o);
    const int cv = cout / VW;
    for (int e = threadIdx.x; e < K * cin * cv; e += NT) {
        const int k = e / (cin * cv), ci = (e / cv) % cin, c = (e % cv) * VW;
        T t[VW];
        ldvec(w + k * wsk + (int64_t)ci * wsci + c, t);
#pragma unroll
        for (int i = 0; i < VW; ++i) ws[(k * cin + ci) * cout + c + i] = t[i];
    }
    __syncthreads();
    if (m >= n_out || gl * 4 >= cout) return;
    T acc[4] = {T(0), T(0), T(0), T(0)};
    while (present) {
        const int k = __ffs(present) - 1;
        present &= present - 1;
        const T *xr = x + (int64_t)__ldg(map + m * ldm + k) * ldx;
        const T *wk = ws + k * cin * cout + gl * 4;
        for (int c0 = 0; c0 < cin; c0 += 8) {
            T xv[8];
#pragma unroll
            for (int c = 0; c < 8; c += VW) ldvec(c0 + c < cin ? xr + c0 + c : nullptr, &xv[c]);
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                if (c0 + c >= cin) break;
                T b[4];
                Vec4<T>::load(wk + (c0 + c) * cout, b);
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[j] = fma(xv[c], b[j], acc[j]);
            }
        }
    }
    const int64_t r = out_rows ? (int64_t)out_rows[m] : m;
    T *dst = y + r * ldy + gl * 4;
#pragma unroll
    for (int j = 0; j < 4; ++j) dst[j] = fin(accumulate ? (T)(dst[j] + acc[j]) : acc[j], gl * 4 + j);
}

template <typename T>
int launch_fwd_simt(const void *x, int64_t n_x, int32_t cin, int64_t ldx, const int32_t *map, int64_t n_out, int32_t K,
                    int64_t ldm, const void *w, int64_t wsk, int64_t wsci, int64_t wsco, void *y, int32_t cout,
                    int64_t ldy, int32_t accumulate, const int32_t *rows, const void *bias, int32_t relu, cudaStream_t s) {
    const Finish<T> fin{(const T *)bias, relu};
    constexpr int VW = 16 / sizeof(T);
    const bool vec = cin % VW == 0 && ldx % VW == 0 && wsco == 1 && cout % VW == 0 && wsk % VW == 0 && wsci % VW == 0 &&
                     (((uintptr_t)x | (uintptr_t)w) & 15) == 0;
    // The short-row kernel: 16 channels and fewer always (a 64-wide tile would be three quarters empty; 16->16,
    // 1.2M surface voxels: 1135 us in 64-wide tiles, 706; 0.9M of a dense block 1385 and 956).  Up to 32
    // channels where rows and channels are few: it multiplies present entries only but reads every weight for
    // four products, so it wins by more the fewer entries rows have, and loses on dense blocks.  16->32, us
    // among other calls, in 32-wide tiles and here: dense blocks 8k rows 33 and 35, 16k 34 and 49, 33k 43 and
    // 86; surfaces 9k 33 and 25, 22k 39 and 46, 56k 48 and 82; random voxels at 8 % 20k 31 and 18, 59k 36 and
    // 37.  8->32: dense 16k 33 and 29, 33k 43 and 50, surfaces 56k 47 and 46, random 59k 36 and 23.
    const int64_t wbytes = (int64_t)K * cin * cout * sizeof(T);
    if (vec && cout % 4 == 0 && K <= 32 && wbytes <= kShortSmem &&
        (cout <= 16 || (cout <= 32 && n_out < ((int64_t)1 << 16) && (cin <= 8 || n_out * cin <= (int64_t)7 << 15)))) {
        int gs = 0;
        while ((4 << gs) < cout) ++gs;
        if (set_dynamic_smem(conv_fwd_short_kernel<T>, kShortSmem) != cudaSuccess) return launch_status();
        conv_fwd_short_kernel<T><<<(unsigned)ceil_div(n_out << gs, (int64_t)NT), NT, (size_t)wbytes, s>>>(
            (const T *)x, n_x, cin, ldx, map, n_out, K, ldm, (const T *)w, wsk, wsci, (T *)y, cout, ldy, accumulate, rows,
            gs, fin);
        return FVGB_OK;
    }
    const bool narrow = cout % 64 != 0 && cout % 64 <= 32;
    const int fm = 128, fn = narrow ? 32 : 64, threads = narrow ? 128 : 256;
    const dim3 grid((unsigned)ceil_div(n_out, fm), (unsigned)ceil_div(cout, fn));
    if (ceil_div(cout, fn) > 65535) return FVGB_EINVAL;
    const int smem = K <= kStageK ? fm * K * 4 : 0;
    auto go = [&](auto kern) {
        if (set_dynamic_smem(kern, smem) != cudaSuccess) return;
        kern<<<grid, threads, smem, s>>>((const T *)x, n_x, cin, ldx, map, n_out, K, ldm, (const T *)w, wsk, wsci, wsco, (T *)y, cout,
                                 ldy, accumulate, rows, fin);
    };
    if (narrow) {
        if (vec) go(conv_fwd_simt_kernel<T, true, 128, 32>);
        else go(conv_fwd_simt_kernel<T, false, 128, 32>);
    } else {
        if (vec) go(conv_fwd_simt_kernel<T, true, 128, 64>);
        else go(conv_fwd_simt_kernel<T, false, 128, 64>);
    }
    return FVGB_OK;
}

// Rows per wgrad chunk so that the grid has enough CTAs; deterministic in the sizes only.
struct WgradPlan {
    int64_t chunks, rows_per_chunk;
    int32_t tm, tn;              // tile of dW: tm input x tn output channels (32 or 64 each)
    int32_t tiles_ci, tiles_co;
};

// 64 wide unless the last 64 would be at most half used
int32_t wgrad_tile(int32_t c) { return c % 64 == 0 || c % 64 > 32 ? 64 : 32; }

WgradPlan wgrad_plan(int64_t n_out, int32_t K, int32_t cin, int32_t cout) {
    WgradPlan p;
    p.tm = wgrad_tile(cin);
    p.tn = wgrad_tile(cout);
    p.tiles_ci = (int32_t)ceil_div(cin, p.tm);
    p.tiles_co = (int32_t)ceil_div(cout, p.tn);
    const int64_t per_chunk_ctas = (int64_t)K * p.tiles_ci * p.tiles_co;
    int64_t chunks = ceil_div(2048, per_chunk_ctas);
    const int64_t max_chunks = ceil_div(n_out > 0 ? n_out : 1, 256);
    if (chunks > max_chunks) chunks = max_chunks;
    if (chunks < 1) chunks = 1;
    p.rows_per_chunk = ceil_div(ceil_div(n_out > 0 ? n_out : 1, chunks), 16) * 16;
    p.chunks = ceil_div(n_out > 0 ? n_out : 1, p.rows_per_chunk);
    return p;
}

// dW partials of one (row chunk, offset, TM x TN channel tile) per CTA.  The chunk's map column is
// read 256 rows at a time and its present entries are queued in row order, so the products run over
// whole batches of BKP present (input row, output row) pairs: an offset of a surface grid is present
// in under half of the rows, which the products would otherwise spend on zeros.  The 256 threads
// form SL slices of TM x TN / 16 threads (4 x 4 outputs each); slice s takes pairs s, s + SL, ... of
// a batch and the slices are added in order at the end, so a narrow tile keeps every thread busy.
// The next batch is loaded into registers while this one is multiplied.  0.11M voxels, 32->64 and
// 64->32 FP32, 3^3: 732 us each with zero rows and 64 x 64 tiles, 203 us here.
constexpr int kPairQueue = 512;  // a batch's leftover and the next 256 rows

template <typename T, int TM, int TN, bool VEC>
__global__ void __launch_bounds__(NT) wgrad_simt_kernel(const T *__restrict__ x, int64_t n_x, int32_t cin, int64_t ldx,
                                                        const int32_t *__restrict__ map, int64_t n_out, int32_t K,
                                                        int64_t ldm, const T *__restrict__ dy, int32_t cout,
                                                        int64_t lddy, int64_t rows_per_chunk, int32_t tiles_co,
                                                        T *__restrict__ partials) {
    constexpr int BKP = sizeof(T) == 8 ? 16 : 32;
    constexpr int TPS = TM * TN / 16, SL = NT / TPS;
    constexpr int VW = VEC ? 16 / sizeof(T) : 1;
    constexpr int XV = BKP * TM / VW, DV = BKP * TN / VW;            // vectors per batch
    constexpr int XQ = (XV + NT - 1) / NT, DQ = (DV + NT - 1) / NT;  // per thread
    __shared__ __align__(16) T pool[2 * BKP * (TM + 4 + TN + 4)];
    T(*Xs)[BKP][TM + 4] = reinterpret_cast<T(*)[BKP][TM + 4]>(pool);
    T(*Ds)[BKP][TN + 4] = reinterpret_cast<T(*)[BKP][TN + 4]>(pool + 2 * BKP * (TM + 4));
    __shared__ int2 queue[kPairQueue];
    __shared__ int32_t wcount[NT / 32];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int slice = tid / TPS, ty = (tid % TPS) / (TN / 4), tx = (tid % TPS) % (TN / 4);
    const int64_t chunk = blockIdx.x;
    const int32_t k = blockIdx.y;
    const int32_t ci0 = (blockIdx.z / tiles_co) * TM, co0 = (blockIdx.z % tiles_co) * TN;
    int64_t r0 = chunk * rows_per_chunk;
    const int64_t r_end = min(n_out, r0 + rows_per_chunk);
    T acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = T(0);
    int32_t head = 0, tail = 0;  // the same in every thread
    // queue present pairs until a batch is full or the chunk ends
    auto fill = [&]() {
        while (tail - head < BKP && r0 < r_end) {
            const int64_t r = r0 + tid;
            int32_t v = r < r_end ? map[r * ldm + k] : -1;
            if (v >= n_x) v = -1;
            const uint32_t present = __ballot_sync(0xffffffffu, v >= 0);
            if (lane == 0) wcount[warp] = __popc(present);
            __syncthreads();
            int before = 0, total = 0;
#pragma unroll
            for (int w = 0; w < NT / 32; ++w) {
                if (w < warp) before += wcount[w];
                total += wcount[w];
            }
            if (v >= 0)
                queue[(tail + before + __popc(present & ((1u << lane) - 1u))) & (kPairQueue - 1)] = make_int2(v, (int32_t)(r - chunk * rows_per_chunk));
            tail += total;
            r0 += NT;
            __syncthreads();
        }
    };
    T rx[XQ * VW], rd[DQ * VW];
    auto fetch = [&]() {
        const int cnt = min(BKP, tail - head);
#pragma unroll
        for (int q = 0; q < XQ; ++q) {
            const int e = tid + q * NT, p = e / (TM / VW), c = (e % (TM / VW)) * VW;
            const T *src = nullptr;
            if (e < XV && p < cnt && ci0 + c < cin)
                src = x + (int64_t)queue[(head + p) & (kPairQueue - 1)].x * ldx + ci0 + c;
            if constexpr (VEC) ldvec(src, &rx[q * VW]);
            else rx[q] = src ? *src : T(0);
        }
#pragma unroll
        for (int q = 0; q < DQ; ++q) {
            const int e = tid + q * NT, p = e / (TN / VW), c = (e % (TN / VW)) * VW;
            const T *src = nullptr;
            if (e < DV && p < cnt && co0 + c < cout)
                src = dy + (chunk * rows_per_chunk + queue[(head + p) & (kPairQueue - 1)].y) * lddy + co0 + c;
            if constexpr (VEC) ldvec(src, &rd[q * VW]);
            else rd[q] = src ? *src : T(0);
        }
        head += cnt;
    };
    auto store = [&](int buf) {
#pragma unroll
        for (int q = 0; q < XQ; ++q) {
            const int e = tid + q * NT, p = e / (TM / VW), c = (e % (TM / VW)) * VW;
            if (e < XV)
#pragma unroll
                for (int v = 0; v < VW; ++v) Xs[buf][p][c + v] = rx[q * VW + v];
        }
#pragma unroll
        for (int q = 0; q < DQ; ++q) {
            const int e = tid + q * NT, p = e / (TN / VW), c = (e % (TN / VW)) * VW;
            if (e < DV)
#pragma unroll
                for (int v = 0; v < VW; ++v) Ds[buf][p][c + v] = rd[q * VW + v];
        }
    };
    fill();
    if (tail > head) {
        fetch();
        store(0);
        __syncthreads();
        int buf = 0;
        while (true) {
            fill();
            const bool more = tail > head;
            if (more) fetch();
#pragma unroll 8
            for (int r = slice; r < BKP; r += SL) {
                T a[4], b[4];
                Vec4<T>::load(&Xs[buf][r][ty * 4], a);
                Vec4<T>::load(&Ds[buf][r][tx * 4], b);
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc[i][j] = fma(a[i], b[j], acc[i][j]);
            }
            if (!more) break;
            store(buf ^ 1);
            __syncthreads();
            buf ^= 1;
        }
    }
    if constexpr (SL > 1) {
        static_assert(2 * BKP * (TM + 4 + TN + 4) >= TM * TN, "the slice sums pass through the operand buffers");
        T *red = pool;
#pragma unroll
        for (int s = 1; s < SL; ++s) {
            __syncthreads();
            if (slice == s)
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) red[(ty * 4 + i) * TN + tx * 4 + j] = acc[i][j];
            __syncthreads();
            if (slice == 0)
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc[i][j] += red[(ty * 4 + i) * TN + tx * 4 + j];
        }
        if (slice != 0) return;
    }
    T *dst = partials + ((chunk * K + k) * (int64_t)cin) * cout;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int32_t ci = ci0 + ty * 4 + i;
        if (ci >= cin) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int32_t co = co0 + tx * 4 + j;
            if (co < cout) dst[(int64_t)ci * cout + co] = acc[i][j];
        }
    }
}

template <typename T, int TM, int TN>
void launch_wgrad_tile(const WgradPlan &p, const void *x, int64_t n_x, int32_t cin, int64_t ldx, const int32_t *map,
                       int64_t n_out, int32_t K, int64_t ldm, const void *dy, int32_t cout, int64_t lddy, void *part,
                       cudaStream_t s) {
    constexpr int VW = 16 / sizeof(T);
    const dim3 grid((unsigned)p.chunks, (unsigned)K, (unsigned)(p.tiles_ci * p.tiles_co));
    const bool vec = cin % VW == 0 && cout % VW == 0 && ldx % VW == 0 && lddy % VW == 0 &&
                     (((uintptr_t)x | (uintptr_t)dy) & 15) == 0;
    if (vec)
        wgrad_simt_kernel<T, TM, TN, true><<<grid, NT, 0, s>>>((const T *)x, n_x, cin, ldx, map, n_out, K, ldm,
                                                               (const T *)dy, cout, lddy, p.rows_per_chunk, p.tiles_co,
                                                               (T *)part);
    else
        wgrad_simt_kernel<T, TM, TN, false><<<grid, NT, 0, s>>>((const T *)x, n_x, cin, ldx, map, n_out, K, ldm,
                                                                (const T *)dy, cout, lddy, p.rows_per_chunk, p.tiles_co,
                                                                (T *)part);
}

template <typename T>
void launch_wgrad_simt(const WgradPlan &p, const void *x, int64_t n_x, int32_t cin, int64_t ldx, const int32_t *map,
                       int64_t n_out, int32_t K, int64_t ldm, const void *dy, int32_t cout, int64_t lddy, void *part,
                       cudaStream_t s) {
    if (p.tm == 64 && p.tn == 64)
        launch_wgrad_tile<T, 64, 64>(p, x, n_x, cin, ldx, map, n_out, K, ldm, dy, cout, lddy, part, s);
    else if (p.tm == 64)
        launch_wgrad_tile<T, 64, 32>(p, x, n_x, cin, ldx, map, n_out, K, ldm, dy, cout, lddy, part, s);
    else if (p.tn == 64)
        launch_wgrad_tile<T, 32, 64>(p, x, n_x, cin, ldx, map, n_out, K, ldm, dy, cout, lddy, part, s);
    else
        launch_wgrad_tile<T, 32, 32>(p, x, n_x, cin, ldx, map, n_out, K, ldm, dy, cout, lddy, part, s);
}

// dW[e] = sum over chunks (ascending) of partials[chunk][e], accumulated in FP64.
template <typename AccT, typename OutT>
__global__ void wgrad_reduce_kernel(const AccT *__restrict__ partials, int64_t chunks, int64_t per_chunk,
                                    OutT *__restrict__ dw) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= per_chunk) return;
    double s = 0.0;
#pragma unroll 16  // loads in flight; the sum keeps its order
    for (int64_t c = 0; c < chunks; ++c) s += (double)partials[c * per_chunk + e];
    dw[e] = (OutT)s;
}

}  // namespace
}  // namespace fvgb

using namespace fvgb;

extern "C" int fvgb_conv_fwd_simt(int32_t dtype, const void *x, int64_t n_x, int32_t c_in, int64_t ldx,
                                  const int32_t *map, int64_t n_out, int32_t K, int64_t ldm, const void *w,
                                  int64_t wsk, int64_t wsci, int64_t wsco, void *y, int32_t c_out, int64_t ldy,
                                  int32_t accumulate, fvgb_stream_t stream) {
    return fvgb_conv_fwd_simt_rows(dtype, x, n_x, c_in, ldx, map, n_out, K, ldm, nullptr, w, wsk, wsci, wsco, y, c_out,
                                   ldy, accumulate, stream);
}

namespace fvgb {
namespace {
int simt_forward(int32_t dtype, const void *x, int64_t n_x, int32_t c_in, int64_t ldx,
                                       const int32_t *map, int64_t n_out, int32_t K, int64_t ldm, const int32_t *rows,
                                       const void *w, int64_t wsk, int64_t wsci, int64_t wsco, void *y, int32_t c_out,
                                       int64_t ldy, int32_t accumulate, const void *bias, int32_t relu, fvgb_stream_t stream) {
    if (c_in < 1 || c_out < 1 || K < 1 || n_out < 0 || n_x < 0 || ldm < K || ldx < c_in || ldy < c_out)
        return FVGB_EINVAL;
    if (n_out == 0) return FVGB_OK;
    if (!map || !w || !y || (n_x > 0 && !x)) return FVGB_EINVAL;
    if (ceil_div(c_out, 64) > 65535) return FVGB_EINVAL;
    cudaStream_t s = as_stream(stream);
    int st;
    if (dtype == FVGB_F32)
        st = launch_fwd_simt<float>(x, n_x, c_in, ldx, map, n_out, K, ldm, w, wsk, wsci, wsco, y, c_out, ldy, accumulate,
                                    rows, bias, relu, s);
    else if (dtype == FVGB_F64)
        st = launch_fwd_simt<double>(x, n_x, c_in, ldx, map, n_out, K, ldm, w, wsk, wsci, wsco, y, c_out, ldy, accumulate,
                                     rows, bias, relu, s);
    else
        return FVGB_ETYPE;
    if (st) return st;
    count_launches(1);
    return launch_status();
}
}  // namespace
}  // namespace fvgb

extern "C" int fvgb_conv_fwd_simt_rows(int32_t dtype, const void *x, int64_t n_x, int32_t c_in, int64_t ldx,
                                       const int32_t *map, int64_t n_out, int32_t K, int64_t ldm, const int32_t *rows,
                                       const void *w, int64_t wsk, int64_t wsci, int64_t wsco, void *y, int32_t c_out,
                                       int64_t ldy, int32_t accumulate, fvgb_stream_t stream) {
    return simt_forward(dtype, x, n_x, c_in, ldx, map, n_out, K, ldm, rows, w, wsk, wsci, wsco, y, c_out, ldy, accumulate, nullptr, 0, stream);
}

extern "C" int fvgb_conv_fwd_simt_finish(int32_t dtype, const void *x, int64_t n_x, int32_t c_in, int64_t ldx,
                                       const int32_t *map, int64_t n_out, int32_t K, int64_t ldm, const int32_t *rows,
                                       const void *w, int64_t wsk, int64_t wsci, int64_t wsco, void *y, int32_t c_out,
                                       int64_t ldy, const void *bias, int32_t relu, fvgb_stream_t stream) {
    return simt_forward(dtype, x, n_x, c_in, ldx, map, n_out, K, ldm, rows, w, wsk, wsci, wsco, y, c_out, ldy, 0, bias, relu, stream);
}

extern "C" int fvgb_wgrad_workspace(int32_t dtype, int64_t n_out, int32_t K, int32_t c_in, int32_t c_out,
                                    size_t *bytes) {
    if (!bytes || K < 1 || c_in < 1 || c_out < 1 || n_out < 0) return FVGB_EINVAL;
    const WgradPlan p = wgrad_plan(n_out, K, c_in, c_out);
    const size_t elem = dtype == FVGB_F64 ? 8 : 4;
    *bytes = (size_t)p.chunks * K * c_in * c_out * elem + 256;
    return FVGB_OK;
}

extern "C" int fvgb_conv_wgrad_simt(int32_t dtype, const void *x, int64_t n_x, int32_t c_in, int64_t ldx,
                                    const int32_t *map, int64_t n_out, int32_t K, int64_t ldm, const void *dy,
                                    int32_t c_out, int64_t lddy, void *dw, void *workspace,
                                    size_t workspace_bytes, fvgb_stream_t stream) {
    if (c_in < 1 || c_out < 1 || K < 1 || n_out < 0 || n_x < 0 || ldm < K || ldx < c_in || lddy < c_out || !dw)
        return FVGB_EINVAL;
    size_t need = 0;
    fvgb_wgrad_workspace(dtype, n_out, K, c_in, c_out, &need);
    if (!workspace || workspace_bytes < need) return FVGB_ENOSPACE;
    const WgradPlan p = wgrad_plan(n_out, K, c_in, c_out);
    cudaStream_t s = as_stream(stream);
    const int64_t per_chunk = (int64_t)K * c_in * c_out;
    const dim3 grid((unsigned)p.chunks, (unsigned)K, (unsigned)(p.tiles_ci * p.tiles_co));
    if (grid.y > 65535 || grid.z > 65535) return FVGB_EINVAL;
    char *base = reinterpret_cast<char *>(((uintptr_t)workspace + 255) & ~(uintptr_t)255);
    if (dtype == FVGB_F32) {
        float *part = reinterpret_cast<float *>(base);
        if (n_out > 0)
            launch_wgrad_simt<float>(p, x, n_x, c_in, ldx, map, n_out, K, ldm, dy, c_out, lddy, part, s);
        wgrad_reduce_kernel<float, float><<<(unsigned)ceil_div(per_chunk, 256), 256, 0, s>>>(
            part, n_out > 0 ? p.chunks : 0, per_chunk, (float *)dw);
    } else if (dtype == FVGB_F64) {
        double *part = reinterpret_cast<double *>(base);
        if (n_out > 0)
            launch_wgrad_simt<double>(p, x, n_x, c_in, ldx, map, n_out, K, ldm, dy, c_out, lddy, part, s);
        wgrad_reduce_kernel<double, double><<<(unsigned)ceil_div(per_chunk, 256), 256, 0, s>>>(
            part, n_out > 0 ? p.chunks : 0, per_chunk, (double *)dw);
    } else {
        return FVGB_ETYPE;
    }
    count_launches(n_out > 0 ? 2 : 1);
    return launch_status();
}

// ---------------------------------------------------------------------------------------------
// Weight gradient that allocates nothing.
//
// Some callers cannot allocate device memory at the point where they need a weight gradient:
// plugins running inside a host runtime that plans every device buffer ahead of time and
// forbids allocation during execution, and latency-bound serving code that must not risk the
// implicit device synchronisation or the out-of-memory failure of cudaMalloc / cudaFree in the
// middle of a request.  fvgb_conv_wgrad_simt needs a caller-provided partials workspace; this
// variant keeps its per-CTA partials in a fixed device array of this file instead (4 MiB per
// device, held by every GPU that loads the library until the process exits).
//
// * The device address of the array is looked up once per device, with that device current,
//   by the first call on that device (cudaGetSymbolAddress); make that first call before any
//   stream capture.
// * Every call shares the one array and it keeps the previous call's contents.  Each call
//   overwrites every partial it later reads (no clearing needed), so consecutive calls are
//   independent -- but calls that overlap on the GPU (different streams, or concurrent host
//   threads) race on the array and must be serialised by the caller.
// * Sizes whose partials of one row chunk (K * c_in * c_out elements) exceed the array are
//   rejected with FVGB_ENOSPACE before any launch.
// ---------------------------------------------------------------------------------------------
#include <mutex>

static constexpr size_t kWgradScratchBytes = size_t(4) << 20;
static __device__ __align__(256) double fvgb_wgrad_scratch[kWgradScratchBytes / sizeof(double)];

namespace fvgb {
namespace {
constexpr int kMaxDevices = 64;
std::mutex g_scratch_mu;
void *g_scratch_ptr[kMaxDevices] = {};

// Device address of fvgb_wgrad_scratch on the current device (looked up once per device).
int wgrad_scratch_address(void **out) {
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return record_cuda(e);
    if (dev < 0 || dev >= kMaxDevices) return FVGB_EINVAL;
    std::lock_guard<std::mutex> lock(g_scratch_mu);
    if (!g_scratch_ptr[dev]) {
        void *p = nullptr;
        e = cudaGetSymbolAddress(&p, fvgb_wgrad_scratch);
        if (e != cudaSuccess) return record_cuda(e);
        g_scratch_ptr[dev] = p;
    }
    *out = g_scratch_ptr[dev];
    return FVGB_OK;
}
}  // namespace
}  // namespace fvgb

extern "C" int fvgb_conv_wgrad_simt_noalloc(int32_t dtype, const void *x, int64_t n_x, int32_t c_in, int64_t ldx,
                                            const int32_t *map, int64_t n_out, int32_t K, int64_t ldm,
                                            const void *dy, int32_t c_out, int64_t lddy, void *dw,
                                            fvgb_stream_t stream) {
    if (c_in < 1 || c_out < 1 || K < 1 || n_out < 0 || n_x < 0 || ldm < K || ldx < c_in || lddy < c_out || !dw)
        return FVGB_EINVAL;
    if (dtype != FVGB_F32 && dtype != FVGB_F64) return FVGB_ETYPE;
    if (K > 65535) return FVGB_EINVAL;  // one grid row per kernel offset
    const size_t elem = dtype == FVGB_F64 ? 8 : 4;
    // K*c_in*c_out*elem <= the array, compared without overflow: K*c_in < 2^47 fits int64, and
    // for integers a*b > c  <=>  a > floor(c / b)
    const int64_t kc = (int64_t)K * c_in;
    if (kc > (int64_t)(kWgradScratchBytes / ((size_t)c_out * elem))) {
        record_message("fvgb_conv_wgrad_simt_noalloc: K*c_in*c_out partials exceed the 4 MiB scratch array");
        return FVGB_ENOSPACE;
    }
    const size_t per_chunk_bytes = (size_t)kc * (size_t)c_out * elem;
    const int64_t cap_chunks = (int64_t)(kWgradScratchBytes / per_chunk_bytes);
    void *scratch = nullptr;
    const int st = wgrad_scratch_address(&scratch);
    if (st != FVGB_OK) return st;
    WgradPlan p = wgrad_plan(n_out, K, c_in, c_out);
    if (p.chunks > cap_chunks) {
        p.rows_per_chunk = ceil_div(ceil_div(n_out > 0 ? n_out : 1, cap_chunks), 16) * 16;
        p.chunks = ceil_div(n_out > 0 ? n_out : 1, p.rows_per_chunk);
    }
    cudaStream_t s = as_stream(stream);
    const int64_t per_chunk = (int64_t)K * c_in * c_out;
    const dim3 grid((unsigned)p.chunks, (unsigned)K, (unsigned)(p.tiles_ci * p.tiles_co));
    if (grid.y > 65535 || grid.z > 65535) return FVGB_EINVAL;
    if (dtype == FVGB_F32) {
        float *part = reinterpret_cast<float *>(scratch);
        if (n_out > 0)
            launch_wgrad_simt<float>(p, x, n_x, c_in, ldx, map, n_out, K, ldm, dy, c_out, lddy, part, s);
        wgrad_reduce_kernel<float, float><<<(unsigned)ceil_div(per_chunk, 256), 256, 0, s>>>(
            part, n_out > 0 ? p.chunks : 0, per_chunk, (float *)dw);
    } else {
        double *part = reinterpret_cast<double *>(scratch);
        if (n_out > 0)
            launch_wgrad_simt<double>(p, x, n_x, c_in, ldx, map, n_out, K, ldm, dy, c_out, lddy, part, s);
        wgrad_reduce_kernel<double, double><<<(unsigned)ceil_div(per_chunk, 256), 256, 0, s>>>(
            part, n_out > 0 ? p.chunks : 0, per_chunk, (double *)dw);
    }
    count_launches(n_out > 0 ? 2 : 1);
    return launch_status();
}
