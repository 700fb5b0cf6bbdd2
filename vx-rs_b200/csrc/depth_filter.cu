// Depth-map post-filters (vx-vision's DepthFilter: kernels/depth_filter.rs,
// shaders/DepthFilter.metal), the step after WTA in vx-vision's depth chain:
// a median filter over the valid (> 0) values of a window, and an
// edge-preserving bilateral filter.
//
// Semantics (DepthFilter.metal:84-120, depth_median): the valid values of the
// (2r+1)^2 window with clamped coordinates, in raster order; the output is the
// element at index count/2 of their ascending order (the upper middle for an
// even count), or 0 when none is valid. Invalid SGM pixels (LR check, value
// -1) are therefore left out. (DepthFilter.metal:20-66, depth_bilateral): a
// centre <= 0 gives 0; otherwise the mean of the valid neighbours weighted by
// exp(-(dx^2+dy^2) / (2 ss^2)) * exp(-(n-c)^2 / (2 sd^2)), or the centre when
// the weights sum to at most 1e-8; single-precision arithmetic in the shader's
// order (up to radius 8 with the products fused into the sums). The exponentials
// are hardware approximations (a few ulp from expf, and Metal's fast-math exp is
// not exact either), so results agree with a host build to about 1e-6 relative
// (1e-7 against 64-bit arithmetic, rms).
//
// Mapping: a CTA stages its tile and the apron (clamped coordinates) in shared
// memory once. Median: column sorts and merges shared between windows (below).
// Bilateral: radii up to 8 four neighbouring pixels a thread (bilateral_rows_kernel),
// larger ones one thread per output pixel of a 32x8 tile; the spatial weights of the
// window are computed once per CTA.
#include <cuda_runtime.h>

#include <cmath>
#include <utility>

#include "launch.hpp"

namespace vxsgm {

namespace {

constexpr int kTileW = 32, kTileH = 8;

__device__ __forceinline__ int clampi(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }

// Stages the tile of the CTA and its apron of r pixels (clamped) into s (row
// stride tw = 32 + 2r).
__device__ __forceinline__ void stage_tile(const float* __restrict__ in, size_t pitch, int W, int H, int r,
                                           float* __restrict__ s) {
    const int tw = kTileW + 2 * r, th = kTileH + 2 * r;
    const int x0 = blockIdx.x * kTileW - r, y0 = blockIdx.y * kTileH - r;
    for (int i = threadIdx.y * kTileW + threadIdx.x; i < tw * th; i += kTileW * kTileH) {
        const int ty = i / tw, tx = i - ty * tw;
        const int gx = clampi(x0 + tx, 0, W - 1), gy = clampi(y0 + ty, 0, H - 1);
        s[i] = *reinterpret_cast<const float*>(reinterpret_cast<const char*>(in) + (size_t)gy * pitch +
                                               (size_t)gx * sizeof(float));
    }
}

// Median for a compile-time radius R >= 1. The window's values taken (> 0, +inf
// included) and the +inf standing in for invalid ones are positive floats, whose
// order is that of their bit patterns, so everything below is on uint32 (equal
// values have equal bits: any order of them gives the shader's pick).
//
// Work is shared between windows in two ways. Each column of 2R+1 values is
// sorted once and used by the 2R+1 windows of its row that hold it. A thread
// takes two neighbouring pixels, whose windows have 2R columns in common: these
// are merged once into the N/2 + 1 smallest values A (N the window size; only
// ranks count/2 <= N/2 are asked for, so the comparators that feed higher ranks
// are dead code), and each pixel's own column B then meets A in
//     rank k of the union = min over i of max(A[k - i], B[i - 1])
// (A, B below index 0 count as 0, below every value), with A in shared memory
// for its run-time index.
//
// Bound by the min / max operations (one every two cycles a scheduler) and, at
// small radii, by the latency of a CTA's four phases. 1920x1080, a quarter of the
// values invalid, whole calls (a call of no work takes 13 us): r = 1 26 us, r = 2
// 35 us (53 with a full sort of each window's 25 values), r = 3 57 us, r = 4 89 us,
// r = 5 171 us (2.4, 6.0 and 13.2 ms with every value ranked against the others).
//
// Sorting and merging are Batcher's odd-even networks, built at compile time as
// lists of comparators over register indices.
struct Net {
    int a[1024] = {}, b[1024] = {};
    int n = 0;
    constexpr void add(int x, int y) {
        a[n] = x;
        b[n] = y;
        ++n;
    }
};
struct Order {           // register indices whose values ascend
    int w[128] = {};
    int n = 0;
};
constexpr Order every_other(const Order& o, int first) {
    Order r;
    for (int i = first; i < o.n; i += 2) r.w[r.n++] = o.w[i];
    return r;
}
// Merge of two ascending runs: merge the even-indexed and the odd-indexed
// elements apart, then exchange neighbours where the results interleave.
constexpr Order merge_runs(Net& net, const Order& x, const Order& y) {
    if (x.n == 0) return y;
    if (y.n == 0) return x;
    if (x.n == 1 && y.n == 1) {
        net.add(x.w[0], y.w[0]);
        Order r;
        r.w[r.n++] = x.w[0];
        r.w[r.n++] = y.w[0];
        return r;
    }
    const Order v = merge_runs(net, every_other(x, 0), every_other(y, 0));
    const Order w = merge_runs(net, every_other(x, 1), every_other(y, 1));
    Order r;
    r.w[r.n++] = v.w[0];
    for (int i = 0; i < w.n || i + 1 < v.n; ++i) {
        if (i < w.n && i + 1 < v.n) net.add(w.w[i], v.w[i + 1]);
        if (i < w.n) r.w[r.n++] = w.w[i];
        if (i + 1 < v.n) r.w[r.n++] = v.w[i + 1];
    }
    return r;
}
constexpr Order sort_run(Net& net, int first, int n) {
    if (n == 1) {
        Order r;
        r.w[r.n++] = first;
        return r;
    }
    const Order x = sort_run(net, first, n / 2), y = sort_run(net, first + n / 2, n - n / 2);
    return merge_runs(net, x, y);
}
// Sorts n registers.
template <int N>
struct ColumnNet {
    Net net;
    Order order;
    constexpr ColumnNet() { order = sort_run(net, 0, N); }
};
// Merges `cols` sorted columns of n registers (column c: registers c*n..), pairs
// first, then pairs of the results.
constexpr Order merge_columns(Net& net, int first, int cols, int n) {
    if (cols == 1) {
        Order r;
        for (int i = 0; i < n; ++i) r.w[r.n++] = first * n + i;
        return r;
    }
    int half = 1;
    while (2 * half < cols) half *= 2;
    const Order x = merge_columns(net, first, half, n), y = merge_columns(net, first + half, cols - half, n);
    return merge_runs(net, x, y);
}
template <int COLS, int N>
struct MergeNet {
    Net net;
    Order order;
    constexpr MergeNet() { order = merge_columns(net, 0, COLS, N); }
};
template <int N>
constexpr ColumnNet<N> kColumnNet{};
template <int COLS, int N>
constexpr MergeNet<COLS, N> kMergeNet{};

template <int A, int B, int M>
__device__ __forceinline__ void compare_exchange(uint32_t (&v)[M]) {
    const uint32_t x = v[A], y = v[B];
    v[A] = min(x, y);
    v[B] = max(x, y);
}
template <int I, int M>
__device__ __forceinline__ uint32_t reg(const uint32_t (&v)[M]) {
    return v[I];
}
// p[i * stride] = the value of rank i.
template <int N, int... I>
__device__ __forceinline__ void store_column(const uint32_t (&v)[N], uint32_t* p, int stride,
                                             std::integer_sequence<int, I...>) {
    ((p[I * stride] = reg<kColumnNet<N>.order.w[I]>(v)), ...);
}
template <int COLS, int N, int... I>
__device__ __forceinline__ void store_merged(const uint32_t (&v)[COLS * N], uint32_t* p, int stride,
                                             std::integer_sequence<int, I...>) {
    ((p[I * stride] = reg<kMergeNet<COLS, N>.order.w[I]>(v)), ...);
}
template <int N, int... I>
__device__ __forceinline__ void sort_column(uint32_t (&v)[N], std::integer_sequence<int, I...>) {
    (compare_exchange<kColumnNet<N>.net.a[I], kColumnNet<N>.net.b[I]>(v), ...);
}
template <int COLS, int N, int... I>
__device__ __forceinline__ void merge_sorted(uint32_t (&v)[COLS * N], std::integer_sequence<int, I...>) {
    (compare_exchange<kMergeNet<COLS, N>.net.a[I], kMergeNet<COLS, N>.net.b[I]>(v), ...);
}

// A CTA's outputs: 64 x kMedianRows(R), two pixels a thread.
__host__ __device__ constexpr int median_rows(int r) { return r <= 2 ? 8 : 4; }
__host__ __device__ constexpr int median_cols(int r) { return 64 + 2 * r; }
// Shared memory: the raw tile, the sorted columns and their counts, the A runs.
template <int R>
struct MedianShape {
    static constexpr int n = 2 * R + 1, N = n * n, K = N / 2;
    static constexpr int rows = median_rows(R), cols = median_cols(R), threads = 32 * rows;
    static constexpr int raw = cols * (rows + 2 * R);
    static constexpr int sorted = n * rows * cols;      // [i][row][column]
    static constexpr int counts = rows * cols;
    static constexpr int runs = (n + K + 1) * threads;  // [n zeros, A[0..K]][thread]
    // The raw tile is dead once the columns are sorted: the runs take its place.
    static constexpr size_t bytes = 4ull * (sorted + counts + (raw > runs ? raw : runs));
};

template <int R>
__global__ void __launch_bounds__(MedianShape<R>::threads)
median_kernel(const float* __restrict__ in, size_t in_pitch, float* __restrict__ out, size_t out_pitch, int W,
              int H, int y_first) {
    using S = MedianShape<R>;
    constexpr int n = S::n;
    extern __shared__ __align__(16) uint32_t median_smem[];
    uint32_t* const sorted = median_smem;
    uint32_t* const counts = sorted + S::sorted;
    uint32_t* const raw = counts + S::counts;
    uint32_t* const runs = raw;
    const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * 32 + tx;
    constexpr uint32_t kInf = 0x7F800000u;

    // The tile and its apron (clamped), as bits.
    const int x0 = blockIdx.x * 64 - R, y0 = y_first + blockIdx.y * S::rows - R;
    for (int r = ty; r < S::rows + 2 * R; r += S::rows) {
        const char* row = reinterpret_cast<const char*>(in) + (size_t)clampi(y0 + r, 0, H - 1) * in_pitch;
        for (int c = tx; c < S::cols; c += 32)
            raw[r * S::cols + c] = reinterpret_cast<const uint32_t*>(row)[clampi(x0 + c, 0, W - 1)];
    }
    __syncthreads();
    // Every column of every output row, sorted, with its count of valid values: two
    // a thread, then the 2R right of the 64 outputs' by as few warps as they fill.
    auto sort_one = [&](int row, int c) {
        uint32_t v[n], count = 0;
#pragma unroll
        for (int i = 0; i < n; ++i) {
            const uint32_t b = raw[(row + i) * S::cols + c];
            const bool ok = __uint_as_float(b) > 0.0f;
            v[i] = ok ? b : kInf;
            count += ok ? 1u : 0u;
        }
        sort_column<n>(v, std::make_integer_sequence<int, kColumnNet<n>.net.n>{});
        store_column<n>(v, sorted + row * S::cols + c, S::rows * S::cols, std::make_integer_sequence<int, n>{});
        counts[row * S::cols + c] = count;
    };
    sort_one(ty, tx);
    sort_one(ty, tx + 32);
    if (tid < 2 * R * S::rows) sort_one(tid / (2 * R), 64 + tid % (2 * R));
    __syncthreads();

    // Pixels x and x + 1 (x even in the tile): columns c0 .. c0 + 2R + 1, the middle 2R shared.
    const int c0 = 2 * tx;
    uint32_t v[2 * R * n], first[n], last[n];
#pragma unroll
    for (int i = 0; i < n; ++i) {
        const uint2* row = reinterpret_cast<const uint2*>(sorted + (i * S::rows + ty) * S::cols + c0);
#pragma unroll
        for (int q = 0; q <= R; ++q) {                 // columns 2q, 2q + 1
            const uint2 p = row[q];
            if (q == 0) first[i] = p.x; else v[(2 * q - 1) * n + i] = p.x;
            if (q == R) last[i] = p.y; else v[2 * q * n + i] = p.y;
        }
    }
    uint32_t shared_count = 0;
#pragma unroll
    for (int c = 1; c <= 2 * R; ++c) shared_count += counts[ty * S::cols + c0 + c];
    const uint32_t count0 = shared_count + counts[ty * S::cols + c0];
    const uint32_t count1 = shared_count + counts[ty * S::cols + c0 + 2 * R + 1];
    merge_sorted<2 * R, n>(v, std::make_integer_sequence<int, kMergeNet<2 * R, n>.net.n>{});
#pragma unroll
    for (int i = 0; i < n; ++i) runs[i * S::threads + tid] = 0u;
    store_merged<2 * R, n>(v, runs + n * S::threads + tid, S::threads, std::make_integer_sequence<int, S::K + 1>{});

    // Rank count/2 of A and the pixel's own column. (A thread reads its own runs only.)
    auto pick = [&](const uint32_t (&b)[n], uint32_t count) {
        const uint32_t* a = runs + (n + (int)(count / 2)) * S::threads + tid;     // A[k]
        uint32_t best = a[0];
#pragma unroll
        for (int i = 1; i <= n; ++i) best = min(best, max(a[-i * S::threads], b[i - 1]));
        return count == 0u ? 0.0f : __uint_as_float(best);
    };
    const int x = blockIdx.x * 64 + c0, y = y_first + blockIdx.y * S::rows + ty;
    if (y >= H || x >= W) return;
    float* dst = reinterpret_cast<float*>(reinterpret_cast<char*>(out) + (size_t)y * out_pitch) + x;
    const float p0 = pick(first, count0), p1 = pick(last, count1);
    if (x + 1 < W && (reinterpret_cast<uintptr_t>(dst) & 7u) == 0) {
        *reinterpret_cast<float2*>(dst) = make_float2(p0, p1);
    } else {
        dst[0] = p0;
        if (x + 1 < W) dst[1] = p1;
    }
}

// Radius 0: the value itself where it is valid, else 0.
__global__ void __launch_bounds__(kTileW * kTileH)
median0_kernel(const float* __restrict__ in, size_t in_pitch, float* __restrict__ out, size_t out_pitch, int W,
               int H) {
    const int x = blockIdx.x * kTileW + threadIdx.x, y = blockIdx.y * kTileH + threadIdx.y;
    if (x >= W || y >= H) return;
    const float d = reinterpret_cast<const float*>(reinterpret_cast<const char*>(in) + (size_t)y * in_pitch)[x];
    reinterpret_cast<float*>(reinterpret_cast<char*>(out) + (size_t)y * out_pitch)[x] = d > 0.0f ? d : 0.0f;
}

template <int R>
cudaError_t launch_median(const float* in, size_t in_pitch, float* out, size_t out_pitch, int W, int H,
                          cudaStream_t stream) {
    using S = MedianShape<R>;
    if (S::bytes > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute((const void*)median_kernel<R>,
                                                   cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::bytes);
        if (e != cudaSuccess) return e;
    }
    // A grid has at most 65535 rows of CTAs; images of up to kTileH times that are taken
    // at every radius, those of radii with smaller tiles in two launches.
    constexpr int kBand = 65535 * S::rows;
    if (H > 65535 * kTileH) return cudaErrorInvalidConfiguration;
    for (int y = 0; y < H; y += kBand) {
        const int rows = H - y < kBand ? H - y : kBand;
        const dim3 block(32, S::rows), grid((W + 63) / 64, (rows + S::rows - 1) / S::rows);
        count_launch();
        median_kernel<R><<<grid, block, S::bytes, stream>>>(in, in_pitch, out, out_pitch, W, H, y);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

__global__ void __launch_bounds__(kTileW * kTileH)
bilateral_kernel(const float* __restrict__ in, size_t in_pitch, float* __restrict__ out, size_t out_pitch, int W,
                 int H, int R, float sigma_s, float sigma_d) {
    extern __shared__ float s[];
    const int n = 2 * R + 1, TW = kTileW + 2 * R;
    float* ws = s + (kTileH + 2 * R) * TW;      // spatial weights, n*n
    stage_tile(in, in_pitch, W, H, R, s);
    const float inv_2ss = __fdiv_rn(1.0f, __fmul_rn(__fmul_rn(2.0f, sigma_s), sigma_s));
    const float inv_2sd = __fdiv_rn(1.0f, __fmul_rn(__fmul_rn(2.0f, sigma_d), sigma_d));
    for (int i = threadIdx.y * kTileW + threadIdx.x; i < n * n; i += kTileW * kTileH) {
        const int dy = i / n - R, dx = i % n - R;
        ws[i] = expf(__fmul_rn(-(float)(dx * dx + dy * dy), inv_2ss));
    }
    __syncthreads();
    const int x = blockIdx.x * kTileW + threadIdx.x, y = blockIdx.y * kTileH + threadIdx.y;
    if (x >= W || y >= H) return;
    const float c = s[(threadIdx.y + R) * TW + threadIdx.x + R];
    float res = 0.0f;
    if (!(c <= 0.0f)) {
        float sum = 0.0f, wsum = 0.0f;
        // Raster order (the shader's): rows dy, then columns dx.
        for (int dy = 0; dy < n; ++dy) {
            const float* row = s + (threadIdx.y + dy) * TW + threadIdx.x;
            const float* wrow = ws + dy * n;
            for (int dx = 0; dx < n; ++dx) {
                const float nb = row[dx];
                if (nb <= 0.0f) continue;
                const float diff = __fsub_rn(nb, c);
                const float wd = __expf(__fmul_rn(__fmul_rn(-diff, diff), inv_2sd));
                const float wt = __fmul_rn(wrow[dx], wd);
                sum = __fadd_rn(sum, __fmul_rn(nb, wt));
                wsum = __fadd_rn(wsum, wt);
            }
        }
        res = wsum > 1e-8f ? __fdiv_rn(sum, wsum) : c;
    }
    *reinterpret_cast<float*>(reinterpret_cast<char*>(out) + (size_t)y * out_pitch + (size_t)x * sizeof(float)) =
        res;
}

// Bilateral for a compile-time radius: four neighbouring pixels a thread, so that a
// window row's values are read once for the four (16-byte loads), and per
// neighbour one exponential of the sum of both exponents (base 2, from the
// precomputed spatial exponents), a select for invalid neighbours and two
// accumulations: 8 operations, of which the exponential takes a special-function
// unit 8 cycles a warp and bounds the kernel (1920x1080, r = 3: 22 us of about 30;
// staging the tile is most of the rest). One neighbour at a time with its loads,
// weights and branch it took 31 instructions a neighbour (whole call 100 us; now 45).
constexpr int kBilateralPx = 4;
constexpr int kBilateralW = 32 * kBilateralPx, kBilateralH = 8;
__host__ __device__ constexpr int bilateral_row(int r) { return (kBilateralW + 2 * r + 3) & ~3; }   // 16-byte rows

// Flushes results below 2^-126 to 0. Beside the centre's own weight of 1 they change
// nothing, unless a neighbour is more than 2^100 times the centre (keeping them for such
// tiles took 2 to 3 us of 35 at 1920x1080, r = 3, from all others).
__device__ __forceinline__ float exp2_approx(float x) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

template <int R>
__global__ void __launch_bounds__(256)
bilateral_rows_kernel(const float* __restrict__ in, size_t in_pitch, float* __restrict__ out, size_t out_pitch, int W,
                      int H, float sigma_s, float sigma_d) {
    constexpr int n = 2 * R + 1, TW = bilateral_row(R), TH = kBilateralH + 2 * R;
    constexpr int kRowWeights = (n + 3) & ~3;
    constexpr int kValues = kBilateralPx + 2 * R, kLoads = (kValues + 3) / 4;
    static_assert((32 - 1) * kBilateralPx + 4 * kLoads <= TW, "the last thread's loads stay in the row");
    __shared__ __align__(16) float s[TH * TW];
    __shared__ __align__(16) float ws[n * kRowWeights];     // spatial exponents, base 2
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int x0 = blockIdx.x * kBilateralW - R, y0 = blockIdx.y * kBilateralH - R;
    for (int r = ty; r < TH; r += kBilateralH) {
        const float* row = reinterpret_cast<const float*>(reinterpret_cast<const char*>(in) +
                                                          (size_t)clampi(y0 + r, 0, H - 1) * in_pitch);
        for (int c = tx; c < TW; c += 32) {
            // Invalid values as 0: their weight is 0 below, and 0 times -inf would not be.
            const float v = row[clampi(x0 + c, 0, W - 1)];
            s[r * TW + c] = v <= 0.0f ? 0.0f : v;
        }
    }
    constexpr float kLog2e = 1.4426950408889634f;
    const float inv_2ss = __fdiv_rn(1.0f, __fmul_rn(__fmul_rn(2.0f, sigma_s), sigma_s));
    const float inv_2sd = __fdiv_rn(1.0f, __fmul_rn(__fmul_rn(2.0f, sigma_d), sigma_d));
    for (int i = ty * 32 + tx; i < n * n; i += 256) {
        const int dy = i / n - R, dx = i % n - R;
        ws[(i / n) * kRowWeights + i % n] = -(float)(dx * dx + dy * dy) * inv_2ss * kLog2e;
    }
    __syncthreads();
    const int x = blockIdx.x * kBilateralW + kBilateralPx * tx, y = blockIdx.y * kBilateralH + ty;
    if (x >= W || y >= H) return;
    const float k = -inv_2sd * kLog2e;
    float c[kBilateralPx], sum[kBilateralPx], wsum[kBilateralPx];
#pragma unroll
    for (int i = 0; i < kBilateralPx; ++i) {
        c[i] = s[(ty + R) * TW + kBilateralPx * tx + R + i];
        sum[i] = wsum[i] = 0.0f;
    }
    // Raster order (the shader's): rows dy, then columns dx.
#pragma unroll 1
    for (int dy = 0; dy < n; ++dy) {
        float v[4 * kLoads], w[kRowWeights];
        const float4* row = reinterpret_cast<const float4*>(s + (ty + dy) * TW + kBilateralPx * tx);
#pragma unroll
        for (int q = 0; q < kLoads; ++q) {
            const float4 f = row[q];
            v[4 * q] = f.x, v[4 * q + 1] = f.y, v[4 * q + 2] = f.z, v[4 * q + 3] = f.w;
        }
#pragma unroll
        for (int q = 0; q < kRowWeights / 4; ++q) {
            const float4 f = reinterpret_cast<const float4*>(ws + dy * kRowWeights)[q];
            w[4 * q] = f.x, w[4 * q + 1] = f.y, w[4 * q + 2] = f.z, w[4 * q + 3] = f.w;
        }
#pragma unroll
        for (int dx = 0; dx < n; ++dx)
#pragma unroll
            for (int i = 0; i < kBilateralPx; ++i) {
                const float nb = v[dx + i];
                const float diff = __fsub_rn(nb, c[i]);
                const float e = exp2_approx(__fmaf_rn(__fmul_rn(diff, k), diff, w[dx]));
                const float wt = nb <= 0.0f ? 0.0f : e;          // invalid neighbours weigh nothing
                sum[i] = __fmaf_rn(nb, wt, sum[i]);
                wsum[i] = __fadd_rn(wsum[i], wt);
            }
    }
    float res[kBilateralPx];
#pragma unroll
    for (int i = 0; i < kBilateralPx; ++i)
        res[i] = c[i] <= 0.0f ? 0.0f : wsum[i] > 1e-8f ? __fdiv_rn(sum[i], wsum[i]) : c[i];
    float* dst = reinterpret_cast<float*>(reinterpret_cast<char*>(out) + (size_t)y * out_pitch) + x;
    if (x + kBilateralPx <= W && (reinterpret_cast<uintptr_t>(dst) & 15u) == 0) {
        *reinterpret_cast<float4*>(dst) = make_float4(res[0], res[1], res[2], res[3]);
    } else {
#pragma unroll
        for (int i = 0; i < kBilateralPx; ++i)
            if (x + i < W) dst[i] = res[i];
    }
}

template <int R>
void launch_bilateral_rows(const float* in, size_t in_pitch, float* out, size_t out_pitch, int W, int H, float sigma_s,
                           float sigma_d, cudaStream_t stream) {
    const dim3 block(32, kBilateralH), grid((W + kBilateralW - 1) / kBilateralW, (H + kBilateralH - 1) / kBilateralH);
    bilateral_rows_kernel<R><<<grid, block, 0, stream>>>(in, in_pitch, out, out_pitch, W, H, sigma_s, sigma_d);
}

size_t tile_floats(int r) { return (size_t)(kTileH + 2 * r) * (kTileW + 2 * r); }

}  // namespace

cudaError_t launch_depth_median(const float* in, size_t in_pitch, float* out, size_t out_pitch, int W, int H,
                                int radius, cudaStream_t stream) {
    switch (radius) {
        case 1: return launch_median<1>(in, in_pitch, out, out_pitch, W, H, stream);
        case 2: return launch_median<2>(in, in_pitch, out, out_pitch, W, H, stream);
        case 3: return launch_median<3>(in, in_pitch, out, out_pitch, W, H, stream);
        case 4: return launch_median<4>(in, in_pitch, out, out_pitch, W, H, stream);
        case 5: return launch_median<5>(in, in_pitch, out, out_pitch, W, H, stream);
    }
    count_launch();
    const dim3 block(kTileW, kTileH), grid((W + kTileW - 1) / kTileW, (H + kTileH - 1) / kTileH);
    median0_kernel<<<grid, block, 0, stream>>>(in, in_pitch, out, out_pitch, W, H);
    return cudaGetLastError();
}

// Radii without an instantiation.
static cudaError_t launch_bilateral_any(const float* in, size_t in_pitch, float* out, size_t out_pitch, int W, int H,
                                        int radius, float sigma_s, float sigma_d, cudaStream_t stream) {
    const dim3 block(kTileW, kTileH), grid((W + kTileW - 1) / kTileW, (H + kTileH - 1) / kTileH);
    const size_t smem = (tile_floats(radius) + (size_t)(2 * radius + 1) * (2 * radius + 1)) * sizeof(float);
    bilateral_kernel<<<grid, block, smem, stream>>>(in, in_pitch, out, out_pitch, W, H, radius, sigma_s, sigma_d);
    return cudaGetLastError();
}

cudaError_t launch_depth_bilateral(const float* in, size_t in_pitch, float* out, size_t out_pitch, int W, int H,
                                   int radius, float sigma_s, float sigma_d, cudaStream_t stream) {
    count_launch();
    switch (radius) {
        case 1: launch_bilateral_rows<1>(in, in_pitch, out, out_pitch, W, H, sigma_s, sigma_d, stream); break;
        case 2: launch_bilateral_rows<2>(in, in_pitch, out, out_pitch, W, H, sigma_s, sigma_d, stream); break;
        case 3: launch_bilateral_rows<3>(in, in_pitch, out, out_pitch, W, H, sigma_s, sigma_d, stream); break;
        case 4: launch_bilateral_rows<4>(in, in_pitch, out, out_pitch, W, H, sigma_s, sigma_d, stream); break;
        case 5: launch_bilateral_rows<5>(in, in_pitch, out, out_pitch, W, H, sigma_s, sigma_d, stream); break;
        case 6: launch_bilateral_rows<6>(in, in_pitch, out, out_pitch, W, H, sigma_s, sigma_d, stream); break;
        case 7: launch_bilateral_rows<7>(in, in_pitch, out, out_pitch, W, H, sigma_s, sigma_d, stream); break;
        case 8: launch_bilateral_rows<8>(in, in_pitch, out, out_pitch, W, H, sigma_s, sigma_d, stream); break;
        default: return launch_bilateral_any(in, in_pitch, out, out_pitch, W, H, radius, sigma_s, sigma_d, stream);
    }
    return cudaGetLastError();
}

size_t depth_bilateral_smem_bytes(int radius) {
    return (tile_floats(radius) + (size_t)(2 * radius + 1) * (2 * radius + 1)) * sizeof(float);
}

}  // namespace vxsgm
