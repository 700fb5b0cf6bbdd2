// Census transform for a batch of stereo pairs (both views in one launch).
//
// Semantics: vx-vision/shaders/SGMStereo.metal:25-66 - bit b of the descriptor
// is set iff neighbour < centre (strict), neighbours in raster order with the
// centre skipped, coordinates clamped to the image. The shader reads R8Unorm
// texels as value/255 floats; comparing those is the same as comparing the
// u8 values, which is what this kernel does.
//
// Layout: each 32x32 tile of one view is staged once in shared memory with its
// (rx, ry) apron, then every thread builds the descriptors of four pixels side by
// side, a neighbour of all four a 4-byte word: large tiles, so that the
// per-CTA costs (finding the pair, staging latency) are paid per 1024 pixels. Descriptors are written row-major (read by
// the cost-volume kernel and by the vertical and diagonal paths of the
// single-scanline aggregation) and, for batches run by the single-scanline
// aggregation only, a second time in 32-row bands, x-major inside a band, word
// (x, y) at ((y/32)*W + x)*32 + y%32 (read by its horizontal paths: the 32
// scanlines of a warp are the 32 rows of a band, so each column is 128
// contiguous bytes). Output word: u32 when the window has <= 32 bits, else u64.
//
// What bounds it: the comparisons' integer instructions and a tile's staging latency.
// One comparison an instruction triple for a byte took 32 us for 1920x1080 with a 5x5
// window, 55 with 9x7 and 90 with 7x5 (radii at run time); four a word 24, 38 and 50
// (64 mixed pairs 380 -> 271 us).
//
// Staging. A tile whose apron lies inside the image, of a view whose base and
// pitch are 16-byte aligned, is copied with asynchronous 16-byte copies
// (cp.async, global -> shared without registers): each staged row is the
// 16-byte aligned segment [bx - rx - lead, +rw) with lead = (-rx) mod 16 (bx is
// a multiple of 32), rw = lead + 32 + 2 rx rounded up to 16, read only inside
// the row. Border tiles (and unaligned views) stage byte by byte with clamped
// coordinates, which reproduces the shader's clamp.
#include <cuda_runtime.h>

#include "kernels.cuh"
#include "launch.hpp"

namespace vxsgm {

namespace {

__device__ __forceinline__ int find_pair_by_tile(const PairDev* pairs, int n, int tile) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (pairs[mid].census_tile_begin <= tile) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// The descriptors of four pixels side by side: the tile's word at `at` (4-byte
// aligned, row stride `stride` a multiple of 4) holds their centres. A neighbour of
// all four is a 4-byte word put together from two aligned ones, compared a byte at a
// time: with the top bits set in the neighbours and cleared in the centres their
// difference borrows in no byte, and its top bits with the two words' give n < c.
// The result bits (bit 7 of each byte) collect in a word, eight neighbours a time,
// whose bytes are then the pixels' next eight descriptor bits. RX, RY < 0: the radii
// at run time.
template <int RX, int RY>
__device__ __forceinline__ void window_bits4(const uint8_t* __restrict__ at, int stride, int rx, int ry,
                                             uint64_t (&bits)[4]) {
    if (RX >= 0) {
        rx = RX;
        ry = RY;
    }
    const uint32_t c = *reinterpret_cast<const uint32_t*>(at), c7 = c & 0x7F7F7F7Fu;
    uint32_t acc = 0u;
    int b = 0;
    bits[0] = bits[1] = bits[2] = bits[3] = 0u;
    auto take = [&](uint32_t n) {
        const uint32_t d = (n | 0x80808080u) - c7;        // bit 7: the low seven bits of n reach c's
        const uint32_t lt = (~n & c) | (~(n ^ c) & ~d);
        acc = (acc >> 1) | (lt & 0x80808080u);
        ++b;
        if ((b & 7) == 0) {
#pragma unroll
            for (int j = 0; j < 4; ++j) bits[j] |= (uint64_t)((acc >> (8 * j)) & 0xFFu) << (b - 8);
            acc = 0u;
        }
    };
#pragma unroll
    for (int dy = -ry; dy <= ry; ++dy) {
        const uint32_t* row = reinterpret_cast<const uint32_t*>(at + dy * stride);
#pragma unroll
        for (int dx = -rx; dx <= rx; ++dx) {
            if (dx == 0 && dy == 0) continue;
            // dx >> 2 rounds down: the word that holds byte dx.
            take((dx & 3) == 0 ? row[dx >> 2] : __funnelshift_r(row[dx >> 2], row[(dx >> 2) + 1], 8 * (dx & 3)));
        }
    }
    if (b & 7) {
        acc >>= 8 - (b & 7);
#pragma unroll
        for (int j = 0; j < 4; ++j) bits[j] |= (uint64_t)((acc >> (8 * j)) & 0xFFu) << (b & ~7);
    }
}

// The words of four pixels at p, those below n: vector stores where p is aligned for them.
__device__ __forceinline__ void store4(uint32_t* p, const uint64_t (&v)[4], int n) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(p);
    if (n >= 4 && (a & 15) == 0) {
        *reinterpret_cast<uint4*>(p) = make_uint4((uint32_t)v[0], (uint32_t)v[1], (uint32_t)v[2], (uint32_t)v[3]);
    } else if (n >= 4 && (a & 7) == 0) {
        reinterpret_cast<uint2*>(p)[0] = make_uint2((uint32_t)v[0], (uint32_t)v[1]);
        reinterpret_cast<uint2*>(p)[1] = make_uint2((uint32_t)v[2], (uint32_t)v[3]);
    } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (j < n) p[j] = (uint32_t)v[j];
    }
}
__device__ __forceinline__ void store4(uint64_t* p, const uint64_t (&v)[4], int n) {
    if (n >= 4 && (reinterpret_cast<uintptr_t>(p) & 15) == 0) {
        reinterpret_cast<ulonglong2*>(p)[0] = make_ulonglong2(v[0], v[1]);
        reinterpret_cast<ulonglong2*>(p)[1] = make_ulonglong2(v[2], v[3]);
    } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (j < n) p[j] = v[j];
    }
}

template <typename CT, bool BANDED>
__global__ void __launch_bounds__(kCensusTileW * kCensusThreadsY)
census_kernel(const PairDev* __restrict__ pairs, int num_pairs) {
    extern __shared__ __align__(16) uint8_t tile_px[];
    __shared__ CT tile_bits[kCensusTileH][kCensusTileW + 1];
    static_assert(kCensusTileW * kCensusThreadsY * 4 == kCensusTileW * kCensusTileH, "four pixels a thread");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");   // the cost kernel waits for this one's end
    const int pi = find_pair_by_tile(pairs, num_pairs, blockIdx.x);
    const PairDev& pr = pairs[pi];
    const int W = pr.width, H = pr.height, rx = pr.rx, ry = pr.ry;
    const int tiles_x = (W + kCensusTileW - 1) / kCensusTileW;
    const int tiles_y = (H + kCensusTileH - 1) / kCensusTileH;
    int t = blockIdx.x - pr.census_tile_begin;
    const int view = t / (tiles_x * tiles_y);  // 0 = left, 1 = right
    t -= view * tiles_x * tiles_y;
    const int bx = (t % tiles_x) * kCensusTileW;
    const int by = (t / tiles_x) * kCensusTileH;
    const uint8_t* img = view ? pr.right : pr.left;
    const size_t pitch = view ? pr.right_pitch : pr.left_pitch;

    const int sw = kCensusTileW + 2 * rx, sh = kCensusTileH + 2 * ry;
    const int tid = threadIdx.y * kCensusTileW + threadIdx.x;
    constexpr int kThreads = kCensusTileW * kCensusThreadsY;
    const int lead = census_stage_lead(rx), rw = census_stage_row_bytes(rx);
    const int x0 = bx - rx - lead;
    const bool async_stage = ((reinterpret_cast<uintptr_t>(img) | (uintptr_t)pitch) & 15) == 0 && x0 >= 0 &&
                             x0 + rw <= W && by - ry >= 0 && by + kCensusTileH + ry <= H;
    // The staged rows are rw bytes apart, column x = bx - rx at byte `lead`, so that the
    // centres of four pixels (x a multiple of 4) are an aligned word.
    if (async_stage) {
        const uint8_t* src = img + (size_t)(by - ry) * pitch + x0;
        const int cpr = rw >> 4;         // 16-byte copies a row
        const uint32_t dst0 = (uint32_t)__cvta_generic_to_shared(tile_px);
        for (int i = tid; i < sh * cpr; i += kThreads) {
            const int r = i / cpr, c = i - r * cpr;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst0 + (uint32_t)(r * rw + 16 * c)),
                         "l"(src + (size_t)r * pitch + 16 * c)
                         : "memory");
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else {
        for (int i = tid; i < sw * sh; i += kThreads) {
            const int r = i / sw, c = i - r * sw;
            const int sx = min(max(bx - rx + c, 0), W - 1);
            const int sy = min(max(by - ry + r, 0), H - 1);
            tile_px[r * rw + lead + c] = img[(size_t)sy * pitch + sx];
        }
    }
    __syncthreads();

    // Clamped reads at the image border equal reads of the staged apron, which
    // was filled with clamped coordinates; interior threads read their window.
    // The common windows (5x5, 9x7) are unrolled; the radii are uniform per CTA.
    CT* rm = static_cast<CT*>(view ? pr.census_r : pr.census_l);
    const int ty = tid / (kCensusTileW / 4), tx = tid % (kCensusTileW / 4) * 4;
    const int x = bx + tx, y = by + ty;
    const uint8_t* at = tile_px + (ty + ry) * rw + lead + rx + tx;
    uint64_t bits[4];
    if (rx == 2 && ry == 2) window_bits4<2, 2>(at, rw, rx, ry, bits);
    else if (rx == 4 && ry == 3) window_bits4<4, 3>(at, rw, rx, ry, bits);
    else window_bits4<-1, -1>(at, rw, rx, ry, bits);
    if (x < W && y < H) store4(rm + (size_t)y * W + x, bits, W - x);
    if constexpr (BANDED) {
#pragma unroll
        for (int j = 0; j < 4; ++j) tile_bits[ty][tx + j] = (CT)bits[j];
    }
    if constexpr (!BANDED) return;   // the scanline-pair and scan aggregations read the cost volume instead
    // Banded copy: the tile is one 32-row band (by is a multiple of 32), so a
    // tile column is 32 consecutive words there; the descriptors go through
    // shared memory and consecutive threads write consecutive words.
    CT* cm = static_cast<CT*>(view ? pr.census_rt : pr.census_lt);
    __syncthreads();
    for (int w = tid; w < kCensusTileW * kCensusTileH; w += kThreads) {
        const int col = w / kCensusTileH, row = w % kCensusTileH;
        const int ox = bx + col, oy = by + row;
        if (ox < W && oy < H) cm[((size_t)(oy >> 5) * W + ox) * 32 + (oy & 31)] = tile_bits[row][col];
    }
}

}  // namespace

cudaError_t launch_census(const PairDev* d_pairs, int num_pairs, int total_tiles, int max_rx,
                          int max_ry, bool census64, bool banded, cudaStream_t stream) {
    if (total_tiles == 0) return cudaSuccess;
    const dim3 block(kCensusTileW, kCensusThreadsY);
    const size_t smem = census_smem_bytes(max_rx, max_ry);
    count_launch();
    if (census64) {
        if (banded) census_kernel<uint64_t, true><<<total_tiles, block, smem, stream>>>(d_pairs, num_pairs);
        else census_kernel<uint64_t, false><<<total_tiles, block, smem, stream>>>(d_pairs, num_pairs);
    } else {
        if (banded) census_kernel<uint32_t, true><<<total_tiles, block, smem, stream>>>(d_pairs, num_pairs);
        else census_kernel<uint32_t, false><<<total_tiles, block, smem, stream>>>(d_pairs, num_pairs);
    }
    return cudaGetLastError();
}

}  // namespace vxsgm
