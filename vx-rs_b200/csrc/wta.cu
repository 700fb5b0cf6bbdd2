// Winner-take-all, parabola subpixel refinement and left-right check, fused
// with the sum of the per-path slabs. One CTA per (pair, image row).
//
// Semantics (vx-vision/shaders/SGMStereo.metal:179-214):
//   S(d)   = sum over paths of L_r(d), modulo 2^16 (the shader's ushort +=)
//   best_d = first minimum of S over d (strict '<' from 0xFFFF)
//   disp   = best_d + (c0 - c2) / (2 (c0 + c2 - 2 c1)) when 0 < best_d < D-1 and
//            the denominator is non-zero, with c0,c1,c2 = S(best_d-1..best_d+1)
//            (IEEE single precision, correctly rounded division).
// Extension: right-view WTA dR(x') = first minimum over d of S(x'+d, d) with
// x'+d < W; a pixel is invalid when x - dL < 0 or |dL - dR(x - dL)| > tol.
// Optional depth output fx*B/disparity for valid pixels with disparity > 0.
//
// Mapping: lanes span disparities (16 per lane: 16 bytes of a byte-slab vector; 8 or
// 16 per lane of a wide one, wta_form), so one round reads a pixel's whole vector of each path;
// a warp covers 32/seg pixels at once and walks a strip of consecutive ones. The
// loads of all paths of a pixel are issued before any is
// used (the path count is a template parameter). Sums are kept as u16 pairs in
// 32-bit words (wide slabs: added per half, wrapping modulo 2^16; byte slabs: bytes
// widened by byte permutes and summed as whole words, see sum_bytes). An escaped
// byte vector (0xFF in byte 0, held by the pixel's first lane) is taken out of the
// byte sum and its exact u16 values are read from the shadow slab instead. The
// argmin is a min over the key (S << 8 | d), which orders by cost then by d, i.e.
// the first minimum; S(bd-1) and S(bd+1) for the subpixel step come through shared
// memory from the lanes that hold them.
//
// Right view: the keys of (x, d) and (x+1, d+1) belong to the same column x - d,
// and a lane meets both when its next pixel is S <= 16 on, so it carries the minima
// of its columns in registers, S places up a round; the S columns that leave its
// disparities go to the row's minima in shared memory (atomicMin; all 16 of a lane
// from D = 32 down, 8 at D = 64, 2 at D = 256). Wide slabs carry alike, one column a
// pixel leaving each lane where a pixel takes the whole warp (without the carry 1920x1080
// D = 192 took 824 us at 4 paths, now 528, and 1148 at 8, now 1016).
//
// What bounds it: HBM for the slabs where the rows are many (8 pairs of 2048x1536 D =
// 256: 7.6 ms, 6.8 TB/s; 8.0 before), the SMs' unequal rows and the latency of a
// round's loads where they are few (1920x1080 D = 192 609 us, 5.2 TB/s; 743 with 580
// rather than 300 instructions a round: 16 atomics and their padded addresses, idle
// lanes' loads filled with zeros; 640x480 D = 64, 4 paths, 25 us from 34).
#include <cuda_runtime.h>

#include <algorithm>

#include "kernels.cuh"
#include "launch.hpp"

namespace vxsgm {

namespace {

constexpr unsigned kFull = 0xffffffffu;

// Position k of the WTA order whose rows hold this row (wta_row_begin rises with k).
__device__ __forceinline__ int find_wta_position(const PairDev* pairs, int n, int row) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (pairs[mid].wta_row_begin <= row) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// Wide slabs: the sums over the NP paths of the 8 disparities d = 8c..8c+7 of the
// pixel at offset `off` (u16 values, row base included by the caller), as pairs
// acc[k] = S(8c+2k) | S(8c+2k+1) << 16, added per half (modulo 2^16). Lanes past Dp
// (Dv can be Dp + 8) and idle lanes read the row's first values; their sums are not used.
// V vectors a path: of the disparities V * 8c .. V * 8c + 8V-1.
template <int NP, int V>
__device__ __forceinline__ void sum_wide(const uint4 (&v)[NP * V], uint32_t (&acc)[4 * V]) {
#pragma unroll
    for (int k = 0; k < 4 * V; ++k) acc[k] = 0u;
#pragma unroll
    for (int p = 0; p < NP; ++p)
#pragma unroll
        for (int q = 0; q < V; ++q) {
            acc[4 * q] = __vadd2(acc[4 * q], v[V * p + q].x);
            acc[4 * q + 1] = __vadd2(acc[4 * q + 1], v[V * p + q].y);
            acc[4 * q + 2] = __vadd2(acc[4 * q + 2], v[V * p + q].z);
            acc[4 * q + 3] = __vadd2(acc[4 * q + 3], v[V * p + q].w);
        }
}

// A 4-byte word's bytes (0, 1) and (2, 3) widened to u16 pairs.
__device__ __forceinline__ uint32_t widen_lo(uint32_t w) { return __byte_perm(w, 0u, 0x4140); }
__device__ __forceinline__ uint32_t widen_hi(uint32_t w) { return __byte_perm(w, 0u, 0x4342); }

// Byte slabs: the sums S(16c .. 16c+15) of pixel x of the row, as pairs acc[k] =
// S(16c+2k) | S(16c+2k+1) << 16, from one 16-byte load per path (byte offset `off`
// from the row; idle lanes read the row's first bytes, their sums are not used). A
// non-escaped byte is at most 254, so 8 of them sum to less than 2^11: widened
// pairs are added as whole 32-bit words, no carry reaching the next half.
// Any marker among the paths: their bytes 0 gathered four to a word (byte
// permutes); a byte 0xFF is a zero byte of the complement, which the borrow test
// (~g - 0x01..01) & g & 0x80..80 finds exactly. Only the pixel's lane c = 0 holds
// markers; the shadow slot is in its bytes 4..7. Escaped vectors are taken out and
// their shadow values put in with per-half wrapping arithmetic (exact modulo 2^16
// in any order), path by path over the paths that any of the warp's pixels needs;
// the byte vector is read again there, so the loads need not stay live.
template <int NP>
__device__ __forceinline__ void sum_bytes(const PairDev& pr, const uint8_t* row, size_t stride, uint32_t off,
                                          size_t pix, int c, bool act, int lead, const uint4 (&v)[NP],
                                          uint32_t (&acc)[8]) {
#pragma unroll
    for (int k = 0; k < 8; ++k) acc[k] = 0u;
#pragma unroll
    for (int p = 0; p < NP; p += 2) {
        acc[0] += widen_lo(v[p].x) + widen_lo(v[p + 1].x);
        acc[1] += widen_hi(v[p].x) + widen_hi(v[p + 1].x);
        acc[2] += widen_lo(v[p].y) + widen_lo(v[p + 1].y);
        acc[3] += widen_hi(v[p].y) + widen_hi(v[p + 1].y);
        acc[4] += widen_lo(v[p].z) + widen_lo(v[p + 1].z);
        acc[5] += widen_hi(v[p].z) + widen_hi(v[p + 1].z);
        acc[6] += widen_lo(v[p].w) + widen_lo(v[p + 1].w);
        acc[7] += widen_hi(v[p].w) + widen_hi(v[p + 1].w);
    }
    uint32_t ff = 0u;
#pragma unroll
    for (int p = 0; p < NP; p += 4) {
        uint32_t g;
        if (NP == 2) {
            g = __byte_perm(v[p].x, v[p + 1].x, 0x4040);
        } else {
            g = __byte_perm(__byte_perm(v[p].x, v[p + 1].x, 0x0040),
                            __byte_perm(v[p + 2].x, v[p + 3].x, 0x0040), 0x5410);
        }
        ff |= (~g - 0x01010101u) & g & 0x80808080u;
    }
    if (__any_sync(kFull, c == 0 && act && ff != 0u)) {
        unsigned e = 0u;
#pragma unroll
        for (int p = 0; p < NP; ++p) e |= ((v[p].x & 0xFFu) == 0xFFu ? 1u : 0u) << p;
        const unsigned em = __shfl_sync(kFull, act ? e : 0u, lead);
        unsigned todo = __reduce_or_sync(kFull, em);
        while (todo) {
            const int p = __ffs((int)todo) - 1;
            todo &= todo - 1u;
            if (!act || !((em >> p) & 1u)) continue;
            const uint8_t* vec = row + stride * p + off;
            const uint4 b = __ldg(reinterpret_cast<const uint4*>(vec));
            acc[0] = __vsub2(acc[0], widen_lo(b.x));
            acc[1] = __vsub2(acc[1], widen_hi(b.x));
            acc[2] = __vsub2(acc[2], widen_lo(b.y));
            acc[3] = __vsub2(acc[3], widen_hi(b.y));
            acc[4] = __vsub2(acc[4], widen_lo(b.z));
            acc[5] = __vsub2(acc[5], widen_hi(b.z));
            acc[6] = __vsub2(acc[6], widen_lo(b.w));
            acc[7] = __vsub2(acc[7], widen_hi(b.w));
            const uint16_t* src = pr.shadow + pr.shadow_stride * p + pix * pr.nd_pad;
            if (pr.shadow_cap != 0) {               // pooled shadow: slots beyond it were never written
                const uint32_t slot = *reinterpret_cast<const uint32_t*>(vec - 16 * c + 4);
                if (slot >= pr.shadow_cap) continue;
                src = pr.shadow + (size_t)slot * pr.nd_pad;
            }
            // Lanes past Dp read no shadow (Dv can be Dp + 8).
            uint4 lo = make_uint4(0u, 0u, 0u, 0u), hi = lo;
            if (16 * c < pr.nd_pad) lo = __ldcs(reinterpret_cast<const uint4*>(src + 16 * c));
            if (16 * c + 8 < pr.nd_pad) hi = __ldcs(reinterpret_cast<const uint4*>(src + 16 * c + 8));
            acc[0] = __vadd2(acc[0], lo.x);
            acc[1] = __vadd2(acc[1], lo.y);
            acc[2] = __vadd2(acc[2], lo.z);
            acc[3] = __vadd2(acc[3], lo.w);
            acc[4] = __vadd2(acc[4], hi.x);
            acc[5] = __vadd2(acc[5], hi.y);
            acc[6] = __vadd2(acc[6], hi.z);
            acc[7] = __vadd2(acc[7], hi.w);
        }
    }
}

// A u16 sum (half HI of w) above byte B of j: key = S << 8 | d. Byte 3 repeats the
// sum's sign bit (a permute's fourth source would be a zero), which keeps the order.
template <int HI, int B>
__device__ __forceinline__ uint32_t make_key(uint32_t w, uint32_t j) {
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(w), "r"(j), "n"((4 + B) | (HI ? 0xB320 : 0x9100)));
    return r;
}

// The disparity loop of one image row: every pixel's first-minimum key, its
// neighbours' sums and (LR) the row's right-view keys into shared memory. The path
// count, the slab form and the carry S (min(K, pixels a warp covers); K: none) are
// template parameters, so each variant is its own straight-line loop.
template <int NP, int FORM, int S>
__device__ __forceinline__ void wta_row(const PairDev& pr, int y, uint32_t* right_key, uint32_t* best_key,
                                        uint32_t* nbr, uint16_t* sums) {
    constexpr int K = wta_disparities_per_lane(FORM);   // disparities a lane sums
    constexpr bool kWide = FORM != kFormBytes;
    constexpr int V = FORM == kFormWide16 ? 2 : 1;  // vectors a path
    constexpr bool kAhead = NP <= 4;                // the next round's vectors are loaded during this one
    const int W = pr.width, D = pr.nd;
    const bool lr = pr.lr_check != 0;
    const int seg = S < K ? 32 / S : wta_lanes_per_pixel(pr.nd_vec, FORM);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int sub = lane / seg, c = lane % seg;
    const int ppw = 32 / seg, warps = blockDim.x >> 5;
    const int rounds = (W + warps * ppw - 1) / (warps * ppw);   // of a warp's strip of the row
    const int d0 = K * c;                           // this lane's first disparity
    const size_t row_pix = (size_t)y * W;
    const size_t stride = kWide ? pr.shadow_stride : pr.slab_stride;
    const uint8_t* const row8 = pr.slabs + row_pix * pr.nd_vec;
    const uint16_t* const row16 = pr.shadow + row_pix * pr.nd_pad;
    const int vec = kWide ? pr.nd_pad : pr.nd_vec;
    uint32_t dj[K / 4];                             // bytes d0 .. d0 + K-1
#pragma unroll
    for (int i = 0; i < K / 4; ++i) dj[i] = 0x03020100u + 0x01010101u * (uint32_t)(d0 + 4 * i);

    // This warp's sums of the current pixels, a chunk a lane (S(d) of a pixel at d),
    // read back for S(bd-1) and S(bd+1).
    uint16_t* const srow = sums + warp * kWtaSumsPerWarp + K * lane;
    uint32_t rk[K];                                 // right-view minima of columns x - d0 - j
#pragma unroll
    for (int j = 0; j < K; ++j) rk[j] = 0xFFFFFFFFu;
    int x = warp * rounds * ppw + sub;
    uint4 v[NP * V];                                // the paths' vectors
    const auto fetch = [&](int xf) {
#pragma unroll
        for (int q = 0; q < V; ++q) {
            const uint32_t off = xf < W && d0 + 8 * q < vec ? (uint32_t)(xf * vec + d0 + 8 * q) : 0u;
#pragma unroll
            for (int p = 0; p < NP; ++p)
                v[V * p + q] = kWide ? __ldcs(reinterpret_cast<const uint4*>(row16 + stride * p + off))
                                     : __ldg(reinterpret_cast<const uint4*>(row8 + stride * p + off));
        }
    };
    if (kAhead) fetch(x);
    for (int i = 0; i < rounds; ++i, x += ppw) {
        const bool act = x < W && d0 < vec;
        if (!kAhead) fetch(x);
        uint32_t acc[K / 2];                        // acc[k] = S(d0 + 2k) | S(d0 + 2k+1) << 16
        if constexpr (kWide) sum_wide<NP, V>(v, acc);
        else sum_bytes<NP>(pr, row8, stride, act ? (uint32_t)(x * vec + d0) : 0u, row_pix + x, c, act, sub * seg, v, acc);
        if (kAhead && i + 1 < rounds) fetch(x + ppw);
#pragma unroll
        for (int q = 0; q < K / 8; ++q)
            *reinterpret_cast<uint4*>(srow + 8 * q) =
                make_uint4(acc[4 * q], acc[4 * q + 1], acc[4 * q + 2], acc[4 * q + 3]);
        uint32_t key[K];
#pragma unroll
        for (int i4 = 0; i4 < K / 4; ++i4) {
            key[4 * i4] = make_key<0, 0>(acc[2 * i4], dj[i4]);
            key[4 * i4 + 1] = make_key<1, 1>(acc[2 * i4], dj[i4]);
            key[4 * i4 + 2] = make_key<0, 2>(acc[2 * i4 + 1], dj[i4]);
            key[4 * i4 + 3] = make_key<1, 3>(acc[2 * i4 + 1], dj[i4]);
        }
        const int nb = act ? D - d0 : 0;            // this lane's keys j < nb take part
        if (nb < K) {
#pragma unroll
            for (int j = 0; j < K; ++j)
                if (j >= nb) key[j] = 0xFFFFFFFFu;
        }
        uint32_t best = key[0];
#pragma unroll
        for (int j = 1; j + 1 < K; j += 2) best = __vimin3_u32(best, key[j], key[j + 1]);
        best = min(best, key[K - 1]);
        if (lr) {
#pragma unroll
            for (int j = K - 1; j >= 0; --j) rk[j] = j >= S ? min(rk[j >= S ? j - S : 0], key[j]) : key[j];
            // The columns that the pixel S on has no key of.
            const int xr = x - d0;
            if (xr >= K - 1 && x < W) {
#pragma unroll
                for (int j = K - S; j < K; ++j) atomicMin(&right_key[xr - j], rk[j]);
            } else {
#pragma unroll
                for (int j = K - S; j < K; ++j)
                    if ((unsigned)(xr - j) < (unsigned)W) atomicMin(&right_key[xr - j], rk[j]);
            }
        }
        for (int o = seg >> 1; o > 0; o >>= 1) best = min(best, __shfl_xor_sync(kFull, best, o));
        __syncwarp();                               // the pixel's sums are in shared memory
        if (c == 0 && x < W) {
            // S(bd-1) and S(bd+1) (only used when 0 < bd < D-1, so both exist).
            const int bd = (int)(best & 0xFFu);
            const uint32_t c0 = srow[max(bd - 1, 0)], c2 = srow[min(bd + 1, D - 1)];
            best_key[x] = best;
            nbr[x] = c0 | (c2 << 16);
        }
        __syncwarp();                               // before the next pixels' sums
    }
    if (lr && S < K) {                              // the columns still carried
        const int xr = x - S - d0;
#pragma unroll
        for (int j = 0; j < K - S; ++j)
            if ((unsigned)(xr - j) < (unsigned)W) atomicMin(&right_key[xr - j], rk[j]);
    }
}

template <int NP>
__device__ __forceinline__ void wta_row_bytes(const PairDev& pr, int y, uint32_t* right_key, uint32_t* best_key,
                                              uint32_t* nbr, uint16_t* sums) {
    switch (wta_lanes_per_pixel(pr.nd_vec, kFormBytes)) {
        case 16: wta_row<NP, kFormBytes, 2>(pr, y, right_key, best_key, nbr, sums); break;
        case 8: wta_row<NP, kFormBytes, 4>(pr, y, right_key, best_key, nbr, sums); break;
        case 4: wta_row<NP, kFormBytes, 8>(pr, y, right_key, best_key, nbr, sums); break;
        default: wta_row<NP, kFormBytes, 16>(pr, y, right_key, best_key, nbr, sums); break;
    }
}

template <int NP>
__device__ __forceinline__ void wta_row_wide(const PairDev& pr, int y, uint32_t* right_key, uint32_t* best_key,
                                             uint32_t* nbr, uint16_t* sums) {
    switch (wta_lanes_per_pixel(pr.nd_vec, kFormWide)) {
        case 32:
            if constexpr (NP == 2) wta_row<2, kFormWide16, 2>(pr, y, right_key, best_key, nbr, sums);   // wta_form's rule
            else wta_row<NP, kFormWide, 1>(pr, y, right_key, best_key, nbr, sums);
            break;
        case 16: wta_row<NP, kFormWide, 2>(pr, y, right_key, best_key, nbr, sums); break;
        case 8: wta_row<NP, kFormWide, 4>(pr, y, right_key, best_key, nbr, sums); break;
        default: wta_row<NP, kFormWide, 8>(pr, y, right_key, best_key, nbr, sums); break;
    }
}

// Pairs of at most MAXP paths. With 8 a thread takes 80 registers (eight 16-byte
// loads, 16 carried minima, 8 words of sums), 24 warps an SM; with at most 4, 64
// registers and 32 warps.
template <int MAXP>
__global__ void __launch_bounds__(wta_max_threads(MAXP), 2)
wta_kernel(const PairDev* __restrict__ pairs, int num_pairs) {
    extern __shared__ __align__(16) uint32_t smem[];
    const int k = find_wta_position(pairs, num_pairs, blockIdx.x);
    const int y = blockIdx.x - pairs[k].wta_row_begin;
    const PairDev pr = pairs[pairs[k].wta_pair];   // fields live in registers
    const int W = pr.width, D = pr.nd, P = pr.num_paths;
    const bool lr = pr.lr_check != 0;

    uint32_t* right_key = smem;                               // W: right-view keys (LR only)
    uint32_t* best_key = smem + W;                            // W: S(bd) << 8 | bd
    uint32_t* nbr = best_key + W;                             // W: S(bd-1) | S(bd+1) << 16
    // then the warps' sums (16-byte aligned)
    uint16_t* sums = reinterpret_cast<uint16_t*>(smem + ((3 * W + 3) & ~3));

    if (lr)
        for (int i = threadIdx.x; i < W; i += blockDim.x) right_key[i] = 0xFFFFFFFFu;
    __syncthreads();

    const bool subpixel = pr.subpixel != 0;
    const bool wide = pr.wide_slabs != 0;           // uniform over the CTA
    if (P == 2) {
        if (wide) wta_row_wide<2>(pr, y, right_key, best_key, nbr, sums);
        else wta_row_bytes<2>(pr, y, right_key, best_key, nbr, sums);
    } else if (MAXP == 4 || P == 4) {
        if (wide) wta_row_wide<4>(pr, y, right_key, best_key, nbr, sums);
        else wta_row_bytes<4>(pr, y, right_key, best_key, nbr, sums);
    } else if constexpr (MAXP == 8) {
        if (wide) wta_row_wide<8>(pr, y, right_key, best_key, nbr, sums);
        else wta_row_bytes<8>(pr, y, right_key, best_key, nbr, sums);
    }
    __syncthreads();

    float* out = reinterpret_cast<float*>(reinterpret_cast<char*>(pr.out_f32) + (size_t)y * pr.out_f32_pitch);
    int16_t* out_i = pr.out_i16
        ? reinterpret_cast<int16_t*>(reinterpret_cast<char*>(pr.out_i16) + (size_t)y * pr.out_i16_pitch)
        : nullptr;
    float* out_z = pr.out_depth
        ? reinterpret_cast<float*>(reinterpret_cast<char*>(pr.out_depth) + (size_t)y * pr.out_depth_pitch)
        : nullptr;
    for (int x = threadIdx.x; x < W; x += blockDim.x) {
        // The parabola step here, one pixel a thread, rather than in the lanes
        // c = 0 of the disparity loop.
        const uint32_t best = best_key[x];
        const int dl = (int)(best & 0xFFu);
        float v = (float)dl;
        if (subpixel && dl > 0 && dl < D - 1) {
            const uint32_t n = nbr[x];
            const float f0 = (float)(n & 0xFFFFu), f1 = (float)((best >> 8) & 0xFFFFu), f2 = (float)(n >> 16);
            const float denom = 2.0f * (f0 + f2 - 2.0f * f1);
            if (fabsf(denom) > 1e-6f) v = __fadd_rn(v, __fdiv_rn(f0 - f2, denom));
        }
        bool valid = true;
        if (lr) {
            const int xr = x - dl;
            valid = xr >= 0 && abs(dl - (int)(right_key[xr] & 0xFFu)) <= pr.lr_tolerance;
        }
        out[x] = valid ? v : pr.invalid_value;
        if (out_i) out_i[x] = (int16_t)(valid ? dl : -1);
        // Depth epilogue: depth = fx * baseline / disparity (the conversion the
        // reference leaves to its caller, kernels/sgm.rs:284-286).
        if (out_z)
            out_z[x] = (valid && v > 0.0f) ? __fdiv_rn(pr.depth_scale, v) : pr.depth_invalid;
    }
}

}  // namespace

namespace {

size_t wta_smem_bytes(int max_width, int threads) {
    return (3 * (size_t)max_width + 3) / 4 * 4 * sizeof(uint32_t) +
           (size_t)(threads / 32) * kWtaSumsPerWarp * sizeof(uint16_t);
}

// CTAs an SM of `warps` warps each.
int wta_ctas(int warps, int max_width, int max_paths) {
    const int by_smem = (int)(227 * 1024 / (wta_smem_bytes(max_width, 32 * warps) + 1024));
    return std::max(1, std::min({2 * wta_max_threads(max_paths) / 32 / warps, 32, by_smem}));
}

// Threads of a CTA. An SM's warps make 2, 3 or 4 CTAs; a launch of few rows takes
// the number whose rounds of CTAs, each as long as its rows are short of warps, end
// first. 1280x720 D = 64, 8 paths: 4 CTAs an SM 125 us, 3: 107, 2: 111; 1242x375 D =
// 128: 110, 105, 124; 640x480 D = 64, 4 paths: 28, 32, 30; many wide rows do not care
// (2048x1536 D = 256: 1012, 1035, 1018).
//
// Many narrow rows take fewer warps each: a warp's steps along the row (row_lanes lanes
// in all) must make up for what a CTA costs, about two steps. 1000 pairs of 32x32 D = 32,
// 16 warps a row 567 us, 4 143, 1 62; 600 of 100x100 D = 128 1287, 639, 521; 30 of
// 640x480 D = 64 500, 406, 490; 20 of 160x120 D = 16 39 with 16, 14 with 1. (Fewer rows
// than 8 an SM are lone pairs, where the rounds decide.)
int wta_threads(int rows, int max_width, int max_paths, int row_lanes, int sms) {
    const int warps = 2 * wta_max_threads(max_paths) / 32;
    int best = 0, best_rounds = 0;
    for (int n = 4; n >= 2; --n) {
        const int w = warps / n, rounds = (rows + sms * n - 1) / (sms * n);
        if (n > 2 && n * (wta_smem_bytes(max_width, 32 * w) + 1024) > 227 * 1024) continue;
        if (best == 0 || rounds * best < best_rounds * w) { best = w; best_rounds = rounds; }
    }
    if (rows < 8 * sms) return 32 * best;
    const auto time = [&](int w) {
        const int at_once = sms * wta_ctas(w, max_width, max_paths);
        return (double)((rows + at_once - 1) / at_once) * (2 + (row_lanes + 32 * w - 1) / (32 * w));
    };
    double limit = 0.95 * time(best);       // many wide rows stay as they are
    for (int w : {4, 3, 2, 1})
        if (w < best && time(w) < limit) { best = w; limit = time(w); }
    return 32 * best;
}

}  // namespace

cudaError_t prepare_wta_kernel() {
    cudaError_t e = cudaFuncSetAttribute(wta_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)wta_smem_bytes(kMaxWidth, wta_max_threads(4)));
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(wta_kernel<8>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)wta_smem_bytes(kMaxWidth, wta_max_threads(8)));
}

cudaError_t launch_wta(const PairDev* d_pairs, int num_pairs, int total_rows, int max_width, int max_paths, int row_lanes,
                       cudaStream_t stream) {
    if (total_rows == 0) return cudaSuccess;
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) (void)cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int threads = wta_threads(total_rows, max_width, max_paths, row_lanes, sms);
    const size_t smem = wta_smem_bytes(max_width, threads);
    count_launch();
    if (max_paths <= 4) wta_kernel<4><<<total_rows, threads, smem, stream>>>(d_pairs, num_pairs);
    else wta_kernel<8><<<total_rows, threads, smem, stream>>>(d_pairs, num_pairs);
    return cudaGetLastError();
}

}  // namespace vxsgm
