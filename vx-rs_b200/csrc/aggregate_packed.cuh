// Path aggregation of semi-global matching, packed across-lanes scan form: as
// aggregate_scan.cu, one segment of lanes per scanline and the recurrence over d
// as a prefix scan with warp shuffles, but on two 16-bit disparities a word and
// with a scan of plain minima. Plans whose penalties keep every intermediate in
// 16 bits (packed_scan_ok) run it instead of the 32-bit scan form.
//
// Semantics (vx-vision/shaders/SGMStereo.metal:120-172), per scanline, per
// pixel, for d = 0..D-1 with ONE array L[] updated in place, all values ushort:
//     o0 = L[d], o1 = u16(Lnew[d-1] + P1) (0xFFFF at d = 0),
//     o2 = u16(L[d+1] + P1) (0xFFFF at d = D-1), o3 = u16(m + P2),
//     Lnew[d] = u16(C + min(o0, o1, o2, o3) - m),   m = min of the previous pixel.
//
// The scan. A_d = min(o0, o2, o3) is formed by per-half 16-bit operations, so
// it is the shader's value whatever wraps. With v_d = sum_{k<=d} (C_k + P1 - m)
// the pixel's recurrence y_d = C_d - m + min(A_d, y_{d-1} + P1) becomes
//     y_d = v_d + min_{k<=d} u_k,      u_k = A_k - P1 - v_{k-1},
// a prefix MINIMUM (one shuffle and one min a round, no second operand), and the
// costs' part of v is a prefix sum that does not depend on the previous pixel,
// so it is formed one step ahead, off the chain. A lane holds K consecutive
// disparities as K/2 words, word j = (d0 + j, d0 + j + K/2): both halves run the
// lane's serial chains at once. V = v + BV and U = u + BU, BU = 65536 - BV,
// BV = 64 Dv + P2 + 65, are unsigned halves that neither carry nor borrow while
// m <= 64 (so plain 32-bit adds serve), and y = V + z per half modulo 2^16.
//
// Exactness. The integers equal the shader's ushort values modulo 2^16 as long
// as m <= 64 and every y_d >= -P1 (then u16(u16(y_d) + P1) = y_d + P1, the
// integer the recurrence needs). A vector without a wrapped value has m <= 64:
// at the previous minimum's disparity y <= C <= 64. A y_d < -P1 is seen by bit 15
// of u16(y_d + P1). Both are tested only where the vector's signed minimum is
// negative (a value wrapped) or the last vector left m > 64; such a pixel is
// recomputed in the shader's own order, lane by lane.
//
// Rest state. Before a scanline's first pixel its costs read as 0, which keeps
// L = 0 and m = 0, and a first pixel with L = 0 and m = 0 gives L = C, the
// shader's step 0: no start test. Pads (d >= D, PADS variants) are set to
// 0xFFFF - P1 after each pixel: o2 of d = D-1 is then 0xFFFF.
//
// Bound and shape. A lone pair is bound by the chain of one pixel step (shuffle
// rounds and dependent 16-bit operations), batches by instructions. Kind
// kPackedLatency takes few disparities a lane (8; 12 where that makes the lanes a
// power of two), which shortens the chain and spreads a pair over more warps;
// kind kPackedThroughput takes many (16, 24, 32), which shares the per-step
// instructions (loads, shuffles, reductions) among more disparities. A 640x480
// D = 64 4-path pair takes 122 us of aggregation (the 32-bit scan form: 405), a
// 1242x375 D = 128 8-path one 327 us (1214; 405 with 8-warp CTAs, whose first warps,
// the longest units, met on one scheduler), a 1920x1080 D = 192 one 1266 us (5096); a
// pixel step of 64 disparities in 8 lanes takes about 120 instructions and 350 cycles
// alone on its scheduler (560 and 1240). A batch of 64 mixed pairs (3.25 G
// pixel-disparities) takes 9.4 ms (scanline pairs: 12.0), 8 pairs of 2048x1536 D = 256
// 18.2 ms (26.1). D = 64 as 32 disparities in two lanes takes 2.74 ms on 16 pairs of
// 1280x720, as 16 in four 3.02. Wide slabs take about twice that (their vectors all go
// through the branch for wrapped and escaped ones), and D whose lanes are far from a power
// of two pay for the idle ones: the planner's pairs_faster.
//
// Minima, maxima, byte permutes and logic run on one 16-lane pipe of a scheduler,
// 16-bit adds (vadd2) and multiply-adds on the other, plain adds on either: an
// operation every 2 cycles on each (measured), so work that can be is put on the
// second (pack_bytes).
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstdio>
#include <cstdlib>

#include "kernels.cuh"
#include "launch.hpp"

namespace vxsgm {
namespace packed {

namespace {

constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ uint32_t vmin2(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("min.u16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ uint32_t smin2(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("min.s16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ uint32_t vmax2(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("max.u16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
// A byte permute with constant selector; selector nibbles with the top bit
// replicate the byte's sign.
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
    return r;
}
// v of the lane `delta` below in the segment (width as a shuffle clamp mask), or
// `own` for lanes without one.
__device__ __forceinline__ uint32_t shfl_up_or(uint32_t v, int delta, uint32_t clamp, uint32_t own) {
    uint32_t r;
    asm volatile(
        "{\n .reg .pred p;\n .reg .b32 t;\n shfl.sync.up.b32 t|p, %1, %2, %3, 0xffffffff;\n"
        " selp.b32 %0, t, %4, p;\n}"
        : "=r"(r)
        : "r"(v), "r"(delta), "r"(clamp), "r"(own));
    return r;
}

// The lane's K cost bytes.
template <int K>
struct Bytes {
    uint32_t w[K / 4];
};
template <int K>
__device__ __forceinline__ void copy_bytes_async(uint32_t dst, const uint8_t* src) {
    if constexpr (K % 16 == 0) {
#pragma unroll
        for (int i = 0; i < K / 16; ++i)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16 * i), "l"(src + 16 * i) : "memory");
    } else if constexpr (K % 8 == 0) {
#pragma unroll
        for (int i = 0; i < K / 8; ++i)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst + 8 * i), "l"(src + 8 * i) : "memory");
    } else {
#pragma unroll
        for (int i = 0; i < K / 4; ++i)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst + 4 * i), "l"(src + 4 * i) : "memory");
    }
}
template <int K>
__device__ __forceinline__ Bytes<K> read_bytes(uint32_t p) {
    Bytes<K> b;
    if constexpr (K % 16 == 0) {
#pragma unroll
        for (int i = 0; i < K / 16; ++i)
            asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                         : "=r"(b.w[4 * i]), "=r"(b.w[4 * i + 1]), "=r"(b.w[4 * i + 2]), "=r"(b.w[4 * i + 3])
                         : "r"(p + 16 * i)
                         : "memory");
    } else if constexpr (K % 8 == 0) {
#pragma unroll
        for (int i = 0; i < K / 8; ++i)
            asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];"
                         : "=r"(b.w[2 * i]), "=r"(b.w[2 * i + 1])
                         : "r"(p + 8 * i)
                         : "memory");
    } else {
#pragma unroll
        for (int i = 0; i < K / 4; ++i)
            asm volatile("ld.shared.b32 %0, [%1];" : "=r"(b.w[i]) : "r"(p + 4 * i) : "memory");
    }
    return b;
}
template <int K>
__device__ __forceinline__ void store_bytes(uint8_t* p, const uint32_t (&w)[K / 4]) {
    if constexpr (K % 16 == 0) {
#pragma unroll
        for (int i = 0; i < K / 16; ++i)
            __stcs(reinterpret_cast<uint4*>(p) + i, make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]));
    } else if constexpr (K % 8 == 0) {
#pragma unroll
        for (int i = 0; i < K / 8; ++i) __stcs(reinterpret_cast<uint2*>(p) + i, make_uint2(w[2 * i], w[2 * i + 1]));
    } else {
#pragma unroll
        for (int i = 0; i < K / 4; ++i) __stcs(reinterpret_cast<uint32_t*>(p) + i, w[i]);
    }
}

// Costs of word j: (byte j, byte j + K/2), widened (costs are at most 64, so the
// sign-replicating selectors give zero high bytes).
template <int K>
__device__ __forceinline__ uint32_t cost_word(const Bytes<K>& b, int j) {
    const int h = j + K / 2;
    const uint32_t lo = j & 3, hi = 4 + (h & 3);
    return prmt(b.w[j >> 2], b.w[h >> 2], lo | (8 | lo) << 4 | hi << 8 | (8 | hi) << 12);
}
template <int K>
__device__ __forceinline__ uint32_t cost_byte(const Bytes<K>& b, int j) {
    return (b.w[j >> 2] >> (8 * (j & 3))) & 0xFFu;
}

// The lane's K values as bytes in d order.
template <int K>
__device__ __forceinline__ void pack_bytes(const uint32_t (&y)[K / 2], uint32_t (&w)[K / 4]) {
    // (y[2i], y[2i+1]) bytes: lo, lo, hi, hi, by a multiply-add (minima and byte
    // permutes fill the other pipe). Values above a byte spill into their
    // neighbours, in vectors whose bytes are not read (escaped ones).
    uint32_t p[K / 4];
#pragma unroll
    for (int i = 0; i < K / 4; ++i) p[i] = y[2 * i + 1] * 256u + y[2 * i];
    // Byte pair q of the lane (q < K/4: the low half of p[q], else the high half of p[q - K/4]).
#pragma unroll
    for (int i = 0; i < K / 4; ++i) {
        const int qa = 2 * i, qb = 2 * i + 1;
        const uint32_t sa = qa < K / 4 ? 0x10 : 0x32, sb = qb < K / 4 ? 0x54 : 0x76;
        w[i] = prmt(p[qa % (K / 4)], p[qb % (K / 4)], sa | sb << 8);
    }
}

// u16 pair q of the lane in d order: (d0 + 2q, d0 + 2q + 1).
template <int K>
__device__ __forceinline__ uint32_t pair16(const uint32_t (&y)[K / 2], int q) {
    const int h = q < K / 4 ? q : q - K / 4;
    return prmt(y[2 * h], y[2 * h + 1], q < K / 4 ? 0x5410 : 0x7632);
}

// Minimum over the segment's lanes as signed words (v = the same 16-bit value in both halves).
template <int SEG>
__device__ __forceinline__ int seg_min(int v) {
    if constexpr (SEG == 1) return v;
    if constexpr (SEG == 32) return __reduce_min_sync(kFull, v);
    if constexpr (SEG == 2) return min(v, __shfl_xor_sync(kFull, v, 1));
    // Lanes 1, 2, 3 away at once, then 4 (8, 12) away: two dependent rounds for 8 and 16 lanes.
    const int a = __shfl_xor_sync(kFull, v, 1), b = __shfl_xor_sync(kFull, v, 2), c = __shfl_xor_sync(kFull, v, 3);
    v = min(__vimin3_s32(v, a, b), c);
    if constexpr (SEG == 8) v = min(v, __shfl_xor_sync(kFull, v, 4));
    if constexpr (SEG == 16) {
        const int d = __shfl_xor_sync(kFull, v, 4), e = __shfl_xor_sync(kFull, v, 8), f = __shfl_xor_sync(kFull, v, 12);
        v = min(__vimin3_s32(v, d, e), f);
    }
    return v;
}

// Minimum over the segment's lanes below this one (0xFFFFFFFF for its first).
template <int SEG>
__device__ __forceinline__ uint32_t scan_min_below(uint32_t v) {
    constexpr uint32_t inf = 0xFFFFFFFFu;
    constexpr uint32_t clamp = (32 - SEG) << 8;
    if constexpr (SEG == 1) return inf;
    uint32_t e = shfl_up_or(v, 1, clamp, inf);
    if constexpr (SEG == 2) return e;
    const uint32_t a = shfl_up_or(v, 2, clamp, inf), b = shfl_up_or(v, 3, clamp, inf);
    e = __vimin3_u32(e, a, b);
    if constexpr (SEG == 4) return e;
    e = min(e, shfl_up_or(v, 4, clamp, inf));        // the four lanes below
    // A lane without a partner gets its own e, which changes nothing.
    if constexpr (SEG == 8) return min(e, __shfl_up_sync(kFull, e, 4, SEG));
    const uint32_t c = __shfl_up_sync(kFull, e, 4, SEG), d = __shfl_up_sync(kFull, e, 8, SEG),
                   f = __shfl_up_sync(kFull, e, 12, SEG);
    e = min(__vimin3_u32(e, c, d), f);               // the sixteen lanes below
    if constexpr (SEG == 32) e = min(e, __shfl_up_sync(kFull, e, 16, SEG));
    return e;
}

// Sum over the segment's lanes below this one.
template <int SEG>
__device__ __forceinline__ uint32_t scan_sum_below(uint32_t v) {
    constexpr uint32_t clamp = (32 - SEG) << 8;
    uint32_t s = v;
#pragma unroll
    for (int o = 1; o < SEG; o <<= 1)
        asm volatile(
            "{\n .reg .pred p;\n .reg .b32 t;\n shfl.sync.up.b32 t|p, %0, %1, %2, 0xffffffff;\n"
            " @p add.u32 %0, %0, t;\n}"
            : "+r"(s)
            : "r"(o), "r"(clamp));
    return s - v;
}

// Cost slots of a thread: the costs of slots_for(K) consecutive steps in shared memory,
// filled by asynchronous copies two steps less ahead. (Loads into
// registers that far ahead make each use wait for the newest of them, since they
// share the few scoreboards of a warp; asynchronous copies are waited for in
// groups, oldest first.)
__host__ __device__ constexpr int slots_for(int k) { return k <= 12 ? 8 : 6; }   // at most 48 KB a CTA
constexpr int kThreads = 128;   // a warp to each of an SM's four schedulers

// One unit: the warp's 32 / SEG scanlines first.. of one (pair, path), each on
// one segment of SEG lanes; lane li of a segment holds disparities
// d0 = li*K .. d0+K-1. All lanes run every step (the shuffles are
// warp-collective). PADS: some of the segment's SEG * K disparities are not real.
// ring: this thread's slot 0 (shared address); slot s is s * 32 * K bytes on (a warp's slots are its own).
template <int K, int SEG, bool PADS, bool CP>
__device__ __forceinline__ void run_unit(const PairDev& pr, const JobDev& job, int first, int lane,
                                         const uint32_t ring) {
    constexpr int N = K / 2;
    constexpr int kSlotBytes = 32 * K, kSlots = slots_for(K);
    const int W = pr.width, H = pr.height, D = pr.nd, Dv = pr.nd_vec;
    const uint32_t P1 = (uint32_t)pr.p1, P2 = (uint32_t)pr.p2;
    const bool wide = pr.wide_slabs != 0;
    const int sl = lane / SEG, li = lane % SEG;
    const int d0 = li * K;
    const bool last = li == SEG - 1;
    const bool lane_on = !PADS || d0 < Dv;
    const int k = first + sl;

    // Steps [tb, tb + len) of this scanline; pixel index base + t * step.
    int tb = INT_MAX, te = INT_MIN;
    ptrdiff_t base = 0;
    const int dx = job.dx, dy = job.dy;
    const ptrdiff_t step = (ptrdiff_t)dy * W + dx;
    if (k < job.num_scanlines) {
        if (dy == 0) {
            tb = 0;
            te = W;
            base = (ptrdiff_t)k * W + (dx > 0 ? 0 : W - 1);
        } else {
            const int kk = job.k_min + k;
            if (dx == 0) { tb = 0; te = H; }
            else if (dx > 0) { tb = max(0, -kk); te = min(H, W - kk); }
            else { tb = max(0, kk - W + 1); te = min(H, kk + 1); }
            base = (ptrdiff_t)(dy > 0 ? 0 : H - 1) * W + kk;
        }
    }
    const int t_lo = __reduce_min_sync(kFull, tb), t_hi = __reduce_max_sync(kFull, te);
    if (t_lo >= t_hi) return;
    const unsigned len = te > tb && lane_on ? (unsigned)(te - tb) : 0u;   // lanes past the vector never read or write
    if (te <= tb) tb = t_lo;
    const unsigned store_len = wide ? 0u : len;
    int rel = t_lo - tb;                                  // step index inside the scanline; active: unsigned(rel) < len

    const ptrdiff_t vstep = step * Dv;                    // bytes between a scanline's vectors
    const ptrdiff_t off0 = (base + (ptrdiff_t)t_lo * step) * Dv + d0;
    const uint8_t* cp = pr.costs + off0;                  // dereferenced on active steps only
    uint8_t* op = pr.slabs + pr.slab_stride * (size_t)job.path + off0;

    const uint32_t P1x2 = P1 * 0x10001u, P2x2 = P2 * 0x10001u;
    const uint32_t BV = 64u * (uint32_t)Dv + P2 + 65u;
    const uint32_t KU = 0x10000u - P1x2;                  // per half 65536 - P1, as one 32-bit addend
    const uint32_t w0 = (uint32_t)d0 | (uint32_t)(d0 + N) << 16;
    const uint32_t e0 = BV * 0x10001u + w0 * P1;          // V before the lane's halves, without costs and m
    const uint32_t nw0 = 0u - w0;
    const uint32_t fill = (0xFFFFu - P1) & 0xFFFFu;
    const uint32_t fillx2 = fill * 0x10001u;
    // A vector with a value above 254 is looked at more closely. Where 64 + P2 <= 254
    // only a wrapped value is above it, and the signed minimum shows that; otherwise
    // (wide slabs, or byte slabs asked for with a larger P2) every vector is.
    constexpr uint32_t plainx2 = 0x00FE00FEu;
    const uint32_t idle = wide || 64u + P2 > 254u ? 0xFFFFFFFFu : 0u;
    uint32_t keep[PADS ? N : 1] = {};                     // real disparities' halves
    if constexpr (PADS) {
#pragma unroll
        for (int j = 0; j < N; ++j)
            keep[j] = (d0 + j < D ? 0xFFFFu : 0u) | (d0 + j + N < D ? 0xFFFF0000u : 0u);
    }
    auto mask = [&](uint32_t v, int j) { return PADS ? v & keep[PADS ? j : 0] : v; };    // pads 0
    auto keep_all = [&](int j) { return PADS ? keep[PADS ? j : 0] : 0xFFFFFFFFu; };
    auto lift = [&](uint32_t v, int j) {                                                  // pads 0x7FFF
        return PADS ? (v & keep[PADS ? j : 0]) | (0x7FFF7FFFu & ~keep[PADS ? j : 0]) : v;
    };

    // Sums of the lane's costs: of its low half and of all of it.
    auto lane_sums = [&](const Bytes<K>& c, uint32_t& lo, uint32_t& all) {
        lo = 0;
        uint32_t hi = 0;
        if constexpr (N % 4 == 0) {
#pragma unroll
            for (int i = 0; i < N / 4; ++i) {
                lo = __dp4a(c.w[i], 0x01010101u, lo);
                hi = __dp4a(c.w[i + N / 4], 0x01010101u, hi);
            }
        } else {                                          // K = 12: bytes 0..5 | 6..11
            lo = __dp4a(c.w[0], 0x01010101u, __dp4a(c.w[1], 0x00000101u, 0u));
            hi = __dp4a(c.w[2], 0x01010101u, __dp4a(c.w[1], 0x01010000u, 0u));
        }
        all = lo + hi;
    };
    // V before the lane's first words of two steps, without m: the costs below the
    // lane (and, in the high half, of the lane's low half). One scan for both
    // steps: a step's sum over the segment is at most 64 * 256.
    auto lane_bases = [&](const Bytes<K>& ca, const Bytes<K>& cb, uint32_t& ea, uint32_t& eb) {
        uint32_t la, lb, ta, tb2;
        lane_sums(ca, la, ta);
        lane_sums(cb, lb, tb2);
        const uint32_t below = scan_sum_below<SEG>(ta + (tb2 << 16));
        ea = e0 + prmt(below, below, 0x1010) + (la << 16);
        eb = e0 + prmt(below, below, 0x3232) + (lb << 16);
    };

    uint32_t L[N];
#pragma unroll
    for (int j = 0; j < N; ++j) L[j] = 0u;
    uint32_t mm = 0u;                                     // m in both halves
    uint32_t forced = idle;                               // all ones after a vector with m > 64

    // Two steps a group of copies; the slots hold kSlots / 2 groups. The slots start at
    // 0, which is what a scanline's steps before its first pixel read.
    asm volatile("cp.async.wait_all;" ::: "memory");
#pragma unroll
    for (int i = 0; i < kSlots; ++i)
#pragma unroll
        for (int w = 0; w < K / 4; ++w)
            asm volatile("st.shared.b32 [%0], %1;" ::"r"(ring + i * kSlotBytes + 4 * w), "r"(0) : "memory");
    auto copy_group = [&](uint32_t slot, int arel) {      // steps arel, arel + 1
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            if ((unsigned)(arel + i) < len) copy_bytes_async<K>(slot + i * kSlotBytes, cp);
            cp += vstep;
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int i = 0; i < kSlots / 2; ++i) copy_group(ring + 2 * i * kSlotBytes, rel + 2 * i);
    asm volatile("cp.async.wait_group %0;" ::"n"(kSlots / 2 - 1) : "memory");
    Bytes<K> c2[2] = {read_bytes<K>(ring), read_bytes<K>(ring + kSlotBytes)};
    uint32_t e2[2];
    lane_bases(c2[0], c2[1], e2[0], e2[1]);

    uint32_t slot = ring;                                 // the slots of this step and the next
#pragma unroll 1
    for (int left = t_hi - t_lo; left > 0; left -= 2) {
        // The next two steps' costs and bases.
        asm volatile("cp.async.wait_group %0;" ::"n"(kSlots / 2 - 2) : "memory");
        const uint32_t next_slot = slot == ring + (kSlots - 2) * kSlotBytes ? ring : slot + 2 * kSlotBytes;
        const Bytes<K> n2[2] = {read_bytes<K>(next_slot), read_bytes<K>(next_slot + kSlotBytes)};
        uint32_t ne2[2];
        lane_bases(n2[0], n2[1], ne2[0], ne2[1]);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const bool active = (unsigned)rel < len;
            // Read again rather than held in registers where a lane has many.
            const Bytes<K> c = K <= 12 ? c2[i] : read_bytes<K>(slot + i * kSlotBytes);
            uint32_t nb = __shfl_down_sync(kFull, L[0], 1, SEG);   // the next lane's L[d0 + K] (low half)
            if (last) nb = fill;
            const uint32_t nbw = prmt(L[0], nb, 0x5432);
            const uint32_t o3 = mm + P2x2, q = P1x2 - mm;
            const uint32_t vb = e2[i] + nw0 * (mm & 0xFFFFu);

            uint32_t V[N], y[N];
#pragma unroll
            for (int j = 0; j < N; ++j) {
                const uint32_t vp = j == 0 ? vb : V[j - 1];
                V[j] = vp + cost_word<K>(c, j) + q;
                const uint32_t o2 = __vadd2(j + 1 < N ? L[j + 1] : nbw, P1x2);
                y[j] = __vimin3_u16x2(L[j], o2, o3) + KU - vp;     // U
            }
            // The lane's minimum of U per half, then over both.
            uint32_t T = y[0];
#pragma unroll
            for (int j = 1; j + 1 < N; j += 2) T = __vimin3_u16x2(T, y[j], y[j + 1]);
            if constexpr (N % 2 == 0) T = vmin2(T, y[N - 1]);
            const uint32_t below = scan_min_below<SEG>(vmin2(T, prmt(T, T, 0x1032)));
            uint32_t z = vmin2(below, prmt(T, 0xFFFFFFFFu, 0x1044));   // low half: below; high: also the low half's
#pragma unroll
            for (int j = 0; j < N; ++j) {
                z = vmin2(z, y[j]);
                y[j] = __vadd2(V[j], z);
                if (PADS) y[j] = (y[j] & keep[PADS ? j : 0]) | (fillx2 & ~keep[PADS ? j : 0]);
            }
            // The vector's minimum, as signed halves: negative where a value wrapped
            // (u16(y) of a y in -P1..-1), which the closer look below takes out again.
            uint32_t mn = lift(y[0], 0);
#pragma unroll
            for (int j = 1; j + 1 < N; j += 2) mn = __vimin3_s16x2(mn, lift(y[j], j), lift(y[j + 1], j + 1));
            if constexpr (N % 2 == 0) mn = smin2(mn, lift(y[N - 1], N - 1));
            mn = smin2(mn, prmt(mn, mn, 0x1032));
            const uint32_t m_prev = mm;
            mm = (uint32_t)seg_min<SEG>((int)mn);
            uint32_t w[K / 4];
            pack_bytes<K>(y, w);
            const bool look = __any_sync(kFull, active && (int)(mn | forced) < 0);
            if (__builtin_expect(look, 0)) {
                const unsigned seg_lanes = SEG == 32 ? kFull : ((1u << (SEG & 31)) - 1u) << ((sl * SEG) & 31);
                const uint32_t m = m_prev & 0xFFFFu;
                bool bad = m > 64u;
#pragma unroll
                for (int j = 0; j < N; ++j) bad |= (mask(__vadd2(y[j], P1x2), j) & 0x80008000u) != 0u;
                const unsigned bad_lanes = __ballot_sync(kFull, active && bad);
                if (bad_lanes) {
                    const bool redo = (bad_lanes & seg_lanes) != 0u;
                    const Bytes<K> rc = read_bytes<K>(slot + i * kSlotBytes);   // not held in registers for this
                    const uint32_t q3 = (m + P2) & 0xFFFFu;
                    uint32_t carry = 0u;                           // Lnew[d0 - 1], from the lane below
#pragma unroll 1
                    for (int s = 0; s < SEG; ++s) {
                        uint32_t prev = carry;
                        if (redo && li == s) {
                            uint32_t r[N];
#pragma unroll
                            for (int j = 0; j < K; ++j) {
                                const int a = j % N;
                                const uint32_t q0 = j < N ? L[a] & 0xFFFFu : L[a] >> 16;
                                const uint32_t nx = j + 1 == K ? nb & 0xFFFFu
                                                    : j + 1 < N ? L[(j + 1) % N] & 0xFFFFu : L[(j + 1) % N] >> 16;
                                if (!PADS || d0 + j < D) {
                                    const uint32_t q1 = d0 + j == 0 ? 0xFFFFu : (prev + P1) & 0xFFFFu;
                                    const uint32_t q2 = d0 + j == D - 1 ? 0xFFFFu : (nx + P1) & 0xFFFFu;
                                    prev = (cost_byte<K>(rc, j) + min(min(q0, q1), min(q2, q3)) - m) & 0xFFFFu;
                                }
                                const uint32_t out = (!PADS || d0 + j < D) ? prev : fill;
                                r[a] = j < N ? out : r[a] | out << 16;
                            }
#pragma unroll
                            for (int j = 0; j < N; ++j) y[j] = r[j];
                        }
                        carry = __shfl_sync(kFull, prev, s, SEG);
                    }
                    pack_bytes<K>(y, w);
                }
                // The shader's minimum (of ushorts) and maximum.
                uint32_t lo = y[0] | ~keep_all(0), mx = mask(y[0], 0);
#pragma unroll
                for (int j = 1; j < N; ++j) {
                    lo = vmin2(lo, y[j] | ~keep_all(j));
                    mx = vmax2(mx, mask(y[j], j));
                }
                lo = min(lo & 0xFFFFu, lo >> 16);
#pragma unroll
                for (int o = SEG / 2; o > 0; o >>= 1) lo = min(lo, __shfl_xor_sync(kFull, lo, o));
                mm = lo * 0x10001u;
                forced = lo > 64u ? 0xFFFFFFFFu : idle;
                // The pixel, from the slab address (used on active steps).
                const uint8_t* slab = pr.slabs + pr.slab_stride * (size_t)job.path;
                const size_t pix = (uint32_t)((size_t)(op - slab) >> 4) / (uint32_t)(Dv >> 4);
                const int Dp = pr.nd_pad;
                const bool esc =
                    (__ballot_sync(kFull, active && !wide && vmax2(mx, plainx2) != plainx2) & seg_lanes) != 0u;
                // Escaped (and wide) vectors' u16 values go to the shadow.
                uint32_t taken = kNoSlot;
                if constexpr (CP) {
                    const EscapeTarget et = escape_target(pr, job.path);
                    if (esc && active && li == 0) taken = take_slot(et, pix);
                    taken = __shfl_sync(kFull, taken, 0, SEG);
                }
                if (active && (wide || esc)) {
                    uint16_t* dst = nullptr;
                    if (!CP || wide) dst = pr.shadow + pr.shadow_stride * (size_t)job.path + pix * Dp + d0;
                    else if (taken != kNoSlot) dst = pr.shadow + (size_t)taken * Dp + d0;
                    if (dst) {
#pragma unroll
                        for (int v = 0; v < K / 4; ++v)
                            if (d0 + 4 * v < Dp)
                                __stcs(reinterpret_cast<uint2*>(dst + 4 * v),
                                       make_uint2(pair16<K>(y, 2 * v), pair16<K>(y, 2 * v + 1)));
                    }
                }
                if (esc && li == 0) {
                    w[0] |= 0xFFu;                                 // the escape marker (byte 0)
                    if (CP) w[1] = taken;                          // the shadow slot (bytes 4..7)
                }
            }
            if ((unsigned)rel < store_len) store_bytes<K>(op, w);
            op += vstep;
            ++rel;
#pragma unroll
            for (int j = 0; j < N; ++j) L[j] = y[j];
        }
        copy_group(slot, rel + kSlots - 2);               // rel is two steps on
        slot = next_slot;
        if (K <= 12) c2[0] = n2[0], c2[1] = n2[1];
        e2[0] = ne2[0], e2[1] = ne2[1];
    }
}

// The variants of a kind: X(K, SEG, PADS).
#define VX_PACKED_LATENCY(X)                                                                         \
    X(8, 2, false) X(8, 4, false) X(8, 8, false) X(8, 16, false) X(8, 32, false) X(12, 4, false)     \
    X(12, 8, false) X(12, 16, false) X(8, 2, true) X(8, 4, true) X(8, 8, true) X(8, 16, true) X(8, 32, true)
#define VX_PACKED_THROUGHPUT(X)                                                                      \
    X(16, 1, false) X(16, 2, false) X(24, 2, false) X(24, 4, false) X(24, 8, false)  \
    X(32, 2, false) X(32, 4, false) X(32, 8, false) X(16, 1, true) X(16, 2, true) X(16, 4, true) X(16, 8, true) X(16, 16, true)

__host__ __device__ constexpr int min_ctas(int k) { return k <= 12 ? 6 : 4; }

// One class of units of a plan: [0, num_units) of `units`, all of this variant.
// The first class is an ordinary launch: started while the cost kernel drains, its
// CTAs would not be spread one to an SM (640x480: 208 -> 233 us a call). A plan's
// classes are launched one after another; the chained ones (all but the first)
// start as soon as the class before has started all its CTAs and frees room for
// theirs, and end after it (their work is independent: no class waits for another's
// results). more: another class follows.
template <int K, int SEG, bool PADS, bool CP>
__global__ void __launch_bounds__(kThreads, min_ctas(K))
packed_kernel(const PairDev* __restrict__ pairs, const JobDev* __restrict__ jobs, const UnitDev* __restrict__ units,
              const int num_units, unsigned* __restrict__ counter, const int sms, const int chained, const int more) {
    __shared__ __align__(16) unsigned char slots[kThreads * slots_for(K) * K];
    const int lane = threadIdx.x & 31;
    const uint32_t ring =
        (uint32_t)__cvta_generic_to_shared(slots) + (threadIdx.x >> 5) * (32 * slots_for(K) * K) + lane * K;
    if (more) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    // First unit of a warp by an interleaved rank: the longest units of the LPT order
    // go one to an SM, then one to each of an SM's schedulers (a warp of the CTA),
    // then to the SMs' second CTAs. Later units come from the counter, after the
    // warps' firsts.
    const int warps = (int)gridDim.x * (kThreads / 32);
    const int round = (int)blockIdx.x / sms, sm = (int)blockIdx.x - round * sms;
    // (Through a shuffle, as below: so the compiler knows that a warp's unit, and all
    // that follows from it, is the same in every lane, and keeps it in uniform
    // registers: 64 mixed pairs (3.25 G pixel-disparities) 10.5 -> 9.7 ms, 1242x375 445 -> 415 us.)
    int u = __shfl_sync(kFull, (round * (kThreads / 32) + (int)(threadIdx.x >> 5)) * sms + sm, 0);
    while (u < num_units) {
        // By reference: what a unit needs rarely is read when it is needed, not held in registers.
        const JobDev& job = jobs[units[u].job];
        run_unit<K, SEG, PADS, CP>(pairs[job.pair], job, units[u].first_scanline, lane, ring);
        __syncwarp();
        if (lane == 0) u = warps + (int)atomicAdd(counter, 1u);
        u = __shfl_sync(kFull, u, 0);
    }
    if (chained) asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <int KIND, bool CP>
const void* kernel_fn(const ScanGeometry& g) {
    const int v = g.k * 128 + g.seg * 2 + (g.pads ? 1 : 0);
#define VX_CASE(K, SEG, PADS) \
    case K * 128 + SEG * 2 + (PADS ? 1 : 0): return (const void*)packed_kernel<K, SEG, PADS, CP>;
    if constexpr (KIND == kPackedLatency) {
        switch (v) { VX_PACKED_LATENCY(VX_CASE) }
    } else {
        switch (v) { VX_PACKED_THROUGHPUT(VX_CASE) }
    }
#undef VX_CASE
    return nullptr;
}

template <int KIND>
cudaError_t launch_kind(const ScanGeometry& g, int ctas, const PairDev* d_pairs, const JobDev* d_jobs, const UnitDev* d_units,
                        int num_units, unsigned* counter, cudaStream_t stream, bool compact, bool chained, bool more) {
    int dev = 0, sms = 148, per_sm = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const void* fn = compact ? kernel_fn<KIND, true>(g) : kernel_fn<KIND, false>(g);
    if (!fn) return cudaErrorInvalidDeviceFunction;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kThreads, 0) != cudaSuccess || per_sm < 1) {
        cudaGetLastError();
        per_sm = 1;
    }
    // Whole rounds of the SMs, so that a warp's first unit is where its rank says.
    const int needed = (num_units + sms * (kThreads / 32) - 1) / (sms * (kThreads / 32));
    const int grid = sms * std::min({per_sm, ctas, needed});
    if (std::getenv("VX_SGM_DEBUG"))
        std::fprintf(stderr, "vx_sgm: aggregation (packed scan, %d x %d%s) %d CTAs x %d threads (%d an SM), %d units\n",
                     g.k, g.seg, g.pads ? " pads" : "", grid, kThreads, per_sm, num_units);
    count_launch();
    int is_chained = chained ? 1 : 0, has_more = more ? 1 : 0;
    void* args[] = {&d_pairs, &d_jobs, &d_units, &num_units, &counter, &sms, &is_chained, &has_more};
    return launch_kernel(fn, dim3(grid), dim3(kThreads), 0, stream, chained, args);
}

}  // namespace
}  // namespace packed
}  // namespace vxsgm
