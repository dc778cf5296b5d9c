// hs_lane.cuh -- the Horner chain over the window sums, on lane-sliced field elements.
//
// The chain's 256 doublings are sequential, so its time is the latency of one
// doubling: three dependent products.  In eight 32-bit limbs on one thread a
// product takes 517 (F_p) / 712 (F_q) clocks.  Here an element is a list of
// radix-2^26 limbs, ten on F_p, eleven on F_q, in shared memory, and a product is
// formed column-wise by a warp: lane l sums a_i b_(l-i) in a 64-bit register.
//
// What a product waits for, in order, and what keeps it short:
// - operands: an element is stored plainly (all lanes read the limbs a_i as the
//   same 16-byte words) and as windows (reversed, zero-padded, in four copies of
//   different alignment, so that lane l reads b_l, b_(l-1), ... as three 16-byte
//   words): six loads instead of two shuffles per limb;
// - sums of products share one set of columns (a b - c d + K with K a multiple of
//   the modulus whose columns exceed the subtrahend's), so that no subtraction is
//   a step of its own;
// - F_p: columns below 2^58, so one shuffle moves what leaves a column; the columns
//   past 2^260 come down times 608 (2^260 == 608) in the same round, then one carry
//   round: four shuffles;
// - F_q: one carry round, one fold of lanes 10..22 by a table of 2^(26(10+h)) mod
//   q, one carry round.  The value is then below 2^286, which an eleventh limb
//   holds (ten would need a second fold and carry).
//
// Bounds, F_p, columns in units of 2^52: norm of columns up to C leaves limbs up to
// 2^26 + 2^16, limb 0 up to (1 + 0.0057 C S) 2^26.  With K = 11 (one product
// subtracted) or 22 (two), the largest columns are 4 Y^2: 41, X': 33, D: 43, Y': 22,
// the M step: 22 with S = 3, the addition's Y': 63; products of the resulting
// elements stay below 10.8 columns, so each K covers what is subtracted, and 64
// (2^58) is never reached.  F_q: stored limbs are below 2^27 + 2^6 (lane 10 below
// 2^26), so a product's columns stay below 11 x 2^54.1 < 2^57.6; K's columns are 2^60;
// the largest sum taken, 3 (a^2 + K - b^2), stays below 2^62.  The fold is a sum below
// 2^27 + 13 x 2^27.1 x 2^26 < 2^57, its lane 9 below 2^52 (the table's limb 9 has 21
// bits), so nothing reaches lane 11.
//
// Measured on GB300: a doubling 1047 (F_p) / 1555 (F_q) clocks; the chain of one MSM at
// c = 16 166 / 259 us against 192 / 306 for ten limbs exchanged by two shuffles per
// limb, with three barriers per doubling; at c = 8 193 / 287 against 222 / 338.  A
// shuffle issues every 4.5 clocks and takes 24, a 16-byte shared load every 11 and
// takes 34; F_q's fold through shared memory instead of shuffles was slower
// (1720 clocks per doubling), as were four chains of multiply-adds per product.
#pragma once
#include "hs_curve.cuh"
#include "hs_internal.h"

namespace hs {

constexpr unsigned LN_ALL = 0xffffffffu;
constexpr uint64_t LN_M26 = (1ull << 26) - 1;

// K: columns that sum to a multiple of the modulus (11 x 2^52 and 22 x 2^52 for F_p, 2^60 for F_q, and a little)
static __constant__ uint64_t LN_KP[2][19] = {
    {0xb0000003c1d9cdull, 0xb0000003ffe5dfull, 0xb0000003ffe5d4ull, 0xb0000003ffe5d4ull, 0xb0000003ffe5d4ull, 0xb0000003ffe5d4ull, 0xb0000003ffe5d4ull, 0xb0000003ffe5d4ull, 0xb0000003ffe5d4ull, 0xb00000001fe5d4ull, 0xb0000000000000ull, 0xb0000000000000ull, 0xb0000000000000ull, 0xb0000000000000ull, 0xb0000000000000ull, 0xb0000000000000ull, 0xb0000000000000ull, 0xb0000000000000ull, 0xb0000000000000ull},
    {0x16000000383b3adull, 0x160000003ffcbbfull, 0x160000003ffcba9ull, 0x160000003ffcba9ull, 0x160000003ffcba9ull, 0x160000003ffcba9ull, 0x160000003ffcba9ull, 0x160000003ffcba9ull, 0x160000003ffcba9ull, 0x1600000001fcba9ull, 0x160000000000000ull, 0x160000000000000ull, 0x160000000000000ull, 0x160000000000000ull, 0x160000000000000ull, 0x160000000000000ull, 0x160000000000000ull, 0x160000000000000ull, 0x160000000000000ull},
};
static __constant__ uint64_t LN_KQ[21] = {
    0x1000000001ef8691ull, 0x100000000238ef9cull, 0x1000000002689ac0ull, 0x1000000002525a6eull, 0x1000000002ad4d04ull, 0x1000000001fd1000ull, 0x10000000005805c8ull, 0x1000000003434d32ull, 0x10000000028670feull, 0x100000000002425bull, 0x1000000000000000ull, 0x1000000000000000ull, 0x1000000000000000ull, 0x1000000000000000ull, 0x1000000000000000ull, 0x1000000000000000ull, 0x1000000000000000ull, 0x1000000000000000ull, 0x1000000000000000ull, 0x1000000000000000ull, 0x1000000000000000ull};
// row h: 2^(26 (10 + h)) mod q in ten limbs
static __constant__ uint32_t LN_RQ[13][10] = {
    {0x3070c20u, 0x16c6c36u, 0x14f2292u, 0x1a44d4au, 0x01010fau, 0x0000002u, 0x0000000u, 0x0000000u, 0x0000000u, 0x0000000u},
    {0x0000000u, 0x3070c20u, 0x16c6c36u, 0x14f2292u, 0x1a44d4au, 0x01010fau, 0x0000002u, 0x0000000u, 0x0000000u, 0x0000000u},
    {0x0000000u, 0x0000000u, 0x3070c20u, 0x16c6c36u, 0x14f2292u, 0x1a44d4au, 0x01010fau, 0x0000002u, 0x0000000u, 0x0000000u},
    {0x0000000u, 0x0000000u, 0x0000000u, 0x3070c20u, 0x16c6c36u, 0x14f2292u, 0x1a44d4au, 0x01010fau, 0x0000002u, 0x0000000u},
    {0x0000000u, 0x0000000u, 0x0000000u, 0x0000000u, 0x3070c20u, 0x16c6c36u, 0x14f2292u, 0x1a44d4au, 0x01010fau, 0x0000002u},
    {0x20e1840u, 0x2d8d86du, 0x29e4524u, 0x3489a94u, 0x02021f4u, 0x3070c24u, 0x16c6c36u, 0x14f2292u, 0x1a44d4au, 0x01010fau},
    {0x09eb42du, 0x1f359fcu, 0x23798c8u, 0x17660e7u, 0x2f5edcbu, 0x0408471u, 0x3070c24u, 0x16c6c36u, 0x14f2292u, 0x0044d4au},
    {0x3a1550au, 0x24f5d25u, 0x36b84ebu, 0x121f2c1u, 0x1a54480u, 0x2fe99a7u, 0x0408471u, 0x3070c24u, 0x16c6c36u, 0x00f2292u},
    {0x2cb966bu, 0x248f1a0u, 0x0cf0f2fu, 0x10edbc3u, 0x1fe917eu, 0x1c3c66fu, 0x2fe99a7u, 0x0408471u, 0x3070c24u, 0x00c6c36u},
    {0x25f57d8u, 0x2f3ea03u, 0x1679a21u, 0x0c9df95u, 0x1650e8du, 0x2179bd1u, 0x1c3c66fu, 0x2fe99a7u, 0x0408471u, 0x0070c24u},
    {0x01fa542u, 0x0c733b9u, 0x04912c4u, 0x3c483d4u, 0x331e04fu, 0x1734323u, 0x2179bd1u, 0x1c3c66fu, 0x2fe99a7u, 0x0008471u},
    {0x1c9ead7u, 0x18d931du, 0x039ce26u, 0x1979b54u, 0x168acbeu, 0x332eb47u, 0x1734323u, 0x2179bd1u, 0x1c3c66fu, 0x01e99a7u},
    {0x36b1e2eu, 0x2bb608fu, 0x30fe555u, 0x1875909u, 0x317af2cu, 0x1a65af5u, 0x332eb47u, 0x1734323u, 0x2179bd1u, 0x003c66fu},
};

// an element in shared memory: limb m at p[m] and, in copy s of the windows, at
// w[40 s + 24 - m + s]; every other word is zero
struct alignas(16) LaneSlot {
    uint32_t p[12];
    uint32_t w[160];
};

template <class F>
struct LaneField {
    static constexpr bool FQ = F::Params::NC != 1;
    static constexpr int NL = FQ ? 11 : 10;       // limbs of an element
    static constexpr int NCOL = 2 * NL - 1;       // columns of a product

    int lane;
    int wofs;        // this lane's window: words b_lane, b_(lane-1), ... of an element start at w[wofs]
    uint64_t k, k2;  // column `lane` of K, for one and for two subtracted products
    uint32_t k1;     // F_p: 608 on lane 0, 1 elsewhere
    int prev;        // F_p: lane - 1, on lane 0 lane 9
    uint32_t m1, m2; // all ones but on lane 0 / lanes 0 and 1
    uint32_t r[13];  // F_q: limb `lane` of the fold table's rows

    __device__ __forceinline__ explicit LaneField(int lane_) : lane(lane_)
    {
        const int t0 = lane <= 24 ? 24 - lane : 0;  // lanes past the columns read zeros
        const int s = lane <= 24 ? (lane & 3) : 0;
        wofs = 40 * s + t0 + s;
        k = lane < NCOL ? (FQ ? LN_KQ[lane < NCOL ? lane : 0] : LN_KP[0][lane < 19 ? lane : 0]) : 0ull;
        k2 = lane < NCOL ? (FQ ? LN_KQ[lane < NCOL ? lane : 0] : LN_KP[1][lane < 19 ? lane : 0]) : 0ull;
        k1 = lane == 0 ? 608u : 1u;
        prev = lane == 0 ? 9 : lane - 1;
        m1 = lane >= 1 ? 0xffffffffu : 0u;
        m2 = lane >= 2 ? 0xffffffffu : 0u;
#pragma unroll
        for (int h = 0; h < 13; h++)
            r[h] = (FQ && lane < 10) ? LN_RQ[h][lane < 10 ? lane : 0] : 0u;
    }

    // column `lane` of a b
    __device__ __forceinline__ uint64_t cols(const uint32_t *__restrict__ a, const LaneSlot &b) const
    {
        const uint4 *pa = reinterpret_cast<const uint4 *>(a);
        const uint4 *pb = reinterpret_cast<const uint4 *>(b.w + wofs);
        const uint4 a0 = pa[0], b0 = pb[0], a1 = pa[1], b1 = pb[1], a2 = pa[2], b2 = pb[2];
        uint64_t c0 = (uint64_t)a0.x * b0.x, c1 = (uint64_t)a0.y * b0.y;
        c0 += (uint64_t)a0.z * b0.z;
        c1 += (uint64_t)a0.w * b0.w;
        c0 += (uint64_t)a1.x * b1.x;
        c1 += (uint64_t)a1.y * b1.y;
        c0 += (uint64_t)a1.z * b1.z;
        c1 += (uint64_t)a1.w * b1.w;
        c0 += (uint64_t)a2.x * b2.x;
        c1 += (uint64_t)a2.y * b2.y;
        if (NL > 10)
            c0 += (uint64_t)a2.z * b2.z;
        return c0 + c1;
    }
    __device__ __forceinline__ uint64_t cols(const LaneSlot &a, const LaneSlot &b) const { return cols(a.p, b); }

    // S times the columns' value -> this lane's limb (lanes past the element's limbs:
    // unspecified; put stores only limbs)
    template <uint32_t S = 1>
    __device__ __forceinline__ uint32_t norm(uint64_t c) const
    {
        const uint32_t lo = (uint32_t)c & (uint32_t)LN_M26;
        if constexpr (!FQ) {
            // columns below 2^58: what leaves a column fits 32 bits.  Positions 10..19
            // (the low part of column 10 + l, the upper part of column 9 + l) come
            // down times 608.
            const uint32_t up = (uint32_t)(c >> 26);
            const uint32_t u = __shfl_up_sync(LN_ALL, up, 1);
            const uint32_t v0 = __shfl_sync(LN_ALL, lo, lane + 10), v1 = __shfl_sync(LN_ALL, up, lane + 9);
            const uint64_t d = (uint64_t)(v0 + v1) * (608u * S) + ((uint64_t)(u & m1) + lo) * S;  // below 2^44
            // one carry round, limb 9's times 608 to limb 0
            const uint32_t e = __shfl_sync(LN_ALL, (uint32_t)(d >> 26), prev);
            return ((uint32_t)d & (uint32_t)LN_M26) + e * k1;
        } else {
            if (S != 1)
                return norm(c * S);
            const uint32_t mid = (uint32_t)(c >> 26) & (uint32_t)LN_M26, hi = (uint32_t)(c >> 52);
            const uint32_t u1 = __shfl_up_sync(LN_ALL, mid, 1), u2 = __shfl_up_sync(LN_ALL, hi, 2);
            const uint32_t cur = lo + (u1 & m1) + (u2 & m2);  // lanes 0..22
            uint64_t d0 = lane < 10 ? (uint64_t)cur : 0ull, d1 = 0;
#pragma unroll
            for (int h = 0; h < 13; h++) {
                const uint32_t x = __shfl_sync(LN_ALL, cur, 10 + h);
                if (h & 1)
                    d1 += (uint64_t)x * r[h];
                else
                    d0 += (uint64_t)x * r[h];
            }
            d0 += d1;
            const uint32_t w1 = __shfl_up_sync(LN_ALL, (uint32_t)(d0 >> 26) & (uint32_t)LN_M26, 1);
            const uint32_t w2 = __shfl_up_sync(LN_ALL, (uint32_t)(d0 >> 52), 2);
            return ((uint32_t)d0 & (uint32_t)LN_M26) + (w1 & m1) + (w2 & m2);
        }
    }

    __device__ __forceinline__ void put_plain(LaneSlot &s, uint32_t v) const
    {
        if (lane < NL)
            s.p[lane] = v;
    }
    __device__ __forceinline__ void put_windows(LaneSlot &s, uint32_t v) const
    {
        if (lane < NL) {
#pragma unroll
            for (int c = 0; c < 4; c++)
                s.w[40 * c + 24 - lane + c] = v;
        }
    }
    __device__ __forceinline__ void put(LaneSlot &s, uint32_t v) const
    {
        put_windows(s, v);
        put_plain(s, v);
    }
    __device__ __forceinline__ uint32_t own(const LaneSlot &s) const { return lane < NL ? s.p[lane] : 0u; }
    // the same from an element stored as windows only
    __device__ __forceinline__ uint32_t own_w(const LaneSlot &s) const { return lane < NL ? s.w[24 - lane] : 0u; }

    // eight 32-bit limbs (any value below 2^256) -> this lane's limb
    __device__ __forceinline__ static uint32_t from_fe(const Fe &a, int lane)
    {
        uint32_t v = 0;
#pragma unroll
        for (int l = 0; l < 10; l++) {
            const int bit = 26 * l, w = bit >> 5, off = bit & 31;
            uint64_t x = a.w[w];
            if (w + 1 < 8)
                x |= (uint64_t)a.w[w + 1] << 32;
            const uint32_t limb = (uint32_t)((x >> off) & LN_M26);
            v = lane == l ? limb : v;
        }
        return v;
    }

    // -> eight 32-bit limbs, weakly reduced (below 2^256), the same on every lane
    __device__ __forceinline__ static Fe to_fe(uint32_t v)
    {
        // every lane gathers the limbs, then carries exactly in registers; the
        // last limb keeps its excess
        uint32_t L[NL];
#pragma unroll
        for (int l = 0; l < NL; l++)
            L[l] = __shfl_sync(LN_ALL, v, l);
#pragma unroll
        for (int l = 0; l < NL - 1; l++) {
            L[l + 1] += L[l] >> 26;
            L[l] &= (uint32_t)LN_M26;
        }
        uint32_t t[16];
#pragma unroll
        for (int i = 0; i < 16; i++)
            t[i] = 0;
#pragma unroll
        for (int l = 0; l < NL; l++) {
            const int bit = 26 * l, w = bit >> 5, off = bit & 31;
            const uint64_t x = (uint64_t)L[l] << off;
            t[w] |= (uint32_t)x;
            t[w + 1] |= (uint32_t)(x >> 32);
        }
        return F::reduce_wide(t);
    }
};

// The running total and the temporaries of a step.  X and M (= 3 (X^2 - ZZ^2), of the
// current total) are double-buffered: a step writes one while others still read.
enum LaneSlotId : int {
    LX0, LX1, LY, LZZ, LZZZ, LM0, LM1,      // running total
    LV, LW, LD,                             // doubling
    LP, LR, LU1, LS1, LPP, LRR, LZ12, LZZZ12, LPPP, LQ,  // addition
    LNSLOTS
};
constexpr int LN_MAX_WINDOWS = 65;  // ceil(257 / 4)

// The chain on one block of four warps, one per scheduler; a step puts its
// independent sums of products on different warps.
template <class C>
struct LaneHorner {
    using F = typename C::F;
    using LF = LaneField<F>;
    LaneSlot *sl;
    LF f;
    int warp;
    int x = 0, m = 0;  // current buffers of X and M

    __device__ __forceinline__ LaneHorner(LaneSlot *slots, int lane, int warp_) : sl(slots), f(lane), warp(warp_) {}

    // M of the current total (by warp 2, which also computes it in a doubling's last step)
    __device__ __forceinline__ void set_m(int xb, int mb)
    {
        const LaneSlot &X = sl[LX0 + xb];
        f.put(sl[LM0 + mb], f.template norm<3>(f.cols(X, X) + f.k - f.cols(sl[LZZ], sl[LZZ])));
    }

    // total = 2 total (not the identity).  dbl-2008-s-1, a = -3, with V = 4 Y^2:
    //   W = 2Y V,  X' = M^2 - 2 X V,  D = S - X' = 3 X V - M^2,  ZZ' = V ZZ,
    //   Y' = M D - W Y,  ZZZ' = W ZZZ,  M' = 3 (X'^2 - ZZ'^2).
    // Two block barriers: V follows Y' on the same warp.
    __device__ __forceinline__ void dbl()
    {
        if (warp == 0)
            f.put_plain(sl[LV], f.norm(f.cols(sl[LY], sl[LY]) << 2));
        __syncthreads();
        const LaneSlot &X = sl[LX0 + x], &M = sl[LM0 + m];
        if (warp == 0) {
            f.put_plain(sl[LW], f.norm(f.cols(sl[LV], sl[LY]) << 1));
        } else if (warp == 1) {
            f.put(sl[LX0 + (x ^ 1)], f.norm(f.cols(M, M) + f.k2 - 2 * f.cols(sl[LV], X)));
        } else if (warp == 2) {
            f.put_windows(sl[LD], f.norm(3 * f.cols(sl[LV], X) + f.k - f.cols(M, M)));
        } else {
            f.put(sl[LZZ], f.norm(f.cols(sl[LV], sl[LZZ])));
        }
        __syncthreads();
        if (warp == 0) {
            const uint32_t y = f.norm(f.cols(M, sl[LD]) + f.k - f.cols(sl[LW], sl[LY]));
            __syncwarp();
            f.put(sl[LY], y);
            __syncwarp();
        } else if (warp == 1) {
            const uint32_t z = f.norm(f.cols(sl[LW], sl[LZZZ]));
            __syncwarp();
            f.put_windows(sl[LZZZ], z);
        } else if (warp == 2) {
            set_m(x ^ 1, m ^ 1);
        }
        x ^= 1;
        m ^= 1;
    }

    // an element (limbs in s) that may be zero: its bits from 234 up are within 3
    // below a multiple of 2^21 (a multiple of the modulus is j 2^255 less at most
    // 2^159), true for 4 in 2^21 of all others
    __device__ __forceinline__ static bool maybe_zero(const LaneSlot &s) { return ((s.p[9] + 3u) & 0x1fffffu) <= 3u; }

    // total += the addend (coordinates X, Y, ZZ, ZZZ at ad, twelve words each; neither
    // is the identity): 0 done, 1 the operands are equal (the caller doubles), 2 they
    // cancel.  add-2008-s.
    __device__ __forceinline__ int add(const uint32_t *__restrict__ ad)
    {
        const uint32_t *X2 = ad, *Y2 = ad + 12, *ZZ2 = ad + 24, *ZZZ2 = ad + 36;
        const LaneSlot &X = sl[LX0 + x];
        __syncthreads();
        if (warp == 0)
            f.put(sl[LP], f.norm(f.cols(X2, sl[LZZ]) + f.k - f.cols(ZZ2, X)));
        else if (warp == 1)
            f.put(sl[LR], f.norm(f.cols(Y2, sl[LZZZ]) + f.k - f.cols(ZZZ2, sl[LY])));
        else if (warp == 2)
            f.put_windows(sl[LU1], f.norm(f.cols(ZZ2, X)));
        else
            f.put_windows(sl[LS1], f.norm(f.cols(ZZZ2, sl[LY])));
        __syncthreads();
        if (maybe_zero(sl[LP])) {  // the same on every thread of the block
            if (F::is_zero(LF::to_fe(f.own(sl[LP]))))
                return F::is_zero(LF::to_fe(f.own(sl[LR]))) ? 1 : 2;
        }
        if (warp == 0)
            f.put_plain(sl[LPP], f.norm(f.cols(sl[LP], sl[LP])));
        else if (warp == 1)
            f.put_plain(sl[LRR], f.norm(f.cols(sl[LR], sl[LR])));
        else if (warp == 2)
            f.put_windows(sl[LZ12], f.norm(f.cols(ZZ2, sl[LZZ])));
        else
            f.put_windows(sl[LZZZ12], f.norm(f.cols(ZZZ2, sl[LZZZ])));
        __syncthreads();
        if (warp == 0)
            f.put_plain(sl[LPPP], f.norm(f.cols(sl[LPP], sl[LP])));
        else if (warp == 1)
            f.put_plain(sl[LQ], f.norm(f.cols(sl[LPP], sl[LU1])));
        else if (warp == 2)
            f.put(sl[LZZ], f.norm(f.cols(sl[LPP], sl[LZ12])));
        __syncthreads();
        if (warp == 0) {  // Y' = R (3Q + PPP - RR) - S1 PPP
            const uint64_t pos = 3 * f.cols(sl[LQ], sl[LR]) + f.cols(sl[LPPP], sl[LR]);
            const uint64_t neg = f.cols(sl[LRR], sl[LR]) + f.cols(sl[LPPP], sl[LS1]);
            f.put(sl[LY], f.norm(pos + f.k2 - neg));
        } else if (warp == 1) {  // X' = RR - PPP - 2Q
            const uint64_t c = (uint64_t)f.own(sl[LRR]) + f.k - f.own(sl[LPPP]) - 2 * (uint64_t)f.own(sl[LQ]);
            f.put(sl[LX0 + (x ^ 1)], f.norm(c));
        } else if (warp == 2) {
            f.put_windows(sl[LZZZ], f.norm(f.cols(sl[LPPP], sl[LZZZ12])));
        }
        __syncthreads();
        x ^= 1;
        if (warp == 2)
            set_m(x, m);
        return 0;
    }

    // total = the addend
    __device__ __forceinline__ void take(const uint32_t *__restrict__ ad)
    {
        __syncthreads();
        const uint32_t v = f.lane < 12 ? ad[12 * warp + f.lane] : 0u;
        f.put(sl[warp == 0 ? LX0 + x : warp == 1 ? LY : warp == 2 ? LZZ : LZZZ], v);
        __syncthreads();
        if (warp == 2)
            set_m(x, m);
    }
};

}  // namespace hs
