// hs_quad.cuh -- point operations on four lanes, for the latency-bound kernels.
//
// A point lies across a quad of lanes: lane j of the quad holds coordinate j
// (X, Y, ZZ, ZZZ).  An XYZZ addition is 14 products that form four dependent
// stages of 4, 4, 4 and 3, a doubling three of 2, 4 and 3, so a quad computes
// one product per lane and stage and exchanges operands by shuffles: four
// product latencies instead of fourteen, at 16 product slots instead of 14.
// One lone warp per scheduler on GB300 takes 517 (F_p) / 712 (F_q) clocks per
// product, so an addition takes about 1.2 / 1.6 us against 3.5 / 5.3 us on one
// thread.  Every function is called by all 32 lanes of a warp (eight quads),
// branches on warp votes only, and is complete: identity operands and equal or
// opposite points are handled, and where no quad of the warp has two points to add
// (or one to double) nothing is computed: small scalars leave most buckets empty, and
// one F_p MSM of 65536 points with scalars 0 and 1 took 346 us, 96 of them in level 2
// on identities (305 with one thread per point, which leaves early), and 271 so.
// The two operations are out of line, the points
// passed by value in registers: a kernel's many uses then share one body, which
// stays in the instruction cache.  Level 2 of one MSM of 2^20 points (F_p / F_q):
// 184 / 287 us with one thread per point, 160 / 217 with inlined quads, 139 / 177
// as here; the reduction of 33 windows of 128 buckets: 84 / 104 us on eight-lane
// groups, 43 / 52 here.
#pragma once
#include "hs_curve.cuh"

namespace hs {

template <class C>
struct Quad {
    using F = typename C::F;
    static constexpr unsigned ALL = 0xffffffffu;
    int j;  // lane within the quad: the coordinate it holds

    __device__ __forceinline__ explicit Quad(uint32_t thread) : j((int)(thread & 3u)) {}

    __device__ __forceinline__ static Fe shx(const Fe &a, int x)
    {
        Fe r;
#pragma unroll
        for (int k = 0; k < 8; k++)
            r.w[k] = __shfl_xor_sync(ALL, a.w[k], x);
        return r;
    }
    __device__ __forceinline__ static Fe bcast(const Fe &a, int src)
    {
        Fe r;
#pragma unroll
        for (int k = 0; k < 8; k++)
            r.w[k] = __shfl_sync(ALL, a.w[k], src, 4);
        return r;
    }
    __device__ __forceinline__ static Fe sel(bool c, const Fe &a, const Fe &b)
    {
        Fe r;
#pragma unroll
        for (int k = 0; k < 8; k++)
            r.w[k] = c ? a.w[k] : b.w[k];
        return r;
    }
    __device__ __forceinline__ static bool flag(bool f, int src) { return __shfl_sync(ALL, (int)f, src, 4) != 0; }
    // the quad's point is the identity (ZZ exactly zero)
    __device__ __forceinline__ static bool is_inf(const Fe &p) { return flag(F::is_exact_zero(p), 2); }

    __device__ __forceinline__ static Fe load(const uint4 *points, size_t i, int j)
    {
        const uint4 a = points[8 * i + 2 * j], b = points[8 * i + 2 * j + 1];
        return Fe{{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w}};
    }
    __device__ __forceinline__ static void store(uint4 *points, size_t i, int j, const Fe &p)
    {
        points[8 * i + 2 * j] = make_uint4(p.w[0], p.w[1], p.w[2], p.w[3]);
        points[8 * i + 2 * j + 1] = make_uint4(p.w[4], p.w[5], p.w[6], p.w[7]);
    }

    // 2p (dbl-2008-s-1, a = -3).  The identity's ZZ stays exactly zero.
    __device__ __forceinline__ Fe dbl(const Fe &p) const { return dbl_v(p, j); }
    static __device__ __noinline__ Fe dbl_v(const Fe p, const int j)
    {
        // lane 0: T = (X - ZZ)(X + ZZ); lane 1: V = (2Y)^2
        const Fe o = bcast(p, 2);
        if (__all_sync(ALL, F::is_exact_zero(o)))
            return p;  // eight identities
        const Fe u = F::dbl(p);
        const Fe r1 = F::mul(sel(j == 0, F::sub(p, o), u), sel(j == 0, F::add(p, o), u));
        const Fe v = bcast(r1, 1), t = bcast(r1, 0);
        const Fe m = F::add(F::dbl(t), t);  // M = 3 (X^2 - ZZ^2)
        // S = X V, W = 2Y V, ZZ' = ZZ V, M^2
        const Fe r2 = F::mul(sel(j == 3, m, sel(j == 1, u, p)), sel(j == 3, m, v));
        const Fe mm = bcast(r2, 3), w = bcast(r2, 1);
        const Fe x3 = F::sub(mm, F::dbl(r2));  // lane 0
        // lane 0: M (S - X'); lane 1: W Y; lane 3: W ZZZ
        const Fe r3 = F::mul(sel(j == 0, m, w), sel(j == 0, F::sub(r2, x3), p));
        const Fe e = bcast(r3, 0);
        Fe r = sel(j == 0, x3, sel(j == 1, F::sub(e, r3), sel(j == 2, r2, r3)));
        // y = 0: no such point on a prime-order curve, kept complete
        if (j == 2 && F::is_zero(r))
            r = F::zero();
        return r;
    }

    // p + q (add-2008-s), or with MIXED p + (x, y) for an affine q that is not the
    // identity (madd-2008-s; lane 0 holds x, lane 1 y).  Where `take` is false
    // (quad-uniform) the result is p.
    template <bool MIXED>
    __device__ __forceinline__ Fe add(const Fe &p, const Fe &q, bool take) const
    {
        return add_v<MIXED>(p, q, take, j);
    }
    template <bool MIXED>
    static __device__ __noinline__ Fe add_v(const Fe p, const Fe q, const bool take, const int j)
    {
        // (flags are shuffles: taken on every lane, never behind a short-circuit)
        const bool p_inf = is_inf(p), q_zero = is_inf(q);
        const bool q_inf = !take || (!MIXED && q_zero);
        const Fe qv = MIXED ? sel(j < 2, q, F::one()) : q;
        if (__all_sync(ALL, p_inf || q_inf))  // no quad has two points to add
            return q_inf ? p : qv;
        // U1 = X1 ZZ2, S1 = Y1 ZZZ2, U2 = X2 ZZ1, S2 = Y2 ZZZ1 on lanes 0..3 (MIXED: U1 = X1, S1 = Y1)
        Fe r1 = F::mul(p, shx(q, 2));
        if (MIXED)
            r1 = sel(j < 2, p, r1);
        const Fe d = F::sub(shx(r1, 2), r1);  // lane 0: P = U2 - U1, lane 1: R = S2 - S1
        const Fe x1 = shx(r1, 1);             // lane 0: S1, lane 1: U1
        const bool zero_d = F::is_zero(d);
        const bool zero_p = flag(zero_d, 0);
        const bool same_x = zero_p && !p_inf && !q_inf;
        // PP, RR, ZZ1 ZZ2, ZZZ1 ZZZ2 (MIXED: ZZ1, ZZZ1)
        Fe r2 = F::mul(sel(j < 2, d, p), sel(j < 2, d, q));
        if (MIXED)
            r2 = sel(j < 2, r2, p);
        const Fe pp = bcast(r2, 0);
        // PPP = P PP, Q = U1 PP, ZZ' = ZZ12 PP, ZZZ12 PP
        const Fe r3 = F::mul(sel(j == 0, d, sel(j == 1, x1, r2)), pp);
        const Fe x3r = shx(r3, 1);  // lane 1: PPP
        const Fe x3 = F::sub(F::sub(r2, x3r), F::dbl(r3));  // lane 1: X' = RR - PPP - 2Q
        // lane 0: S1 PPP; lane 1: R (Q - X'); lane 3: ZZZ12 PP P
        const Fe pd = bcast(d, 0);
        const Fe r4 = F::mul(sel(j == 0, x1, sel(j == 1, d, r3)), sel(j == 0, r3, sel(j == 1, F::sub(r3, x3), pd)));
        const Fe ex = shx(sel(j == 1, x3, r4), 1);  // lane 0: X', lane 1: S1 PPP
        Fe r = sel(j == 0, ex, sel(j == 1, F::sub(r4, ex), sel(j == 2, r3, r4)));
        if (__any_sync(ALL, same_x)) {  // equal (double) or opposite (identity) points
            const bool same_y = flag(zero_d, 1);
            Fe z = p;
            if (MIXED)  // double the affine point
                z = sel(j < 2, q, F::one());
            const Fe two = dbl_v(z, j);
            r = same_x ? sel(same_y, two, F::zero()) : r;
        }
        return q_inf ? p : sel(p_inf, qv, r);
    }
};

}  // namespace hs
