// hs_curve.cuh -- Helios / Selene group law on the device.
//
// Both curves are y^2 = x^3 - 3x + b (helios/include/helios_constants.h:36-41 over
// F_p, selene/include/selene_constants.h:36-41 over F_q).  The reference adds in
// Jacobian coordinates (add-2007-bl, dbl-2001-b, helios/src/x64/helios_add.cpp:52-107,
// helios_dbl.cpp:45-88) behind an edge-case wrapper (helios_msm_vartime.cpp:59-104).
//
// Bucket arithmetic here uses extended Jacobian "XYZZ" coordinates
// (x = X/ZZ, y = Y/ZZZ, ZZ^3 = ZZZ^2): mixed addition of an affine base costs
// 8M+2S instead of 7M+4S, and the doubling / inverse cases are detected from
// the same intermediate values.  The identity is ZZ = 0 exactly (a non-identity
// point never has ZZ congruent to 0, and the identity is only ever produced by
// an explicit store of zeros).

#pragma once
#include "hs_field.cuh"

namespace hs {

struct HeliosCurve {
    using F = Fp;
    static constexpr int ID = 0;
    // b = 15789920373731020205926570676277057129217619222203920395806844808978996083412
    __device__ __forceinline__ static Fe b()
    {
        return Fe{{0xedd73ad4u, 0x22b49ee1u, 0x4113bf35u, 0x043f6f38u, 0x3ebb7b3bu, 0xbe94a76bu, 0xb0ea70b8u,
                   0x22e8c739u}};
    }
    static constexpr int SSWU_Z = 7;  // helios/src/x64/helios_map_to_curve.cpp:54
};

struct SeleneCurve {
    using F = Fq;
    static constexpr int ID = 1;
    // b = 50691664119640283727448954162351551669994268339720539671652090628799494505816
    __device__ __forceinline__ static Fe b()
    {
        return Fe{{0xcb5a4558u, 0x68de0983u, 0x06ae900eu, 0xf3944bdfu, 0x95ffe279u, 0x7f51bba5u, 0x695876c1u,
                   0x70127713u}};
    }
    static constexpr int SSWU_Z = -4;  // selene/src/x64/selene_map_to_curve.cpp
};

struct Xyzz {
    Fe X, Y, ZZ, ZZZ;
};

template <class C>
struct Group {
    using F = typename C::F;

    __device__ __forceinline__ static Fe b() { return C::b(); }

    __device__ __forceinline__ static Xyzz inf()
    {
        Xyzz r;
        r.X = F::zero();
        r.Y = F::zero();
        r.ZZ = F::zero();
        r.ZZZ = F::zero();
        return r;
    }

    __device__ __forceinline__ static bool is_inf(const Xyzz &p) { return F::is_exact_zero(p.ZZ); }

    __device__ __forceinline__ static Xyzz from_affine(const Fe &x, const Fe &y)
    {
        Xyzz r;
        r.X = x;
        r.Y = y;
        r.ZZ = F::one();
        r.ZZZ = F::one();
        return r;
    }

    // dbl-2008-s-1 for a = -3: M = 3(X - ZZ)(X + ZZ).  7M + 2S.
    __device__ static Xyzz dbl(const Xyzz &p)
    {
        if (is_inf(p))
            return p;
        Fe U = F::dbl(p.Y);
        Fe V = F::sqr(U);
        Fe W = F::mul(U, V);
        Fe S = F::mul(p.X, V);
        Fe t0 = F::sub(p.X, p.ZZ);
        Fe t1 = F::add(p.X, p.ZZ);
        Fe M = F::mul(t0, t1);
        M = F::add(F::dbl(M), M);
        Xyzz r;
        r.X = F::sub(F::sqr(M), F::dbl(S));
        r.Y = F::sub(F::mul(M, F::sub(S, r.X)), F::mul(W, p.Y));
        r.ZZ = F::mul(V, p.ZZ);
        r.ZZZ = F::mul(W, p.ZZZ);
        if (F::is_zero(r.ZZ))  // y == 0 (no such point on a prime-order curve; kept complete)
            return inf();
        return r;
    }

    // mdbl-2008-s-1: doubling of an affine point, M = 3x^2 - 3.
    __device__ static Xyzz dbl_affine(const Fe &x, const Fe &y)
    {
        Fe U = F::dbl(y);
        Fe V = F::sqr(U);
        Fe W = F::mul(U, V);
        Fe S = F::mul(x, V);
        Fe M = F::sub(F::sqr(x), F::one());
        M = F::add(F::dbl(M), M);
        Xyzz r;
        r.X = F::sub(F::sqr(M), F::dbl(S));
        r.Y = F::mul_sub(M, F::sub(S, r.X), W, y);
        r.ZZ = V;
        r.ZZZ = W;
        if (F::is_zero(r.ZZ))
            return inf();
        return r;
    }

    // acc += (x2, y2), the affine point never being the identity.  madd-2008-s.
    __device__ __forceinline__ static void add_affine(Xyzz &acc, const Fe &x2, const Fe &y2)
    {
        if (is_inf(acc)) {
            acc = from_affine(x2, y2);
            return;
        }
        Fe U2 = F::mul(x2, acc.ZZ);
        Fe S2 = F::mul(y2, acc.ZZZ);
        Fe P = F::sub(U2, acc.X);
        Fe R = F::sub(S2, acc.Y);
        if (F::is_zero(P)) {
            if (F::is_zero(R))
                acc = dbl_affine(x2, y2);  // same point: double
            else
                acc = inf();  // opposite points
            return;
        }
        Fe PP = F::sqr(P);
        Fe PPP = F::mul(P, PP);
        Fe Q = F::mul(acc.X, PP);
        Fe X3 = F::sub(F::sub(F::sqr(R), PPP), F::dbl(Q));
        Fe Y3 = F::mul_sub(R, F::sub(Q, X3), acc.Y, PPP);
        acc.ZZ = F::mul(acc.ZZ, PP);
        acc.ZZZ = F::mul(acc.ZZZ, PPP);
        acc.X = X3;
        acc.Y = Y3;
    }

    // p + q, complete.  add-2008-s: 12M + 2S.
    __device__ static Xyzz add(const Xyzz &p, const Xyzz &q)
    {
        if (is_inf(p))
            return q;
        if (is_inf(q))
            return p;
        Fe U1 = F::mul(p.X, q.ZZ);
        Fe U2 = F::mul(q.X, p.ZZ);
        Fe S1 = F::mul(p.Y, q.ZZZ);
        Fe S2 = F::mul(q.Y, p.ZZZ);
        Fe P = F::sub(U2, U1);
        Fe R = F::sub(S2, S1);
        if (F::is_zero(P)) {
            if (F::is_zero(R))
                return dbl(p);
            return inf();
        }
        Fe PP = F::sqr(P);
        Fe PPP = F::mul(P, PP);
        Fe Q = F::mul(U1, PP);
        Xyzz r;
        r.X = F::sub(F::sub(F::sqr(R), PPP), F::dbl(Q));
        r.Y = F::sub(F::mul(R, F::sub(Q, r.X)), F::mul(S1, PPP));
        r.ZZ = F::mul(F::mul(p.ZZ, q.ZZ), PP);
        r.ZZZ = F::mul(F::mul(p.ZZZ, q.ZZZ), PPP);
        return r;
    }

    // r = p + q for operands that are not the identity; 1 when they are equal and 2
    // when they are opposite (r is then unset).  The operands are dead after the first
    // six products, so a caller that can get q again keeps fewer registers than with
    // add().
    __device__ __forceinline__ static int add_lean(Xyzz &r, const Xyzz &p, const Xyzz &q)
    {
        const Fe U1 = F::mul(p.X, q.ZZ);
        const Fe P = F::sub(F::mul(q.X, p.ZZ), U1);
        const Fe S1 = F::mul(p.Y, q.ZZZ);
        const Fe R = F::sub(F::mul(q.Y, p.ZZZ), S1);
        const Fe zz = F::mul(p.ZZ, q.ZZ), zzz = F::mul(p.ZZZ, q.ZZZ);
        if (F::is_zero(P))
            return F::is_zero(R) ? 1 : 2;
        const Fe PP = F::sqr(P);
        const Fe Q = F::mul(U1, PP);
        const Fe PPP = F::mul(P, PP);
        r.ZZ = F::mul(zz, PP);
        r.ZZZ = F::mul(zzz, PPP);
        r.X = F::sub(F::sub(F::sqr(R), PPP), F::dbl(Q));
        r.Y = F::sub(F::mul(R, F::sub(Q, r.X)), F::mul(S1, PPP));
        return 0;
    }

    // ---- Jacobian points (x = X/Z^2, y = Y/Z^3; the identity is Z exactly zero), for
    // chains of doublings: dbl-2001-b is 3M + 5S against XYZZ's 7M + 2S ----
    struct Jac {
        Fe X, Y, Z;
    };
    // an addend with the powers of its Z that an addition needs
    struct JacEntry {
        Fe X, Y, Z, ZZ, ZZZ;
    };
    __device__ __forceinline__ static bool is_inf(const Jac &p) { return F::is_exact_zero(p.Z); }
    __device__ __forceinline__ static Jac jac_inf() { return Jac{F::one(), F::one(), F::zero()}; }

    // 2p, a = -3 (the identity's Z stays exactly zero)
    __device__ __forceinline__ static Jac dbl(const Jac &p)
    {
        const Fe delta = F::sqr(p.Z), gamma = F::sqr(p.Y);
        const Fe t = F::mul(F::sub(p.X, delta), F::add(p.X, delta));
        const Fe alpha = F::add(F::dbl(t), t);
        Jac r;
        r.Z = F::sub(F::sub(F::sqr(F::add(p.Y, p.Z)), gamma), delta);
        const Fe g2 = F::dbl(gamma);
        const Fe b4 = F::dbl(F::mul(p.X, g2));  // 4 X gamma
        r.X = F::sub(F::sqr(alpha), F::dbl(b4));
        r.Y = F::sub(F::mul(alpha, F::sub(b4, r.X)), F::dbl(F::sqr(g2)));
        if (F::is_zero(r.Z))  // y = 0: no such point on a prime-order curve, kept complete
            r.Z = F::zero();
        return r;
    }

    // p + (q, or -q), complete
    __device__ __forceinline__ static Jac add(const Jac &p, const JacEntry &q, bool negate)
    {
        const Fe y2 = negate ? F::neg(q.Y) : q.Y;
        if (F::is_exact_zero(q.ZZ))
            return p;
        if (is_inf(p))
            return Jac{q.X, y2, q.Z};
        const Fe z1z1 = F::sqr(p.Z);
        const Fe U1 = F::mul(p.X, q.ZZ), S1 = F::mul(p.Y, q.ZZZ);
        const Fe H = F::sub(F::mul(q.X, z1z1), U1);
        const Fe R = F::sub(F::mul(y2, F::mul(p.Z, z1z1)), S1);
        if (F::is_zero(H))
            return F::is_zero(R) ? dbl(p) : jac_inf();
        const Fe HH = F::sqr(H), HHH = F::mul(H, HH), V = F::mul(U1, HH);
        Jac r;
        r.Z = F::mul(F::mul(p.Z, q.Z), H);
        r.X = F::sub(F::sub(F::sqr(R), HHH), F::dbl(V));
        r.Y = F::mul_sub(R, F::sub(V, r.X), S1, HHH);
        return r;
    }

    // XYZZ -> Jacobian without inversion: Z = ZZ*ZZZ, X = X*ZZ*ZZZ^2, Y = Y*ZZ^3*ZZZ^2.
    // Identity -> (1:1:0), the reference's encoding (helios/include/helios_ops.h:45-50).
    __device__ static void to_jacobian(Fe &X, Fe &Y, Fe &Z, const Xyzz &p)
    {
        if (is_inf(p)) {
            X = F::one();
            Y = F::one();
            Z = F::zero();
            return;
        }
        Fe zzz2 = F::sqr(p.ZZZ);
        Fe zz2 = F::sqr(p.ZZ);
        Z = F::mul(p.ZZ, p.ZZZ);
        X = F::mul(F::mul(p.X, p.ZZ), zzz2);
        Y = F::mul(F::mul(p.Y, F::mul(zz2, p.ZZ)), zzz2);
    }
};

}  // namespace hs
