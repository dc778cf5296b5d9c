// hs_field.cuh -- F_p and F_q arithmetic for sm_103a on the integer-multiply pipe.
//
//   F_p, p = 2^255 - 19      (Helios coordinates)   2^256 == 38       (mod p)
//   F_q, q = 2^255 - gamma   (Selene coordinates)   2^256 == 2*gamma  (mod q)
//
// The reference keeps radix-2^51 limbs and folds by 19 / gamma
// (fp/include/x64/fp51_inline.h:46-243, fq/include/x64/fq51_inline.h:1087-1225,
// constants fq/include/x64/fq51.h:38-86).  Here an element is eight 32-bit
// limbs (little endian) holding any value in [0, 2^256) congruent to it
// ("weakly reduced"); the canonical value < m is produced only at the edges.
// Products are 8x8 schoolbook rows of multiply-add carry chains, followed by a
// fold of the high half by c = 2^256 mod m.

#pragma once
#include <cstdint>

namespace hs {

struct Fe {
    uint32_t w[8];
};

// ---------------------------------------------------------------------------
// field parameter sets
// ---------------------------------------------------------------------------
struct FpParams {
    // p = 2^255 - 19
    static constexpr uint32_t M[8] = {0xffffffedu, 0xffffffffu, 0xffffffffu, 0xffffffffu,
                                      0xffffffffu, 0xffffffffu, 0xffffffffu, 0x7fffffffu};
    // c = 2^256 mod p = 38 (one limb)
    static constexpr int NC = 1;
    static constexpr uint32_t C[4] = {38u, 0u, 0u, 0u};
};

struct FqParams {
    // q = 2^255 - gamma, gamma = 85737960593035654572250192257530476641
    static constexpr uint32_t M[8] = {0x7927c79fu, 0x6eb6d272u, 0xb7656b58u, 0xbf7f782cu,
                                      0xffffffffu, 0xffffffffu, 0xffffffffu, 0x7fffffffu};
    // c = 2^256 mod q = 2*gamma (four limbs)
    static constexpr int NC = 4;
    static constexpr uint32_t C[4] = {0x0db070c2u, 0x22925b1bu, 0x9135294fu, 0x81010fa6u};
};

// ---------------------------------------------------------------------------
// raw 256-bit helpers
// ---------------------------------------------------------------------------
// A 32 x 32 -> 64 product with accumulation is one multiply-add whose 64-bit
// addend is an aligned register pair, and costs about 4 issue cycles of a
// scheduler against about 1.9 for an add with carry; the two do not overlap, so
// a product's time is close to 4 x products + 1.9 x adds.  Products are therefore
// kept in two accumulators whose pairs are aligned: e[k] holds word k (products
// a_i b_j with i + j even), o[k] word k + 1 (i + j odd); with one array, the
// odd products fall on unaligned pairs and cost more.  Measured on GB300, four
// warps per scheduler, clocks per SM and product, one array -> two arrays with
// the folds below: F_p multiplication 3.01 -> 2.64 and square 2.03 -> 1.88,
// F_q 4.56 -> 3.80 and 3.68 -> 2.96.  (Karatsuba on 4 x 4 halves saves 16
// products for about 70 adds: 2.84.  Limbs of 29 bits in 64-bit columns: 3.64.)

// Every output of these statements is early-clobbered (&): a statement is many
// instructions, and without it an output may share the register of an input of the
// same value -- a zero accumulator and a zero operand, as in the square of the
// constant one, which then came out as 39.

// acc[0..2N-1] += sum_k a[2k] b 2^(64k), k < N; with CARRY, acc[2N] = the carry out
// (without, the caller's bound says there is none)
template <int N, bool CARRY>
__device__ __forceinline__ void mad_chain(uint32_t *acc, const uint32_t *a, uint32_t b)
{
    if (N == 4 && CARRY)
        asm("{\n\t"
            "mad.lo.cc.u32  %0, %9, %13, %0;\n\t"
            "madc.hi.cc.u32 %1, %9, %13, %1;\n\t"
            "madc.lo.cc.u32 %2, %10, %13, %2;\n\t"
            "madc.hi.cc.u32 %3, %10, %13, %3;\n\t"
            "madc.lo.cc.u32 %4, %11, %13, %4;\n\t"
            "madc.hi.cc.u32 %5, %11, %13, %5;\n\t"
            "madc.lo.cc.u32 %6, %12, %13, %6;\n\t"
            "madc.hi.cc.u32 %7, %12, %13, %7;\n\t"
            "addc.u32       %8, 0, 0;\n\t"
            "}"
            : "+&r"(acc[0]), "+&r"(acc[1]), "+&r"(acc[2]), "+&r"(acc[3]), "+&r"(acc[4]), "+&r"(acc[5]), "+&r"(acc[6]),
              "+&r"(acc[7]), "=&r"(acc[8])
            : "r"(a[0]), "r"(a[2]), "r"(a[4]), "r"(a[6]), "r"(b));
    else if (N == 4)
        asm("{\n\t"
            "mad.lo.cc.u32  %0, %8, %12, %0;\n\t"
            "madc.hi.cc.u32 %1, %8, %12, %1;\n\t"
            "madc.lo.cc.u32 %2, %9, %12, %2;\n\t"
            "madc.hi.cc.u32 %3, %9, %12, %3;\n\t"
            "madc.lo.cc.u32 %4, %10, %12, %4;\n\t"
            "madc.hi.cc.u32 %5, %10, %12, %5;\n\t"
            "madc.lo.cc.u32 %6, %11, %12, %6;\n\t"
            "madc.hi.u32    %7, %11, %12, %7;\n\t"
            "}"
            : "+&r"(acc[0]), "+&r"(acc[1]), "+&r"(acc[2]), "+&r"(acc[3]), "+&r"(acc[4]), "+&r"(acc[5]), "+&r"(acc[6]),
              "+&r"(acc[7])
            : "r"(a[0]), "r"(a[2]), "r"(a[4]), "r"(a[6]), "r"(b));
    else if (N == 3 && CARRY)
        asm("{\n\t"
            "mad.lo.cc.u32  %0, %7, %10, %0;\n\t"
            "madc.hi.cc.u32 %1, %7, %10, %1;\n\t"
            "madc.lo.cc.u32 %2, %8, %10, %2;\n\t"
            "madc.hi.cc.u32 %3, %8, %10, %3;\n\t"
            "madc.lo.cc.u32 %4, %9, %10, %4;\n\t"
            "madc.hi.cc.u32 %5, %9, %10, %5;\n\t"
            "addc.u32       %6, 0, 0;\n\t"
            "}"
            : "+&r"(acc[0]), "+&r"(acc[1]), "+&r"(acc[2]), "+&r"(acc[3]), "+&r"(acc[4]), "+&r"(acc[5]), "=&r"(acc[6])
            : "r"(a[0]), "r"(a[2]), "r"(a[4]), "r"(b));
    else if (N == 3)
        asm("{\n\t"
            "mad.lo.cc.u32  %0, %6, %9, %0;\n\t"
            "madc.hi.cc.u32 %1, %6, %9, %1;\n\t"
            "madc.lo.cc.u32 %2, %7, %9, %2;\n\t"
            "madc.hi.cc.u32 %3, %7, %9, %3;\n\t"
            "madc.lo.cc.u32 %4, %8, %9, %4;\n\t"
            "madc.hi.u32    %5, %8, %9, %5;\n\t"
            "}"
            : "+&r"(acc[0]), "+&r"(acc[1]), "+&r"(acc[2]), "+&r"(acc[3]), "+&r"(acc[4]), "+&r"(acc[5])
            : "r"(a[0]), "r"(a[2]), "r"(a[4]), "r"(b));
    else if (N == 2 && CARRY)
        asm("{\n\t"
            "mad.lo.cc.u32  %0, %5, %7, %0;\n\t"
            "madc.hi.cc.u32 %1, %5, %7, %1;\n\t"
            "madc.lo.cc.u32 %2, %6, %7, %2;\n\t"
            "madc.hi.cc.u32 %3, %6, %7, %3;\n\t"
            "addc.u32       %4, 0, 0;\n\t"
            "}"
            : "+&r"(acc[0]), "+&r"(acc[1]), "+&r"(acc[2]), "+&r"(acc[3]), "=&r"(acc[4])
            : "r"(a[0]), "r"(a[2]), "r"(b));
    else if (N == 2)
        asm("{\n\t"
            "mad.lo.cc.u32  %0, %4, %6, %0;\n\t"
            "madc.hi.cc.u32 %1, %4, %6, %1;\n\t"
            "madc.lo.cc.u32 %2, %5, %6, %2;\n\t"
            "madc.hi.u32    %3, %5, %6, %3;\n\t"
            "}"
            : "+&r"(acc[0]), "+&r"(acc[1]), "+&r"(acc[2]), "+&r"(acc[3])
            : "r"(a[0]), "r"(a[2]), "r"(b));
    else if (N == 1 && CARRY)
        asm("{\n\t"
            "mad.lo.cc.u32  %0, %3, %4, %0;\n\t"
            "madc.hi.cc.u32 %1, %3, %4, %1;\n\t"
            "addc.u32       %2, 0, 0;\n\t"
            "}"
            : "+&r"(acc[0]), "+&r"(acc[1]), "=&r"(acc[2])
            : "r"(a[0]), "r"(b));
    else
        asm("{\n\t"
            "mad.lo.cc.u32  %0, %2, %3, %0;\n\t"
            "madc.hi.u32    %1, %2, %3, %1;\n\t"
            "}"
            : "+&r"(acc[0]), "+&r"(acc[1])
            : "r"(a[0]), "r"(b));
}
__device__ __forceinline__ void mul_pair(uint32_t *acc, uint32_t a, uint32_t b)
{
    const uint64_t p = (uint64_t)a * b;
    acc[0] = (uint32_t)p;
    acc[1] = (uint32_t)(p >> 32);
}

// a b = sum e[k] 2^(32k) + sum o[k] 2^(32(k+1)), e[0..15], o[0..14].  Row i adds
// a b[i]; the sums of either accumulator after row i stay below 2^(32(i+9)),
// so a chain that ends on word i + 8 has no carry out, and one that ends on
// word i + 7 carries one bit into a word not yet used.
__device__ __forceinline__ void mul_eo(uint32_t e[16], uint32_t o[16], const uint32_t a[8], const uint32_t b[8])
{
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
        mul_pair(e + j, a[j], b[0]);
        mul_pair(o + j, a[j + 1], b[0]);
    }
    e[8] = 0;
#pragma unroll
    for (int i = 1; i < 8; i += 2) {
        mad_chain<4, true>(o + i - 1, a, b[i]);  // words i .. i+7, carry into i+8
        e[i + 8] = 0;
        mad_chain<4, false>(e + i + 1, a + 1, b[i]);  // words i+1 .. i+8
        if (i < 7) {
            mad_chain<4, true>(e + i + 1, a, b[i + 1]);
            o[i + 8] = 0;
            mad_chain<4, false>(o + i + 1, a + 1, b[i + 1]);
        }
    }
}

// the 28 cross products a_i a_j (i < j), in the same form: e[2..13], o[0..13]
__device__ __forceinline__ void cross_eo(uint32_t e[16], uint32_t o[16], const uint32_t a[8])
{
#pragma unroll
    for (int j = 1; j < 8; j += 2)
        mul_pair(o + j - 1, a[0], a[j]);  // words j, j+1
#pragma unroll
    for (int j = 2; j < 8; j += 2)
        mul_pair(e + j, a[0], a[j]);
    mad_chain<3, true>(o + 2, a + 2, a[1]);  // words 3..8, carry 9
    e[8] = e[9] = 0;
    mad_chain<3, false>(e + 4, a + 3, a[1]);  // words 4..9
    o[9] = 0;
    mad_chain<3, false>(o + 4, a + 3, a[2]);  // words 5..10
    mad_chain<2, true>(e + 6, a + 4, a[2]);   // words 6..9, carry 10
    mad_chain<2, true>(o + 6, a + 4, a[3]);   // words 7..10, carry 11
    e[11] = 0;
    mad_chain<2, false>(e + 8, a + 5, a[3]);  // words 8..11
    o[11] = 0;
    mad_chain<2, false>(o + 8, a + 5, a[4]);  // words 9..12
    mad_chain<1, true>(e + 10, a + 6, a[4]);  // words 10, 11, carry 12
    mad_chain<1, true>(o + 10, a + 6, a[5]);  // words 11, 12, carry 13
    e[13] = 0;
    mad_chain<1, false>(e + 12, a + 7, a[5]);  // words 12, 13
    o[13] = 0;
    mad_chain<1, false>(o + 12, a + 7, a[6]);  // words 13, 14
}

// r = x + y over eight words; returns the carry out
__device__ __forceinline__ uint32_t add8(uint32_t *r, const uint32_t *x, const uint32_t *y)
{
    uint32_t c;
    asm("add.cc.u32  %0, %9, %17;\n\taddc.cc.u32 %1, %10, %18;\n\taddc.cc.u32 %2, %11, %19;\n\taddc.cc.u32 %3, %12, %20;\n\t"
        "addc.cc.u32 %4, %13, %21;\n\taddc.cc.u32 %5, %14, %22;\n\taddc.cc.u32 %6, %15, %23;\n\taddc.cc.u32 %7, %16, %24;\n\t"
        "addc.u32 %8, 0, 0;"
        : "=&r"(r[0]), "=&r"(r[1]), "=&r"(r[2]), "=&r"(r[3]), "=&r"(r[4]), "=&r"(r[5]), "=&r"(r[6]), "=&r"(r[7]), "=&r"(c)
        : "r"(x[0]), "r"(x[1]), "r"(x[2]), "r"(x[3]), "r"(x[4]), "r"(x[5]), "r"(x[6]), "r"(x[7]), "r"(y[0]), "r"(y[1]),
          "r"(y[2]), "r"(y[3]), "r"(y[4]), "r"(y[5]), "r"(y[6]), "r"(y[7]));
    return c;
}

// r = x - y over eight words, less 1 when bw is not 0; returns the borrow out (0 or 0xffffffff)
__device__ __forceinline__ uint32_t sub8(uint32_t *r, const uint32_t *x, const uint32_t *y, uint32_t bw)
{
    uint32_t m = bw;
    asm("sub.cc.u32 %8, 0, %8;\n\t"
        "subc.cc.u32 %0, %9, %17;\n\tsubc.cc.u32 %1, %10, %18;\n\tsubc.cc.u32 %2, %11, %19;\n\tsubc.cc.u32 %3, %12, %20;\n\t"
        "subc.cc.u32 %4, %13, %21;\n\tsubc.cc.u32 %5, %14, %22;\n\tsubc.cc.u32 %6, %15, %23;\n\tsubc.cc.u32 %7, %16, %24;\n\t"
        "subc.u32 %8, 0, 0;"
        : "=&r"(r[0]), "=&r"(r[1]), "=&r"(r[2]), "=&r"(r[3]), "=&r"(r[4]), "=&r"(r[5]), "=&r"(r[6]), "=&r"(r[7]), "+&r"(m)
        : "r"(x[0]), "r"(x[1]), "r"(x[2]), "r"(x[3]), "r"(x[4]), "r"(x[5]), "r"(x[6]), "r"(x[7]), "r"(y[0]), "r"(y[1]),
          "r"(y[2]), "r"(y[3]), "r"(y[4]), "r"(y[5]), "r"(y[6]), "r"(y[7]));
    return m;
}

// t[0..14] += o[0..14] (no carry out by the caller's bound)
__device__ __forceinline__ void merge15(uint32_t *t, const uint32_t *o)
{
    asm("add.cc.u32  %0, %0, %15;\n\t"
        "addc.cc.u32 %1, %1, %16;\n\t"
        "addc.cc.u32 %2, %2, %17;\n\t"
        "addc.cc.u32 %3, %3, %18;\n\t"
        "addc.cc.u32 %4, %4, %19;\n\t"
        "addc.cc.u32 %5, %5, %20;\n\t"
        "addc.cc.u32 %6, %6, %21;\n\t"
        "addc.cc.u32 %7, %7, %22;\n\t"
        "addc.cc.u32 %8, %8, %23;\n\t"
        "addc.cc.u32 %9, %9, %24;\n\t"
        "addc.cc.u32 %10, %10, %25;\n\t"
        "addc.cc.u32 %11, %11, %26;\n\t"
        "addc.cc.u32 %12, %12, %27;\n\t"
        "addc.cc.u32 %13, %13, %28;\n\t"
        "addc.u32    %14, %14, %29;"
        : "+&r"(t[0]), "+&r"(t[1]), "+&r"(t[2]), "+&r"(t[3]), "+&r"(t[4]), "+&r"(t[5]), "+&r"(t[6]), "+&r"(t[7]), "+&r"(t[8]),
          "+&r"(t[9]), "+&r"(t[10]), "+&r"(t[11]), "+&r"(t[12]), "+&r"(t[13]), "+&r"(t[14])
        : "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3]), "r"(o[4]), "r"(o[5]), "r"(o[6]), "r"(o[7]), "r"(o[8]),
          "r"(o[9]), "r"(o[10]), "r"(o[11]), "r"(o[12]), "r"(o[13]), "r"(o[14]));
}

template <class P>
struct Field {
    using Params = P;
    static constexpr uint32_t M0 = P::M[0], M1 = P::M[1], M2 = P::M[2], M3 = P::M[3];
    static constexpr uint32_t M4 = P::M[4], M5 = P::M[5], M6 = P::M[6], M7 = P::M[7];
    static constexpr uint32_t C0 = P::C[0], C1 = P::C[1], C2 = P::C[2], C3 = P::C[3];

    __device__ __forceinline__ static Fe zero()
    {
        Fe r;
#pragma unroll
        for (int i = 0; i < 8; i++)
            r.w[i] = 0;
        return r;
    }
    __device__ __forceinline__ static Fe one()
    {
        Fe r = zero();
        r.w[0] = 1;
        return r;
    }
    __device__ __forceinline__ static Fe from_u32(uint32_t v)
    {
        Fe r = zero();
        r.w[0] = v;
        return r;
    }

    // r += k*c for k in {0,1}-like masks: adds (c & mask), returns carry out
    __device__ __forceinline__ static uint32_t add_c_masked(Fe &r, uint32_t mask)
    {
        uint32_t cy;
        asm("{\n\t"
            "add.cc.u32  %0, %0, %9;\n\t"
            "addc.cc.u32 %1, %1, %10;\n\t"
            "addc.cc.u32 %2, %2, %11;\n\t"
            "addc.cc.u32 %3, %3, %12;\n\t"
            "addc.cc.u32 %4, %4, 0;\n\t"
            "addc.cc.u32 %5, %5, 0;\n\t"
            "addc.cc.u32 %6, %6, 0;\n\t"
            "addc.cc.u32 %7, %7, 0;\n\t"
            "addc.u32    %8, 0, 0;\n\t"
            "}"
            : "+&r"(r.w[0]), "+&r"(r.w[1]), "+&r"(r.w[2]), "+&r"(r.w[3]), "+&r"(r.w[4]), "+&r"(r.w[5]), "+&r"(r.w[6]),
              "+&r"(r.w[7]), "=&r"(cy)
            : "r"(C0 & mask), "r"(C1 & mask), "r"(C2 & mask), "r"(C3 & mask));
        return cy;
    }

    __device__ __forceinline__ static uint32_t sub_c_masked(Fe &r, uint32_t mask)
    {
        uint32_t bw;
        asm("{\n\t"
            "sub.cc.u32  %0, %0, %9;\n\t"
            "subc.cc.u32 %1, %1, %10;\n\t"
            "subc.cc.u32 %2, %2, %11;\n\t"
            "subc.cc.u32 %3, %3, %12;\n\t"
            "subc.cc.u32 %4, %4, 0;\n\t"
            "subc.cc.u32 %5, %5, 0;\n\t"
            "subc.cc.u32 %6, %6, 0;\n\t"
            "subc.cc.u32 %7, %7, 0;\n\t"
            "subc.u32    %8, 0, 0;\n\t"
            "}"
            : "+&r"(r.w[0]), "+&r"(r.w[1]), "+&r"(r.w[2]), "+&r"(r.w[3]), "+&r"(r.w[4]), "+&r"(r.w[5]), "+&r"(r.w[6]),
              "+&r"(r.w[7]), "=&r"(bw)
            : "r"(C0 & mask), "r"(C1 & mask), "r"(C2 & mask), "r"(C3 & mask));
        return bw;  // 0 or 0xffffffff
    }

    // Sums and differences wrap at 2^256, which is worth c.  c is added (or
    // subtracted) to its own words and the one above; a carry that goes further
    // (one in 2^32 for values spread over their range) takes a branch instead of
    // six (F_p) or three (F_q) more adds with carry for everyone: 0.25 clocks
    // per SM against 0.46 on F_p, 0.35 against 0.50 on F_q.

    // a carry of 1 into word K; another wrap is worth c (what is left is then small)
    template <int K>
    __device__ __forceinline__ static void carry_from(Fe &r)
    {
        uint32_t cy = 1;
#pragma unroll
        for (int i = K; i < 8; i++) {
            r.w[i] += cy;
            cy = cy & (uint32_t)(r.w[i] == 0);
        }
        if (cy)
            add_c_masked(r, 0xffffffffu);
    }
    template <int K>
    __device__ __forceinline__ static void borrow_from(Fe &r)
    {
        uint32_t bw = 1;
#pragma unroll
        for (int i = K; i < 8; i++) {
            const uint32_t v = r.w[i];
            r.w[i] = v - bw;
            bw = bw & (uint32_t)(v == 0);
        }
        if (bw)
            sub_c_masked(r, 0xffffffffu);
    }

    // r + cy c (mod m), cy 0 or 1
    __device__ __forceinline__ static void add_c(Fe &r, uint32_t cy)
    {
        uint32_t more;
        if (P::NC == 1) {
            asm("mad.lo.cc.u32 %0, %3, %4, %0;\n\taddc.cc.u32 %1, %1, 0;\n\taddc.u32 %2, 0, 0;"
                : "+&r"(r.w[0]), "+&r"(r.w[1]), "=&r"(more)
                : "r"(cy), "r"(C0));
            if (more)
                carry_from<2>(r);
        } else {
            asm("mad.lo.cc.u32 %0, %6, %7, %0;\n\tmadc.lo.cc.u32 %1, %6, %8, %1;\n\tmadc.lo.cc.u32 %2, %6, %9, %2;\n\t"
                "madc.lo.cc.u32 %3, %6, %10, %3;\n\taddc.cc.u32 %4, %4, 0;\n\taddc.u32 %5, 0, 0;"
                : "+&r"(r.w[0]), "+&r"(r.w[1]), "+&r"(r.w[2]), "+&r"(r.w[3]), "+&r"(r.w[4]), "=&r"(more)
                : "r"(cy), "r"(C0), "r"(C1), "r"(C2), "r"(C3));
            if (more)
                carry_from<5>(r);
        }
    }
    // r - c (mod m) where mask is 0xffffffff, r where it is 0
    __device__ __forceinline__ static void sub_c(Fe &r, uint32_t mask)
    {
        uint32_t more;
        if (P::NC == 1) {
            asm("sub.cc.u32 %0, %0, %3;\n\tsubc.cc.u32 %1, %1, 0;\n\tsubc.u32 %2, 0, 0;"
                : "+&r"(r.w[0]), "+&r"(r.w[1]), "=&r"(more)
                : "r"(C0 & mask));
            if (more)
                borrow_from<2>(r);
        } else {
            asm("sub.cc.u32 %0, %0, %6;\n\tsubc.cc.u32 %1, %1, %7;\n\tsubc.cc.u32 %2, %2, %8;\n\tsubc.cc.u32 %3, %3, %9;\n\t"
                "subc.cc.u32 %4, %4, 0;\n\tsubc.u32 %5, 0, 0;"
                : "+&r"(r.w[0]), "+&r"(r.w[1]), "+&r"(r.w[2]), "+&r"(r.w[3]), "+&r"(r.w[4]), "=&r"(more)
                : "r"(C0 & mask), "r"(C1 & mask), "r"(C2 & mask), "r"(C3 & mask));
            if (more)
                borrow_from<5>(r);
        }
    }

    __device__ __forceinline__ static Fe add(const Fe &a, const Fe &b)
    {
        Fe r;
        add_c(r, add8(r.w, a.w, b.w));
        return r;
    }
    __device__ __forceinline__ static Fe sub(const Fe &a, const Fe &b)
    {
        Fe r;
        uint32_t m;
        asm("sub.cc.u32  %0, %9, %17;\n\tsubc.cc.u32 %1, %10, %18;\n\tsubc.cc.u32 %2, %11, %19;\n\tsubc.cc.u32 %3, %12, %20;\n\t"
            "subc.cc.u32 %4, %13, %21;\n\tsubc.cc.u32 %5, %14, %22;\n\tsubc.cc.u32 %6, %15, %23;\n\tsubc.cc.u32 %7, %16, %24;\n\t"
            "subc.u32 %8, 0, 0;"
            : "=&r"(r.w[0]), "=&r"(r.w[1]), "=&r"(r.w[2]), "=&r"(r.w[3]), "=&r"(r.w[4]), "=&r"(r.w[5]), "=&r"(r.w[6]), "=&r"(r.w[7]),
              "=&r"(m)
            : "r"(a.w[0]), "r"(a.w[1]), "r"(a.w[2]), "r"(a.w[3]), "r"(a.w[4]), "r"(a.w[5]), "r"(a.w[6]), "r"(a.w[7]),
              "r"(b.w[0]), "r"(b.w[1]), "r"(b.w[2]), "r"(b.w[3]), "r"(b.w[4]), "r"(b.w[5]), "r"(b.w[6]), "r"(b.w[7]));
        sub_c(r, m);
        return r;
    }

    __device__ __forceinline__ static Fe neg(const Fe &a) { return sub(zero(), a); }
    __device__ __forceinline__ static Fe dbl(const Fe &a) { return add(a, a); }

    // F_p: e + 2^32 o + 2^256 (c h) for h = the eight words 8..15, as e (words
    // 0..7, loaded), o (words 1..8, loaded, word 8 below 2^32 - 38) and h
    __device__ __forceinline__ static Fe fold_p(uint32_t e[9], uint32_t o[8], const uint32_t *h)
    {
        mad_chain<4, true>(e, h, C0);
        mad_chain<4, false>(o, h + 1, C0);
        Fe r;
        uint32_t r8;  // below 2^7
        r.w[0] = e[0];
        asm("add.cc.u32  %0, %8, %16;\n\taddc.cc.u32 %1, %9, %17;\n\taddc.cc.u32 %2, %10, %18;\n\taddc.cc.u32 %3, %11, %19;\n\t"
            "addc.cc.u32 %4, %12, %20;\n\taddc.cc.u32 %5, %13, %21;\n\taddc.cc.u32 %6, %14, %22;\n\taddc.u32 %7, %15, %23;"
            : "=&r"(r.w[1]), "=&r"(r.w[2]), "=&r"(r.w[3]), "=&r"(r.w[4]), "=&r"(r.w[5]), "=&r"(r.w[6]), "=&r"(r.w[7]), "=&r"(r8)
            : "r"(e[1]), "r"(e[2]), "r"(e[3]), "r"(e[4]), "r"(e[5]), "r"(e[6]), "r"(e[7]), "r"(e[8]), "r"(o[0]),
              "r"(o[1]), "r"(o[2]), "r"(o[3]), "r"(o[4]), "r"(o[5]), "r"(o[6]), "r"(o[7]));
        // r8 c back into the low words; a wrap leaves less than 2^13 in r, so adding c is safe
        uint32_t cy;
        asm("mad.lo.cc.u32 %0, %9, %10, %0;\n\taddc.cc.u32 %1, %1, 0;\n\taddc.cc.u32 %2, %2, 0;\n\t"
            "addc.cc.u32 %3, %3, 0;\n\taddc.cc.u32 %4, %4, 0;\n\taddc.cc.u32 %5, %5, 0;\n\t"
            "addc.cc.u32 %6, %6, 0;\n\taddc.cc.u32 %7, %7, 0;\n\taddc.u32 %8, 0, 0;"
            : "+&r"(r.w[0]), "+&r"(r.w[1]), "+&r"(r.w[2]), "+&r"(r.w[3]), "+&r"(r.w[4]), "+&r"(r.w[5]), "+&r"(r.w[6]),
              "+&r"(r.w[7]), "=&r"(cy)
            : "r"(r8), "r"(C0));
        r.w[0] += C0 & (0u - cy);
        return r;
    }

    // F_q: p = h c, four words by four
    __device__ __forceinline__ static void mul_c(uint32_t p[8], const uint32_t h[4])
    {
        uint32_t o[8];
        mul_pair(p, h[0], C0);
        mul_pair(p + 2, h[2], C0);
        mul_pair(o, h[1], C0);
        mul_pair(o + 2, h[3], C0);
        p[4] = 0;
        mad_chain<2, true>(o, h, C1);
        p[5] = 0;
        mad_chain<2, false>(p + 2, h + 1, C1);
        mad_chain<2, true>(p + 2, h, C2);
        o[5] = 0;
        mad_chain<2, false>(o + 2, h + 1, C2);
        mad_chain<2, true>(o + 2, h, C3);
        p[7] = 0;
        mad_chain<2, false>(p + 4, h + 1, C3);
        asm("add.cc.u32 %0, %0, %7;\n\taddc.cc.u32 %1, %1, %8;\n\taddc.cc.u32 %2, %2, %9;\n\taddc.cc.u32 %3, %3, %10;\n\t"
            "addc.cc.u32 %4, %4, %11;\n\taddc.cc.u32 %5, %5, %12;\n\taddc.u32 %6, %6, %13;"
            : "+&r"(p[1]), "+&r"(p[2]), "+&r"(p[3]), "+&r"(p[4]), "+&r"(p[5]), "+&r"(p[6]), "+&r"(p[7])
            : "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3]), "r"(o[4]), "r"(o[5]), "r"(o[6]));
    }

    // Fold a 512-bit value t[0..15] to a weakly reduced element.  F_q (c of four
    // words) folds from the top in two steps of four words, 16 products each:
    //   p = t[4..11] + t[12..15] c          (carry c1, worth 2^384 = 2^128 c)
    //   r = t[0..3] + 2^128 p[0..3] + p[4..7] c + c1 2^128 c.
    // (Folding the eight high words at once takes 32, then 16 for the words it
    // leaves above 2^256.)  One carry at most leaves r: c < 0.51 2^128, and c1 = 1
    // means p < t[12..15] c < 2^128 c, so p[4..7] < c and r < (1 + 0.27 + 0.51)
    // 2^256; with c1 = 0, r < 1.51 2^256.
    __device__ __forceinline__ static Fe reduce_wide(const uint32_t t[16])
    {
        if (P::NC == 1) {
            uint32_t e[9], o[8];
#pragma unroll
            for (int i = 0; i < 8; i++) {
                e[i] = t[i];
                o[i] = 0;
            }
            return fold_p(e, o, t + 8);
        }
        uint32_t p[8], q[8];
        mul_c(p, t + 12);
        const uint32_t c1 = add8(p, p, t + 4);
        mul_c(q, p + 4);
        Fe r;
        const uint32_t lo[8] = {t[0], t[1], t[2], t[3], p[0], p[1], p[2], p[3]};
        const uint32_t cy = add8(r.w, q, lo);
        uint32_t k;
        asm("mad.lo.cc.u32 %0, %5, %6, %0;\n\tmadc.lo.cc.u32 %1, %5, %7, %1;\n\tmadc.lo.cc.u32 %2, %5, %8, %2;\n\t"
            "madc.lo.cc.u32 %3, %5, %9, %3;\n\taddc.u32 %4, %10, 0;"
            : "+&r"(r.w[4]), "+&r"(r.w[5]), "+&r"(r.w[6]), "+&r"(r.w[7]), "=&r"(k)
            : "r"(c1), "r"(C0), "r"(C1), "r"(C2), "r"(C3), "r"(cy));
        add_c(r, k);
        return r;
    }

    __device__ __forceinline__ static Fe mul(const Fe &a, const Fe &b)
    {
        uint32_t e[16], o[16];
        mul_eo(e, o, a.w, b.w);
        if (P::NC == 1) {
            // only the high words are merged before the fold (without the low words'
            // carry, which the fold's own sum keeps): the low ones go in as they are
            uint32_t h[8];
            add8(h, e + 8, o + 7);
            o[7] = 0;
            uint32_t e9[9];
#pragma unroll
            for (int i = 0; i < 8; i++)
                e9[i] = e[i];
            return fold_p(e9, o, h);
        }
        merge15(e + 1, o);
        return reduce_wide(e);
    }

    __device__ __forceinline__ static Fe sqr(const Fe &a)
    {
        uint32_t t[16], o[16];
        cross_eo(t, o, a.w);
        t[1] = 0;
        t[14] = t[15] = o[14] = 0;
        merge15(t + 1, o);
        // double the cross sum (below 2^511, so nothing leaves word 15), then the squares at words 2i
#pragma unroll
        for (int k = 15; k > 1; k--)
            t[k] = __funnelshift_l(t[k - 1], t[k], 1);
        t[1] <<= 1;
        t[0] = 0;
        asm("{\n\t"
            "mad.lo.cc.u32  %0, %16, %16, %0;\n\t"
            "madc.hi.cc.u32 %1, %16, %16, %1;\n\t"
            "madc.lo.cc.u32 %2, %17, %17, %2;\n\t"
            "madc.hi.cc.u32 %3, %17, %17, %3;\n\t"
            "madc.lo.cc.u32 %4, %18, %18, %4;\n\t"
            "madc.hi.cc.u32 %5, %18, %18, %5;\n\t"
            "madc.lo.cc.u32 %6, %19, %19, %6;\n\t"
            "madc.hi.cc.u32 %7, %19, %19, %7;\n\t"
            "madc.lo.cc.u32 %8, %20, %20, %8;\n\t"
            "madc.hi.cc.u32 %9, %20, %20, %9;\n\t"
            "madc.lo.cc.u32 %10, %21, %21, %10;\n\t"
            "madc.hi.cc.u32 %11, %21, %21, %11;\n\t"
            "madc.lo.cc.u32 %12, %22, %22, %12;\n\t"
            "madc.hi.cc.u32 %13, %22, %22, %13;\n\t"
            "madc.lo.cc.u32 %14, %23, %23, %14;\n\t"
            "madc.hi.u32    %15, %23, %23, %15;\n\t"
            "}"
            : "+&r"(t[0]), "+&r"(t[1]), "+&r"(t[2]), "+&r"(t[3]), "+&r"(t[4]), "+&r"(t[5]), "+&r"(t[6]), "+&r"(t[7]),
              "+&r"(t[8]), "+&r"(t[9]), "+&r"(t[10]), "+&r"(t[11]), "+&r"(t[12]), "+&r"(t[13]), "+&r"(t[14]), "+&r"(t[15])
            : "r"(a.w[0]), "r"(a.w[1]), "r"(a.w[2]), "r"(a.w[3]), "r"(a.w[4]), "r"(a.w[5]), "r"(a.w[6]), "r"(a.w[7]));
        return reduce_wide(t);
    }

    // a b - c d.  On F_q the difference is taken before the reduction, which saves
    // one fold (32 products) for eight adds; on F_p the fold is 8 products and the
    // two products' difference would only hold more registers.
    __device__ __forceinline__ static Fe mul_sub(const Fe &a, const Fe &b, const Fe &c, const Fe &d)
    {
        if (P::NC == 1)
            return sub(mul(a, b), mul(c, d));
        uint32_t e[16], o[16], f[16];
        mul_eo(e, o, a.w, b.w);
        merge15(e + 1, o);
        mul_eo(f, o, c.w, d.w);
        merge15(f + 1, o);
        const uint32_t m = sub8(e + 8, e + 8, f + 8, sub8(e, e, f, 0u));
        // a borrow out of 2^512 is worth -2^256 c: the high half as a field element, less c
        Fe h;
#pragma unroll
        for (int i = 0; i < 8; i++)
            h.w[i] = e[8 + i];
        sub_c(h, m);
#pragma unroll
        for (int i = 0; i < 8; i++)
            e[8 + i] = h.w[i];
        return reduce_wide(e);
    }

    // canonical representative in [0, m): a < 2^256 = 2m + c
    __device__ __forceinline__ static Fe canon(const Fe &a)
    {
        Fe t = a;
        uint32_t cy = add_c_masked(t, 0xffffffffu);  // t = a + c; carry <=> a >= 2m
        Fe v = cy ? t : a;
        Fe d;
        uint32_t bw;
        asm("{\n\t"
            "sub.cc.u32  %0, %9, %17;\n\t"
            "subc.cc.u32 %1, %10, %18;\n\t"
            "subc.cc.u32 %2, %11, %19;\n\t"
            "subc.cc.u32 %3, %12, %20;\n\t"
            "subc.cc.u32 %4, %13, %21;\n\t"
            "subc.cc.u32 %5, %14, %22;\n\t"
            "subc.cc.u32 %6, %15, %23;\n\t"
            "subc.cc.u32 %7, %16, %24;\n\t"
            "subc.u32    %8, 0, 0;\n\t"
            "}"
            : "=&r"(d.w[0]), "=&r"(d.w[1]), "=&r"(d.w[2]), "=&r"(d.w[3]), "=&r"(d.w[4]), "=&r"(d.w[5]), "=&r"(d.w[6]),
              "=&r"(d.w[7]), "=&r"(bw)
            : "r"(v.w[0]), "r"(v.w[1]), "r"(v.w[2]), "r"(v.w[3]), "r"(v.w[4]), "r"(v.w[5]), "r"(v.w[6]),
              "r"(v.w[7]), "r"(M0), "r"(M1), "r"(M2), "r"(M3), "r"(M4), "r"(M5), "r"(M6), "r"(M7));
        return bw ? v : d;
    }

    __device__ __forceinline__ static bool is_zero(const Fe &a)
    {
        // a == 0 (mod m) <=> a in {0, m, 2m}; the top word screens the common case
        uint32_t top = a.w[7];
        if (top != 0u && top != M7 && top != ((M7 << 1) | (M6 >> 31)))
            return false;
        Fe c = canon(a);
        uint32_t o = 0;
#pragma unroll
        for (int i = 0; i < 8; i++)
            o |= c.w[i];
        return o == 0;
    }

    __device__ __forceinline__ static bool is_exact_zero(const Fe &a)
    {
        uint32_t o = 0;
#pragma unroll
        for (int i = 0; i < 8; i++)
            o |= a.w[i];
        return o == 0;
    }

    __device__ __forceinline__ static bool eq(const Fe &a, const Fe &b) { return is_zero(sub(a, b)); }

    // a^(2^n), n >= 0
    __device__ __forceinline__ static Fe sqr_n(Fe a, int n)
    {
#pragma unroll 1
        for (int i = 0; i < n; i++)
            a = sqr(a);
        return a;
    }

    // a^(2^k - 1), k >= 1: a run of n ones doubles to 2n by n squarings and one product
    __device__ static Fe pow_ones(const Fe &a, int k)
    {
        Fe r = a;
        int n = 1;
#pragma unroll 1
        for (int b = 30 - __clz(k); b >= 0; b--) {
            r = mul(sqr_n(r, n), r);
            n *= 2;
            if ((k >> b) & 1) {
                r = mul(sqr(r), a);
                n++;
            }
        }
        return r;
    }

    // ---- inversion by batched divsteps ----------------------------------------
    // The variable-time binary-GCD inversion of Bernstein and Yang ("Fast
    // constant-time gcd computation and modular inversion", 2019), with the
    // half-delta divstep: starting from (f, g) = (m, a), each divstep maps
    //     delta > 0 and g odd:  (delta, f, g) -> (1 - delta, g, (g - f) / 2)
    //     g odd:                (delta, f, g) -> (1 + delta, f, (g + f) / 2)
    //     g even:               (delta, f, g) -> (1 + delta, f, g / 2)
    // until g = 0, where f = +-gcd = +-1.  Steps run in batches of 30 on the low
    // 32 bits of f and g, which give a transition matrix T (entries at most 2^30)
    // with 2^30 (f', g') = T (f, g); T is then applied to the full f and g, held
    // in nine signed 30-bit limbs, and to (d, e) with f = d a, g = e a (mod m),
    // where the division by 2^30 is made exact by adding a multiple of m.  At the
    // end a^-1 = +-d.  A 256-bit input needs at most 590 divsteps (20 batches);
    // the loop is capped at 40.  Against Fermat's a^(m-2) (255 dependent
    // squarings) the dependent chain is about a tenth as long.  Within a batch,
    // runs of even steps are one shift, and runs of steps without a swap one
    // multiple of f (below): about a quarter as many turns as steps.
    struct L30 {
        int32_t l[9];  // value = sum l[i] 2^(30 i); l[0..7] in [0, 2^30), l[8] signed
    };

    __device__ __forceinline__ static L30 to_l30(const Fe &a)
    {
        L30 r;
#pragma unroll
        for (int i = 0; i < 9; i++) {
            const int b = 30 * i, k = b >> 5, sh = b & 31;
            const uint64_t lo = a.w[k], hi = k + 1 < 8 ? a.w[k + 1] : 0u;
            r.l[i] = (int32_t)(((lo | (hi << 32)) >> sh) & 0x3fffffffu);
        }
        return r;
    }

    // (x, y) <- (s x + t y + k m) / 2^30 for one row; the low 30 bits vanish
    __device__ __forceinline__ static void l30_row(L30 &out, const L30 &x, const L30 &y, int32_t s, int32_t t,
                                                   int32_t k, const L30 &m)
    {
        int64_t c = (int64_t)s * x.l[0] + (int64_t)t * y.l[0] + (int64_t)k * m.l[0];
        c >>= 30;
#pragma unroll
        for (int i = 1; i < 9; i++) {
            c += (int64_t)s * x.l[i] + (int64_t)t * y.l[i] + (int64_t)k * m.l[i];
            out.l[i - 1] = (int32_t)(c & 0x3fffffff);
            c >>= 30;
        }
        out.l[8] = (int32_t)c;
    }

    __device__ static Fe inv(const Fe &a)
    {
        const Fe x = canon(a);
        if (is_exact_zero(x))
            return zero();  // 0 -> 0
        const Fe mf = {{M0, M1, M2, M3, M4, M5, M6, M7}};
        const L30 m = to_l30(mf);
        L30 zero30;
#pragma unroll
        for (int i = 0; i < 9; i++)
            zero30.l[i] = 0;
        // m^-1 mod 2^32 by Newton's iteration (m odd: m m = 1 mod 8 to start)
        uint32_t minv = M0;
#pragma unroll
        for (int i = 0; i < 4; i++)
            minv *= 2u - M0 * minv;
        L30 f = m, g = to_l30(x), d = zero30, e = zero30;
        e.l[0] = 1;
        int32_t D = 1;  // 2 delta, delta = 1/2
        for (int batch = 0; batch < 40; batch++) {
            uint32_t any = 0;
#pragma unroll
            for (int i = 0; i < 9; i++)
                any |= (uint32_t)g.l[i];
            if (!any)
                break;
            uint32_t fl = (uint32_t)f.l[0] | ((uint32_t)f.l[1] << 30);
            uint32_t gl = (uint32_t)g.l[0] | ((uint32_t)g.l[1] << 30);
            int32_t u = 1, v = 0, q = 0, r = 1;
            int left = 30;
            for (;;) {
                // the even steps up to the next odd g
                const int z = __ffs((int)(gl | (1u << left))) - 1;
                gl >>= z;
                u = (int32_t)((uint32_t)u << z);
                v = (int32_t)((uint32_t)v << z);
                D += 2 * z;
                left -= z;
                if (left == 0)
                    break;
                if (D > 0) {  // the swap of a first-form step: what remains is g + f, halved
                    const uint32_t t = fl;
                    const int32_t tu = u, tv = v;
                    D = -D;
                    fl = gl;
                    gl = 0u - t;
                    u = q;
                    v = r;
                    q = -tu;
                    r = -tv;
                }
                // no swap is due for (1 - D) / 2 steps: of these, up to six at once, by
                // the multiple w f that clears as many low bits of g (the halvings
                // are the next turn's even steps), a step known from the variable-time
                // inversion of libsecp256k1.  f (2 - f^2) = 1/f mod 64.
                int lim = (1 - D) >> 1;
                lim = lim < left ? lim : left;
                lim = lim < 6 ? lim : 6;
                const uint32_t w = (0u - gl * (fl * (2u - fl * fl))) & ((1u << lim) - 1u);
                gl += fl * w;
                q += u * (int32_t)w;
                r += v * (int32_t)w;
            }
            L30 nf, ng, nd, ne;
            l30_row(nf, f, g, u, v, 0, m);
            l30_row(ng, f, g, q, r, 0, m);
            const uint32_t td = (uint32_t)u * (uint32_t)d.l[0] + (uint32_t)v * (uint32_t)e.l[0];
            const uint32_t te = (uint32_t)q * (uint32_t)d.l[0] + (uint32_t)r * (uint32_t)e.l[0];
            const int32_t md = (int32_t)(((0u - td) * minv) << 2) >> 2;  // in [-2^29, 2^29)
            const int32_t me = (int32_t)(((0u - te) * minv) << 2) >> 2;
            l30_row(nd, d, e, u, v, md, m);
            l30_row(ne, d, e, q, r, me, m);
            f = nf;
            g = ng;
            d = nd;
            e = ne;
        }
        // d + 16 m > 0 (|d| < m here), packed into nine 32-bit words, folded mod m
        int64_t c = 0;
        uint32_t w[9];
        {
            L30 t;
#pragma unroll
            for (int i = 0; i < 9; i++) {
                c += (int64_t)d.l[i] + 16 * (int64_t)m.l[i];
                t.l[i] = i < 8 ? (int32_t)(c & 0x3fffffff) : (int32_t)c;
                c >>= 30;
            }
            uint64_t acc = 0;
            int bits = 0, k = 0;
#pragma unroll
            for (int i = 0; i < 9; i++) {
                acc |= (uint64_t)(uint32_t)t.l[i] << bits;
                bits += 30;
                while (bits >= 32 && k < 9) {
                    w[k++] = (uint32_t)acc;
                    acc >>= 32;
                    bits -= 32;
                }
            }
            while (k < 9) {
                w[k++] = (uint32_t)acc;
                acc >>= 32;
            }
        }
        Fe lo;
#pragma unroll
        for (int i = 0; i < 8; i++)
            lo.w[i] = w[i];
        Fe cfe = zero();
        add_c_masked(cfe, 0xffffffffu);  // 2^256 mod m
        Fe res = add(lo, mul(from_u32(w[8]), cfe));
        return f.l[8] < 0 ? neg(res) : res;
    }
};

using Fp = Field<FpParams>;
using Fq = Field<FqParams>;

}  // namespace hs
