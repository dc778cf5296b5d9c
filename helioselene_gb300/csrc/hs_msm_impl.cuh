// hs_msm_impl.cuh -- curve-templated device kernels of the MSM path.
//
// Pipeline of one MSM (n points, c-bit signed windows, W = ceil(257/c) windows,
// B = 2^(c-1) buckets per window), following the reference Pippenger
// (helios/src/x64/helios_msm_vartime.cpp:265-388) but laid out for the GPU:
//   1. recode + counting sort (hs_runtime.cu): every (point, window) with a
//      nonzero digit becomes one entry "point index | sign" placed
//      contiguously per bucket;
//   2. k_accumulate: buckets are cut into segments of at most L entries, one
//      thread sums one segment of affine bases into an XYZZ point;
//   3. k_merge / k_merge_heavy: buckets with several segments are folded
//      (sequentially when few, by a block-wide tree when many);
//   4. k_reduce_groups / k_window_chunks / k_window_sum (k_window_serial for many
//      windows, k_window_quads instead of all for small plans): per window
//      S = sum_j (j+1) B_j by running sums over groups of 8 buckets, then
//      suffix scans and trees over the groups (no scalar multiples);
//   5. k_combine: Horner over the windows, S = 2^c S + S_k (the reference's
//      per-window doublings, :285-289) on lane-sliced elements, a cluster of blocks
//      per MSM; result as canonical Jacobian.
#pragma once

#include <cooperative_groups.h>

#include "hs_curve.cuh"
#include "hs_internal.h"
#include "hs_lane.cuh"
#include "hs_quad.cuh"

namespace hs {

// ---------------------------------------------------------------------------
// memory helpers
// ---------------------------------------------------------------------------
// One field element per access: 32-byte loads and stores of global memory.  A warp's
// gather of 64-byte points is then two requests per point instead of four, and a
// stream of elements is full sectors.  The library's own buffers are 256-byte
// aligned; the caller's points need only 16 bytes, so their loads take `wide`, the
// same for a whole launch.
__device__ __forceinline__ Fe ldg_fe(const uint4 *p)
{
    Fe f;
    asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(f.w[0]), "=r"(f.w[1]), "=r"(f.w[2]), "=r"(f.w[3]), "=r"(f.w[4]), "=r"(f.w[5]), "=r"(f.w[6]), "=r"(f.w[7])
        : "l"(p));
    return f;
}
__device__ __forceinline__ Fe ldg_fe(const uint4 *p, bool wide)
{
    if (wide)
        return ldg_fe(p);
    const uint4 a = __ldg(p), b = __ldg(p + 1);
    return Fe{{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w}};
}
__device__ __forceinline__ bool wide_points(const uint4 *pts) { return (reinterpret_cast<uintptr_t>(pts) & 31) == 0; }

__device__ __forceinline__ void stg_fe(uint4 *p, const Fe &f)
{
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(f.w[0]), "r"(f.w[1]),
                 "r"(f.w[2]), "r"(f.w[3]), "r"(f.w[4]), "r"(f.w[5]), "r"(f.w[6]), "r"(f.w[7])
                 : "memory");
}

__device__ __forceinline__ void load_affine(const uint4 *__restrict__ pts, uint32_t idx, Fe &x, Fe &y, bool wide)
{
    const uint4 *p = pts + 4 * (size_t)idx;
    x = ldg_fe(p, wide);
    y = ldg_fe(p + 2, wide);
}

__device__ __forceinline__ void store_fe(uint4 *o, const Fe &f)
{
    o[0] = make_uint4(f.w[0], f.w[1], f.w[2], f.w[3]);
    o[1] = make_uint4(f.w[4], f.w[5], f.w[6], f.w[7]);
}

__device__ __forceinline__ Fe load_fe(const uint4 *o)
{
    Fe f;
    uint4 a = o[0], b = o[1];
    f.w[0] = a.x; f.w[1] = a.y; f.w[2] = a.z; f.w[3] = a.w;
    f.w[4] = b.x; f.w[5] = b.y; f.w[6] = b.z; f.w[7] = b.w;
    return f;
}

__device__ __forceinline__ void store_xyzz(uint4 *o, const Xyzz &p)
{
    store_fe(o, p.X);
    store_fe(o + 2, p.Y);
    store_fe(o + 4, p.ZZ);
    store_fe(o + 6, p.ZZZ);
}

__device__ __forceinline__ Xyzz load_xyzz(const uint4 *o)
{
    Xyzz p;
    p.X = load_fe(o);
    p.Y = load_fe(o + 2);
    p.ZZ = load_fe(o + 4);
    p.ZZZ = load_fe(o + 6);
    return p;
}

// the library's own buffers in global memory
__device__ __forceinline__ void stg_xyzz(uint4 *o, const Xyzz &p)
{
    stg_fe(o, p.X);
    stg_fe(o + 2, p.Y);
    stg_fe(o + 4, p.ZZ);
    stg_fe(o + 6, p.ZZZ);
}

// ---------------------------------------------------------------------------
// 2. bucket accumulation: one thread per segment of <= L entries (segments come
//    longest first, so the lanes of a warp do equal work).  The launch takes the
//    descriptors [*seg_lo, *seg_hi) (device values: one list, or one part of
//    host inputs in two parts); with RESUME, a descriptor with d.w set
//    continues the sum stored in its slot by the earlier part.
// ---------------------------------------------------------------------------
template <class C, bool RESUME>
__global__ void __launch_bounds__(128, 4) k_accumulate(const uint4 *__restrict__ segs, const uint32_t *__restrict__ seg_lo,
                                                   const uint32_t *__restrict__ seg_hi,
                                                   const uint32_t *__restrict__ sorted, const uint4 *__restrict__ pts,
                                                   uint4 *__restrict__ seg_sum)
{
    using G = Group<C>;
    using F = typename C::F;
    const uint32_t S0 = *seg_lo, S = *seg_hi;
    const bool wide = wide_points(pts);
    for (uint32_t s = S0 + blockIdx.x * blockDim.x + threadIdx.x; s < S; s += gridDim.x * blockDim.x) {
        const uint4 d = segs[s];  // start, length, destination slot, continue
        Xyzz acc = (RESUME && d.w) ? load_xyzz(seg_sum + 8 * (size_t)d.z) : G::inf();
        for (uint32_t i = 0; i < d.y; i++) {
            const uint32_t e = __ldg(sorted + d.x + i);
            Fe x, y;
            load_affine(pts, e & 0x7fffffffu, x, y, wide);
            if (F::is_exact_zero(x) && F::is_exact_zero(y))
                continue;  // identity base (the reference's Z == 0 input) contributes nothing
            if (e >> 31)
                y = F::neg(y);
            G::add_affine(acc, x, y);
        }
        stg_xyzz(seg_sum + 8 * (size_t)d.z, acc);
    }
}

// ---------------------------------------------------------------------------
// 2'. batch-affine bucket accumulation (plans with ba_rounds = R > 0)
// ---------------------------------------------------------------------------
// Every bucket's entry list is padded to a multiple of 2^R (padding entries are
// PAD_ENTRY, the identity), so the lists of every round start at even
// positions.  Round r then adds the items of the previous level in flat pairs:
// output q = item 2q + item 2q+1 (round 1: entries, later: affine sums), by
//     lambda = (y_b - y_a) / (x_b - x_a)   (doubling: (3 x_a^2 - 3) / (2 y_a)),
//     x = lambda^2 - x_a - x_b,  y = lambda (x_a - x) - y_a,
// and bucket k's round-r list is [off_k >> r, off_{k+1} >> r) with no scan:
// a round is a pure stream over the level, every warp reading 32 consecutive
// pairs.  The divisions of a round share inversions by Montgomery's trick
// (fp/include/fp_batch_invert.h:61-114 applied across a wave of additions):
//   k_ba_pairs   lane l of warp tile w takes outputs w*32K + l + 32k (k < K):
//                denominators and their running product (each output's exclusive
//                prefix and the thread's total are stored);
//   k_ba_invert  the totals' inverses, one inversion shared by a block's BA_G *
//                BA_INV_BT totals (so by BA_K times as many additions);
//   k_ba_finish  each output walks back from the thread's inverse:
//                1/d = (1/prefix through d) * (prefix before d), and the sum.
// (A product tree over each block of k_ba_pairs, one inversion per block, held up
// its warps at the tree's fourteen barriers: 248 + 30 us and 199 + 30 us on F_q and F_p
// for one MSM of 2^20 points.)
// Pairs with equal x double (d = 2 y_a) or cancel (the identity, d = 1); an
// identity operand (affine (0,0), or a padding entry) takes d = 1 and the
// other operand is copied.  The last round's sums are folded into XYZZ bucket
// sums by k_accumulate_level.
constexpr int BA_K = (int)BA_PLAN_K;    // outputs per thread
constexpr int BA_BT = (int)BA_PLAN_BT;  // threads per block

enum BaKind : int { BA_ADD, BA_DBL, BA_COPY_A, BA_COPY_B, BA_ZERO };

// The two items of an output.  Round 1 reads entries 2q and 2q + 1 (point index |
// sign << 31; PAD_ENTRY is the identity), later rounds items 2q and 2q + 1 of the
// previous level's affine sums.
template <class C, bool FIRST>
struct BaInput {
    using F = typename C::F;
    const uint2 *entries;
    const uint4 *base;  // the points, or the previous level
    bool wide;

    __device__ __forceinline__ BaInput(const uint32_t *sorted, const uint4 *pts, const uint4 *lvl)
        : entries(reinterpret_cast<const uint2 *>(sorted)), base(FIRST ? pts : lvl), wide(!FIRST || wide_points(pts))
    {
    }
    __device__ __forceinline__ uint2 entry(uint64_t q) const
    {
        return FIRST ? __ldg(entries + q) : make_uint2((uint32_t)(2 * q), (uint32_t)(2 * q + 1));
    }
    __device__ __forceinline__ static bool pad(uint32_t e) { return FIRST && e == PAD_ENTRY; }
    // (a padding entry reads element 0, and what it read is dropped)
    __device__ __forceinline__ const uint4 *src(uint32_t e) const
    {
        return base + 4 * (size_t)(FIRST ? (pad(e) ? 0u : e & 0x7fffffffu) : e);
    }
    __device__ __forceinline__ Fe x(uint32_t e) const { return ldg_fe(src(e), wide); }
    __device__ __forceinline__ Fe y(uint32_t e) const  // negated for a negative digit; the identity's 0 stays 0
    {
        const Fe v = ldg_fe(src(e) + 2, wide);
        return FIRST && (e >> 31) ? F::neg(v) : v;
    }
    // an item that may be the identity (padding, or an x whose low word is 0), or
    // equal x: the cases that kind() sorts out
    __device__ __forceinline__ bool rare(const uint2 &e, const Fe &xa, const Fe &xb, const Fe &dx) const
    {
        return pad(e.x) || pad(e.y) || xa.w[0] == 0 || xb.w[0] == 0 || F::is_zero(dx);
    }
    // kind and denominator of a rare pair (d: x_b - x_a on entry); the coordinates of
    // a padding item become 0
    __device__ __forceinline__ int kind(const uint2 &e, Fe &xa, Fe &ya, Fe &xb, Fe &yb, Fe &d) const
    {
        if (pad(e.x))
            xa = ya = F::zero();
        if (pad(e.y))
            xb = yb = F::zero();
        if (F::is_exact_zero(xb) && F::is_exact_zero(yb))
            return BA_COPY_A;  // b is the identity
        if (F::is_exact_zero(xa) && F::is_exact_zero(ya))
            return BA_COPY_B;  // a is the identity
        if (!F::is_zero(d))
            return BA_ADD;
        if (!F::is_zero(F::sub(yb, ya)) || F::is_zero(ya))
            return BA_ZERO;  // b = -a (or a point of order 2, which doubles to the identity)
        d = F::dbl(ya);  // b = a: double
        return BA_DBL;
    }
};

// first output of this thread's warp tile, plus its lane (outputs base + 32 k),
// in a launch over outputs [E0, E)
__device__ __forceinline__ uint64_t ba_tile_base(uint32_t E0)
{
    const uint64_t tile = (uint64_t)blockIdx.x * (BA_BT / 32) + (threadIdx.x >> 5);
    return E0 + tile * 32 * BA_K + (threadIdx.x & 31);
}

// A launch covers round r's outputs [*lo >> r, *hi >> r) (lo null: from 0):
// the whole level, or the lists of one part of host inputs in two parts.
__device__ __forceinline__ uint32_t ba_first(const uint32_t *lo, uint32_t r) { return lo ? __ldg(lo) >> r : 0u; }

template <class C, bool FIRST>
__global__ void __launch_bounds__(BA_BT) k_ba_pairs(const uint32_t *__restrict__ lo, const uint32_t *__restrict__ hi,
                                                   uint32_t r, const uint32_t *__restrict__ sorted,
                                                   const uint4 *__restrict__ pts, const uint4 *__restrict__ lvl,
                                                   uint4 *__restrict__ pre, uint4 *__restrict__ tot)
{
    using F = typename C::F;
    const uint32_t E0 = ba_first(lo, r), E = __ldg(hi) >> r;  // outputs of this launch
    if (E0 + (uint64_t)blockIdx.x * BA_BT * BA_K >= E)
        return;  // the whole block is past the launch's outputs
    const BaInput<C, FIRST> in(sorted, pts, lvl);
    const uint64_t base = ba_tile_base(E0);
    Fe run = F::one();
    bool any = false;
    if (base < E) {
        const int kmax = (int)((E - 1 - base) / 32) < BA_K - 1 ? (int)((E - 1 - base) / 32) : BA_K - 1;
        uint2 e = in.entry(base), next = kmax > 0 ? in.entry(base + 32) : e;
#pragma unroll 1
        for (int k = 0; k <= kmax; k++) {
            const uint64_t q = base + 32 * (uint64_t)k;
            const uint2 after = k + 2 <= kmax ? in.entry(q + 64) : next;
            Fe xa = in.x(e.x), xb = in.x(e.y);
            Fe d = F::sub(xb, xa);
            int kind = BA_ADD;
            if (in.rare(e, xa, xb, d)) {
                Fe ya = in.y(e.x), yb = in.y(e.y);
                kind = in.kind(e, xa, ya, xb, yb, d);
            }
            if (kind <= BA_DBL) {
                stg_fe(pre + 2 * q, run);  // exclusive prefix of this output (1 for the first)
                run = any ? F::mul(run, d) : d;
                any = true;
            }
            e = next;
            next = after;
        }
    }
    stg_fe(tot + 2 * ((size_t)blockIdx.x * BA_BT + threadIdx.x), run);
}

// The thread totals' inverses, in place (a total is never zero: every factor is not).
// A block takes BA_G totals per thread: their running products per thread, a
// product tree over the threads, one inversion, and the way back.  One inversion per
// BA_G totals without the tree took 85 us for the 524288 totals of an MSM of 2^20
// points, against 44 (twice as many, K = 16) and less now.
constexpr int BA_G = 8;
constexpr int BA_INV_BT = 128;

template <class C>
__global__ void __launch_bounds__(BA_INV_BT) k_ba_invert(const uint32_t *__restrict__ lo,
                                                        const uint32_t *__restrict__ hi, uint32_t r, uint4 *tot)
{
    using F = typename C::F;
    __shared__ Fe tree[2 * BA_INV_BT], cop[2 * BA_INV_BT];
    const uint32_t E0 = ba_first(lo, r), E = __ldg(hi) >> r;
    const uint64_t count = (((uint64_t)(E - E0) + BA_BT * BA_K - 1) / (BA_BT * BA_K)) * BA_BT;
    const uint32_t t = threadIdx.x;
    const uint64_t first = blockIdx.x * (uint64_t)(BA_G * BA_INV_BT) + t;  // totals first + j BA_INV_BT
    if (first - t >= count)
        return;  // the whole block
    Fe pre[BA_G];  // products of this thread's totals up to j (1 past the end)
#pragma unroll
    for (int j = 0; j < BA_G; j++) {
        const uint64_t i = first + (uint64_t)j * BA_INV_BT;
        const Fe v = i < count ? load_fe(tot + 2 * i) : F::one();
        pre[j] = j ? F::mul(pre[j - 1], v) : v;
    }
    // product tree over the threads (leaf t at BA_INV_BT + t), then top down
    // cop[node] = the inverse of the node's product
    tree[BA_INV_BT + t] = pre[BA_G - 1];
    __syncthreads();
    for (uint32_t s = BA_INV_BT / 2; s >= 1; s >>= 1) {
        if (t < s)
            tree[s + t] = F::mul(tree[2 * (s + t)], tree[2 * (s + t) + 1]);
        __syncthreads();
    }
    if (t == 0)
        cop[1] = F::inv(tree[1]);
    __syncthreads();
    for (uint32_t s = 1; s < BA_INV_BT; s <<= 1) {
        if (t < 2 * s) {  // node 2 s + t, by its sibling
            const uint32_t nd = 2 * s + t;
            cop[nd] = F::mul(cop[nd >> 1], tree[nd ^ 1]);
        }
        __syncthreads();
    }
    Fe inv = cop[BA_INV_BT + t];
#pragma unroll
    for (int j = BA_G - 1; j >= 0; j--) {
        const uint64_t i = first + (uint64_t)j * BA_INV_BT;
        if (i < count) {
            const Fe v = load_fe(tot + 2 * i);
            stg_fe(tot + 2 * i, j ? F::mul(inv, pre[j - 1]) : inv);
            inv = F::mul(inv, v);
        }
    }
}

template <class C, bool FIRST>
__global__ void __launch_bounds__(BA_BT) k_ba_finish(const uint32_t *__restrict__ lo, const uint32_t *__restrict__ hi,
                                                    uint32_t r, const uint32_t *__restrict__ sorted,
                                                    const uint4 *__restrict__ pts, const uint4 *__restrict__ lvl,
                                                    const uint4 *__restrict__ pre, const uint4 *__restrict__ tot,
                                                    uint4 *__restrict__ out)
{
    using F = typename C::F;
    const uint32_t E0 = ba_first(lo, r), E = __ldg(hi) >> r;
    const uint64_t base = ba_tile_base(E0);
    if (base >= E)
        return;
    const BaInput<C, FIRST> in(sorted, pts, lvl);
    // 1 / (this thread's total)
    Fe inv_run = ldg_fe(tot + 2 * ((size_t)blockIdx.x * BA_BT + threadIdx.x));
    const int kmax = (int)((E - 1 - base) / 32) < BA_K - 1 ? (int)((E - 1 - base) / 32) : BA_K - 1;
    uint2 e = in.entry(base + 32 * (uint64_t)kmax), next = kmax > 0 ? in.entry(base + 32 * (uint64_t)(kmax - 1)) : e;
#pragma unroll 1
    for (int k = kmax; k >= 0; k--) {
        const uint64_t q = base + 32 * (uint64_t)k;
        const uint2 after = k >= 2 ? in.entry(q - 64) : next;
        Fe xa = in.x(e.x), xb = in.x(e.y), ya = in.y(e.x), yb = in.y(e.y);
        Fe d = F::sub(xb, xa);
        int kind = BA_ADD;
        if (in.rare(e, xa, xb, d))
            kind = in.kind(e, xa, ya, xb, yb, d);
        Fe x3, y3;
        if (kind <= BA_DBL) {
            const Fe inv_d = F::mul(inv_run, ldg_fe(pre + 2 * q));
            inv_run = F::mul(inv_run, d);
            Fe num = F::sub(yb, ya);
            if (kind == BA_DBL) {
                const Fe t = F::sub(F::sqr(xa), F::one());
                num = F::add(F::dbl(t), t);  // 3 x^2 + a, a = -3
                xb = xa;
            }
            const Fe lam = F::mul(num, inv_d);
            x3 = F::sub(F::sub(F::sqr(lam), xa), xb);
            y3 = F::sub(F::mul(lam, F::sub(xa, x3)), ya);
        } else {
            x3 = kind == BA_COPY_A ? xa : kind == BA_COPY_B ? xb : F::zero();
            y3 = kind == BA_COPY_A ? ya : kind == BA_COPY_B ? yb : F::zero();
        }
        uint4 *dst = out + 4 * q;
        stg_fe(dst, x3);
        stg_fe(dst + 2, y3);
        e = next;
        next = after;
    }
}

// The batch-affine rounds' last sums, folded per segment into XYZZ bucket sums
// (segments of a bucket's list in the last level buffer, longest first, as in
// k_accumulate; the items are affine points, (0,0) the identity).  With
// RESUME (part 1 of host inputs in two parts), a descriptor with d.w set
// continues the sum stored in its slot by part 0.
template <class C, bool RESUME>
__global__ void __launch_bounds__(128) k_accumulate_level(const uint4 *__restrict__ segs,
                                                         const uint32_t *__restrict__ seg_lo,
                                                         const uint32_t *__restrict__ seg_hi,
                                                         const uint4 *__restrict__ lvl, uint4 *__restrict__ seg_sum)
{
    using G = Group<C>;
    using F = typename C::F;
    const uint32_t S0 = *seg_lo, S = *seg_hi;
    for (uint32_t s = S0 + blockIdx.x * blockDim.x + threadIdx.x; s < S; s += gridDim.x * blockDim.x) {
        const uint4 d = segs[s];  // start, length, destination slot, continue
        Xyzz acc = (RESUME && d.w) ? load_xyzz(seg_sum + 8 * (size_t)d.z) : G::inf();
        for (uint32_t i = 0; i < d.y; i++) {
            Fe x, y;
            load_affine(lvl, d.x + i, x, y, true);
            if (F::is_exact_zero(x) && F::is_exact_zero(y))
                continue;
            G::add_affine(acc, x, y);
        }
        stg_xyzz(seg_sum + 8 * (size_t)d.z, acc);
    }
}

// ---------------------------------------------------------------------------
// 3. folding buckets that were cut into several segments
// ---------------------------------------------------------------------------
// Both kernels work on quads: a bucket's few additions in sequence and a heavy
// bucket's tree are latency, which one thread's 14 products per addition set: 66 + 70 us
// for one F_q MSM of 65521 points, 38 + 23 so.
template <class C>
__global__ void __launch_bounds__(128) k_merge(const uint32_t *__restrict__ seg_off, uint32_t NB,
                                              uint4 *__restrict__ seg_sum, uint32_t *__restrict__ heavy,
                                              uint32_t *__restrict__ heavy_n, uint32_t heavy_min)
{
    using F = typename C::F;
    using Q = Quad<C>;
    const Q op(threadIdx.x);
    const uint32_t stride = gridDim.x * (blockDim.x >> 2);
    for (uint32_t w = blockIdx.x * (blockDim.x >> 2) + (threadIdx.x >> 5) * 8; w < NB; w += stride) {
        const uint32_t kb = w + ((threadIdx.x >> 2) & 7);
        uint32_t s0 = 0, ns = 0;
        if (kb < NB) {
            s0 = seg_off[kb];
            ns = seg_off[kb + 1] - s0;
            if (ns > heavy_min) {
                if (op.j == 0)
                    heavy[atomicAdd(heavy_n, 1u)] = kb;
                ns = 0;
            }
        }
        const uint32_t most = __reduce_max_sync(Q::ALL, ns);
        if (most < 2)
            continue;
        Fe acc = ns > 1 ? Q::load(seg_sum, s0, op.j) : F::zero();
        for (uint32_t i = 1; i < most; i++) {
            const bool take = i < ns;
            const Fe o = take ? Q::load(seg_sum, s0 + i, op.j) : F::zero();
            acc = op.template add<false>(acc, o, take);
        }
        if (ns > 1)
            Q::store(seg_sum, s0, op.j, acc);
    }
}

constexpr int HEAVY_QUADS = 64;

template <class C>
__global__ void __launch_bounds__(HEAVY_QUADS * 4) k_merge_heavy(const uint32_t *__restrict__ seg_off,
                                                                const uint32_t *__restrict__ heavy,
                                                                const uint32_t *__restrict__ heavy_n,
                                                                uint4 *__restrict__ seg_sum)
{
    using F = typename C::F;
    using Q = Quad<C>;
    __shared__ uint4 sh[HEAVY_QUADS * 8];
    const Q op(threadIdx.x);
    const uint32_t g = threadIdx.x >> 2;
    const uint32_t cnt = *heavy_n;
    for (uint32_t h = blockIdx.x; h < cnt; h += gridDim.x) {
        const uint32_t kb = heavy[h];
        const uint32_t s0 = seg_off[kb], ns = seg_off[kb + 1] - s0;
        Fe acc = g < ns ? Q::load(seg_sum, s0 + g, op.j) : F::zero();
        const uint32_t first = g & ~7u;  // the warp's first quad: its quads loop together
        for (uint32_t i = first + HEAVY_QUADS; i < ns; i += HEAVY_QUADS) {
            const uint32_t mine = i + (g - first);
            const bool take = mine < ns;
            const Fe o = take ? Q::load(seg_sum, s0 + mine, op.j) : F::zero();
            acc = op.template add<false>(acc, o, take);
        }
        Q::store(sh, g, op.j, acc);
        __syncthreads();
        // the tree spans only the quads that hold a segment (a power of two)
        uint32_t width = 1;
        while (width < ns && width < (uint32_t)HEAVY_QUADS)
            width <<= 1;
        for (uint32_t stride = width / 2; stride > 0; stride >>= 1) {
            if (first < stride) {  // whole warps
                const bool take = g < stride;
                const Fe o = take ? Q::load(sh, g + stride, op.j) : F::zero();
                acc = op.template add<false>(acc, o, take);
            }
            __syncthreads();
            if (g < stride)
                Q::store(sh, g, op.j, acc);
            __syncthreads();
        }
        if (g == 0)
            Q::store(seg_sum, s0, op.j, acc);
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// 4. bucket reduction: S = sum_j (j+1) B_j per window, in two levels
// ---------------------------------------------------------------------------
// Level 1, k_reduce_groups: thread (k, t) owns the m0 buckets [t m0, (t+1) m0)
// of window k and runs the reference's top-down running sum over them
// (helios_msm_vartime.cpp:334-361), giving
//     run_t = sum_j B_j,   acc_t = sum_j (j - t m0 + 1) B_j,
// so that S = sum_t acc_t + m0 sum_t t run_t.
// One addition in the loop, used for run += B_j and acc += run in turn, and acc kept in
// shared memory between its turns (one uint4 column per thread, conflict-free): with
// two inlined additions and both sums in registers the kernel missed the
// instruction cache and spilled: 157 / 256 us (F_p / F_q) for one MSM of 2^20
// points, 145 / 219 so; three blocks per SM measured a little better than four
template <class C>
__global__ void __launch_bounds__(128, 3) k_reduce_groups(const uint32_t *__restrict__ seg_off,
                                                      const uint4 *__restrict__ seg_sum,
                                                      const MsmDesc *__restrict__ desc, uint32_t M, uint32_t G,
                                                      uint4 *__restrict__ out)
{
    using G_ = Group<C>;
    using F = typename C::F;
    __shared__ uint4 sa[8][128];
    const uint32_t tid = threadIdx.x;
    const uint32_t gid = blockIdx.x * blockDim.x + tid;
    if (gid >= G)
        return;
    const uint32_t mi = find_msm(M, gid, [&](uint32_t k) { return desc[k].group_base; });
    const MsmDesc d = desc[mi];
    const uint32_t local = gid - d.group_base;
    const uint32_t k = local / d.T, t = local % d.T;
    const uint32_t m = d.m0;
    const uint32_t kb0 = d.bucket_base + k * d.B + t * m;
#pragma unroll
    for (int c = 0; c < 8; c++)
        sa[c][tid] = make_uint4(0, 0, 0, 0);
    auto ld = [&](int c) {
        const uint4 a = sa[2 * c][tid], b = sa[2 * c + 1][tid];
        return Fe{{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w}};
    };
    auto st = [&](int c, const Fe &f) {
        sa[2 * c][tid] = make_uint4(f.w[0], f.w[1], f.w[2], f.w[3]);
        sa[2 * c + 1][tid] = make_uint4(f.w[4], f.w[5], f.w[6], f.w[7]);
    };
    Xyzz run = G_::inf();
    uint32_t end = seg_off[kb0 + m];
#pragma unroll 1
    for (uint32_t j = 2 * m; j-- > 0;) {  // odd j: run += bucket j / 2; even j: acc += run
        const bool odd = j & 1;
        Xyzz p;  // the other operand is run either way
        if (odd) {
            const uint32_t s0 = seg_off[kb0 + (j >> 1)];
            const bool empty = s0 == end;
            end = s0;
            if (empty)
                continue;
            const uint4 *src = seg_sum + 8 * (size_t)s0;
            p = Xyzz{ldg_fe(src), ldg_fe(src + 2), ldg_fe(src + 4), ldg_fe(src + 6)};
        } else {
            p = Xyzz{ld(0), ld(1), ld(2), ld(3)};
        }
        if (G_::is_inf(run)) {
            if (odd)
                run = p;
            continue;
        }
        if (G_::is_inf(p)) {
            p = run;
        } else {
            const int c = G_::add_lean(p, p, run);
            if (c)
                p = c == 2 ? G_::inf() : G_::dbl(run);
        }
        if (odd) {
            run = p;
        } else {
            st(0, p.X);
            st(1, p.Y);
            st(2, p.ZZ);
            st(3, p.ZZZ);
        }
    }
    uint4 *o = out + 16 * (size_t)gid;
#pragma unroll
    for (int c = 0; c < 8; c++)
        o[c] = sa[c][tid];
    stg_xyzz(o + 8, run);
}

// Level 2 spreads each window's T groups over chunks of up to RED_CHUNK groups,
// one block per chunk (k_window_chunks), then adds the chunks of a window
// (k_window_sum).  Both use one identity: for points x_0..x_{m-1},
//     sum_i i x_i = sum_{i >= 1} X_i,   X_i = sum_{j >= i} x_j,
// where the suffix sums X_i come from a scan over the threads of a block.
// Chunk b of window k (groups from t0 = b RED_CHUNK) yields
//     C_b = sum_t acc_t + m0 sum_t (t - t0) run_t,     R_b = sum_t run_t,
// and the window sum is S = sum_b C_b + m0 RED_CHUNK sum_b b R_b.  Each step
// is a short running sum, a log-depth scan or tree, and log2 of a power of two
// doublings: no scalar multiples by group index.
// Both kernels work on quads (hs_quad.cuh): with one thread per point, an
// addition's 14 products in sequence set their time (113 + 71 us on F_p and 171 +
// 115 us on F_q for one MSM of 2^20 points).

// inclusive suffix scan over the first nt quads of the block (sh: one point per
// quad); quad g holds r and returns sum_{h >= g} r_h
template <class C>
__device__ __forceinline__ Fe block_suffix_scan(const Quad<C> &op, uint4 *sh, Fe r, uint32_t g, uint32_t nt)
{
    using Q = Quad<C>;
    Q::store(sh, g, op.j, r);
    __syncthreads();
    for (uint32_t dl = 1; dl < nt; dl <<= 1) {
        const bool take = g + dl < nt;
        const Fe o = take ? Q::load(sh, g + dl, op.j) : C::F::zero();
        __syncthreads();
        if (__any_sync(Q::ALL, take)) {
            r = op.template add<false>(r, o, take);
            Q::store(sh, g, op.j, r);
        }
        __syncthreads();
    }
    return r;
}

// sum of v over the first nt (a power of two) quads; quad 0 returns it
template <class C>
__device__ __forceinline__ Fe block_tree_sum(const Quad<C> &op, uint4 *sh, Fe v, uint32_t g, uint32_t nt)
{
    using Q = Quad<C>;
    Q::store(sh, g, op.j, v);
    __syncthreads();
    for (uint32_t stride = nt / 2; stride > 0; stride >>= 1) {
        if ((g & ~7u) < stride) {  // whole warps
            const bool take = g < stride;
            const Fe o = take ? Q::load(sh, g + stride, op.j) : C::F::zero();
            v = op.template add<false>(v, o, take);
        }
        __syncthreads();
        if (g < stride)
            Q::store(sh, g, op.j, v);
        __syncthreads();
    }
    return v;
}

// One step of level 2 on a block: over the nt pairs (acc_t, run_t) at in[lo0 ..],
//     sum_t acc_t + mult sum_t t run_t   (returned on quad 0; mult a power of two),
// and sum_t run_t (quad 0's r).  Quad g first runs a top-down running sum over
// its q consecutive pairs (first one t = g q):
//     r_g = sum run_t,  w_g = sum (t - g q) run_t,  a_g = sum acc_t,
// then the block scans r (X_g = sum_{h >= g} r_h) and quad g contributes
//     a_g + mult (w_g + q X_g [g >= 1]).
template <class C>
__device__ __forceinline__ Fe weighted_sum(const Quad<C> &op, uint4 *sh, const uint4 *__restrict__ in, size_t lo0,
                                           uint32_t nt, uint32_t q, uint32_t mult, Fe &r)
{
    using F = typename C::F;
    using Q = Quad<C>;
    const uint32_t g = threadIdx.x >> 2, P = nt / q;
    const bool warp_in = (g & ~7u) < P, in_p = g < P;
    Fe a = F::zero(), w = F::zero();
    r = F::zero();
    if (warp_in) {
        const size_t lo = lo0 + (size_t)g * q;
        for (int u = (int)q - 1; u >= 0; u--) {
            const Fe ta = in_p ? Q::load(in, 2 * (lo + u), op.j) : F::zero();
            const Fe tr = in_p ? Q::load(in, 2 * (lo + u) + 1, op.j) : F::zero();
            a = op.template add<false>(a, ta, in_p);
            r = op.template add<false>(r, tr, in_p);
            if (u > 0)
                w = op.template add<false>(w, r, in_p);
        }
    }
    r = block_suffix_scan<C>(op, sh, r, g, P);
    Fe v = F::zero();
    if (warp_in) {
        v = g >= 1 ? r : F::zero();
        for (uint32_t m = q; m > 1; m >>= 1)
            v = op.dbl(v);
        v = op.template add<false>(v, w, true);
        for (uint32_t m = mult; m > 1; m >>= 1)
            v = op.dbl(v);
        v = op.template add<false>(v, a, true);
    }
    return block_tree_sum<C>(op, sh, v, g, P);
}

// quads of a level-2 block, and groups per quad: RED_CHUNK_Q keeps both the
// sequential part and the scans' extra work small; in a plan of few windows
// (wide: latency-bound) as few as fill the block, so that only the scan is serial
constexpr uint32_t RED_CHUNK_Q = 4;
constexpr uint32_t RED_QUADS = RED_CHUNK / RED_CHUNK_Q;

// DIRECT: every window of the batch is one chunk (T <= RED_CHUNK), so C_b is
// already the window sum and goes straight to S (k_window_sum is skipped).
template <class C, bool DIRECT>
__global__ void __launch_bounds__(RED_QUADS * 4) k_window_chunks(const uint4 *__restrict__ in,
                                                                const MsmDesc *__restrict__ desc, uint32_t M,
                                                                uint4 *__restrict__ outC, int wide)
{
    using Q = Quad<C>;
    __shared__ uint4 sh[RED_QUADS * 8];
    const Q op(threadIdx.x);
    const uint32_t ch = blockIdx.x;
    const uint32_t mi = find_msm(M, ch, [&](uint32_t k) { return desc[k].chunk_base; });
    const MsmDesc d = desc[mi];
    const uint32_t nbk = d.T > RED_CHUNK ? d.T / RED_CHUNK : 1;
    const uint32_t nt = d.T < RED_CHUNK ? d.T : RED_CHUNK;
    const uint32_t q = wide ? (nt > RED_QUADS ? nt / RED_QUADS : 1) : (nt < RED_CHUNK_Q ? nt : RED_CHUNK_Q);
    const uint32_t local = ch - d.chunk_base;
    const uint32_t k = local / nbk, b = local % nbk;
    Fe r;
    const Fe v = weighted_sum<C>(op, sh, in, (size_t)d.group_base + (size_t)k * d.T + (size_t)b * RED_CHUNK, nt, q,
                                 d.m0, r);
    if (threadIdx.x < 4) {
        Q::store(outC, DIRECT ? (size_t)ch : 2 * (size_t)ch, op.j, v);
        if (!DIRECT)
            Q::store(outC, 2 * (size_t)ch + 1, op.j, r);  // quad 0's suffix sum is the chunk's run total
    }
}

template <class C>
__global__ void __launch_bounds__(RED_QUADS * 4) k_window_sum(const uint4 *__restrict__ inC,
                                                             const MsmDesc *__restrict__ desc, uint32_t M,
                                                             uint4 *__restrict__ S)
{
    using Q = Quad<C>;
    __shared__ uint4 sh[RED_QUADS * 8];
    const Q op(threadIdx.x);
    const uint32_t s = blockIdx.x;
    const uint32_t mi = find_msm(M, s, [&](uint32_t k) { return desc[k].win_base; });
    const MsmDesc d = desc[mi];
    const uint32_t nbk = d.T > RED_CHUNK ? d.T / RED_CHUNK : 1;
    const uint32_t q = nbk > RED_QUADS ? nbk / RED_QUADS : 1;
    Fe r;
    const Fe v = weighted_sum<C>(op, sh, inC, (size_t)d.chunk_base + (size_t)(s - d.win_base) * nbk, nbk, q,
                                 d.m0 * RED_CHUNK, r);
    if (threadIdx.x < 4)
        Q::store(S, s, op.j, v);
}

// Level 2 of a plan of many windows: one quad per window, which runs the window's T
// groups down in turn,
//     sum_t acc_t + m0 sum_t t run_t,   sum_t t run_t = sum_{t >= 1} sum_{h >= t} run_h.
// Three additions per group and no scan, tree or barrier: where the windows fill the
// device, this does with some 3 steps of a whole warp per window of 8 groups what
// k_window_chunks' block per window did with 13.  Bound by the multiplier.  GB300: 256
// verifications (as many MSMs a curve) 2.10 -> 1.79 ms, 1024 MSMs of 64 to 65536 points 28.4 ->
// 27.2 ms, 8192 commitments to 228 generators 7.02 -> 6.64 ms, 4096 x 64 points 6.33 |
// 9.73 -> 4.28 | 6.98 ms (Helios | Selene).
// The chain of 3 T additions has to be outweighed by the windows there are, 64 per group
// (GB300, us, Helios: 64 x 512 points, 2752 windows of 8 groups, 527 without and 512
// with; 100 x 2048, 3300 of 16, 1147 and 1098; 40 x 2048, 1320 of 16, 644 and 746;
// 100 x 8192, 2600 of 64, 2658 and 2803).
constexpr int WS_QUADS = 32;
constexpr uint32_t WS_MIN_WINDOWS = 2048;
constexpr uint32_t WS_WINDOWS_PER_GROUP = 64;

template <class C>
__global__ void __launch_bounds__(WS_QUADS * 4) k_window_serial(const uint4 *__restrict__ in,
                                                               const MsmDesc *__restrict__ desc, uint32_t M,
                                                               uint32_t WS, uint4 *__restrict__ S)
{
    using F = typename C::F;
    using Q = Quad<C>;
    const Q op(threadIdx.x);
    const uint32_t s = blockIdx.x * WS_QUADS + (threadIdx.x >> 2);
    uint32_t T = 0, doublings = 0;
    size_t lo = 0;
    if (s < WS) {
        const MsmDesc &d = desc[find_msm(M, s, [&](uint32_t k) { return desc[k].win_base; })];
        T = d.T;
        doublings = d.log2m0;
        lo = (size_t)d.group_base + (size_t)(s - d.win_base) * T;
    }
    const uint32_t tmax = __reduce_max_sync(Q::ALL, T), dmax = __reduce_max_sync(Q::ALL, doublings);
    Fe a = F::zero(), r = F::zero(), w = F::zero();
    for (uint32_t t = tmax; t-- > 0;) {
        const bool take = t < T;
        const Fe ta = take ? Q::load(in, 2 * (lo + t), op.j) : F::zero();
        const Fe tr = take ? Q::load(in, 2 * (lo + t) + 1, op.j) : F::zero();
        a = op.template add<false>(a, ta, take);
        r = op.template add<false>(r, tr, take);
        if (t > 0)
            w = op.template add<false>(w, r, take);
    }
    for (uint32_t m = 0; m < dmax; m++) {
        const Fe x = op.dbl(w);
        w = Q::sel(m < doublings, x, w);
    }
    w = op.template add<false>(w, a, true);
    if (s < WS)
        Q::store(S, s, op.j, w);
}

// ---------------------------------------------------------------------------
// 5. window combination (Horner) -> canonical Jacobian
// ---------------------------------------------------------------------------
constexpr uint32_t COMBINE_MAX_GROUPS = 8;  // a cluster's blocks

template <class C>
__device__ void store_jacobian_canon(uint32_t *out, const Xyzz &p)
{
    using G = Group<C>;
    using F = typename C::F;
    Fe X, Y, Z;
    G::to_jacobian(X, Y, Z, p);
    X = F::canon(X);
    Y = F::canon(Y);
    Z = F::canon(Z);
#pragma unroll
    for (int i = 0; i < 8; i++) {
        out[i] = X.w[i];
        out[8 + i] = Y.w[i];
        out[16 + i] = Z.w[i];
    }
}

// One block of four warps per group of an MSM's windows (hs_lane.cuh), the G groups of
// an MSM a cluster.  The chain's doublings can't be shortened, but its additions can:
// block r of the cluster sums the r-th group from the top by itself, in the time that
// block 0 takes for the top group, and hands the sum to block 0, whose chain goes on
// with one addition per group instead of one per window.  Blocks of a cluster with
// no windows left hand over nothing.
template <class C>
__global__ void __launch_bounds__(128, 1) k_combine(const uint4 *__restrict__ S, const MsmDesc *__restrict__ desc,
                                                   uint32_t *__restrict__ out, uint32_t G)
{
    using F = typename C::F;
    using LF = LaneField<F>;
    __shared__ LaneSlot sl[LNSLOTS];
    __shared__ alignas(16) uint32_t ad[LN_MAX_WINDOWS][48];  // the window sums' limbs, coordinate by coordinate
    __shared__ uint32_t nonzero[LN_MAX_WINDOWS];
    __shared__ alignas(16) uint32_t gsum[COMBINE_MAX_GROUPS][48];  // block 0: the groups' sums
    __shared__ uint32_t gnonzero[COMBINE_MAX_GROUPS];
    const uint32_t mi = blockIdx.x / G, rank = blockIdx.x - mi * G;
    const MsmDesc d = desc[mi];
    if (d.Wr == 1 && d.shift == 0) {  // one window (fixed base): nothing to combine
        if (rank == 0 && threadIdx.x == 0)
            store_jacobian_canon<C>(out + 24 * (size_t)mi, load_xyzz(S + 8 * (size_t)d.win_base));
        return;
    }
    const uint32_t per = (d.Wr + G - 1) / G;
    const uint32_t top = d.Wr > rank * per ? d.Wr - rank * per : 0;  // this block's windows: [low, top)
    const uint32_t low = top > per ? top - per : 0;
    const uint4 *Sm = S + 8 * ((size_t)d.win_base + low);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    LaneHorner<C> h(sl, lane, warp);
    for (uint32_t i = threadIdx.x; i < sizeof(sl) / 4; i += blockDim.x)
        reinterpret_cast<uint32_t *>(sl)[i] = 0;
    // every window sum's limbs up front (the chain then waits for no global load)
    for (uint32_t i = warp; i < 4 * (top - low); i += 4) {
        const uint32_t k = i >> 2, c = i & 3;
        const Fe v = load_fe(Sm + 8 * (size_t)k + 2 * c);
        const uint32_t limb = LF::from_fe(v, lane);
        if (lane < 12)
            ad[k][12 * c + lane] = limb;
        if (c == 2 && lane == 0)
            nonzero[k] = F::is_exact_zero(v) ? 0u : 1u;
    }
    __syncthreads();
    bool ident = true;
    const auto step = [&](uint32_t doublings, const uint32_t *a, uint32_t nz) {
        if (!ident)
            for (uint32_t i = 0; i < doublings; i++)
                h.dbl();
        if (!nz)
            return;
        if (ident) {
            h.take(a);
            ident = false;
            return;
        }
        const int r = h.add(a);
        if (r == 1) {  // equal operands: double
            __syncthreads();
            h.dbl();
        } else if (r == 2) {  // they cancel
            ident = true;
        }
    };
    for (uint32_t k = top - low; k-- > 0;)
        step(d.c, ad[k], nonzero[k]);
    if (G > 1) {
        namespace cg = cooperative_groups;
        cg::cluster_group cluster = cg::this_cluster();
        cluster.sync();  // block 0 runs and its shared memory may be written
        if (rank) {
            __syncthreads();
            // coordinate `warp` in exact limbs, as a window sum's
            const LaneSlot &co = sl[warp == 0 ? LX0 + h.x : warp == 1 ? LY : warp == 2 ? LZZ : LZZZ];
            const uint32_t limb = LF::from_fe(LF::to_fe(warp == 3 ? h.f.own_w(co) : h.f.own(co)), lane);
            uint32_t *dst = cluster.map_shared_rank(&gsum[0][0], 0);
            if (lane < 12)
                dst[48 * rank + 12 * warp + lane] = limb;
            if (threadIdx.x == 0)
                *cluster.map_shared_rank(&gnonzero[rank], 0) = ident ? 0u : 1u;
        }
        cluster.sync();
        if (rank)
            return;
        for (uint32_t r = 1, t = low; t; r++) {  // group r: windows [t - size, t)
            const uint32_t size = t < per ? t : per;
            step(d.c * size, gsum[r], gnonzero[r]);
            t -= size;
        }
    }
    if (!ident)
        for (uint32_t i = 0; i < d.shift; i++)  // upper window-split half: times 2^(c w_lo)
            h.dbl();
    __syncthreads();
    if (warp == 0) {
        Xyzz t = Group<C>::inf();
        if (!ident) {
            t.X = LF::to_fe(h.f.own(sl[LX0 + h.x]));
            t.Y = LF::to_fe(h.f.own(sl[LY]));
            t.ZZ = LF::to_fe(h.f.own(sl[LZZ]));
            t.ZZZ = LF::to_fe(h.f.own_w(sl[LZZZ]));
        }
        if (lane == 0)
            store_jacobian_canon<C>(out + 24 * (size_t)mi, t);
    }
}

// Groups of windows per MSM, while every block has an SM to itself: two on one slow each
// other's chains by more than the additions were worth (GB300, 64-point MSMs, Helios |
// Selene, us: 19 of them 369 | 499 without groups, 360 | 488 with; 38 of them 423 |
// 562 and 426 | 600).  With them one MSM of 16 points from host memory takes 267 us
// instead of 289, 65521 encodings 945 instead of 962.  By width, without and with (one
// MSM, Helios | Selene, us): 33 windows of 8 bits 299 | 403 and 272 | 361; 26 of 10 bits
// 475 | 626 and 452 | 593; 20 of 13 bits 559 | 730 and 544 | 707; 17 of 16 bits 841 | 1110
// and 832 | 1115; 15 of 18 bits 1370 | 1935 and 1363 | 1927.
static uint32_t combine_groups(const BatchPlan &p, int sm_count)
{
    uint32_t wr = 1;
    for (const MsmDesc &d : p.msms)
        wr = std::max(wr, d.Wr);
    const uint32_t G = wr >= 28 ? COMBINE_MAX_GROUPS : wr >= 16 ? 5 : wr >= 8 ? 3 : 1;
    return (uint64_t)p.M * G <= (uint64_t)sm_count ? G : 1;
}

template <class C>
static cudaError_t launch_combine(Context &ctx, const BatchPlan &p, const BatchBuffers &b, cudaStream_t st)
{
    const uint32_t G = combine_groups(p, ctx.sm_count);
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = G;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(p.M * G);
    cfg.blockDim = dim3(128);
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, k_combine<C>, (const uint4 *)b.redS, (const MsmDesc *)b.desc,
                                             (uint32_t *)b.out_jac, G);
    if (e != cudaSuccess)
        return e;
    HS_LAUNCH_CHECK(ctx);
    return cudaSuccess;
}

// Window sums of a plan of few windows of at most WQ_MAX_B buckets, where the
// two-level reduction's chains of additions set the time: one block of WQ_QUADS
// four-lane quads per window, quad g taking the q = B / quads buckets
// [g q, (g + 1) q):
//     run_g = sum_j B_j,   acc_g = sum_j (j - g q + 1) B_j   (top-down running sum),
// then S = sum_g acc_g + q sum_{g >= 1} R_g with R_g = sum_{h >= g} run_h (a
// suffix scan over the quads), q R_g by doublings, and a tree sum.  Additions
// that no quad of a warp needs (empty buckets, identities) are skipped.
constexpr int WQ_QUADS = 64;
constexpr uint32_t WQ_MAX_B = 256;

template <class C>
__global__ void __launch_bounds__(WQ_QUADS * 4) k_window_quads(const uint32_t *__restrict__ seg_off,
                                                              const uint4 *__restrict__ seg_sum,
                                                              const MsmDesc *__restrict__ desc, uint32_t M,
                                                              uint4 *__restrict__ S)
{
    using F = typename C::F;
    using Q = Quad<C>;
    __shared__ uint4 sh[WQ_QUADS * 8];
    const uint32_t s = blockIdx.x;
    const uint32_t mi = find_msm(M, s, [&](uint32_t k) { return desc[k].win_base; });
    const MsmDesc d = desc[mi];
    const uint32_t k = s - d.win_base;
    const uint32_t g = threadIdx.x >> 2;
    const Q op(threadIdx.x);
    const uint32_t nga = d.B < (uint32_t)WQ_QUADS ? d.B : (uint32_t)WQ_QUADS;  // B is a power of two
    const uint32_t q = d.B / nga;
    const bool active = g < nga;
    Fe run = F::zero(), acc = F::zero();
    for (int u = (int)q - 1; u >= 0; u--) {
        Fe t = F::zero();
        bool take = false;
        if (active) {
            const uint32_t kb = d.bucket_base + k * d.B + g * q + (uint32_t)u;
            const uint32_t s0 = seg_off[kb];
            take = seg_off[kb + 1] != s0;
            if (take)
                t = Q::load(seg_sum, s0, op.j);
        }
        if (__any_sync(Q::ALL, take))
            run = op.template add<false>(run, t, take);
        const bool more = !Q::is_inf(run);
        if (__any_sync(Q::ALL, more))
            acc = op.template add<false>(acc, run, more);
    }
    Q::store(sh, g, op.j, run);
    __syncthreads();
    for (uint32_t dl = 1; dl < nga; dl <<= 1) {  // R_g
        bool take = g + dl < nga;
        const Fe o = take ? Q::load(sh, g + dl, op.j) : F::zero();
        const bool o_inf = Q::is_inf(o);
        take = take && !o_inf;
        __syncthreads();
        if (__any_sync(Q::ALL, take)) {
            run = op.template add<false>(run, o, take);
            Q::store(sh, g, op.j, run);
        }
        __syncthreads();
    }
    // v_g = q R_g [g >= 1] + acc_g
    Fe v = g >= 1 ? run : F::zero();
    for (uint32_t m = q; m > 1; m >>= 1)
        v = op.dbl(v);
    v = op.template add<false>(v, acc, true);
    Q::store(sh, g, op.j, v);
    __syncthreads();
    for (uint32_t st = nga / 2; st > 0; st >>= 1) {
        if ((threadIdx.x >> 5) * 8 < st) {  // whole warps
            const bool take = g < st;
            const Fe o = take ? Q::load(sh, g + st, op.j) : F::zero();
            v = op.template add<false>(v, o, take);
        }
        __syncthreads();
        if (g < st)
            Q::store(sh, g, op.j, v);
        __syncthreads();
    }
    if (g == 0)
        Q::store(S, s, op.j, v);
}

// Bucket accumulation of small plans on quads (a mixed addition is 4 product stages
// against 10 products on one thread), one quad per segment.  16 product slots per
// entry against 10, so only for plans of at most ACC_QUADS_MAX_ENTRIES entries.
constexpr uint64_t ACC_QUADS_MAX_ENTRIES = 98304;

template <class C>
__global__ void __launch_bounds__(128) k_accumulate_quads(const uint4 *__restrict__ segs,
                                                         const uint32_t *__restrict__ seg_lo,
                                                         const uint32_t *__restrict__ seg_hi,
                                                         const uint32_t *__restrict__ sorted,
                                                         const uint4 *__restrict__ pts, uint4 *__restrict__ seg_sum)
{
    using F = typename C::F;
    using Q = Quad<C>;
    const Q op(threadIdx.x);
    const uint32_t S0 = *seg_lo, S = *seg_hi;
    const uint32_t stride = gridDim.x * (blockDim.x >> 2);
    // a warp's eight quads take consecutive segments and leave the loop together
    for (uint32_t w = S0 + blockIdx.x * (blockDim.x >> 2) + (threadIdx.x >> 5) * 8; w < S; w += stride) {
        const uint32_t s = w + ((threadIdx.x >> 2) & 7);
        const uint4 d = s < S ? segs[s] : make_uint4(0, 0, 0, 0);  // start, length, destination slot
        const uint32_t len = __reduce_max_sync(Q::ALL, d.y);
        Fe acc = F::zero();
        for (uint32_t i = 0; i < len; i++) {
            bool take = i < d.y;
            Fe c = F::zero();
            uint32_t e = 0;
            if (take) {
                e = __ldg(sorted + d.x + i);
                if (op.j < 2) {
                    const uint4 *src = pts + 4 * (size_t)(e & 0x7fffffffu) + 2 * op.j;
                    const uint4 a = __ldg(src), b = __ldg(src + 1);
                    c = Fe{{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w}};
                }
            }
            // an identity base contributes nothing (both flags on every lane: they are shuffles)
            const bool z = F::is_exact_zero(c);
            const bool zx = Q::flag(z, 0), zy = Q::flag(z, 1);
            take = take && !(zx && zy);
            if (op.j == 1 && (e >> 31))
                c = F::neg(c);
            if (__any_sync(Q::ALL, take))
                acc = op.template add<true>(acc, c, take);
        }
        if (s < S)
            Q::store(seg_sum, d.z, op.j, acc);
    }
}

template <class C>
cudaError_t msm_tail(Context &ctx, const BatchPlan &p, const BatchBuffers &b)
{
    cudaStream_t st = ctx.stream;
    // a small plan: accumulation on quads
    const bool small = !p.ba_rounds && !p.part_slice && p.entries_bound <= ACC_QUADS_MAX_ENTRIES;
    // 2. accumulate: a grid of short blocks (up to 32 per SM, several waves), each
    //    thread taking segments at a stride of the grid.  Segments come longest
    //    first, so every block gets a like mix of long and short ones; blocks end
    //    wave by wave, so kernels of other streams (another MSM's tail) get SM
    //    slots while this one runs.  Threads past the device-side count exit.
    if (p.ba_rounds) {
        // Host inputs in two parts: bucket k's part-j entries form list NB*j + k
        // (offsets has 2 NB + 1 entries), so each part's lists are one range of
        // every level; its rounds and its fold run once that part is in, and
        // the first part-1 segment of a bucket continues its part-0 sum.
        const int parts = p.part_slice ? 2 : 1;
        const size_t nh = (size_t)(p.L + 1) * p.hist_blocks * (p.part_slice ? 2 : 1);
        const uint32_t *bound[3] = {b.len_scan, b.len_scan + (p.part_slice ? nh / 2 : nh), b.len_scan + nh};
        const uint4 *last = b.ba_lvl[(p.ba_rounds - 1) & 1];
        for (int j = 0; j < parts; j++) {
            if (b.ready[j]) {  // host inputs: this part of the bases arrives on another stream
                const cudaError_t e =
                    cudaStreamWaitEvent(st, b.ready[j], ctx.capturing_host ? cudaEventWaitExternal : 0);
                if (e != cudaSuccess)
                    return e;
            }
            cudaEvent_t ev0 = nullptr;
            prof_begin(ctx, &ev0);
            const uint32_t *lo = j ? b.offsets + p.NB : nullptr;
            const uint32_t *hi = b.offsets + (size_t)p.NB * (j + 1);
            for (uint32_t r = 1; r <= p.ba_rounds; r++) {
                const uint4 *in_lvl = r == 1 ? nullptr : b.ba_lvl[(r - 2) & 1];
                uint4 *out_lvl = b.ba_lvl[(r - 1) & 1];
                const uint32_t blocks = std::max<uint32_t>(1, p.ba_blocks[r - 1]);
                const uint32_t iblocks = (uint32_t)(((uint64_t)blocks * BA_BT + BA_G * BA_INV_BT - 1) / (BA_G * BA_INV_BT));
                if (r == 1)
                    k_ba_pairs<C, true><<<blocks, BA_BT, 0, st>>>(lo, hi, r, b.sorted, b.points, in_lvl, b.ba_pre,
                                                                  b.ba_tot);
                else
                    k_ba_pairs<C, false><<<blocks, BA_BT, 0, st>>>(lo, hi, r, b.sorted, b.points, in_lvl, b.ba_pre,
                                                                   b.ba_tot);
                HS_LAUNCH_CHECK(ctx);
                k_ba_invert<C><<<iblocks, BA_INV_BT, 0, st>>>(lo, hi, r, b.ba_tot);
                HS_LAUNCH_CHECK(ctx);
                if (r == 1)
                    k_ba_finish<C, true><<<blocks, BA_BT, 0, st>>>(lo, hi, r, b.sorted, b.points, in_lvl, b.ba_pre,
                                                                   b.ba_tot, out_lvl);
                else
                    k_ba_finish<C, false><<<blocks, BA_BT, 0, st>>>(lo, hi, r, b.sorted, b.points, in_lvl,
                                                                    b.ba_pre, b.ba_tot, out_lvl);
                HS_LAUNCH_CHECK(ctx);
            }
            const int threads = 128;
            const uint64_t want = (p.max_segs + threads - 1) / threads;
            const int blocks = (int)std::max<uint64_t>(1, std::min<uint64_t>(want, (uint64_t)ctx.sm_count * 32));
            if (j == 0)
                k_accumulate_level<C, false><<<blocks, threads, 0, st>>>(b.segs, bound[0], bound[1], last, b.seg_sum);
            else
                k_accumulate_level<C, true><<<blocks, threads, 0, st>>>(b.segs, bound[1], bound[2], last, b.seg_sum);
            HS_LAUNCH_CHECK(ctx);
            prof_end(ctx, ev0, j == 0 ? p.entries_pinned : 0);
        }
    } else if (small) {
        const uint64_t want = (p.max_segs + 31) / 32;
        const int blocks = (int)std::max<uint64_t>(1, std::min<uint64_t>(want, (uint64_t)ctx.sm_count * 8));
        const size_t nh = (size_t)(p.L + 1) * p.hist_blocks;
        if (b.ready[0]) {  // host inputs: the bases arrive on another stream
            const cudaError_t e = cudaStreamWaitEvent(st, b.ready[0], ctx.capturing_host ? cudaEventWaitExternal : 0);
            if (e != cudaSuccess)
                return e;
        }
        cudaEvent_t ev0 = nullptr;
        prof_begin(ctx, &ev0);
        k_accumulate_quads<C><<<blocks, 128, 0, st>>>(b.segs, b.len_scan, b.len_scan + nh, b.sorted, b.points,
                                                      b.seg_sum);
        HS_LAUNCH_CHECK(ctx);
        prof_end(ctx, ev0, p.entries_pinned);
    } else {
        const int threads = 128;
        const uint64_t want = (p.max_segs + threads - 1) / threads;
        const int blocks = (int)std::max<uint64_t>(1, std::min<uint64_t>(want, (uint64_t)ctx.sm_count * 32));
        // the segment lists: [0, total), or per part [0, P1) and [P1, total) with P1
        // the scan position where the part-1 histogram starts
        const size_t nh = (size_t)(p.L + 1) * p.hist_blocks * (p.part_slice ? 2 : 1);
        const int parts = p.part_slice ? 2 : 1;
        const uint32_t *bound[3] = {b.len_scan, b.len_scan + (p.part_slice ? nh / 2 : nh), b.len_scan + nh};
        for (int j = 0; j < parts; j++) {
            if (b.ready[j]) {  // host inputs: this part of the bases arrives on another stream
                const cudaError_t e = cudaStreamWaitEvent(st, b.ready[j], ctx.capturing_host ? cudaEventWaitExternal : 0);
                if (e != cudaSuccess)
                    return e;
            }
            cudaEvent_t ev0 = nullptr;
            prof_begin(ctx, &ev0);
            if (j == 0)
                k_accumulate<C, false><<<blocks, threads, 0, st>>>(b.segs, bound[0], bound[1], b.sorted, b.points,
                                                                   b.seg_sum);
            else
                k_accumulate<C, true><<<blocks, threads, 0, st>>>(b.segs, bound[1], bound[2], b.sorted, b.points,
                                                                  b.seg_sum);
            HS_LAUNCH_CHECK(ctx);
            prof_end(ctx, ev0, j == 0 ? p.entries_pinned : 0);
        }
    }
    // 3. merge multi-segment buckets: a bucket holds at most one entry per point (per
    //    point and window in a fixed-base MSM), so plans of few points have none, or
    //    none of more than HEAVY_MIN segments
    constexpr uint32_t HEAVY_MIN = 8;
    uint64_t most = 0;
    for (const MsmDesc &d : p.msms)
        most = std::max<uint64_t>(most, (uint64_t)d.n * (d.fixed ? d.w_cnt : 1u));
    if (p.ba_rounds || most > p.L) {
        const bool any_heavy = p.ba_rounds || most > (uint64_t)HEAVY_MIN * p.L;
        if (any_heavy) {
            cudaError_t e = cudaMemsetAsync(b.heavy_n, 0, sizeof(uint32_t), st);
            if (e != cudaSuccess)
                return e;
        }
        const unsigned mb =
            (unsigned)std::max<uint32_t>(1, std::min<uint32_t>((p.NB + 31) / 32, (uint32_t)ctx.sm_count * 64));
        k_merge<C><<<mb, 128, 0, st>>>(b.seg_off, p.NB, b.seg_sum, b.heavy, b.heavy_n, HEAVY_MIN);
        HS_LAUNCH_CHECK(ctx);
        if (any_heavy) {
            k_merge_heavy<C><<<ctx.sm_count, HEAVY_QUADS * 4, 0, st>>>(b.seg_off, b.heavy, b.heavy_n, b.seg_sum);
            HS_LAUNCH_CHECK(ctx);
        }
    }
    // 4. bucket reduction: group running sums, then one block per window; a
    //    plan of few windows of at most WQ_MAX_B buckets reduces each window on
    //    one block of quads
    if (p.max_B <= WQ_MAX_B && p.WS <= 4u * (uint32_t)ctx.sm_count) {
        k_window_quads<C><<<p.WS, WQ_QUADS * 4, 0, st>>>(b.seg_off, b.seg_sum, b.desc, p.M, b.redS);
        HS_LAUNCH_CHECK(ctx);
    } else {
        const int threads = 128;
        k_reduce_groups<C><<<(p.G + threads - 1) / threads, threads, 0, st>>>(b.seg_off, b.seg_sum, b.desc, p.M,
                                                                            p.G, b.redA);
        HS_LAUNCH_CHECK(ctx);
        if (p.WS >= std::max(WS_MIN_WINDOWS, WS_WINDOWS_PER_GROUP * p.max_T)) {
            k_window_serial<C><<<(p.WS + WS_QUADS - 1) / WS_QUADS, WS_QUADS * 4, 0, st>>>(b.redA, b.desc, p.M, p.WS,
                                                                                        b.redS);
            HS_LAUNCH_CHECK(ctx);
            return launch_combine<C>(ctx, p, b, st);
        }
        // A plan of few chunks (one or a few MSMs) is latency-bound, and so are
        // windows of at most 16 groups: one quad per group up to RED_QUADS groups.
        // Many chunks of more groups (a batch of larger MSMs) fill the device, and
        // RED_CHUNK_Q groups per quad keep the scans' extra work small.  (Measured with
        // one thread where a quad is now: 256 verifications, 16 groups per window, 51k ->
        // 65k per second with one group each; 1024 MSMs of 64 to 65536 points 1.5% faster
        // with four.)
        const int wide = p.CH <= 4u * (uint32_t)ctx.sm_count || p.max_T <= 16;
        const uint32_t t2 =
            std::max<uint32_t>(32, 4 * std::min<uint32_t>(RED_QUADS, wide ? p.max_T : p.max_T / RED_CHUNK_Q));
        if (p.max_nbk == 1) {  // one chunk per window: chunk index == window slot
            k_window_chunks<C, true><<<p.CH, t2, 0, st>>>(b.redA, b.desc, p.M, b.redS, wide);
            HS_LAUNCH_CHECK(ctx);
        } else {
            k_window_chunks<C, false><<<p.CH, t2, 0, st>>>(b.redA, b.desc, p.M, b.redC, wide);
            HS_LAUNCH_CHECK(ctx);
            const uint32_t t3 = std::max<uint32_t>(32, 4 * std::min<uint32_t>(RED_QUADS, p.max_nbk));
            k_window_sum<C><<<p.WS, t3, 0, st>>>(b.redC, b.desc, p.M, b.redS);
            HS_LAUNCH_CHECK(ctx);
        }
    }
    // 5. Horner over windows, a cluster of blocks of four warps per MSM
    return launch_combine<C>(ctx, p, b, st);
}

// ---------------------------------------------------------------------------
// input conversion: radix-2^51 limbs -> 8 x 32-bit words (weakly reduced)
// ---------------------------------------------------------------------------
template <class C>
__device__ Fe fe_from_51(const uint64_t *l)
{
    using F = typename C::F;
    // sum l_i * 2^(51 i) into five 64-bit words (limbs may exceed 51 bits)
    unsigned __int128 acc = 0;
    uint64_t w[5];
    // word j covers bits [64j, 64j+64)
    unsigned __int128 v0 = (unsigned __int128)l[0];
    unsigned __int128 v1 = (unsigned __int128)l[1] << 51;  // bits 51..115
    unsigned __int128 v2 = (unsigned __int128)l[2] << 38;  // 102 = 64 + 38
    unsigned __int128 v3 = (unsigned __int128)l[3] << 25;  // 153 = 128 + 25
    unsigned __int128 v4 = (unsigned __int128)l[4] << 12;  // 204 = 192 + 12
    acc = (unsigned __int128)(uint64_t)v0 + (uint64_t)v1;
    w[0] = (uint64_t)acc;
    acc = (acc >> 64) + (uint64_t)(v0 >> 64) + (uint64_t)(v1 >> 64) + (uint64_t)v2;
    w[1] = (uint64_t)acc;
    acc = (acc >> 64) + (uint64_t)(v2 >> 64) + (uint64_t)v3;
    w[2] = (uint64_t)acc;
    acc = (acc >> 64) + (uint64_t)(v3 >> 64) + (uint64_t)v4;
    w[3] = (uint64_t)acc;
    acc = (acc >> 64) + (uint64_t)(v4 >> 64);
    w[4] = (uint64_t)acc;  // < 2^13
    Fe r;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        r.w[2 * i] = (uint32_t)w[i];
        r.w[2 * i + 1] = (uint32_t)(w[i] >> 32);
    }
    // fold w[4] * 2^256 == w[4] * c, one bit at a time (w[4] is tiny, usually 0)
    uint64_t top = w[4];
    Fe c1 = F::zero();
    F::add_c_masked(c1, 0xffffffffu);  // c1 = c = 2^256 mod m
    while (top) {
        if (top & 1)
            r = F::add(r, c1);
        c1 = F::dbl(c1);
        top >>= 1;
    }
    return r;
}

template <class C>
__device__ void fe_to_51(uint64_t *l, const Fe &canon)
{
    uint64_t w[4];
#pragma unroll
    for (int i = 0; i < 4; i++)
        w[i] = (uint64_t)canon.w[2 * i] | ((uint64_t)canon.w[2 * i + 1] << 32);
    const uint64_t M51 = (1ull << 51) - 1;
    l[0] = w[0] & M51;
    l[1] = ((w[0] >> 51) | (w[1] << 13)) & M51;
    l[2] = ((w[1] >> 38) | (w[2] << 26)) & M51;
    l[3] = ((w[2] >> 25) | (w[3] << 39)) & M51;
    l[4] = (w[3] >> 12) & M51;
}

// batch Jacobian -> affine: each thread owns a chunk, multiplies the Z values
// that are neither 0 nor 1 (Montgomery's trick, fp/include/fp_batch_invert.h:61-114),
// inverts the chunk product once and walks back.  Identity (Z == 0) -> (0,0).
constexpr int AFF_CHUNK = 16;

template <class C>
__global__ void k_jac_to_affine(const uint64_t *__restrict__ in, int fmt, size_t n, uint4 *__restrict__ out,
                                uint4 *__restrict__ scratch)
{
    using F = typename C::F;
    // thread t takes points t, t + T, t + 2T, ... (T threads in the grid, at most
    // AFF_CHUNK points each): a warp reads consecutive records
    const size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    const size_t T = (size_t)gridDim.x * blockDim.x;
    if (t >= n)
        return;
    const size_t cnt = (n - t + T - 1) / T;
    const size_t stride = (fmt == HS_FMT_JACOBIAN51) ? 15 : (fmt == HS_FMT_AFFINE51 ? 10 : 8);
    // pass 1: prefix products of the Z values that need inverting
    Fe run = F::one();
    bool any = false;
    for (size_t j = 0; j < cnt; j++) {
        const size_t i = t + j * T;
        Fe z;
        if (fmt == HS_FMT_JACOBIAN51) {
            z = fe_from_51<C>(in + stride * i + 10);
            Fe zc = F::canon(z);
            bool is0 = F::is_exact_zero(zc);
            Fe one = F::one();
            bool is1 = true;
#pragma unroll
            for (int k = 0; k < 8; k++)
                is1 = is1 && (zc.w[k] == one.w[k]);
            if (!is0 && !is1) {
                run = F::mul(run, z);
                any = true;
            }
        }
        store_fe(scratch + 2 * i, run);
    }
    Fe inv = any ? F::inv(run) : F::one();
    // pass 2: walk back
    for (size_t j = cnt; j-- > 0;) {
        const size_t i = t + j * T;
        Fe x, y;
        if (fmt == HS_FMT_JACOBIAN51) {
            x = fe_from_51<C>(in + stride * i);
            y = fe_from_51<C>(in + stride * i + 5);
        } else if (fmt == HS_FMT_AFFINE51) {
            x = fe_from_51<C>(in + stride * i);
            y = fe_from_51<C>(in + stride * i + 5);
        } else {
            const uint4 *src = reinterpret_cast<const uint4 *>(in) + 4 * i;
            x = load_fe(src);
            y = load_fe(src + 2);
        }
        bool ident = false;
        if (fmt == HS_FMT_JACOBIAN51) {
            Fe z = fe_from_51<C>(in + stride * i + 10);
            Fe zc = F::canon(z);
            bool is0 = F::is_exact_zero(zc);
            Fe one = F::one();
            bool is1 = true;
#pragma unroll
            for (int k = 0; k < 8; k++)
                is1 = is1 && (zc.w[k] == one.w[k]);
            if (is0) {
                ident = true;
            } else if (!is1) {
                Fe prev = (j > 0) ? load_fe(scratch + 2 * (i - T)) : F::one();
                Fe zi = F::mul(inv, prev);  // 1/z
                inv = F::mul(inv, z);
                Fe zi2 = F::sqr(zi);
                x = F::mul(x, zi2);
                y = F::mul(y, F::mul(zi2, zi));
            }
        } else {
            Fe xc = F::canon(x), yc = F::canon(y);
            ident = F::is_exact_zero(xc) && F::is_exact_zero(yc);
        }
        if (ident) {
            x = F::zero();
            y = F::zero();
        }
        store_fe(out + 4 * i, F::canon(x));
        store_fe(out + 4 * i + 2, F::canon(y));
    }
}

template <class C>
cudaError_t decompress(Context &ctx, const void *d_in, size_t n, uint4 *d_out, uint8_t *d_valid, uint32_t *d_bad);

// HS_FMT_COMPRESSED input decodes on the device; the count of invalid
// encodings is left in the first word of scratch for the caller to check.
template <class C>
cudaError_t to_affine(Context &ctx, const void *d_in, int fmt, size_t n, uint4 *d_out, void *scratch)
{
    if (n == 0)
        return cudaSuccess;
    if (fmt == HS_FMT_COMPRESSED) {
        cudaError_t e = cudaMemsetAsync(scratch, 0, sizeof(uint32_t), ctx.stream);
        if (e != cudaSuccess)
            return e;
        return decompress<C>(ctx, d_in, n, d_out, nullptr, static_cast<uint32_t *>(scratch));
    }
    const size_t chunks = (n + AFF_CHUNK - 1) / AFF_CHUNK;
    const int threads = 128;
    k_jac_to_affine<C><<<(unsigned)((chunks + threads - 1) / threads), threads, 0, ctx.stream>>>(
        reinterpret_cast<const uint64_t *>(d_in), fmt, n, d_out, reinterpret_cast<uint4 *>(scratch));
    HS_LAUNCH_CHECK(ctx);
    return cudaSuccess;
}

inline size_t to_affine_scratch(size_t n) { return n * 32; }

// ---------------------------------------------------------------------------
// output formatting of canonical Jacobians (24 words each)
// ---------------------------------------------------------------------------
template <class C>
__global__ void k_format_out(const uint32_t *__restrict__ jac, size_t count, int fmt, void *__restrict__ out)
{
    using F = typename C::F;
    const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i >= count)
        return;
    Fe X, Y, Z;
#pragma unroll
    for (int k = 0; k < 8; k++) {
        X.w[k] = jac[24 * i + k];
        Y.w[k] = jac[24 * i + 8 + k];
        Z.w[k] = jac[24 * i + 16 + k];
    }
    const bool ident = F::is_zero(Z);
    if (fmt == HS_FMT_JACOBIAN51) {
        uint64_t *o = reinterpret_cast<uint64_t *>(out) + 15 * i;
        fe_to_51<C>(o, F::canon(X));
        fe_to_51<C>(o + 5, F::canon(Y));
        fe_to_51<C>(o + 10, F::canon(Z));
        return;
    }
    Fe x = F::zero(), y = F::zero();
    Fe zc = F::canon(Z);
    bool z_one = zc.w[0] == 1u;
#pragma unroll
    for (int k = 1; k < 8; k++)
        z_one = z_one && zc.w[k] == 0u;
    if (z_one) {
        x = F::canon(X);
        y = F::canon(Y);
    } else if (!ident) {
        Fe zi = F::inv(Z);
        Fe zi2 = F::sqr(zi);
        x = F::canon(F::mul(X, zi2));
        y = F::canon(F::mul(Y, F::mul(zi2, zi)));
    }
    if (fmt == HS_FMT_AFFINE51) {
        uint64_t *o = reinterpret_cast<uint64_t *>(out) + 10 * i;
        fe_to_51<C>(o, x);
        fe_to_51<C>(o + 5, y);
    } else if (fmt == HS_FMT_AFFINE) {
        uint4 *o = reinterpret_cast<uint4 *>(out) + 4 * i;
        store_fe(o, x);
        store_fe(o + 2, y);
    } else {  // compressed: x with parity of y in bit 255
        uint32_t *o = reinterpret_cast<uint32_t *>(out) + 8 * i;
#pragma unroll
        for (int k = 0; k < 8; k++)
            o[k] = x.w[k];
        if (!ident)
            o[7] |= (y.w[0] & 1u) << 31;
    }
}

template <class C>
cudaError_t format_out(Context &ctx, const uint32_t *d_jac, size_t count, int out_fmt, void *d_out)
{
    if (count == 0)
        return cudaSuccess;
    const int threads = 64;
    k_format_out<C><<<(unsigned)((count + threads - 1) / threads), threads, 0, ctx.stream>>>(d_jac, count, out_fmt,
                                                                                           d_out);
    HS_LAUNCH_CHECK(ctx);
    return cudaSuccess;
}

// ---------------------------------------------------------------------------
// simplified SWU map (RFC 9380 6.6.2) as the reference computes it
// (helios/src/x64/helios_map_to_curve.cpp:98-198): output affine, Z = 1.
// ---------------------------------------------------------------------------
// the low 125 bits of (q + 1)/4 as (squarings, then times a^odd), and 3 squarings
constexpr int SQRT_Q_STEPS = 26;
static __constant__ uint8_t SQRT_Q[SQRT_Q_STEPS][2] = {
    {5, 15}, {4, 13}, {4, 15}, {4, 13}, {3, 7}, {9, 11}, {6, 11}, {4, 7}, {3, 3}, {5, 5}, {5, 13}, {5,
    13}, {3, 3}, {8, 13}, {4, 13}, {5, 13}, {4, 11}, {5, 9}, {5, 7}, {6, 9}, {3, 7}, {6, 9}, {6, 15},
    {1, 1}, {7, 15}, {2, 1}};

template <class C>
__device__ bool fsqrt(Fe &r, const Fe &a);

template <>
__device__ inline bool fsqrt<HeliosCurve>(Fe &r, const Fe &a)
{
    // p = 5 (mod 8): x = a^((p+3)/8), (p+3)/8 = 2 (2^251 - 1); if x^2 = -a multiply by
    // sqrt(-1) = 2^((p-1)/4)
    const Fe sqrtm1 = {{0x4a0ea0b0u, 0xc4ee1b27u, 0xad2fe478u, 0x2f431806u,
                        0x3dfbd7a7u, 0x2b4d0099u, 0x4fc1df0bu, 0x2b832480u}};
    Fe x = Fp::sqr(Fp::pow_ones(a, 251));
    Fe x2 = Fp::sqr(x);
    if (!Fp::eq(x2, a)) {
        if (!Fp::eq(x2, Fp::neg(a)))
            return false;
        x = Fp::mul(x, sqrtm1);
    }
    r = x;
    return true;
}

template <>
__device__ inline bool fsqrt<SeleneCurve>(Fe &r, const Fe &a)
{
    // q = 3 (mod 4): x = a^((q+1)/4).  The exponent is 128 ones, then 125 bits taken in
    // 26 windows of at most four bits (odd values: a table of a, a^3, .. a^15): 253
    // squarings and 40 products.  (A table of sixteen powers, one selected per nibble,
    // took 76 products and as many passes over the table: 279 us for 65521
    // encodings against 231 now.)
    Fe odd[8];
    odd[0] = a;
    const Fe a2 = Fq::sqr(a);
#pragma unroll 1
    for (int i = 1; i < 8; i++)
        odd[i] = Fq::mul(odd[i - 1], a2);
    Fe x = Fq::pow_ones(a, 128);
#pragma unroll 1
    for (int i = 0; i < SQRT_Q_STEPS; i++)
        x = Fq::mul(Fq::sqr_n(x, SQRT_Q[i][0]), odd[SQRT_Q[i][1] >> 1]);
    x = Fq::sqr_n(x, 3);
    if (!Fq::eq(Fq::sqr(x), a))
        return false;
    r = x;
    return true;
}

template <class C>
__global__ void k_map_to_curve(const uint4 *__restrict__ u, size_t n, uint4 *__restrict__ out)
{
    using F = typename C::F;
    using G = Group<C>;
    const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    Fe uu = load_fe(u + 2 * i);
    uu.w[7] &= 0x7fffffffu;  // fp_frombytes masks bit 255
    const Fe A = F::neg(F::from_u32(3));
    const Fe Z = (C::SSWU_Z < 0) ? F::neg(F::from_u32((uint32_t)(-C::SSWU_Z))) : F::from_u32((uint32_t)C::SSWU_Z);
    const Fe B = G::b();
    Fe u2 = F::sqr(uu);
    Fe Zu2 = F::mul(Z, u2);
    Fe den = F::add(F::sqr(Zu2), Zu2);
    Fe x1;
    if (F::is_zero(den)) {
        x1 = F::mul(B, F::inv(F::mul(Z, A)));  // B / (Z A)
    } else {
        // x1 = (-B/A) (1 + 1/den) = -B (den + 1) / (A den)
        Fe num = F::neg(F::mul(B, F::add(den, F::one())));
        x1 = F::mul(num, F::inv(F::mul(A, den)));
    }
    Fe gx1 = F::add(F::sub(F::mul(F::sqr(x1), x1), F::add(F::dbl(x1), x1)), B);
    Fe x, y;
    if (fsqrt<C>(y, gx1)) {
        x = x1;
    } else {
        x = F::mul(Zu2, x1);
        Fe gx2 = F::add(F::sub(F::mul(F::sqr(x), x), F::add(F::dbl(x), x)), B);
        fsqrt<C>(y, gx2);
    }
    y = F::canon(y);
    Fe uc = F::canon(uu);
    if ((uc.w[0] & 1u) != (y.w[0] & 1u))
        y = F::canon(F::neg(y));
    store_fe(out + 4 * i, F::canon(x));
    store_fe(out + 4 * i + 2, y);
}

template <class C>
cudaError_t map_to_curve(Context &ctx, const void *d_u, size_t n, uint4 *d_out)
{
    if (n == 0)
        return cudaSuccess;
    const int threads = 64;
    k_map_to_curve<C><<<(unsigned)((n + threads - 1) / threads), threads, 0, ctx.stream>>>(
        reinterpret_cast<const uint4 *>(d_u), n, d_out);
    HS_LAUNCH_CHECK(ctx);
    return cudaSuccess;
}

// ---------------------------------------------------------------------------
// point decoding (helios/src/x64/helios_frombytes.cpp:59-109, selene twin):
// bit 255 is the parity of y; x must be canonical (the reference re-encodes and
// compares); y = sqrt(x^3 - 3x + b), negated when its parity differs.  An
// invalid encoding (x >= m, or no square root: this includes the 32 zero bytes
// of the identity's encoding) gives (0, 0), valid[i] = 0 and one count in *bad.
// ---------------------------------------------------------------------------
template <class C>
__global__ void k_decompress(const uint4 *__restrict__ in, size_t n, uint4 *__restrict__ out,
                             uint8_t *__restrict__ valid, uint32_t *__restrict__ bad)
{
    using F = typename C::F;
    using G = Group<C>;
    const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    Fe x = load_fe(in + 2 * i);
    const uint32_t parity = x.w[7] >> 31;
    x.w[7] &= 0x7fffffffu;
    const Fe xc = F::canon(x);
    bool ok = true;
#pragma unroll
    for (int k = 0; k < 8; k++)
        ok = ok && (xc.w[k] == x.w[k]);
    Fe y = F::zero();
    if (ok) {
        const Fe rhs = F::add(F::sub(F::mul(F::sqr(x), x), F::add(F::dbl(x), x)), G::b());
        ok = fsqrt<C>(y, rhs);
    }
    if (ok) {
        y = F::canon(y);
        if ((y.w[0] & 1u) != parity)
            y = F::canon(F::neg(y));
    } else {
        x = F::zero();
        y = F::zero();
        atomicAdd(bad, 1u);
    }
    store_fe(out + 4 * i, x);
    store_fe(out + 4 * i + 2, y);
    if (valid)
        valid[i] = ok ? 1 : 0;
}

template <class C>
cudaError_t decompress(Context &ctx, const void *d_in, size_t n, uint4 *d_out, uint8_t *d_valid, uint32_t *d_bad)
{
    if (n == 0)
        return cudaSuccess;
    const int threads = 64;
    k_decompress<C><<<(unsigned)((n + threads - 1) / threads), threads, 0, ctx.stream>>>(
        reinterpret_cast<const uint4 *>(d_in), n, d_out, d_valid, d_bad);
    HS_LAUNCH_CHECK(ctx);
    return cudaSuccess;
}

// any input format -> canonical Jacobian (24 words); affine inputs get Z = 1,
// the affine identity (0,0) becomes (1:1:0)
template <class C>
__global__ void k_to_jac24(const uint64_t *__restrict__ in, int fmt, size_t n, uint32_t *__restrict__ out)
{
    using F = typename C::F;
    const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    Fe X, Y, Z;
    if (fmt == HS_FMT_JACOBIAN51) {
        X = fe_from_51<C>(in + 15 * i);
        Y = fe_from_51<C>(in + 15 * i + 5);
        Z = fe_from_51<C>(in + 15 * i + 10);
    } else {
        if (fmt == HS_FMT_AFFINE51) {
            X = fe_from_51<C>(in + 10 * i);
            Y = fe_from_51<C>(in + 10 * i + 5);
        } else {
            const uint4 *src = reinterpret_cast<const uint4 *>(in) + 4 * i;
            X = load_fe(src);
            Y = load_fe(src + 2);
        }
        const bool ident = F::is_zero(X) && F::is_zero(Y);
        Z = ident ? F::zero() : F::one();
        if (ident) {
            X = F::one();
            Y = F::one();
        }
    }
    X = F::canon(X);
    Y = F::canon(Y);
    Z = F::canon(Z);
#pragma unroll
    for (int k = 0; k < 8; k++) {
        out[24 * i + k] = X.w[k];
        out[24 * i + 8 + k] = Y.w[k];
        out[24 * i + 16 + k] = Z.w[k];
    }
}

template <class C>
cudaError_t to_jac24(Context &ctx, const void *d_in, int fmt, size_t n, uint32_t *d_out)
{
    if (n == 0)
        return cudaSuccess;
    const int threads = 128;
    k_to_jac24<C><<<(unsigned)((n + threads - 1) / threads), threads, 0, ctx.stream>>>(
        reinterpret_cast<const uint64_t *>(d_in), fmt, n, d_out);
    HS_LAUNCH_CHECK(ctx);
    return cudaSuccess;
}

template <class C>
__global__ void k_field_op(int op, const uint4 *__restrict__ a, const uint4 *__restrict__ b, size_t n,
                           uint4 *__restrict__ out)
{
    using F = typename C::F;
    const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    const Fe x = load_fe(a + 2 * i);
    const Fe y = (op == 2 || op == 3 || op == 0) ? load_fe(b + 2 * i) : F::zero();
    Fe r;
    switch (op) {
    case 0: r = F::mul(x, y); break;
    case 1: r = F::sqr(x); break;
    case 2: r = F::add(x, y); break;
    case 3: r = F::sub(x, y); break;
    case 4: r = x; break;
    case 5: r = F::inv(x); break;
    default: r = F::neg(x); break;
    }
    store_fe(out + 2 * i, F::canon(r));
}

// The lane-sliced field of the Horner chain, one warp per element: op 7
// a*b, 8 (a - b)(a + b) = a^2 - b^2 (a difference of products in one set of
// columns), 9 a^(2^32) by 32 squarings (repeated products of products), 10 the
// conversion in and out.
template <class C>
__global__ void __launch_bounds__(128) k_field_lane_op(int op, const uint4 *__restrict__ a, const uint4 *__restrict__ b,
                                                      size_t n, uint4 *__restrict__ out)
{
    using F = typename C::F;
    using LF = LaneField<F>;
    __shared__ LaneSlot sl[4][2];
    LaneSlot *w = sl[threadIdx.x >> 5];
    const size_t i = blockIdx.x * (size_t)(blockDim.x / 32) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    for (uint32_t k = lane; k < 2 * sizeof(LaneSlot) / 4; k += 32)
        reinterpret_cast<uint32_t *>(w)[k] = 0;
    if (i >= n)  // whole warps leave together
        return;
    __syncwarp();
    const LF f(lane);
    uint32_t r = LF::from_fe(load_fe(a + 2 * i), lane);
    f.put(w[0], r);
    f.put(w[1], op == 7 || op == 8 ? LF::from_fe(load_fe(b + 2 * i), lane) : 0u);
    __syncwarp();
    switch (op) {
    case 7: r = f.norm(f.cols(w[0], w[1])); break;
    case 8: r = f.norm(f.cols(w[0], w[0]) + f.k - f.cols(w[1], w[1])); break;
    case 9:
        for (int k = 0; k < 32; k++) {
            r = f.norm(f.cols(w[0], w[0]));
            __syncwarp();
            f.put(w[0], r);
            __syncwarp();
        }
        break;
    default: break;
    }
    const Fe v = LF::to_fe(r);
    if (lane == 0)
        store_fe(out + 2 * i, F::canon(v));
}

template <class C>
cudaError_t field_op(Context &ctx, int op, const void *d_a, const void *d_b, size_t n, void *d_out)
{
    if (n == 0)
        return cudaSuccess;
    const int threads = 128;
    if (op >= 7) {
        k_field_lane_op<C><<<(unsigned)((n + 3) / 4), threads, 0, ctx.stream>>>(op, (const uint4 *)d_a,
                                                                               (const uint4 *)d_b, n, (uint4 *)d_out);
        HS_LAUNCH_CHECK(ctx);
        return cudaSuccess;
    }
    k_field_op<C><<<(unsigned)((n + threads - 1) / threads), threads, 0, ctx.stream>>>(
        op, (const uint4 *)d_a, (const uint4 *)d_b, n, (uint4 *)d_out);
    HS_LAUNCH_CHECK(ctx);
    return cudaSuccess;
}

// ---------------------------------------------------------------------------
// fixed-base window tables: table[i*W + k] = 2^(c k) * G_i, affine
// ---------------------------------------------------------------------------
template <class C>
__global__ void k_fb_expand(const uint4 *__restrict__ gens, size_t n, int c, int W, uint4 *__restrict__ tmp)
{
    using G = Group<C>;
    using F = typename C::F;
    const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    Fe x, y;
    load_affine(gens, (uint32_t)i, x, y, wide_points(gens));
    Xyzz acc = (F::is_exact_zero(x) && F::is_exact_zero(y)) ? G::inf() : G::from_affine(x, y);
    for (int k = 0; k < W; k++) {
        store_xyzz(tmp + 8 * ((size_t)i * W + k), acc);
        if (k + 1 < W)
            for (int d = 0; d < c; d++)
                acc = G::dbl(acc);
    }
}

// XYZZ -> affine in chunks of 16 with one inversion per chunk (Montgomery's
// trick on ZZ*ZZZ); identity -> (0,0)
template <class C>
__global__ void k_fb_normalize(const uint4 *__restrict__ tmp, size_t m, uint4 *__restrict__ table,
                               uint4 *__restrict__ prefix)
{
    using G = Group<C>;
    using F = typename C::F;
    const size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    const size_t lo = t * AFF_CHUNK;
    if (lo >= m)
        return;
    const size_t hi = lo + AFF_CHUNK < m ? lo + AFF_CHUNK : m;
    Fe run = F::one();
    for (size_t i = lo; i < hi; i++) {
        const Xyzz p = load_xyzz(tmp + 8 * i);
        if (!G::is_inf(p))
            run = F::mul(run, F::mul(p.ZZ, p.ZZZ));
        store_fe(prefix + 2 * i, run);
    }
    Fe inv = F::inv(run);
    for (size_t i = hi; i-- > lo;) {
        const Xyzz p = load_xyzz(tmp + 8 * i);
        Fe x = F::zero(), y = F::zero();
        if (!G::is_inf(p)) {
            const Fe z = F::mul(p.ZZ, p.ZZZ);
            const Fe prev = (i > lo) ? load_fe(prefix + 2 * (i - 1)) : F::one();
            const Fe zi = F::mul(inv, prev);  // 1 / (ZZ ZZZ)
            inv = F::mul(inv, z);
            x = F::canon(F::mul(p.X, F::mul(p.ZZZ, zi)));
            y = F::canon(F::mul(p.Y, F::mul(p.ZZ, zi)));
        }
        store_fe(table + 4 * i, x);
        store_fe(table + 4 * i + 2, y);
    }
}

template <class C>
cudaError_t fixed_table(Context &ctx, const uint4 *d_gens, size_t n, int c, int W, uint4 *d_tmp, uint4 *d_table)
{
    if (n == 0)
        return cudaSuccess;
    const size_t m = n * (size_t)W;
    uint4 *prefix = d_tmp + 8 * m;  // tmp holds m XYZZ points then m prefix products
    k_fb_expand<C><<<(unsigned)((n + 127) / 128), 128, 0, ctx.stream>>>(d_gens, n, c, W, d_tmp);
    HS_LAUNCH_CHECK(ctx);
    const size_t chunks = (m + AFF_CHUNK - 1) / AFF_CHUNK;
    k_fb_normalize<C><<<(unsigned)((chunks + 127) / 128), 128, 0, ctx.stream>>>(d_tmp, m, d_table, prefix);
    HS_LAUNCH_CHECK(ctx);
    return cudaSuccess;
}

// out = a + b over canonical Jacobians (the two halves of a window-split MSM)
template <class C>
__device__ Xyzz xyzz_from_jac24(const uint32_t *j)
{
    using F = typename C::F;
    using G = Group<C>;
    Fe X, Y, Z;
#pragma unroll
    for (int k = 0; k < 8; k++) {
        X.w[k] = j[k];
        Y.w[k] = j[8 + k];
        Z.w[k] = j[16 + k];
    }
    if (F::is_zero(Z))
        return G::inf();
    Xyzz p;
    p.X = X;
    p.Y = Y;
    p.ZZ = F::sqr(Z);
    p.ZZZ = F::mul(p.ZZ, Z);
    return p;
}

template <class C>
__global__ void k_join(const uint32_t *__restrict__ a, const uint32_t *__restrict__ b, size_t count,
                       uint32_t *__restrict__ out)
{
    using G = Group<C>;
    const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i >= count)
        return;
    store_jacobian_canon<C>(out + 24 * i, G::add(xyzz_from_jac24<C>(a + 24 * i), xyzz_from_jac24<C>(b + 24 * i)));
}

template <class C>
cudaError_t join(Context &ctx, const uint32_t *d_a, const uint32_t *d_b, size_t count, uint32_t *d_out)
{
    if (count == 0)
        return cudaSuccess;
    const int threads = 64;
    k_join<C><<<(unsigned)((count + threads - 1) / threads), threads, 0, ctx.stream>>>(d_a, d_b, count, d_out);
    HS_LAUNCH_CHECK(ctx);
    return cudaSuccess;
}

// ---------------------------------------------------------------------------
// independent variable-time scalar multiplications s_i * P_i
// (helios/include/helios_scalarmult_vartime.h:39-57, the n = 1 case of the MSM)
// ---------------------------------------------------------------------------
// One thread per pair, from the top digit four doublings and one addition per signed
// 4-bit digit.  With s' = s + 8 (1 + 16 + 16^2 + ...) the digits are the nibbles of s'
// less 8, in [-8, 7], and the carry of s' is the top digit.  The chain is in
// Jacobian coordinates (a doubling 3M + 5S against XYZZ's 7M + 2S, and 24 registers
// less); the table P..8P keeps each entry's Z^2 and Z^3, so that an addition is
// 11M + 3S.  2^17 pairs on F_p: 4.50 ms in XYZZ, 4.02 so (4.15 with three blocks per SM).
template <class C>
__global__ void __launch_bounds__(128, 4) k_scalar_mul(const uint4 *__restrict__ scalars, const uint4 *__restrict__ pts,
                                                      size_t n, uint32_t *__restrict__ out)
{
    using G = Group<C>;
    using F = typename C::F;
    const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    Fe x, y;
    load_affine(pts, (uint32_t)i, x, y, wide_points(pts));
    typename G::Jac Q = G::jac_inf();
    if (!(F::is_exact_zero(x) && F::is_exact_zero(y))) {
        const uint4 sa = __ldg(scalars + 2 * i), sb = __ldg(scalars + 2 * i + 1);
        const uint32_t s[8] = {sa.x, sa.y, sa.z, sa.w, sb.x, sb.y, sb.z, sb.w};
        const uint32_t eights[8] = {0x88888888u, 0x88888888u, 0x88888888u, 0x88888888u,
                                    0x88888888u, 0x88888888u, 0x88888888u, 0x88888888u};
        uint32_t d[8];
        const uint32_t top = add8(d, s, eights);
        typename G::JacEntry T[8];
        T[0] = typename G::JacEntry{x, y, F::one(), F::one(), F::one()};
        typename G::Jac P = G::dbl(typename G::Jac{x, y, F::one()});
        for (int j = 1; j < 8; j++) {
            if (j > 1)
                P = G::add(P, T[0], false);
            const Fe zz = F::sqr(P.Z);
            T[j] = typename G::JacEntry{P.X, P.Y, P.Z, zz, F::mul(zz, P.Z)};
        }
        if (top)
            Q = typename G::Jac{x, y, F::one()};
#pragma unroll 1
        for (int k = 63; k >= 0; k--) {
#pragma unroll 1
            for (int b = 0; b < 4; b++)
                Q = G::dbl(Q);
            const int dk = (int)((d[k >> 3] >> (4 * (k & 7))) & 15u) - 8;
            if (dk != 0)
                Q = G::add(Q, T[(dk > 0 ? dk : -dk) - 1], dk < 0);
        }
    }
    const bool inf = G::is_inf(Q);
    const Fe v[3] = {F::canon(inf ? F::one() : Q.X), F::canon(inf ? F::one() : Q.Y), F::canon(Q.Z)};
#pragma unroll
    for (int c = 0; c < 3; c++)
#pragma unroll
        for (int w = 0; w < 8; w++)
            out[24 * i + 8 * c + w] = v[c].w[w];
}

template <class C>
cudaError_t scalar_mul(Context &ctx, const void *d_scalars, const uint4 *d_points, size_t n, uint32_t *d_out)
{
    if (n == 0)
        return cudaSuccess;
    const int threads = 128;
    k_scalar_mul<C><<<(unsigned)((n + threads - 1) / threads), threads, 0, ctx.stream>>>(
        static_cast<const uint4 *>(d_scalars), d_points, n, d_out);
    HS_LAUNCH_CHECK(ctx);
    return cudaSuccess;
}

template <class C>
CurveOps make_ops()
{
    return CurveOps{&msm_tail<C>, &to_affine<C>, &to_affine_scratch, &format_out<C>, &map_to_curve<C>,
                    &to_jac24<C>, &field_op<C>,  &fixed_table<C>,    &join<C>,       &decompress<C>,
                    &scalar_mul<C>};
}

}  // namespace hs
