// Point operations by two lanes of a warp, for kernels whose time is a chain of
// dependent point additions in a few warps.
//
// A lone warp runs at the latency of its instructions, so a chain's time is
// the number of instructions of one addition.  An XYZZ addition is 14
// products, but only 7 deep two at a time: the two lanes of a pair (lane & 1)
// hold the same operands, take one of two products in the same instruction
// and swap the results.  Both lanes end with the whole sum.  About 1500
// instructions against 2700; a Jacobian doubling is 4 products deep instead
// of 7.  (Four lanes would be 5 deep and shuffle more.)
//
// Every lane of `mask` has to take part; operands are the same in both lanes
// of a pair.
#pragma once

#include "bn254.cuh"

namespace impeller {

using namespace ec;

template <class F>
__device__ __forceinline__ Fe<F> fe_swap(const Fe<F> &a, u32 mask) {
    Fe<F> r;
#pragma unroll
    for (int i = 0; i < F::N; i++) r.l[i] = __shfl_xor_sync(mask, a.l[i], 1);
    return r;
}

// a in the pair's even lane, b in its odd one
template <class F>
__device__ __forceinline__ Fe<F> fe_pick(bool odd, const Fe<F> &a, const Fe<F> &b) {
    Fe<F> r;
#pragma unroll
    for (int i = 0; i < F::N; i++) r.l[i] = odd ? b.l[i] : a.l[i];
    return r;
}

// 2p on one lane, out of line: equal operands are rare.
template <class F>
__device__ __noinline__ XyzzT<F> xyzz_dbl_call(XyzzT<F> p) {
    return xyzz_dbl<F, MulCall>(p);
}

// Whether zz can be zero, from its low word.
template <class F>
__device__ __forceinline__ bool pair_maybe_identity(const XyzzT<F> &p) {
    constexpr Words<F::N> m = words(F::M);
    return p.zz.l[0] == 0 || p.zz.l[0] == m.v[0];
}

// add-2008-s; every special case.  Empty buckets are common (a zero polynomial;
// a column of small values leaves all windows but the lowest empty), so lanes
// that all add the identity leave early: 2^10 to 2^20 zero scalars on plain
// windows 0.40 to 0.51 ms without, 0.08 to 0.17 with.
template <class F>
__device__ __forceinline__ XyzzT<F> xyzz_add_pair(const XyzzT<F> &p, const XyzzT<F> &q, bool odd, u32 mask) {
    if (__all_sync(mask, pair_maybe_identity(p) || pair_maybe_identity(q))) {
        const bool id = xyzz_is_identity(p);
        if (__all_sync(mask, id || xyzz_is_identity(q))) return id ? q : p;
    }
    const Fe<F> u = fe_mul(fe_pick(odd, p.x, q.x), fe_pick(odd, q.zz, p.zz));    // u1 | u2
    const Fe<F> s = fe_mul(fe_pick(odd, p.y, q.y), fe_pick(odd, q.zzz, p.zzz));  // s1 | s2
    // P and R in the even lane, their negatives in the odd one
    const Fe<F> P = fe_sub(fe_swap(u, mask), u), R = fe_sub(fe_swap(s, mask), s);
    const Fe<F> sq = fe_sqr(fe_pick(odd, P, R));  // pp | rr
    const Fe<F> sqo = fe_swap(sq, mask);          // rr | pp
    const Fe<F> pp = fe_pick(odd, sq, sqo);
    const Fe<F> a = fe_mul(fe_pick(odd, P, p.zz), fe_pick(odd, pp, q.zz));    // ppp | zz zz'
    const Fe<F> b = fe_mul(fe_pick(odd, u, p.zzz), fe_pick(odd, pp, q.zzz));  // Q = u1 pp | zzz zzz'
    const Fe<F> c = fe_mul(fe_pick(odd, s, a), fe_pick(odd, a, pp));          // s1 ppp | zz3
    const Fe<F> ao = fe_swap(a, mask);
    const Fe<F> x3 = fe_sub(fe_sub(fe_sub(sqo, a), b), b);                     // (even lane)
    const Fe<F> d = fe_mul(fe_pick(odd, R, b), fe_pick(odd, fe_sub(b, x3), ao));  // R (Q - x3) | zzz3
    const Fe<F> y3 = fe_sub(d, c);
    const Fe<F> f = fe_swap(fe_pick(odd, x3, c), mask), g = fe_swap(fe_pick(odd, y3, d), mask);
    XyzzT<F> r;
    r.x = fe_pick(odd, x3, f);
    r.y = fe_pick(odd, y3, g);
    r.zz = fe_pick(odd, f, c);
    r.zzz = fe_pick(odd, g, d);
    if (xyzz_is_identity(p)) return q;
    if (xyzz_is_identity(q)) return p;
    if (fe_is_zero(P)) return fe_is_zero(R) ? xyzz_dbl_call(p) : xyzz_identity<F>();
    return r;
}

// dbl-2009-l with a = 0.
template <class F>
__device__ __forceinline__ JacT<F> jac_dbl_pair(const JacT<F> &p, bool odd, u32 mask) {
    const Fe<F> s1 = fe_sqr(fe_pick(odd, p.x, p.y));  // a | b
    const Fe<F> o1 = fe_swap(s1, mask);
    const Fe<F> a = fe_pick(odd, s1, o1), b = fe_pick(odd, o1, s1);
    const Fe<F> m = fe_mul(fe_pick(odd, p.y, b), fe_pick(odd, p.z, b));  // y z | c = b^2
    const Fe<F> e = fe_add(fe_dbl(a), a);
    const Fe<F> s3 = fe_sqr(fe_pick(odd, e, fe_add(p.x, b)));  // e^2 | (x + b)^2
    const Fe<F> om = fe_swap(m, mask), o3 = fe_swap(s3, mask);
    const Fe<F> c = fe_pick(odd, om, m);
    const Fe<F> d = fe_dbl(fe_sub(fe_sub(fe_pick(odd, o3, s3), a), c));
    JacT<F> r;
    r.x = fe_sub(fe_pick(odd, s3, o3), fe_dbl(d));
    r.y = fe_sub(fe_mul(e, fe_sub(d, r.x)), fe_dbl(fe_dbl(fe_dbl(c))));
    r.z = fe_dbl(fe_pick(odd, m, om));
    return r;
}

// 2^k p through Jacobian coordinates (xyzz_dbl_n); the identity stays so.
template <class F>
__device__ __forceinline__ XyzzT<F> xyzz_dbl_n_pair(const XyzzT<F> &p, u32 k, bool odd, u32 mask) {
    if (k == 0 || __all_sync(mask, xyzz_is_identity(p))) return p;
    JacT<F> j;
    j.x = fe_mul(p.x, fe_sqr(p.zz));
    j.y = fe_mul(p.y, fe_sqr(p.zzz));
    j.z = p.zzz;
#pragma unroll 1
    for (u32 i = 0; i < k; i++) j = jac_dbl_pair(j, odd, mask);
    XyzzT<F> r;
    r.x = j.x;
    r.y = j.y;
    r.zz = fe_sqr(j.z);
    r.zzz = fe_mul(j.z, r.zz);
    return r;
}

}  // namespace impeller
