// Modular inversion by Bernstein-Yang divsteps, variable time.
//
// Used for the few conversions to affine form at the end of an MSM, where a
// single thread's latency is what counts.  The inputs are public (curve
// points), so variable time is fine.
//
// The method (D. J. Bernstein and B.-Y. Yang, "Fast constant-time gcd
// computation and modular inversion", 2019; the form that starts at
// delta = 1/2 is P. Wuille's, 2021, and this way of batching the steps is that
// of the description of libsecp256k1's modular inversion by P. Dettman and
// P. Wuille) keeps an odd f (initially the modulus p), a g (initially the
// input x) and zeta = -(delta + 1/2), and applies divsteps: with g odd and
// zeta < 0, (f, g) <- (g, (g - f) / 2) and zeta <- -zeta - 2; with g odd and
// zeta >= 0, g <- (g + f) / 2 and zeta <- zeta - 1; with g even, g <- g / 2
// and zeta <- zeta - 1.  g reaches 0 with f = +-1.  Divsteps look only at the
// low bits of f and g, so 30 of them at a time run on the low 32-bit words
// alone, collecting a 2x2 transition matrix T = [u v; q r] with
// 2^30 (f', g') = T (f, g); the full-width numbers are then updated once per
// batch.  Beside f and g the method carries d and e with d x = f and e x = g
// (mod p); they take the same matrix, divided by 2^30 modulo p, so at the end
// x^-1 = +-d.
//
// The 30 steps of a batch are straight-line code on masks (18 instructions a
// step): taking runs of even steps at once and merging odd steps needs fewer
// instructions for one input, but its loop depends on the input, so the lanes
// of a warp wait for the longest, and its count of trailing zeros and Newton
// steps are one long chain.  |u| + |v| <= 2^30 and |q| + |r| <= 2^30 after a
// batch, so the matrix fits 32-bit signed integers (the words wrap
// consistently modulo 2^32).
//
// d and e are not reduced between batches: an update takes a pair bounded by
// B p to one bounded by (B + 1/2) p (the multiple of p that makes the sum
// divisible by 2^30 is below 2^29 in magnitude), which the limbs hold through
// the last batch; one reduction at the end.
//
// Multi-precision numbers are signed radix-2^30: limbs 0..L-2 in [0, 2^30),
// the top limb signed.  Written for host and device so that the host build
// of this header can be checked against big-integer arithmetic.
#pragma once

#include <cstdint>

#if defined(__CUDACC__)
#define SG_HD __host__ __device__ __forceinline__
#define SG_CX __host__ __device__ constexpr
#else
#define SG_HD inline
#define SG_CX constexpr
#endif

namespace ec {
namespace sg {

static constexpr uint32_t M30 = 0x3fffffffu;

template <int L>
struct S30 {
    int32_t v[L];
};

struct Trans {
    int32_t u, v, q, r;
};

// Limb count for an N-word (32-bit) modulus: room for the unreduced d and e
// (magnitude below 2^5 p for 8 words, 2^6 p for 12; the fields' moduli leave
// two and three bits of their words free) and a sign.
SG_CX int limbs_for(int N) { return (32 * N + 2 + 29) / 30; }

// Upper bound of batches: Bernstein-Yang's bound of (49 d + 57) / 17 divsteps
// for d-bit inputs (the delta = 1/2 form needs fewer), in batches of 30, plus
// one.
SG_CX int max_batches(int N) { return ((49 * 32 * N + 57) / 17 + 29) / 30 + 1; }

// 30 divsteps on the low words of f (odd) and g; returns the new zeta.
SG_HD int divsteps30(int zeta, uint32_t f, uint32_t g, Trans &t) {
    uint32_t u = 1, v = 0, q = 0, r = 1;
#if defined(__CUDA_ARCH__)
#pragma unroll 10
#endif
    for (int i = 0; i < 30; i++) {
        const uint32_t odd = 0u - (g & 1u);
        const uint32_t swap = odd & (uint32_t)(zeta >> 31);
        // (x ^ swap) & odd, less swap: 0, x or -x
        const uint32_t df = (f ^ swap) & odd, du = (u ^ swap) & odd, dv = (v ^ swap) & odd;
        f ^= (f ^ g) & swap;
        u ^= (u ^ q) & swap;
        v ^= (v ^ r) & swap;
        g = (g + df - swap) >> 1;
        q = q + du - swap;
        r = r + dv - swap;
        u <<= 1;
        v <<= 1;
        zeta = (zeta ^ (int)swap) - 1;
    }
    t.u = (int32_t)u;
    t.v = (int32_t)v;
    t.q = (int32_t)q;
    t.r = (int32_t)r;
    return zeta;
}

// (f, g) <- T (f, g) / 2^30 (exact).
template <int L>
SG_HD void update_fg(S30<L> &f, S30<L> &g, const Trans &t) {
    const int64_t u = t.u, v = t.v, q = t.q, r = t.r;
    int64_t cf = u * f.v[0] + v * g.v[0];
    int64_t cg = q * f.v[0] + r * g.v[0];
    cf >>= 30;
    cg >>= 30;
#pragma unroll
    for (int i = 1; i < L; i++) {
        cf += u * f.v[i] + v * g.v[i];
        cg += q * f.v[i] + r * g.v[i];
        f.v[i - 1] = (int32_t)(cf & M30);
        g.v[i - 1] = (int32_t)(cg & M30);
        cf >>= 30;
        cg >>= 30;
    }
    f.v[L - 1] = (int32_t)cf;
    g.v[L - 1] = (int32_t)cg;
}

// x < 0 (normalised form: the sign is the top limb's)
template <int L>
SG_HD bool s30_neg(const S30<L> &x) {
    return x.v[L - 1] < 0;
}

// s x + k p for s = +-1 and a small k, the limbs renormalised
template <int L>
SG_HD S30<L> s30_mul_add(const S30<L> &x, int32_t s, const S30<L> &p, int32_t k) {
    S30<L> y;
    int64_t c = 0;
#pragma unroll
    for (int i = 0; i < L - 1; i++) {
        c += (int64_t)s * x.v[i] + (int64_t)k * p.v[i];
        y.v[i] = (int32_t)(c & M30);
        c >>= 30;
    }
    y.v[L - 1] = (int32_t)(c + (int64_t)s * x.v[L - 1] + (int64_t)k * p.v[L - 1]);
    return y;
}

// (d, e) <- T (d, e) / 2^30 mod p, unreduced.  pinv = p^-1 mod 2^30.
template <int L>
SG_HD void update_de(S30<L> &d, S30<L> &e, const Trans &t, const S30<L> &p, uint32_t pinv) {
    const int64_t u = t.u, v = t.v, q = t.q, r = t.r;
    int64_t cd = u * d.v[0] + v * e.v[0];
    int64_t ce = q * d.v[0] + r * e.v[0];
    // md, me in [-2^29, 2^29) make the low 30 bits of cd + md p and ce + me p zero
    const int64_t md = (int32_t)((0u - (uint32_t)cd * pinv) << 2) >> 2;
    const int64_t me = (int32_t)((0u - (uint32_t)ce * pinv) << 2) >> 2;
    cd += md * p.v[0];
    ce += me * p.v[0];
    cd >>= 30;
    ce >>= 30;
#pragma unroll
    for (int i = 1; i < L; i++) {
        cd += u * d.v[i] + v * e.v[i] + md * p.v[i];
        ce += q * d.v[i] + r * e.v[i] + me * p.v[i];
        d.v[i - 1] = (int32_t)(cd & M30);
        e.v[i - 1] = (int32_t)(ce & M30);
        cd >>= 30;
        ce >>= 30;
    }
    d.v[L - 1] = (int32_t)cd;
    e.v[L - 1] = (int32_t)ce;
}

template <int L>
SG_HD bool s30_is_zero(const S30<L> &x) {
    int32_t o = 0;
#pragma unroll
    for (int i = 0; i < L; i++) o |= x.v[i];
    return o == 0;
}

// N 32-bit words (little-endian, value < 2^(32 N)) -> radix 2^30
template <int L, int N>
SG_HD S30<L> to_s30(const uint32_t *w) {
    S30<L> x;
#pragma unroll
    for (int i = 0; i < L; i++) {
        const int bit = 30 * i, k = bit >> 5, s = bit & 31;
        uint64_t lo = k < N ? w[k] : 0u;
        uint64_t hi = k + 1 < N ? w[k + 1] : 0u;
        x.v[i] = (int32_t)(((lo | (hi << 32)) >> s) & M30);
    }
    return x;
}

// radix 2^30 (non-negative, below 2^(32 N)) -> N 32-bit words
template <int L, int N>
SG_HD void from_s30(const S30<L> &x, uint32_t *w) {
#pragma unroll
    for (int k = 0; k < N; k++) {
        const int bit = 32 * k, i = bit / 30, s = bit % 30;
        uint64_t acc = (uint64_t)(uint32_t)x.v[i] >> s;
        int have = 30 - s;
        if (i + 1 < L) acc |= (uint64_t)(uint32_t)x.v[i + 1] << have;
        have += 30;
        if (have < 32 && i + 2 < L) acc |= (uint64_t)(uint32_t)x.v[i + 2] << have;
        w[k] = (uint32_t)acc;
    }
}

// p^-1 mod 2^30 for odd p0 (Newton from 5 bits)
SG_CX uint32_t inv30(uint32_t p0) {
    uint32_t x = (3u * p0) ^ 2u;
    x *= 2u - p0 * x;
    x *= 2u - p0 * x;
    x *= 2u - p0 * x;
    return x & M30;
}

// x^-1 mod p for the canonical x (N words, 0 <= x < p, p an odd prime);
// zero gives zero, as does a run that exceeds the step bound (no input in
// [0, p) does).  out: N words, canonical.
template <int N>
SG_HD void inverse(const uint32_t *x, const uint32_t *pw, uint32_t *out) {
    constexpr int L = limbs_for(N);
    const S30<L> p = to_s30<L, N>(pw);
    const uint32_t pinv = inv30(pw[0]);
    S30<L> f = p, g = to_s30<L, N>(x), d, e;
#pragma unroll
    for (int i = 0; i < L; i++) {
        d.v[i] = 0;
        e.v[i] = 0;
    }
    e.v[0] = 1;
#pragma unroll
    for (int k = 0; k < N; k++) out[k] = 0;
    if (s30_is_zero(g)) return;
    // |d| <= (1 + max_batches / 2) p < K p at the end
    constexpr int K = N == 8 ? 16 : 32;
    static_assert(1 + max_batches(N) / 2 < K, "the last batch's d");
    int zeta = -1;
#pragma unroll 1
    for (int b = 0; b < max_batches(N); b++) {
        Trans t;
        zeta = divsteps30(zeta, (uint32_t)f.v[0] | ((uint32_t)f.v[1] << 30),
                          (uint32_t)g.v[0] | ((uint32_t)g.v[1] << 30), t);
        update_fg(f, g, t);
        update_de(d, e, t, p, pinv);
        if (s30_is_zero(g)) {
            // f = +-1: x^-1 = +-d; into [0, 2 K p), then below p
            d = s30_mul_add(d, s30_neg(f) ? -1 : 1, p, K);
#pragma unroll 1
            for (int k = K; k; k >>= 1) {
                const S30<L> r = s30_mul_add(d, 1, p, -k);
                if (!s30_neg(r)) d = r;
            }
            from_s30<L, N>(d, out);
            return;
        }
    }
}

}  // namespace sg
}  // namespace ec
