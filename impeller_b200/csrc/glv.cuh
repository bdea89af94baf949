// BN254's endomorphism and the scalar decomposition that goes with it
// (R. Gallant, R. Lambert, S. Vanstone, "Faster point multiplication on
// elliptic curves with efficient endomorphisms", 2001).
//
// beta^3 = 1 mod p gives phi(x, y) = (beta x, y) on y^2 = x^3 + 3; on G1 (the
// whole curve: its order is the prime r) phi(P) = lambda P with
// lambda^2 + lambda + 1 = 0 mod r.  The lattice of (a, b) with
// a + b lambda = 0 mod r has the reduced basis (A, -N1), (N2, A), of
// determinant r, so with c1 = round(A k / r), c2 = round(N1 k / r)
//   k1 = k - c1 A - c2 N2,   k2 = c1 N1 - c2 A,   k = k1 + k2 lambda mod r.
// The rounded quotients come from products with G = round(2^256 A / r) and
// round(2^256 N1 / r), off by at most 1/2 + 2^-3 for k < 2^254, so
// |k1|, |k2| <= 0.625 (A + N2) < 2^127.
//
// An MSM over plain windows then has 128-bit scalars over twice the points:
// as many digits, but half the bucket sets to reduce and half the doublings
// between the windows' totals.
#pragma once

#include <cstdint>

#if defined(__CUDACC__)
#define GLV_HD __host__ __device__ __forceinline__
#else
#define GLV_HD inline
#endif

namespace ec {
namespace glv {

// beta in Montgomery form
#define GLV_BETA {0xd782e155u, 0x71930c11u, 0xffbe3323u, 0xa6bb947cu, 0xd4741444u, 0xaa303344u, 0x26594943u, 0x2c3b3f0du}

// Signed-digit windows of width c for one half: the top digit plus its
// incoming carry stays at most 2^(c-1) for magnitudes below 2^127.
GLV_HD uint32_t windows(uint32_t c) { return (128u + c - 1u) / c; }

// acc (NR words) += or -= a (NA words) * b (NB words), modulo 2^(32 NR)
template <int NR, int NA, int NB, bool SUB>
GLV_HD void mul_acc(uint32_t (&acc)[NR], const uint32_t (&a)[NA], const uint32_t (&b)[NB]) {
    uint32_t t[NR];
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
    for (int i = 0; i < NR; i++) t[i] = 0;
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
    for (int i = 0; i < NA; i++) {
        uint64_t c = 0;
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
        for (int j = 0; j < NB; j++) {
            if (i + j >= NR) break;
            c += (uint64_t)a[i] * b[j] + t[i + j];
            t[i + j] = (uint32_t)c;
            c >>= 32;
        }
        if (i + NB < NR) t[i + NB] = (uint32_t)c;
    }
    uint64_t c = SUB ? 1 : 0;
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
    for (int i = 0; i < NR; i++) {
        c += (uint64_t)acc[i] + (SUB ? ~t[i] : t[i]);
        acc[i] = (uint32_t)c;
        c >>= 32;
    }
}

// Two's complement x (5 words) -> magnitude (4 words); returns 1 when negative.
GLV_HD uint32_t magnitude(const uint32_t (&x)[5], uint32_t (&m)[4]) {
    const uint32_t neg = x[4] >> 31, mask = 0u - neg;
    uint64_t c = neg;
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
    for (int i = 0; i < 4; i++) {
        c += x[i] ^ mask;
        m[i] = (uint32_t)c;
        c >>= 32;
    }
    return neg;
}

// k (8 words, below r) = (-1)^neg1 k1 + (-1)^neg2 k2 lambda mod r
GLV_HD void split(const uint32_t (&k)[8], uint32_t (&k1)[4], uint32_t &neg1, uint32_t (&k2)[4], uint32_t &neg2) {
    const uint32_t g1[3] = {0xc7e0b3d7u, 0xd91d232eu, 0x00000002u};
    const uint32_t g2[5] = {0x391eb18eu, 0x7a7bd9d4u, 0xa773d2cfu, 0x4ccef014u, 0x00000002u};
    const uint32_t a[2] = {0x94d213e3u, 0x89d32568u};
    const uint32_t n1[4] = {0x7d4f1128u, 0x8211bbebu, 0xeeb859fcu, 0x6f4d8248u};
    const uint32_t n2[4] = {0x1221250bu, 0x0be4e154u, 0xeeb859fdu, 0x6f4d8248u};
    // quotients rounded to nearest: the accumulators start at 2^255
    uint32_t q1[11] = {0, 0, 0, 0, 0, 0, 0, 0x80000000u}, q2[13] = {0, 0, 0, 0, 0, 0, 0, 0x80000000u};
    mul_acc<11, 8, 3, false>(q1, k, g1);
    mul_acc<13, 8, 5, false>(q2, k, g2);
    const uint32_t c1[3] = {q1[8], q1[9], q1[10]}, c2[4] = {q2[8], q2[9], q2[10], q2[11]};
    uint32_t x[5] = {k[0], k[1], k[2], k[3], k[4]}, y[5] = {0, 0, 0, 0, 0};
    mul_acc<5, 3, 2, true>(x, c1, a);
    mul_acc<5, 4, 4, true>(x, c2, n2);
    mul_acc<5, 3, 4, false>(y, c1, n1);
    mul_acc<5, 4, 2, true>(y, c2, a);
    neg1 = magnitude(x, k1);
    neg2 = magnitude(y, k2);
}

}  // namespace glv
}  // namespace ec
