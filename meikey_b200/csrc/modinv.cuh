// Inversion modulo p = 2^255 - 19 by division steps (Bernstein and Yang, "Fast constant-time gcd
// computation and modular inversion", CHES 2019).  The half-integer start of delta with its bound of
// 590 steps, the nine signed limbs of 30 bits, the limb-by-limb application of a matrix with two
// running sums, and the names zeta, cf, cg, cd, ce are those of libsecp256k1 (src/modinv32 and
// doc/safegcd_implementation.md, by Pieter Wuille and Peter Dettman; MIT licence).  The step on
// wrapping words, the correction by a centred multiple of p = -19 + 2^255 and the final sign and fold
// are this file's own.
//
// A division step on (delta, f, g), f odd, needs only the lowest bits of f and g, so 30 of them
// run on 32-bit words and are collected in a 2x2 matrix of integers below 2^30 in magnitude, which
// is then applied to the full f, g (nine signed limbs of 30 bits) and to d, e, which keep
// d·x = f and e·x = g (mod p) up to the common power of two.  When g reaches 0, f is ±1 and ±d the
// inverse.  It takes at most 590 steps from a 256-bit start, about 530 on random values.
//
// Why not x^(p-2): that is 254 dependent squarings, about 100 instructions each, on the one
// warp that inverts; a division step is about 15 instructions with a short dependent chain.  The
// inverting warp is what short iterations wait for: with the powering, 5 M incremental candidates
// at 8 keys per thread took 0.99 ms on B200, with the division steps 0.71 ms; 2^30 of them at
// 16 keys 114.0 and 109.0 ms; a 72-needle job, where the inversion rotates over the warps, 214.7
// and 207.9 ms; one secure iteration, whose inversion nothing hides, 1.54 and 1.50 ms.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define MKI_FN __device__ __forceinline__
#else
#define MKI_FN inline
#endif

namespace mkinv {

constexpr uint32_t M30 = (1u << 30) - 1;
constexpr uint32_t INV19 = 678152731u;  // 19^-1 mod 2^30
constexpr int MAX_BATCHES = 25;         // 750 division steps

// 30 division steps on the low words of f and g.  zeta = -(delta + 1/2).  The matrix (u v; q r)
// takes (f, g) to 2^30 times their new values.
MKI_FN void divsteps30(int32_t& zeta, uint32_t f, uint32_t g, int32_t m[4]) {
    uint32_t u = 1, v = 0, q = 0, r = 1;
#ifdef __CUDACC__
#pragma unroll 6
#endif
    for (int i = 0; i < 30; i++) {
        const uint32_t neg = (uint32_t)(zeta >> 31);             // all ones: delta > 0
        const uint32_t k = neg & g & 1u;                         // 1: swap (delta > 0 and g odd)
        const uint32_t a = (neg | 1u) & (0u - (g & 1u));         // g odd: -1 if delta > 0, else 1
        g += a * f;
        q += a * u;
        r += a * v;
        f += k * g;  // a swap leaves the old g: f + (g - f)
        u += k * q;
        v += k * r;
        zeta = (zeta ^ (int32_t)(0u - k)) - 1;
        g >>= 1;
        u <<= 1;
        v <<= 1;
    }
    m[0] = (int32_t)u;
    m[1] = (int32_t)v;
    m[2] = (int32_t)q;
    m[3] = (int32_t)r;
}

// (f, g) = matrix · (f, g) / 2^30 (exact)
MKI_FN void update_fg(int32_t f[9], int32_t g[9], const int32_t m[4]) {
    int64_t cf = (int64_t)m[0] * f[0] + (int64_t)m[1] * g[0];
    int64_t cg = (int64_t)m[2] * f[0] + (int64_t)m[3] * g[0];
    cf >>= 30;
    cg >>= 30;
#ifdef __CUDACC__
#pragma unroll
#endif
    for (int i = 1; i < 9; i++) {
        cf += (int64_t)m[0] * f[i] + (int64_t)m[1] * g[i];
        cg += (int64_t)m[2] * f[i] + (int64_t)m[3] * g[i];
        f[i - 1] = (int32_t)((uint32_t)cf & M30);
        g[i - 1] = (int32_t)((uint32_t)cg & M30);
        cf >>= 30;
        cg >>= 30;
    }
    f[8] = (int32_t)cf;
    g[8] = (int32_t)cg;
}

// (d, e) = matrix · (d, e) / 2^30 mod p: a multiple of p in [-p/2, p/2)·2^30 makes the low limb
// divisible (p = -19 + 2^15·2^240).  |d|, |e| grow by at most p/2 a call, to 13.5 p after 25;
// limb 8 has room for 2^16 p.
MKI_FN void update_de(int32_t d[9], int32_t e[9], const int32_t m[4]) {
    int64_t cd = (int64_t)m[0] * d[0] + (int64_t)m[1] * e[0];
    int64_t ce = (int64_t)m[2] * d[0] + (int64_t)m[3] * e[0];
    const int32_t kd = (int32_t)(((uint32_t)cd * INV19) << 2) >> 2;
    const int32_t ke = (int32_t)(((uint32_t)ce * INV19) << 2) >> 2;
    cd -= (int64_t)kd * 19;
    ce -= (int64_t)ke * 19;
    cd >>= 30;
    ce >>= 30;
#ifdef __CUDACC__
#pragma unroll
#endif
    for (int i = 1; i < 9; i++) {
        cd += (int64_t)m[0] * d[i] + (int64_t)m[1] * e[i];
        ce += (int64_t)m[2] * d[i] + (int64_t)m[3] * e[i];
        if (i == 8) {
            cd += (int64_t)kd << 15;
            ce += (int64_t)ke << 15;
        }
        d[i - 1] = (int32_t)((uint32_t)cd & M30);
        e[i - 1] = (int32_t)((uint32_t)ce & M30);
        cd >>= 30;
        ce >>= 30;
    }
    d[8] = (int32_t)cd;
    e[8] = (int32_t)ce;
}

// out = x^-1 mod p for any 256-bit x (not necessarily below p), 0 for a multiple of p; the result
// is below 2^256, not canonical.
MKI_FN void invert(const uint32_t x[8], uint32_t out[8]) {
    int32_t f[9], g[9], d[9], e[9];
#ifdef __CUDACC__
#pragma unroll
#endif
    for (int i = 0; i < 9; i++) {
        const int w = 30 * i / 32, s = 30 * i % 32;
        uint64_t pair = (uint64_t)x[w] | (uint64_t)(w < 7 ? x[w + 1] : 0u) << 32;
        g[i] = (int32_t)((uint32_t)(pair >> s) & M30);
        f[i] = (int32_t)M30;
        d[i] = e[i] = 0;
    }
    f[0] = (int32_t)M30 - 18;  // p
    f[8] = (1 << 15) - 1;
    e[0] = 1;
    int32_t zeta = -1;
#ifdef __CUDACC__
#pragma unroll 1
#endif
    for (int b = 0; b < MAX_BATCHES; b++) {
        int32_t any = 0;
#ifdef __CUDACC__
#pragma unroll
#endif
        for (int i = 0; i < 9; i++) any |= g[i];
        if (any == 0) break;
        int32_t m[4];
        divsteps30(zeta, (uint32_t)f[0], (uint32_t)g[0], m);
        update_de(d, e, m);
        update_fg(f, g, m);
    }
    // ±d + 16 p in [0, 30 p), the sign from f = ±1 (its limbs 0..7 hold the two's complement); a
    // multiple of p ends with f = ±p, whose limb 8 is not just a sign, and gives 16 p
    const int32_t s = f[8] >> 31;
    const int32_t unit = f[8] == s ? -1 : 0;
    int32_t c = -16 * 19;
    uint32_t l[9];
#ifdef __CUDACC__
#pragma unroll
#endif
    for (int i = 0; i < 9; i++) {
        c += ((d[i] ^ s) - s) & unit;
        if (i == 8) c += 16 << 15;
        l[i] = i < 8 ? (uint32_t)c & M30 : (uint32_t)c;
        c >>= 30;
    }
    // words, with the bits from 256 up (below 2^5) folded as 38 each
    const uint32_t top = l[8] >> 16;
    uint64_t carry = (uint64_t)38 * top;
#ifdef __CUDACC__
#pragma unroll
#endif
    for (int j = 0; j < 8; j++) {
        carry += l[j] >> (2 * j) | l[j + 1] << (30 - 2 * j);
        out[j] = (uint32_t)carry;
        carry >>= 32;
    }
    out[0] += 38u * (uint32_t)carry;  // a carry leaves the value below 38·31
}

}  // namespace mkinv
