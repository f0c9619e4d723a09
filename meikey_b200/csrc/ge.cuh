// edwards25519 point arithmetic over the radix-2^32 field (fe32.cuh).
//
// Points are extended (X:Y:Z:T), x = X/Z, y = Y/Z, xy = T/Z.  Table points are
// affine "Niels" triples (y+x, y-x, 2d·x·y) stored canonical as 8 LE words each.
// The mixed addition is the a = -1 complete formula (Hisil-Wong-Carter-Dawson 2008,
// also RFC 8032 5.1.4 with Z2 = 1): 7 multiplications, or 3 when only y = Y/Z of the
// sum is wanted (then y = (B+A)/(2Z-C) and x = (B-A)/(2Z+C)).
#pragma once
#include "fe32.cuh"
#include "modinv.cuh"

namespace mk32 {

struct ge {
    fe X, Y, Z, T;
};

struct niels {
    fe ypx, ymx, t2d;
};

// -q when neg: swaps y+x and y-x and negates 2dxy
__device__ __forceinline__ niels niels_signed(const niels& q, bool neg) {
    const fe nt = fe_sub_t(fe_zero(), q.t2d);
    niels r;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        r.ypx.v[i] = neg ? q.ymx.v[i] : q.ypx.v[i];
        r.ymx.v[i] = neg ? q.ypx.v[i] : q.ymx.v[i];
        r.t2d.v[i] = neg ? nt.v[i] : q.t2d.v[i];
    }
    return r;
}

// P + Q for a table point Q, P's coordinates tight (so are the sum's).
__device__ __forceinline__ ge ge_add_niels(const ge& p, const niels& q) {
    const fe a = fe_mul(fe_sub_t(p.Y, p.X), q.ymx);
    const fe b = fe_mul(fe_add_t(p.Y, p.X), q.ypx);
    const fe c = fe_mul(p.T, q.t2d);
    const fe d = fe_add_t(p.Z, p.Z);
    const fe e = fe_sub_t(b, a), h = fe_add_t(b, a);
    const fe f = fe_sub_t(d, c), g = fe_add_1(d, c);
    ge r;
    r.X = fe_mul(e, f);
    r.Y = fe_mul(g, h);
    r.Z = fe_mul(f, g);
    r.T = fe_mul(e, h);
    return r;
}

// The last addition (P tight): the sum's y as a fraction yn/yd and, optionally, x as xn/xd.
__device__ __forceinline__ void ge_add_niels_frac(const ge& p, const niels& q, fe& yn, fe& yd, fe* xn, fe* xd) {
    const fe a = fe_mul(fe_sub_t(p.Y, p.X), q.ymx);
    const fe b = fe_mul(fe_add_t(p.Y, p.X), q.ypx);
    const fe c = fe_mul(p.T, q.t2d);
    const fe d = fe_add_t(p.Z, p.Z);
    yn = fe_add_t(b, a);
    yd = fe_sub_t(d, c);
    if (xn) {
        *xn = fe_sub_t(b, a);
        *xd = fe_add_1(d, c);
    }
}

// General addition P + Q of two extended points (9 multiplications; used for table building).
__device__ __forceinline__ ge ge_add(const ge& p, const ge& q, const fe& d2) {
    fe a = fe_mul(fe_sub(p.Y, p.X), fe_sub(q.Y, q.X));
    fe b = fe_mul(fe_add(p.Y, p.X), fe_add(q.Y, q.X));
    fe c = fe_mul(fe_mul(p.T, d2), q.T);
    fe zz = fe_mul(p.Z, q.Z);
    fe d = fe_add(zz, zz);
    fe e = fe_sub(b, a), h = fe_add(b, a);
    fe f = fe_sub(d, c), g = fe_add(d, c);
    ge r;
    r.X = fe_mul(e, f);
    r.Y = fe_mul(g, h);
    r.Z = fe_mul(f, g);
    r.T = fe_mul(e, h);
    return r;
}

__device__ __forceinline__ ge ge_identity() {
    ge r;
    r.X = fe_zero();
    r.Y = fe_small(1);
    r.Z = fe_small(1);
    r.T = fe_zero();
    return r;
}

// 1/z (0 for z = 0 mod p), not canonical
__device__ __noinline__ fe fe_invert(const fe z) {
    fe r;
    mkinv::invert(z.v, r.v);
    return r;
}

}  // namespace mk32
