// GF(2^255 - 19) in eight 32-bit limbs (radix 2^32), values kept below 2^256
// (congruent mod p, not canonical).  "Tight" values are below 2^255 + 1500: canonical ones and
// every product.  Sums and differences of tight values need half the carries (fe_add_t, fe_add_1,
// fe_sub_t) and may reach 2^256; products take either.  Products use hand-written mad.lo.cc /
// madc.hi.cc carry chains; 2^256 is folded back as 38.  Exact integer math, no FP.
#pragma once
#include <stdint.h>

namespace mk32 {

typedef uint32_t u32;
typedef uint64_t u64;

struct fe {
    u32 v[8];
};

__device__ __forceinline__ fe fe_zero() {
    fe r;
#pragma unroll
    for (int i = 0; i < 8; i++) r.v[i] = 0;
    return r;
}

__device__ __forceinline__ fe fe_small(u32 x) {
    fe r = fe_zero();
    r.v[0] = x;
    return r;
}

// r = a + b mod 2^256 folded: a carry out of bit 256 adds 38
__device__ __forceinline__ fe fe_add(const fe& a, const fe& b) {
    fe r;
    u32 c;
    asm("add.cc.u32 %0, %9, %17;\n\t"
        "addc.cc.u32 %1, %10, %18;\n\t"
        "addc.cc.u32 %2, %11, %19;\n\t"
        "addc.cc.u32 %3, %12, %20;\n\t"
        "addc.cc.u32 %4, %13, %21;\n\t"
        "addc.cc.u32 %5, %14, %22;\n\t"
        "addc.cc.u32 %6, %15, %23;\n\t"
        "addc.cc.u32 %7, %16, %24;\n\t"
        "addc.u32 %8, 0, 0;\n\t"
        : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]), "=r"(r.v[6]),
          "=r"(r.v[7]), "=r"(c)
        : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]), "r"(a.v[6]), "r"(a.v[7]),
          "r"(b.v[0]), "r"(b.v[1]), "r"(b.v[2]), "r"(b.v[3]), "r"(b.v[4]), "r"(b.v[5]), "r"(b.v[6]), "r"(b.v[7]));
    // fold: r += 38·c; a second carry is impossible to miss: it leaves r < 38, and 38 more fits
    u32 add = 38u * c, c2;
    asm("add.cc.u32 %0, %0, %9;\n\t"
        "addc.cc.u32 %1, %1, 0;\n\t"
        "addc.cc.u32 %2, %2, 0;\n\t"
        "addc.cc.u32 %3, %3, 0;\n\t"
        "addc.cc.u32 %4, %4, 0;\n\t"
        "addc.cc.u32 %5, %5, 0;\n\t"
        "addc.cc.u32 %6, %6, 0;\n\t"
        "addc.cc.u32 %7, %7, 0;\n\t"
        "addc.u32 %8, 0, 0;\n\t"
        : "+r"(r.v[0]), "+r"(r.v[1]), "+r"(r.v[2]), "+r"(r.v[3]), "+r"(r.v[4]), "+r"(r.v[5]), "+r"(r.v[6]),
          "+r"(r.v[7]), "=r"(c2)
        : "r"(add));
    r.v[0] += 38u * c2;
    return r;
}

// r = a - b; a borrow subtracts 38 (2^256 ≡ 38)
__device__ __forceinline__ fe fe_sub(const fe& a, const fe& b) {
    fe r;
    u32 bw;
    asm("sub.cc.u32 %0, %9, %17;\n\t"
        "subc.cc.u32 %1, %10, %18;\n\t"
        "subc.cc.u32 %2, %11, %19;\n\t"
        "subc.cc.u32 %3, %12, %20;\n\t"
        "subc.cc.u32 %4, %13, %21;\n\t"
        "subc.cc.u32 %5, %14, %22;\n\t"
        "subc.cc.u32 %6, %15, %23;\n\t"
        "subc.cc.u32 %7, %16, %24;\n\t"
        "subc.u32 %8, 0, 0;\n\t"
        : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]), "=r"(r.v[6]),
          "=r"(r.v[7]), "=r"(bw)
        : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]), "r"(a.v[6]), "r"(a.v[7]),
          "r"(b.v[0]), "r"(b.v[1]), "r"(b.v[2]), "r"(b.v[3]), "r"(b.v[4]), "r"(b.v[5]), "r"(b.v[6]), "r"(b.v[7]));
    // bw is 0 or 0xffffffff
    u32 sub = 38u & bw, b2;
    asm("sub.cc.u32 %0, %0, %9;\n\t"
        "subc.cc.u32 %1, %1, 0;\n\t"
        "subc.cc.u32 %2, %2, 0;\n\t"
        "subc.cc.u32 %3, %3, 0;\n\t"
        "subc.cc.u32 %4, %4, 0;\n\t"
        "subc.cc.u32 %5, %5, 0;\n\t"
        "subc.cc.u32 %6, %6, 0;\n\t"
        "subc.cc.u32 %7, %7, 0;\n\t"
        "subc.u32 %8, 0, 0;\n\t"
        : "+r"(r.v[0]), "+r"(r.v[1]), "+r"(r.v[2]), "+r"(r.v[3]), "+r"(r.v[4]), "+r"(r.v[5]), "+r"(r.v[6]),
          "+r"(r.v[7]), "=r"(b2)
        : "r"(sub));
    // a second borrow leaves r >= 2^256 - 38, so 38 less cannot borrow again
    r.v[0] -= 38u & b2;
    return r;
}

// a + b, both tight: a carry out leaves less than 3000, so adding 38 stays in word 0
__device__ __forceinline__ fe fe_add_t(const fe& a, const fe& b) {
    fe r;
    u32 c;
    asm("add.cc.u32 %0, %9, %17;\n\t"
        "addc.cc.u32 %1, %10, %18;\n\t"
        "addc.cc.u32 %2, %11, %19;\n\t"
        "addc.cc.u32 %3, %12, %20;\n\t"
        "addc.cc.u32 %4, %13, %21;\n\t"
        "addc.cc.u32 %5, %14, %22;\n\t"
        "addc.cc.u32 %6, %15, %23;\n\t"
        "addc.cc.u32 %7, %16, %24;\n\t"
        "addc.u32 %8, 0, 0;"
        : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]), "=r"(r.v[6]),
          "=r"(r.v[7]), "=r"(c)
        : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]), "r"(a.v[6]), "r"(a.v[7]),
          "r"(b.v[0]), "r"(b.v[1]), "r"(b.v[2]), "r"(b.v[3]), "r"(b.v[4]), "r"(b.v[5]), "r"(b.v[6]), "r"(b.v[7]));
    r.v[0] += 38u * c;
    return r;
}

// a + b, b tight: a carry out leaves less than 2^255 + 1500, so adding 38 carries no further
__device__ __forceinline__ fe fe_add_1(const fe& a, const fe& b) {
    fe r;
    u32 c;
    asm("add.cc.u32 %0, %9, %17;\n\t"
        "addc.cc.u32 %1, %10, %18;\n\t"
        "addc.cc.u32 %2, %11, %19;\n\t"
        "addc.cc.u32 %3, %12, %20;\n\t"
        "addc.cc.u32 %4, %13, %21;\n\t"
        "addc.cc.u32 %5, %14, %22;\n\t"
        "addc.cc.u32 %6, %15, %23;\n\t"
        "addc.cc.u32 %7, %16, %24;\n\t"
        "addc.u32 %8, 0, 0;"
        : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]), "=r"(r.v[6]),
          "=r"(r.v[7]), "=r"(c)
        : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]), "r"(a.v[6]), "r"(a.v[7]),
          "r"(b.v[0]), "r"(b.v[1]), "r"(b.v[2]), "r"(b.v[3]), "r"(b.v[4]), "r"(b.v[5]), "r"(b.v[6]), "r"(b.v[7]));
    const u32 add = 38u * c;
    asm("add.cc.u32 %0, %0, %8;\n\t"
        "addc.cc.u32 %1, %1, 0;\n\t"
        "addc.cc.u32 %2, %2, 0;\n\t"
        "addc.cc.u32 %3, %3, 0;\n\t"
        "addc.cc.u32 %4, %4, 0;\n\t"
        "addc.cc.u32 %5, %5, 0;\n\t"
        "addc.cc.u32 %6, %6, 0;\n\t"
        "addc.u32 %7, %7, 0;"
        : "+r"(r.v[0]), "+r"(r.v[1]), "+r"(r.v[2]), "+r"(r.v[3]), "+r"(r.v[4]), "+r"(r.v[5]), "+r"(r.v[6]), "+r"(r.v[7])
        : "r"(add));
    return r;
}

// a - b, b tight: a borrow leaves at least 2^255 - 1500, so taking 38 off borrows no further
__device__ __forceinline__ fe fe_sub_t(const fe& a, const fe& b) {
    fe r;
    u32 bw;
    asm("sub.cc.u32 %0, %9, %17;\n\t"
        "subc.cc.u32 %1, %10, %18;\n\t"
        "subc.cc.u32 %2, %11, %19;\n\t"
        "subc.cc.u32 %3, %12, %20;\n\t"
        "subc.cc.u32 %4, %13, %21;\n\t"
        "subc.cc.u32 %5, %14, %22;\n\t"
        "subc.cc.u32 %6, %15, %23;\n\t"
        "subc.cc.u32 %7, %16, %24;\n\t"
        "subc.u32 %8, 0, 0;"
        : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]), "=r"(r.v[6]),
          "=r"(r.v[7]), "=r"(bw)
        : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]), "r"(a.v[6]), "r"(a.v[7]),
          "r"(b.v[0]), "r"(b.v[1]), "r"(b.v[2]), "r"(b.v[3]), "r"(b.v[4]), "r"(b.v[5]), "r"(b.v[6]), "r"(b.v[7]));
    const u32 sub = 38u & bw;
    asm("sub.cc.u32 %0, %0, %8;\n\t"
        "subc.cc.u32 %1, %1, 0;\n\t"
        "subc.cc.u32 %2, %2, 0;\n\t"
        "subc.cc.u32 %3, %3, 0;\n\t"
        "subc.cc.u32 %4, %4, 0;\n\t"
        "subc.cc.u32 %5, %5, 0;\n\t"
        "subc.cc.u32 %6, %6, 0;\n\t"
        "subc.u32 %7, %7, 0;"
        : "+r"(r.v[0]), "+r"(r.v[1]), "+r"(r.v[2]), "+r"(r.v[3]), "+r"(r.v[4]), "+r"(r.v[5]), "+r"(r.v[6]), "+r"(r.v[7])
        : "r"(sub));
    return r;
}

// a as a tight value: bit 255 comes back as 19
__device__ __forceinline__ fe fe_tight(const fe& a) {
    fe r = a;
    const u32 add = 19u * (a.v[7] >> 31);
    r.v[7] &= 0x7fffffffu;
    asm("add.cc.u32 %0, %0, %8;\n\t"
        "addc.cc.u32 %1, %1, 0;\n\t"
        "addc.cc.u32 %2, %2, 0;\n\t"
        "addc.cc.u32 %3, %3, 0;\n\t"
        "addc.cc.u32 %4, %4, 0;\n\t"
        "addc.cc.u32 %5, %5, 0;\n\t"
        "addc.cc.u32 %6, %6, 0;\n\t"
        "addc.u32 %7, %7, 0;"
        : "+r"(r.v[0]), "+r"(r.v[1]), "+r"(r.v[2]), "+r"(r.v[3]), "+r"(r.v[4]), "+r"(r.v[5]), "+r"(r.v[6]), "+r"(r.v[7])
        : "r"(add));
    return r;
}

// ---- products in even/odd accumulators ----
//
// A product of two limbs a_i·b_j is added at words i+j, i+j+1.  The integer pipe adds a full
// 64-bit product to an aligned register pair in one instruction (with the carry in and out), so
// the products at even words go to one accumulator e (pairs e[2k], e[2k+1]) and those at odd
// words to a second one o, one word up (o[k] stands for word k+1): every pair is aligned, and
// the two are added once at the end.  Rows that add all products into one array put every other
// chain on misaligned pairs, which splits its products into low and high halves (three issue
// slots instead of two).  On B200, one chain per thread and 16 warps per SM: 111 G
// multiplications/s against 102 G for the one-array rows and 100 G for Karatsuba on them
// (117 against 91 and 103 with four chains); Karatsuba on even/odd accumulators runs at 106 G:
// its 25 % fewer products do not pay for about 60 more adds.  The search kernel gains 3 % on hashed
// seeds (2^29 candidates: 696 -> 675 ms; it multiplied in the Karatsuba form) and 12 % on the
// incremental source (2^30: 128.0 -> 114.0 ms).

// w[0..1] = x·y
__device__ __forceinline__ void wide(u32* w, u32 x, u32 y) {
    asm("mul.lo.u32 %0, %2, %3;\n\t"
        "mul.hi.u32 %1, %2, %3;"
        : "=&r"(w[0]), "=r"(w[1])
        : "r"(x), "r"(y));
}

// One chain of n products by the same limb y on consecutive pairs, w[2i..2i+1] += x_i·y:
//   rown_carry  every pair holds a sum already; the carry starts the next pair, w[2n] = carry;
//   rown_add    the same, the carry added to the next pair, which holds a sum;
//   rown_open   the last pair is new, and rown_top new but for a carry `top` (0 or 1) of an earlier
//               row; neither overflows (x·y + 2 < 2^64).
__device__ __forceinline__ void row2_carry(u32* w, u32 x0, u32 x1, u32 y) {
    asm("mad.lo.cc.u32 %0, %5, %7, %0;\n\t"
        "madc.hi.cc.u32 %1, %5, %7, %1;\n\t"
        "madc.lo.cc.u32 %2, %6, %7, %2;\n\t"
        "madc.hi.cc.u32 %3, %6, %7, %3;\n\t"
        "addc.u32 %4, 0, 0;"
        : "+r"(w[0]), "+r"(w[1]), "+r"(w[2]), "+r"(w[3]), "=r"(w[4])
        : "r"(x0), "r"(x1), "r"(y));
}

__device__ __forceinline__ void row2_top(u32* w, u32 x0, u32 x1, u32 y, u32 top) {
    asm("mad.lo.cc.u32 %0, %4, %6, %0;\n\t"
        "madc.hi.cc.u32 %1, %4, %6, %1;\n\t"
        "madc.lo.cc.u32 %2, %5, %6, %7;\n\t"
        "madc.hi.u32 %3, %5, %6, 0;"
        : "+r"(w[0]), "+r"(w[1]), "=&r"(w[2]), "=r"(w[3])
        : "r"(x0), "r"(x1), "r"(y), "r"(top));
}

__device__ __forceinline__ void row4_carry(u32* w, u32 x0, u32 x1, u32 x2, u32 x3, u32 y) {
    asm("mad.lo.cc.u32 %0, %9, %13, %0;\n\t"
        "madc.hi.cc.u32 %1, %9, %13, %1;\n\t"
        "madc.lo.cc.u32 %2, %10, %13, %2;\n\t"
        "madc.hi.cc.u32 %3, %10, %13, %3;\n\t"
        "madc.lo.cc.u32 %4, %11, %13, %4;\n\t"
        "madc.hi.cc.u32 %5, %11, %13, %5;\n\t"
        "madc.lo.cc.u32 %6, %12, %13, %6;\n\t"
        "madc.hi.cc.u32 %7, %12, %13, %7;\n\t"
        "addc.u32 %8, 0, 0;"
        : "+r"(w[0]), "+r"(w[1]), "+r"(w[2]), "+r"(w[3]), "+r"(w[4]), "+r"(w[5]), "+r"(w[6]), "+r"(w[7]),
          "=r"(w[8])
        : "r"(x0), "r"(x1), "r"(x2), "r"(x3), "r"(y));
}

__device__ __forceinline__ void row4_open(u32* w, u32 x0, u32 x1, u32 x2, u32 x3, u32 y) {
    asm("mad.lo.cc.u32 %0, %8, %12, %0;\n\t"
        "madc.hi.cc.u32 %1, %8, %12, %1;\n\t"
        "madc.lo.cc.u32 %2, %9, %12, %2;\n\t"
        "madc.hi.cc.u32 %3, %9, %12, %3;\n\t"
        "madc.lo.cc.u32 %4, %10, %12, %4;\n\t"
        "madc.hi.cc.u32 %5, %10, %12, %5;\n\t"
        "madc.lo.cc.u32 %6, %11, %12, 0;\n\t"
        "madc.hi.u32 %7, %11, %12, 0;"
        : "+r"(w[0]), "+r"(w[1]), "+r"(w[2]), "+r"(w[3]), "+r"(w[4]), "+r"(w[5]), "=&r"(w[6]), "=r"(w[7])
        : "r"(x0), "r"(x1), "r"(x2), "r"(x3), "r"(y));
}

__device__ __forceinline__ void row4_add(u32* w, u32 x0, u32 x1, u32 x2, u32 x3, u32 y) {
    asm("mad.lo.cc.u32 %0, %10, %14, %0;\n\t"
        "madc.hi.cc.u32 %1, %10, %14, %1;\n\t"
        "madc.lo.cc.u32 %2, %11, %14, %2;\n\t"
        "madc.hi.cc.u32 %3, %11, %14, %3;\n\t"
        "madc.lo.cc.u32 %4, %12, %14, %4;\n\t"
        "madc.hi.cc.u32 %5, %12, %14, %5;\n\t"
        "madc.lo.cc.u32 %6, %13, %14, %6;\n\t"
        "madc.hi.cc.u32 %7, %13, %14, %7;\n\t"
        "addc.cc.u32 %8, %8, 0;\n\t"
        "addc.u32 %9, %9, 0;"
        : "+r"(w[0]), "+r"(w[1]), "+r"(w[2]), "+r"(w[3]), "+r"(w[4]), "+r"(w[5]), "+r"(w[6]), "+r"(w[7]),
          "+r"(w[8]), "+r"(w[9])
        : "r"(x0), "r"(x1), "r"(x2), "r"(x3), "r"(y));
}

// t = e + o·2^32 over n+1 words (t[0] = e[0]); the sum fits
__device__ __forceinline__ void merge7(const u32* e, const u32* o, u32* t) {
    t[0] = e[0];
    asm("add.cc.u32 %0, %7, %14;\n\t"
        "addc.cc.u32 %1, %8, %15;\n\t"
        "addc.cc.u32 %2, %9, %16;\n\t"
        "addc.cc.u32 %3, %10, %17;\n\t"
        "addc.cc.u32 %4, %11, %18;\n\t"
        "addc.cc.u32 %5, %12, %19;\n\t"
        "addc.u32 %6, %13, %20;"
        : "=r"(t[1]), "=r"(t[2]), "=r"(t[3]), "=r"(t[4]), "=r"(t[5]), "=r"(t[6]), "=r"(t[7])
        : "r"(e[1]), "r"(e[2]), "r"(e[3]), "r"(e[4]), "r"(e[5]), "r"(e[6]), "r"(e[7]),
          "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3]), "r"(o[4]), "r"(o[5]), "r"(o[6]));
}

__device__ __forceinline__ void merge15(const u32* e, const u32* o, u32* t) {
    t[0] = e[0];
    asm("add.cc.u32 %0, %15, %30;\n\t"
        "addc.cc.u32 %1, %16, %31;\n\t"
        "addc.cc.u32 %2, %17, %32;\n\t"
        "addc.cc.u32 %3, %18, %33;\n\t"
        "addc.cc.u32 %4, %19, %34;\n\t"
        "addc.cc.u32 %5, %20, %35;\n\t"
        "addc.cc.u32 %6, %21, %36;\n\t"
        "addc.cc.u32 %7, %22, %37;\n\t"
        "addc.cc.u32 %8, %23, %38;\n\t"
        "addc.cc.u32 %9, %24, %39;\n\t"
        "addc.cc.u32 %10, %25, %40;\n\t"
        "addc.cc.u32 %11, %26, %41;\n\t"
        "addc.cc.u32 %12, %27, %42;\n\t"
        "addc.cc.u32 %13, %28, %43;\n\t"
        "addc.u32 %14, %29, %44;"
        : "=r"(t[1]), "=r"(t[2]), "=r"(t[3]), "=r"(t[4]), "=r"(t[5]), "=r"(t[6]), "=r"(t[7]), "=r"(t[8]),
          "=r"(t[9]), "=r"(t[10]), "=r"(t[11]), "=r"(t[12]), "=r"(t[13]), "=r"(t[14]), "=r"(t[15])
        : "r"(e[1]), "r"(e[2]), "r"(e[3]), "r"(e[4]), "r"(e[5]), "r"(e[6]), "r"(e[7]), "r"(e[8]),
          "r"(e[9]), "r"(e[10]), "r"(e[11]), "r"(e[12]), "r"(e[13]), "r"(e[14]), "r"(e[15]),
          "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3]), "r"(o[4]), "r"(o[5]), "r"(o[6]), "r"(o[7]),
          "r"(o[8]), "r"(o[9]), "r"(o[10]), "r"(o[11]), "r"(o[12]), "r"(o[13]), "r"(o[14]));
}

// Fold a 512-bit product t[0..15] to 8 words (tight): t_lo + 38·t_hi, then the bits from 255 up.  The
// products 38·t[8+j] of even j extend the pairs of t_lo, those of odd j go one word up.
__device__ __forceinline__ fe fe_reduce512(const u32 t[16]) {
    u32 s[8], w[9];
#pragma unroll
    for (int k = 0; k < 4; k++) wide(s + 2 * k, t[9 + 2 * k], 38u);
#pragma unroll
    for (int i = 0; i < 8; i++) w[i] = t[i];
    row4_carry(w, t[8], t[10], t[12], t[14], 38u);
    fe r;
    u32 top = w[8];
#pragma unroll
    for (int i = 0; i < 8; i++) r.v[i] = w[i];
    asm("add.cc.u32 %0, %0, %8;\n\t"
        "addc.cc.u32 %1, %1, %9;\n\t"
        "addc.cc.u32 %2, %2, %10;\n\t"
        "addc.cc.u32 %3, %3, %11;\n\t"
        "addc.cc.u32 %4, %4, %12;\n\t"
        "addc.cc.u32 %5, %5, %13;\n\t"
        "addc.cc.u32 %6, %6, %14;\n\t"
        "addc.u32 %7, %7, %15;"
        : "+r"(r.v[1]), "+r"(r.v[2]), "+r"(r.v[3]), "+r"(r.v[4]), "+r"(r.v[5]), "+r"(r.v[6]), "+r"(r.v[7]), "+r"(top)
        : "r"(s[0]), "r"(s[1]), "r"(s[2]), "r"(s[3]), "r"(s[4]), "r"(s[5]), "r"(s[6]), "r"(s[7]));
    // top < 40: what stands above bit 255, below 78, comes back as 19 each and carries no further
    const u32 add = 19u * __funnelshift_l(r.v[7], top, 1);
    r.v[7] &= 0x7fffffffu;
    asm("add.cc.u32 %0, %0, %8;\n\t"
        "addc.cc.u32 %1, %1, 0;\n\t"
        "addc.cc.u32 %2, %2, 0;\n\t"
        "addc.cc.u32 %3, %3, 0;\n\t"
        "addc.cc.u32 %4, %4, 0;\n\t"
        "addc.cc.u32 %5, %5, 0;\n\t"
        "addc.cc.u32 %6, %6, 0;\n\t"
        "addc.u32 %7, %7, 0;"
        : "+r"(r.v[0]), "+r"(r.v[1]), "+r"(r.v[2]), "+r"(r.v[3]), "+r"(r.v[4]), "+r"(r.v[5]), "+r"(r.v[6]), "+r"(r.v[7])
        : "r"(add));
    return r;
}

// r = a·b mod p (tight), schoolbook: 64 products.  Limb b_i meets the limbs a_j of its own parity
// on the even words and the others on the odd ones.  Of two rows whose chains end on one pair, the
// one that opens it goes first and the other's carry is added to it: a pair opened on top of a
// waiting carry would need that carry moved into a pair with a zero.
__device__ __forceinline__ fe fe_mul_schoolbook(const fe& a, const fe& b) {
    u32 e[16], o[16], t[16];
    const u32 a0 = a.v[0], a1 = a.v[1], a2 = a.v[2], a3 = a.v[3], a4 = a.v[4], a5 = a.v[5], a6 = a.v[6], a7 = a.v[7];
    wide(e, a0, b.v[0]); wide(e + 2, a2, b.v[0]); wide(e + 4, a4, b.v[0]); wide(e + 6, a6, b.v[0]);
    wide(o, a1, b.v[0]); wide(o + 2, a3, b.v[0]); wide(o + 4, a5, b.v[0]); wide(o + 6, a7, b.v[0]);
    row4_open(e + 2, a1, a3, a5, a7, b.v[1]);
#pragma unroll
    for (int i = 2; i < 8; i += 2) {
        row4_open(e + i + 2, a1, a3, a5, a7, b.v[i + 1]);
        row4_add(e + i, a0, a2, a4, a6, b.v[i]);
        row4_open(o + i, a1, a3, a5, a7, b.v[i]);
        row4_add(o + i - 2, a0, a2, a4, a6, b.v[i - 1]);
    }
    row4_carry(o + 6, a0, a2, a4, a6, b.v[7]);
    merge15(e, o, t);
    return fe_reduce512(t);
}

// t[0..7] = x · y for 128-bit x, y (four limbs each): 16 products
__device__ __forceinline__ void mul128(const u32 x[4], const u32 y[4], u32 t[8]) {
    u32 e[8], o[8];
    wide(e, x[0], y[0]); wide(e + 2, x[2], y[0]);
    wide(o, x[1], y[0]); wide(o + 2, x[3], y[0]);
    row2_top(e + 2, x[1], x[3], y[1], 0u);
    row2_carry(o, x[0], x[2], y[1]);
    row2_carry(e + 2, x[0], x[2], y[2]);
    row2_top(o + 2, x[1], x[3], y[2], o[4]);
    row2_top(e + 4, x[1], x[3], y[3], e[6]);
    row2_carry(o + 2, x[0], x[2], y[3]);
    merge7(e, o, t);
}

// d = |x - y| for 128-bit x, y; returns all ones when x < y, else 0
__device__ __forceinline__ u32 absdiff128(const u32 x[4], const u32 y[4], u32 d[4]) {
    u32 s;
    asm("sub.cc.u32 %0, %5, %9;\n\t"
        "subc.cc.u32 %1, %6, %10;\n\t"
        "subc.cc.u32 %2, %7, %11;\n\t"
        "subc.cc.u32 %3, %8, %12;\n\t"
        "subc.u32 %4, 0, 0;\n\t"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]), "=r"(s)
        : "r"(x[0]), "r"(x[1]), "r"(x[2]), "r"(x[3]), "r"(y[0]), "r"(y[1]), "r"(y[2]), "r"(y[3]));
    // negative: (d ^ s) - s = 2^128 - d, the magnitude
#pragma unroll
    for (int i = 0; i < 4; i++) d[i] ^= s;
    asm("sub.cc.u32 %0, %0, %4;\n\t"
        "subc.cc.u32 %1, %1, %4;\n\t"
        "subc.cc.u32 %2, %2, %4;\n\t"
        "subc.u32 %3, %3, %4;\n\t"
        : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
        : "r"(s));
    return s;
}

// r = a·b mod p by one level of subtractive Karatsuba on the 128-bit halves
// (a = A1·2^128 + A0): A0·B1 + A1·B0 = L + H - (A0 - A1)·(B0 - B1) with L = A0·B0 and
// H = A1·B1, so the 512-bit product takes 48 lo + 48 hi products and about 60 adds and
// logic operations instead of 64 + 64.  Both operands use the same difference X0 - X1, so an
// operand that enters several products (the point-addition outputs' E, F, G, H) has one
// |X0 - X1| the compiler can share.  The product t is the same 512-bit integer as the
// schoolbook's, and so is the folded result.
__device__ __forceinline__ fe fe_mul_karatsuba(const fe& a, const fe& b) {
    u32 da[4], db[4], mm[8], lo[8], hi[8], mid[9];
    const u32 sa = absdiff128(&a.v[0], &a.v[4], da);
    const u32 sb = absdiff128(&b.v[0], &b.v[4], db);
    // (A0 - A1)(B0 - B1) is subtracted, so |..|·|..| is subtracted when the signs agree
    const u32 s = ~(sa ^ sb);  // all ones: the middle product is subtracted
    mul128(da, db, mm);
    mul128(&a.v[0], &b.v[0], lo);
    mul128(&a.v[4], &b.v[4], hi);
    // mid = L + H, nine words
    asm("add.cc.u32 %0, %9, %17;\n\t"
        "addc.cc.u32 %1, %10, %18;\n\t"
        "addc.cc.u32 %2, %11, %19;\n\t"
        "addc.cc.u32 %3, %12, %20;\n\t"
        "addc.cc.u32 %4, %13, %21;\n\t"
        "addc.cc.u32 %5, %14, %22;\n\t"
        "addc.cc.u32 %6, %15, %23;\n\t"
        "addc.cc.u32 %7, %16, %24;\n\t"
        "addc.u32 %8, 0, 0;\n\t"
        : "=r"(mid[0]), "=r"(mid[1]), "=r"(mid[2]), "=r"(mid[3]), "=r"(mid[4]), "=r"(mid[5]), "=r"(mid[6]),
          "=r"(mid[7]), "=r"(mid[8])
        : "r"(lo[0]), "r"(lo[1]), "r"(lo[2]), "r"(lo[3]), "r"(lo[4]), "r"(lo[5]), "r"(lo[6]), "r"(lo[7]),
          "r"(hi[0]), "r"(hi[1]), "r"(hi[2]), "r"(hi[3]), "r"(hi[4]), "r"(hi[5]), "r"(hi[6]), "r"(hi[7]));
    // mid += ±M mod 2^288: (M ^ s) with a ninth word s, plus a carry-in of s & 1 (set by s + s);
    // the true value A0·B1 + A1·B0 lies in [0, 2^257)
#pragma unroll
    for (int i = 0; i < 8; i++) mm[i] ^= s;
    asm("{\n\t"
        ".reg .u32 cf;\n\t"
        "add.cc.u32 cf, %9, %9;\n\t"
        "addc.cc.u32 %0, %0, %10;\n\t"
        "addc.cc.u32 %1, %1, %11;\n\t"
        "addc.cc.u32 %2, %2, %12;\n\t"
        "addc.cc.u32 %3, %3, %13;\n\t"
        "addc.cc.u32 %4, %4, %14;\n\t"
        "addc.cc.u32 %5, %5, %15;\n\t"
        "addc.cc.u32 %6, %6, %16;\n\t"
        "addc.cc.u32 %7, %7, %17;\n\t"
        "addc.u32 %8, %8, %9;\n\t"
        "}"
        : "+r"(mid[0]), "+r"(mid[1]), "+r"(mid[2]), "+r"(mid[3]), "+r"(mid[4]), "+r"(mid[5]), "+r"(mid[6]),
          "+r"(mid[7]), "+r"(mid[8])
        : "r"(s), "r"(mm[0]), "r"(mm[1]), "r"(mm[2]), "r"(mm[3]), "r"(mm[4]), "r"(mm[5]), "r"(mm[6]), "r"(mm[7]));
    // t = L + mid·2^128 + H·2^256 (below 2^512: no carry out of word 15)
    u32 t[16];
    t[0] = lo[0];
    t[1] = lo[1];
    t[2] = lo[2];
    t[3] = lo[3];
    asm("add.cc.u32 %0, %12, %24;\n\t"
        "addc.cc.u32 %1, %13, %25;\n\t"
        "addc.cc.u32 %2, %14, %26;\n\t"
        "addc.cc.u32 %3, %15, %27;\n\t"
        "addc.cc.u32 %4, %16, %28;\n\t"
        "addc.cc.u32 %5, %17, %29;\n\t"
        "addc.cc.u32 %6, %18, %30;\n\t"
        "addc.cc.u32 %7, %19, %31;\n\t"
        "addc.cc.u32 %8, %20, %32;\n\t"
        "addc.cc.u32 %9, %21, 0;\n\t"
        "addc.cc.u32 %10, %22, 0;\n\t"
        "addc.u32 %11, %23, 0;\n\t"
        : "=r"(t[4]), "=r"(t[5]), "=r"(t[6]), "=r"(t[7]), "=r"(t[8]), "=r"(t[9]), "=r"(t[10]), "=r"(t[11]),
          "=r"(t[12]), "=r"(t[13]), "=r"(t[14]), "=r"(t[15])
        : "r"(lo[4]), "r"(lo[5]), "r"(lo[6]), "r"(lo[7]), "r"(hi[0]), "r"(hi[1]), "r"(hi[2]), "r"(hi[3]),
          "r"(hi[4]), "r"(hi[5]), "r"(hi[6]), "r"(hi[7]), "r"(mid[0]), "r"(mid[1]), "r"(mid[2]), "r"(mid[3]),
          "r"(mid[4]), "r"(mid[5]), "r"(mid[6]), "r"(mid[7]), "r"(mid[8]));
    return fe_reduce512(t);
}

// r = a·b mod p (tight) for any values below 2^256
__device__ __forceinline__ fe fe_mul(const fe& a, const fe& b) { return fe_mul_schoolbook(a, b); }

// Canonical value (mod p) as 8 words
__device__ __forceinline__ void fe_to_words(const fe& a, u32 out[8]) {
    // fold bit 255: x = lo255 + 19·bit255  (< 2^255 + 19)
    u32 w[8];
#pragma unroll
    for (int i = 0; i < 8; i++) w[i] = a.v[i];
    u32 hb = w[7] >> 31;
    w[7] &= 0x7fffffffu;
    u64 c = 19ull * hb;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        c += w[i];
        w[i] = (u32)c;
        c >>= 32;
    }
    // subtract p if x >= p: compute x + 19 and test bit 255
    u32 t[8];
    c = 19;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        c += w[i];
        t[i] = (u32)c;
        c >>= 32;
    }
    u32 ge = t[7] >> 31;
    t[7] &= 0x7fffffffu;
#pragma unroll
    for (int i = 0; i < 8; i++) out[i] = ge ? t[i] : w[i];
}

__device__ __forceinline__ fe fe_from_words(const u32 w[8]) {
    fe r;
#pragma unroll
    for (int i = 0; i < 8; i++) r.v[i] = w[i];
    return r;
}

}  // namespace mk32
