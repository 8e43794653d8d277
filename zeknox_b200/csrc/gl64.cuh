// Goldilocks field arithmetic, p = 2^64 - 2^32 + 1, for sm_100a.
//
// Every value handed between functions is canonical (in [0, p)), so results
// are bit-identical to zeknox's gl64_t (native/ff/gl64_t.cuh:93-369) and
// cpp_gl64_t (native/ff/goldilocks.hpp:139-177), whose outputs are canonical
// for canonical inputs.  The 64x64 -> 128-bit product is formed from 32-bit
// IMAD chains; the reductions use 2^64 = 2^32 - 1 and 2^96 = -1 (mod p).
#pragma once
#include <stdint.h>

#define ZK_P 0xffffffff00000001ull
#define ZK_EPS 0x00000000ffffffffull  // 2^64 mod p

namespace zk {

__device__ __forceinline__ uint64_t gl_canon_fwd(uint64_t x) { return x >= ZK_P ? x - ZK_P : x; }

// a + b mod p for a, b < p.  With s = a + b (mod 2^64) the result is s + EPS
// (mod 2^64) exactly when the sum carried out or s >= p (i.e. s + EPS carries).
__device__ __forceinline__ uint64_t gl_add(uint64_t a, uint64_t b) {
    uint64_t s, t;
    uint32_t c;
    asm("{\n\t"
        ".reg .u32 c0;\n\t"
        "add.cc.u64 %0, %3, %4;\n\t"
        "addc.u32 c0, 0, 0;\n\t"
        "add.cc.u64 %1, %0, %5;\n\t"
        "addc.u32 %2, c0, 0;\n\t"
        "}"
        : "=l"(s), "=l"(t), "=r"(c)
        : "l"(a), "l"(b), "l"(ZK_EPS));
    return c ? t : s;
}

// Full 64 x 64 -> 128-bit product from 32-bit limbs.
__device__ __forceinline__ void mul_wide(uint64_t a, uint64_t b, uint64_t &lo, uint64_t &hi) {
    uint32_t a0 = (uint32_t)a, a1 = (uint32_t)(a >> 32);
    uint32_t b0 = (uint32_t)b, b1 = (uint32_t)(b >> 32);
    uint32_t r0, r1, r2, r3;
    asm("{\n\t"
        "mul.lo.u32 %0, %4, %6;\n\t"
        "mul.hi.u32 %1, %4, %6;\n\t"
        "mul.lo.u32 %2, %5, %7;\n\t"
        "mul.hi.u32 %3, %5, %7;\n\t"
        "mad.lo.cc.u32 %1, %4, %7, %1;\n\t"
        "madc.hi.cc.u32 %2, %4, %7, %2;\n\t"
        "addc.u32 %3, %3, 0;\n\t"
        "mad.lo.cc.u32 %1, %5, %6, %1;\n\t"
        "madc.hi.cc.u32 %2, %5, %6, %2;\n\t"
        "addc.u32 %3, %3, 0;\n\t"
        "}"
        : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
        : "r"(a0), "r"(a1), "r"(b0), "r"(b1));
    lo = ((uint64_t)r1 << 32) | r0;
    hi = ((uint64_t)r3 << 32) | r2;
}

__device__ __forceinline__ uint64_t pr_mul(uint64_t a, uint64_t b);

// Canonical product: the partially reduced product (below) then one
// conditional subtraction.
__device__ __forceinline__ uint64_t gl_mul(uint64_t a, uint64_t b) { return gl_canon_fwd(pr_mul(a, b)); }

// Canonical representative of an arbitrary u64.
__device__ __forceinline__ uint64_t gl_canon(uint64_t x) { return x >= ZK_P ? x - ZK_P : x; }

}  // namespace zk

// ---------------------------------------------------------------------------
// Partially reduced arithmetic for the hash permutations: a value is any u64
// congruent to the field element (so in [0, 2^64), not necessarily < p).
// Results are exact modulo p; callers canonicalise (gl_canon) before storing.
// ---------------------------------------------------------------------------
namespace zk {

// (h1, h0, l1, l0) 128-bit -> u64 congruent mod p:
//   x = (l1:l0) - h1 + h0 * (2^32 - 1).
__device__ __forceinline__ uint64_t pr_reduce128(uint32_t l0, uint32_t l1, uint32_t h0, uint32_t h1) {
    uint32_t r0, r1;
    asm("{\n\t"
        ".reg .u32 b, k;\n\t"
        "sub.cc.u32  %0, %2, %5;\n\t"   // r = (l1:l0) - h1
        "subc.cc.u32 %1, %3, 0;\n\t"
        "subc.u32    b, 0, 0;\n\t"      // b = all-ones on borrow
        "sub.cc.u32  %0, %0, b;\n\t"    // on borrow: r -= EPS (r + p mod 2^64)
        "subc.u32    %1, %1, 0;\n\t"
        "add.cc.u32  %1, %1, %4;\n\t"   // r += h0 * 2^32
        "addc.u32    k, 0, 0;\n\t"
        "sub.cc.u32  %0, %0, %4;\n\t"   // r -= h0
        "subc.cc.u32 %1, %1, 0;\n\t"
        "subc.u32    k, k, 0;\n\t"      // k = 1 iff r + h0*EPS overflowed 2^64
        "neg.s32     k, k;\n\t"
        "add.cc.u32  %0, %0, k;\n\t"    // then add 2^64 mod p = EPS
        "addc.u32    %1, %1, 0;\n\t"
        "}"
        : "=r"(r0), "=r"(r1)
        : "r"(l0), "r"(l1), "r"(h0), "r"(h1));
    return ((uint64_t)r1 << 32) | r0;
}

// a * b for any u64 a, b; result partially reduced.  The 128-bit product
// comes from the 32-bit multiply-add chain of mul_wide (cheaper here than
// 64-bit-accumulating wide multiplies).
__device__ __forceinline__ uint64_t pr_mul(uint64_t a, uint64_t b) {
    uint64_t lo, hi;
    mul_wide(a, b, lo, hi);
    return pr_reduce128((uint32_t)lo, (uint32_t)(lo >> 32), (uint32_t)hi, (uint32_t)(hi >> 32));
}

// a + c for any u64 a and c < p: one wrap at most, fixed by adding EPS.
__device__ __forceinline__ uint64_t pr_add_c(uint64_t a, uint64_t c) {
    const uint64_t s = a + c;
    return s < a ? s + ZK_EPS : s;
}

// a b + c as 128 bits (c any u64) from four 32 x 32 -> 64-bit products: the
// two middle ones are summed first (65 bits) and added once, and the halves of
// c start the first two products, so the addend costs no instruction of its
// own.  Counted per application: 6.5 instructions against 7.5 of mul_wide.
__device__ __forceinline__ void mul_add_words(uint64_t a, uint64_t b, uint32_t c0, uint32_t c1, uint32_t w[4]) {
    asm("{\n\t"
        ".reg .u64 l, m, h, e;\n\t"
        ".reg .u32 l1, m0, m1, h0, h1, c, z;\n\t"
        "mov.u32 z, 0;\n\t"
        "mov.b64 e, {%8, z};\n\t"
        "mad.wide.u32 l, %4, %6, e;\n\t"
        "mov.b64 e, {%9, z};\n\t"
        "mad.wide.u32 m, %4, %7, e;\n\t"
        "mul.wide.u32 h, %5, %7;\n\t"
        "mov.b64 {%0, l1}, l;\n\t"
        "mov.b64 {m0, m1}, m;\n\t"
        "mov.b64 {h0, h1}, h;\n\t"
        "mad.lo.cc.u32 m0, %5, %6, m0;\n\t"
        "madc.hi.cc.u32 m1, %5, %6, m1;\n\t"
        "addc.u32 c, h1, 0;\n\t"
        "add.cc.u32 %1, l1, m0;\n\t"
        "addc.cc.u32 %2, h0, m1;\n\t"
        "addc.u32 %3, c, 0;\n\t"
        "}"
        : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3])
        : "r"((uint32_t)a), "r"((uint32_t)(a >> 32)), "r"((uint32_t)b), "r"((uint32_t)(b >> 32)), "r"(c0), "r"(c1));
}

// a^2 as 128 bits from three products, the cross term doubled by shifts: one
// multiply fewer for three ALU instructions.  A 32 x 32 -> 64-bit product takes
// two issue slots on this GPU, so this is the cheaper form in the S-box.
__device__ __forceinline__ void sqr_words(uint64_t a, uint32_t w[4]) {
    asm("{\n\t"
        ".reg .u64 l, m, h;\n\t"
        ".reg .u32 l1, m0, m1, h0, h1, c;\n\t"
        "mul.wide.u32 l, %4, %4;\n\t"
        "mul.wide.u32 m, %4, %5;\n\t"
        "mul.wide.u32 h, %5, %5;\n\t"
        "mov.b64 {%0, l1}, l;\n\t"
        "mov.b64 {m0, m1}, m;\n\t"
        "mov.b64 {h0, h1}, h;\n\t"
        "shr.u32 c, m1, 31;\n\t"             // bit 64 of 2 a0 a1
        "shf.l.wrap.b32 m1, m0, m1, 1;\n\t"
        "shl.b32 m0, m0, 1;\n\t"
        "add.cc.u32 %1, l1, m0;\n\t"
        "addc.cc.u32 %2, h0, m1;\n\t"
        "addc.u32 %3, h1, c;\n\t"
        "}"
        : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3])
        : "r"((uint32_t)a), "r"((uint32_t)(a >> 32)));
}

// Montgomery reduction: (w3 w2 w1 w0) 2^-64 mod p, partially reduced, for any
// 128-bit value.  2^128 = -2^32 (mod p), so 2^-64 (w1 w0) = -(w1 w0) 2^32 =
// (w1 + e) - (s + e) 2^32 with s + e 2^32 = w0 + w1; the subtrahend below is
// the negative of that, in [0, p), and a borrow from the high half adds p
// back.  For a product of two canonical values the result is canonical.
// Nine instructions, no multiply, against 13 of pr_reduce128.
__device__ __forceinline__ uint64_t mont_reduce(uint32_t w0, uint32_t w1, uint32_t w2, uint32_t w3) {
    uint32_t r0, r1;
    asm("{\n\t"
        ".reg .u32 s, t, b0, b1, k;\n\t"
        "add.cc.u32 s, %3, %2;\n\t"
        "addc.u32 t, s, 0;\n\t"          // s + e: no carry (s <= 2^32 - 2 when e = 1)
        "sub.cc.u32 b0, %2, t;\n\t"      // (s + e) 2^32 - (w1 + e) = (s : w0) - t
        "subc.u32 b1, s, 0;\n\t"
        "sub.cc.u32 %0, %4, b0;\n\t"
        "subc.cc.u32 %1, %5, b1;\n\t"
        "subc.u32 k, 0, 0;\n\t"          // all-ones on borrow: then - (2^32 - 1)
        "sub.cc.u32 %0, %0, k;\n\t"
        "subc.u32 %1, %1, 0;\n\t"
        "}"
        : "=r"(r0), "=r"(r1)
        : "r"(w0), "r"(w1), "r"(w2), "r"(w3));
    return ((uint64_t)r1 << 32) | r0;
}
__device__ __forceinline__ uint64_t mont_mul(uint64_t a, uint64_t b) {  // a b 2^-64
    uint32_t w[4];
    mul_add_words(a, b, 0, 0, w);
    return mont_reduce(w[0], w[1], w[2], w[3]);
}
__device__ __forceinline__ uint64_t mont_sqr(uint64_t a) {  // a^2 2^-64
    uint32_t w[4];
    sqr_words(a, w);
    return mont_reduce(w[0], w[1], w[2], w[3]);
}

// x^7 with partial reduction, from four Montgomery products on plain values.
// With R = 2^64: x^2 R^-1, x^3 R^-2, x^4 R^-3 and their product x^7 R^-6; 2 has
// order 192 mod p, so R^3 = 1 and the result is x^7 itself: no conversion in
// or out.  Per application 62 instructions; with the folding reduction 86.
// kMulSqr: the squares as plain products, three ALU instructions fewer for one
// multiply more each.
template <bool kMulSqr = false>
__device__ __forceinline__ uint64_t pr_pow7(uint64_t x) {
    const uint64_t x2 = kMulSqr ? mont_mul(x, x) : mont_sqr(x);
    const uint64_t x3 = mont_mul(x, x2);
    const uint64_t x4 = kMulSqr ? mont_mul(x2, x2) : mont_sqr(x2);
    return mont_mul(x3, x4);
}

// a^2 + c for any u64 a, c; partially reduced.
__device__ __forceinline__ uint64_t pr_sqr_add(uint64_t a, uint64_t c) {
    uint32_t w[4];
    mul_add_words(a, a, (uint32_t)c, (uint32_t)(c >> 32), w);
    return pr_reduce128(w[0], w[1], w[2], w[3]);
}

// (x1 x0) + t (2^32 - 1) mod p for t < 2^32 - 1, i.e. x0 + x1 2^32 + t 2^64;
// partially reduced.  Written as (x1 x0) - (p - t (2^32 - 1)), whose
// subtrahend is (2^32 - 1 - t) 2^32 + t + 1 <= p: a borrow adds p back.
__device__ __forceinline__ uint64_t pr_fold(uint32_t x0, uint32_t x1, uint32_t t) {
    uint32_t r0, r1;
    asm("{\n\t"
        ".reg .u32 n0, n1, k;\n\t"
        "add.u32 n0, %4, 1;\n\t"
        "not.b32 n1, %4;\n\t"
        "sub.cc.u32 %0, %2, n0;\n\t"
        "subc.cc.u32 %1, %3, n1;\n\t"
        "subc.u32 k, 0, 0;\n\t"
        "sub.cc.u32 %0, %0, k;\n\t"
        "subc.u32 %1, %1, 0;\n\t"
        "}"
        : "=r"(r0), "=r"(r1)
        : "r"(x0), "r"(x1), "r"(t));
    return ((uint64_t)r1 << 32) | r0;
}

// al + ah * 2^32 for al < 2^64 and ah < 2^63; partially reduced.
__device__ __forceinline__ uint64_t pr_reduce_split(uint64_t al, uint64_t ah) {
    uint32_t x1, t;
    asm("add.cc.u32 %0, %2, %3;\n\t"
        "addc.u32   %1, %4, 0;"
        : "=r"(x1), "=r"(t)
        : "r"((uint32_t)(al >> 32)), "r"((uint32_t)ah), "r"((uint32_t)(ah >> 32)));
    return pr_fold((uint32_t)al, x1, t);
}
// The same plus c, any u64.
__device__ __forceinline__ uint64_t pr_reduce_split_add(uint64_t al, uint64_t ah, uint64_t c) {
    uint32_t x0, x1, t;
    asm("{\n\t"
        ".reg .u32 k;\n\t"
        "add.cc.u32  %0, %3, %7;\n\t"
        "addc.cc.u32 %1, %4, %8;\n\t"
        "addc.u32    k, %6, 0;\n\t"
        "add.cc.u32  %1, %1, %5;\n\t"
        "addc.u32    %2, k, 0;\n\t"
        "}"
        : "=r"(x0), "=r"(x1), "=r"(t)
        : "r"((uint32_t)al), "r"((uint32_t)(al >> 32)), "r"((uint32_t)ah), "r"((uint32_t)(ah >> 32)),
          "r"((uint32_t)c), "r"((uint32_t)(c >> 32)));
    return pr_fold(x0, x1, t);
}

}  // namespace zk
