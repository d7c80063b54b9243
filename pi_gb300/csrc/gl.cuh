// Goldilocks field arithmetic for sm_103a: p = 2^64 - 2^32 + 1.
//
// Same field as the reference's CPU code (crates/bignum/src/ntt.rs:159-284).
// Inside the transforms values are kept "weak": any 64-bit word congruent to
// the field element (so possibly in [p, 2^64)).  add / mul accept weak
// inputs and return weak outputs; canon() gives the canonical representative
// in [0, p), which is what leaves the engine.  The reduction uses
// 2^64 = 2^32 - 1 (mod p) and 2^96 = -1 (mod p), written as 32-bit carry
// chains in inline PTX (the integer ALU pipe is the binding resource).
#pragma once
#include <cstdint>

namespace gl {

constexpr uint64_t P = 0xFFFFFFFF00000001ull;
constexpr uint64_t EPS = 0xFFFFFFFFull;  // 2^64 mod p

__device__ __forceinline__ uint32_t lo32(uint64_t x) { return (uint32_t)x; }
__device__ __forceinline__ uint32_t hi32(uint64_t x) { return (uint32_t)(x >> 32); }
__device__ __forceinline__ uint64_t mk64(uint32_t lo, uint32_t hi) { return ((uint64_t)hi << 32) | lo; }

// a + b (weak in, weak out).  A carry out of 64 bits is worth 2^64 = EPS;
// adding EPS back can carry once more (only when both inputs are >= p-ish),
// and that second carry is folded the same way.
__device__ __forceinline__ uint64_t add(uint64_t a, uint64_t b) {
  uint32_t z0, z1;
  asm("{\n\t.reg .u32 c, m;\n\t"
      "add.cc.u32 %0, %2, %4;\n\t"
      "addc.cc.u32 %1, %3, %5;\n\t"
      "addc.u32 c, 0, 0;\n\t"
      "neg.s32 m, c;\n\t"
      "add.cc.u32 %0, %0, m;\n\t"
      "addc.cc.u32 %1, %1, 0;\n\t"
      "addc.u32 c, 0, 0;\n\t"
      "neg.s32 m, c;\n\t"
      "add.cc.u32 %0, %0, m;\n\t"
      "addc.u32 %1, %1, 0;\n\t"
      "}"
      : "=&r"(z0), "=&r"(z1)
      : "r"(lo32(a)), "r"(hi32(a)), "r"(lo32(b)), "r"(hi32(b)));
  return mk64(z0, z1);
}

// Canonical representative in [0, p).
__device__ __forceinline__ uint64_t canon(uint64_t x) { return x >= P ? x - P : x; }

// 128-bit value (x3 x2 x1 x0) -> weak 64-bit:  (x1:x0) + x2 * (2^32 - 1) - x3.
// The multiply-add of x2 (on the FMA pipe) carries at most once; the sum's
// net carry k in {-1, 0, 1} is worth k * 2^64 = k * EPS, and adding that
// cannot carry again (|k * EPS| is far from both ends of the 64-bit range).
__device__ __forceinline__ uint64_t reduce_words(uint32_t r0, uint32_t r1, uint32_t r2, uint32_t r3) {
  uint32_t z0, z1;
  asm("{\n\t.reg .u32 k, nk, hk;\n\t"
      "mad.lo.cc.u32 %0, %4, 0xFFFFFFFF, %2;\n\t"
      "madc.hi.cc.u32 %1, %4, 0xFFFFFFFF, %3;\n\t"
      "addc.u32 k, 0, 0;\n\t"
      "sub.cc.u32 %0, %0, %5;\n\t"
      "subc.cc.u32 %1, %1, 0;\n\t"
      "subc.u32 k, k, 0;\n\t"
      "neg.s32 nk, k;\n\t"           // k * EPS = (k >> 31 : -k) for k in {-1, 0, 1}
      "shr.s32 hk, k, 31;\n\t"
      "add.cc.u32 %0, %0, nk;\n\t"
      "addc.u32 %1, %1, hk;\n\t"
      "}"
      : "=&r"(z0), "=&r"(z1)
      : "r"(r0), "r"(r1), "r"(r2), "r"(r3));
  return mk64(z0, z1);
}

// 64x64 -> 128 product from four 32x32 partial products.
__device__ __forceinline__ void mul128(uint64_t a, uint64_t b, uint32_t& r0, uint32_t& r1, uint32_t& r2,
                                       uint32_t& r3) {
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
      : "=&r"(r0), "=&r"(r1), "=&r"(r2), "=&r"(r3)
      : "r"(lo32(a)), "r"(hi32(a)), "r"(lo32(b)), "r"(hi32(b)));
}

// a * b mod p (weak in, weak out).
__device__ __forceinline__ uint64_t mul(uint64_t a, uint64_t b) {
  uint32_t r0, r1, r2, r3;
  mul128(a, b, r0, r1, r2, r3);
  return reduce_words(r0, r1, r2, r3);
}

// ------------------------------------------------------------ lazy values
// Inside the butterflies values are carried "lazy": a
// 64-bit word plus a small signed count k of 2^64 overflows,
//   value = l + h 2^32 + k 2^64   (= l + h 2^32 + k EPS  mod p).
// Adding or subtracting two lazy values is one 96-bit add (three carry-chain
// instructions) with no modular fix-up; fold() turns a lazy value back into a
// weak 64-bit word once, at the end of the butterfly network.
struct Lz {
  uint32_t l, h;
  int32_t k;
};

__device__ __forceinline__ Lz lz(uint64_t x) { return Lz{lo32(x), hi32(x), 0}; }

__device__ __forceinline__ Lz lz_add(Lz x, Lz y) {
  Lz z;
  asm("add.cc.u32 %0, %3, %6;\n\taddc.cc.u32 %1, %4, %7;\n\taddc.u32 %2, %5, %8;"
      : "=r"(z.l), "=r"(z.h), "=r"(z.k)
      : "r"(x.l), "r"(x.h), "r"(x.k), "r"(y.l), "r"(y.h), "r"(y.k));
  return z;
}

__device__ __forceinline__ Lz lz_sub(Lz x, Lz y) {
  Lz z;
  asm("sub.cc.u32 %0, %3, %6;\n\tsubc.cc.u32 %1, %4, %7;\n\tsubc.u32 %2, %5, %8;"
      : "=r"(z.l), "=r"(z.h), "=r"(z.k)
      : "r"(x.l), "r"(x.h), "r"(x.k), "r"(y.l), "r"(y.h), "r"(y.k));
  return z;
}

// Lazy value + 2^30 p.  A DFT adds what is added to its first input to every
// output (and never shifts that input), so one biased input makes all outputs'
// overflow counts non-negative (|k| < 2^29 before), which is what fold() takes.
__device__ __forceinline__ Lz lz_bias(Lz x) {
  Lz z;
  asm("add.cc.u32 %0, %3, 0x40000000;\n\taddc.cc.u32 %1, %4, 0xC0000000;\n\taddc.u32 %2, %5, 0x3FFFFFFF;"
      : "=r"(z.l), "=r"(z.h), "=r"(z.k)
      : "r"(x.l), "r"(x.h), "r"(x.k));
  return z;
}

// Lazy value with a non-negative overflow count -> weak 64-bit word:
// (h:l) + k EPS is one multiply-add on the FMA pipe; it carries at most once
// (c), and the c EPS = c 2^32 - c which that is worth cannot carry again (the
// wrapped sum is below k EPS <= (2^32 - 1)^2).
__device__ __forceinline__ uint64_t fold(Lz x) {
  uint32_t z0, z1;
  asm("{\n\t.reg .u32 c;\n\t"
      "mad.lo.cc.u32 %0, %4, 0xFFFFFFFF, %2;\n\t"
      "madc.hi.cc.u32 %1, %4, 0xFFFFFFFF, %3;\n\t"
      "addc.u32 c, 0, 0;\n\t"
      "sub.cc.u32 %0, %0, c;\n\t"
      "subc.u32 %1, %1, 0;\n\t"
      "add.u32 %1, %1, c;\n\t"
      "}"
      : "=&r"(z0), "=&r"(z1)
      : "r"(x.l), "r"(x.h), "r"((uint32_t)x.k));
  return mk64(z0, z1);
}

// a * b as a lazy value with k in {-1, 0}: with u = x2 EPS + (EPS - x3)
// (which cannot overflow 64 bits), a b = (x1:x0) + u - EPS and -EPS = -2^64.
__device__ __forceinline__ Lz lz_mul(uint64_t a, uint64_t b) {
  uint32_t r0, r1, r2, r3;
  mul128(a, b, r0, r1, r2, r3);
  uint64_t u;
  asm("mad.wide.u32 %0, %1, 0xFFFFFFFF, %2;" : "=l"(u) : "r"(r2), "l"((uint64_t)(~r3)));
  Lz z;
  asm("add.cc.u32 %0, %3, %5;\n\taddc.cc.u32 %1, %4, %6;\n\taddc.u32 %2, 0xFFFFFFFF, 0;"
      : "=r"(z.l), "=r"(z.h), "=r"(z.k)
      : "r"(r0), "r"(r1), "r"(lo32(u)), "r"(hi32(u)));
  return z;
}

// Shifts that leave their result lazy (no fold), for the butterflies: x 2^S
// for a compile-time 0 < S < 96, S = 32 Q + r.  The 96-bit shift by r gives
// words v0, v1 and a signed top v2 = funnel(h, k, r) (|k| 2^r < 2^31; r > 28
// takes one more word), in all (v0 + v1 2^32 + v2 2^64) 2^(32 Q).  With
// 2^64 = EPS = 2^32 - 1, 2^96 = -1 and 2^128 = -2^32:
//  * Q = 0: (v1:v0) + v2 2^32 - v2, k in {-1 .. 1};
//  * Q = 1: v0 2^32 + v1 EPS - v2.  u = v1 EPS + (EPS - v2), v2 taken unsigned,
//    fits 64 bits; -EPS = -2^64, and a negative v2 counts 2^32 too much, which
//    enters as a carry (the sign bit of k): k in {-1, 0};
//  * Q = 2: v0 EPS - v1 - v2 2^32 = u - v2 2^32 - 2^64 for u = v0 EPS + (EPS - v1),
//    k in {-2 .. 0}.
template <int S>
__device__ __forceinline__ Lz lz_shl(Lz x) {
  static_assert(S > 0 && S < 96, "shift out of range");
  constexpr int Q = S / 32, r = S % 32;
  uint32_t v0 = x.l, v1 = x.h, v2 = (uint32_t)x.k;
  if constexpr (r > 0) {
    v0 = x.l << r;
    v1 = __funnelshift_l(x.l, x.h, r);
    v2 = __funnelshift_l(x.h, (uint32_t)x.k, r);
  }
  Lz z;
  if constexpr (Q == 0 && r > 28) {
    // v2 unsigned and a fourth word v3 = k >> (32 - r): v3 2^96 = -v3
    const int32_t v3 = x.k >> (32 - r);
    asm("{\n\t.reg .u32 c;\n\t"
        "mad.lo.cc.u32 %0, %5, 0xFFFFFFFF, %3;\n\t"
        "madc.hi.cc.u32 %1, %5, 0xFFFFFFFF, %4;\n\t"
        "addc.u32 c, 0, 0;\n\t"
        "sub.cc.u32 %0, %0, %6;\n\t"
        "subc.cc.u32 %1, %1, %7;\n\t"
        "subc.u32 %2, c, %7;\n\t"
        "}"
        : "=&r"(z.l), "=&r"(z.h), "=&r"(z.k)
        : "r"(v0), "r"(v1), "r"(v2), "r"(v3), "r"(v3 >> 31));
  } else if constexpr (Q == 0) {
    asm("{\n\t.reg .u32 c;\n\t"
        "sub.cc.u32 %0, %3, %5;\n\t"
        "subc.cc.u32 %1, %4, %6;\n\t"
        "subc.u32 c, 0, %6;\n\t"
        "add.cc.u32 %1, %1, %5;\n\t"
        "addc.u32 %2, c, %6;\n\t"
        "}"
        : "=&r"(z.l), "=&r"(z.h), "=&r"(z.k)
        : "r"(v0), "r"(v1), "r"(v2), "r"((int32_t)v2 >> 31));
  } else if constexpr (Q == 1) {
    uint64_t u;
    asm("mad.wide.u32 %0, %1, 0xFFFFFFFF, %2;" : "=l"(u) : "r"(v1), "l"((uint64_t)(~v2)));
    z.l = lo32(u);
    asm("{\n\t.reg .u32 t;\n\t"
        "add.cc.u32 t, %4, %4;\n\t"
        "addc.cc.u32 %0, %2, %3;\n\t"
        "addc.u32 %1, 0xFFFFFFFF, 0;\n\t"
        "}"
        : "=&r"(z.h), "=r"(z.k)
        : "r"(hi32(u)), "r"(v0), "r"(x.k));
  } else {
    uint64_t u;
    asm("mad.wide.u32 %0, %1, 0xFFFFFFFF, %2;" : "=l"(u) : "r"(v0), "l"((uint64_t)(~v1)));
    z.l = lo32(u);
    asm("sub.cc.u32 %0, %2, %3;\n\tsubc.u32 %1, 0xFFFFFFFF, %4;"
        : "=r"(z.h), "=r"(z.k)
        : "r"(hi32(u)), "r"(v2), "r"(x.k >> 31));
  }
  return z;
}

// x 2^24 with the shifted-out word left as the overflow count (|k| < 2^28 for
// |x.k| < 2^4), which lz_add, lz_sub and fold accept but another shift does not.
__device__ __forceinline__ Lz lz_shl24_wide(Lz x) {
  Lz z;
  z.l = x.l << 24;
  z.h = __funnelshift_l(x.l, x.h, 24);
  z.k = (int32_t)__funnelshift_l(x.h, (uint32_t)x.k, 24);
  return z;
}

}  // namespace gl
