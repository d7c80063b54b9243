// Goldilocks NTT building blocks shared by the multiply kernels.
//
// Transform structure (this engine's design, not the reference's): a
// length-N = 2^L transform is split into HBM passes of radix R_p = 2^r_p.
// Pass p works on blocks of M_p = R_p * S_p consecutive words and, inside a
// block, on R_p rows of stride S_p.  The forward direction is a
// decimation-in-frequency split: per column j it takes the R_p-point DFT
// over the rows, multiplies output row f by w_M^(f*j) and stores it back in
// place, so every output row is an independent length-S_p problem for the
// next pass.  The spectrum ends in a fixed digit-reversed order; the
// pointwise product does not care, and the inverse passes (the exact mirror)
// restore natural order.  This is the reference's four-step decomposition
// (crates/bignum/src/ntt.rs:905-1105) without the transposes: strided tiles
// are read as coalesced 64-byte (or wider) row segments.
//
// Inside a pass the R_p-point DFT runs as two rounds of radix 4 to 32 held in
// registers; the short products and the merged splitting levels run two or three
// rounds of radix 8 or 16.  2 is a 192nd root of unity mod p, and the root tables
// are built so that the 64th root of unity is 2^3: the butterflies' internal
// twiddles are constant shifts.
#pragma once
#include <cstdint>
#include <type_traits>
#include "gl.cuh"

namespace pimul {

// Root tables.  rho is a primitive 2^32-th root of unity with
// rho^(2^26) = 8 (the 64th root of unity is 2^3).  Every twiddle of every
// transform length is a power of rho.
struct Roots {
  const uint64_t* lo;   // rho^e, e in [0, 2^16)
  const uint64_t* hi;   // rho^(e * 2^16), e in [0, 2^16)
  const uint64_t* w12;  // w_4096^t = rho^(t * 2^20), t in [0, 4096)
  const uint64_t* lvl;  // per-level tables: w_(2^k)^x at lvl[2^k + x], 1 <= k <= LVL_MAX
  const uint64_t* near; // w_(2^L)^(+-x) for x < 4096, LVL_MAX < L <= 32 (see near_table)
  const uint64_t* rt;   // round twiddles of the two-round passes (see rt_offset)
};

constexpr int LVL_MAX = 20;
constexpr int NEAR_LEVELS = 32 - LVL_MAX;  // transform lengths 2^21 .. 2^32

// The 4096 powers w_(2^L)^x (inverse: w_(2^L)^-x), x < 4096, of a length
// 2^L > 2^LVL_MAX.  A first-pass twiddle w^(f (j0 + jj)) with f jj < 4096
// is w^(f j0) (staged per CTA) times one entry of this 32 KB table, which
// stays in L1, instead of two loads from the 512 KB rho tables.
__device__ __forceinline__ const uint64_t* near_table(const Roots& R, int L, bool inverse) {
  return R.near + ((size_t)(L - LVL_MAX - 1) * 2 + (inverse ? 1 : 0)) * 4096;
}

// rho^e for e in [0, 2^32).
__device__ __forceinline__ uint64_t rho_pow(const Roots& R, uint32_t e) {
  uint64_t a = __ldg(R.lo + (e & 0xFFFFu));
  uint32_t h = e >> 16;
  return h ? gl::mul(a, __ldg(R.hi + h)) : a;
}

// w_M^x for M = 2^mlog and x mod 2^mlog; inverse gives w_M^(-x).  Levels up to
// 2^20 read one contiguous table; longer ones combine two table entries.
__device__ __forceinline__ uint64_t root_pow32(const Roots& R, int mlog, uint32_t x, bool inverse) {
  const uint32_t mask = mlog >= 32 ? 0xFFFFFFFFu : (1u << mlog) - 1;
  x &= mask;
  if (inverse) x = (0u - x) & mask;
  if (mlog <= LVL_MAX) return __ldg(R.lvl + (1u << mlog) + x);
  return rho_pow(R, x << (32 - mlog));
}

// Shared-memory index with one pad word per 16 to spread 8-byte banks.
__host__ __device__ __forceinline__ constexpr uint32_t spad(uint32_t lin) { return lin + (lin >> 4); }

// 8-point DFT (INV: unscaled inverse) of lazy values, folded outputs at
// v[STEP k]; x[0] carries the bias of lz_bias.  w^-s = -w^(96 - s) turns the
// inverse's twiddles into shifts with the signs swapped.
template <bool INV, int STEP>
__device__ __forceinline__ void dft8_lz(const gl::Lz* x, uint64_t* v) {
  using namespace gl;
  if constexpr (!INV) {
    // stage 1: x_m +- x_(m+4); the differences d_m carry the twiddle w^m
    Lz a0 = lz_add(x[0], x[4]), d0 = lz_sub(x[0], x[4]);
    Lz a1 = lz_add(x[1], x[5]), d1 = lz_sub(x[1], x[5]);
    Lz a2 = lz_add(x[2], x[6]), d2 = lz_sub(x[2], x[6]);
    Lz a3 = lz_add(x[3], x[7]), d3 = lz_sub(x[3], x[7]);
    // even outputs: radix 4 on the sums
    Lz c0 = lz_add(a0, a2), c2 = lz_sub(a0, a2);
    Lz c1 = lz_add(a1, a3), c3 = lz_shl<48>(lz_sub(a1, a3));
    v[0] = fold(lz_add(c0, c1));
    v[4 * STEP] = fold(lz_sub(c0, c1));
    v[2 * STEP] = fold(lz_add(c2, c3));
    v[6 * STEP] = fold(lz_sub(c2, c3));
    // odd outputs: radix 4 on b_m = w^m d_m.  With g = w^2 d3,
    // b1 + b3 = w (d1 + g) and (b1 - b3) w^2 = w^3 (d1 - g), so every shift
    // acts on a value with a small overflow count and the one by w (24 bits)
    // can stay lazy
    Lz b2 = lz_shl<48>(d2);
    Lz e0 = lz_add(d0, b2), e2 = lz_sub(d0, b2);
    Lz g = lz_shl<48>(d3);
    Lz e1 = lz_shl24_wide(lz_add(d1, g)), e3 = lz_shl<72>(lz_sub(d1, g));
    v[1 * STEP] = fold(lz_add(e0, e1));
    v[5 * STEP] = fold(lz_sub(e0, e1));
    v[3 * STEP] = fold(lz_add(e2, e3));
    v[7 * STEP] = fold(lz_sub(e2, e3));
  } else {
    // radix 2 on the bit-reversed inputs (x0, x4, x2, x6, x1, x5, x3, x7)
    Lz s01 = lz_add(x[0], x[4]), d01 = lz_sub(x[0], x[4]);
    Lz s23 = lz_add(x[2], x[6]), d23 = lz_sub(x[2], x[6]);
    Lz s45 = lz_add(x[1], x[5]), d45 = lz_sub(x[1], x[5]);
    Lz s67 = lz_add(x[3], x[7]), d67 = lz_sub(x[3], x[7]);
    Lz t23 = lz_shl<48>(d23), t67 = lz_shl<48>(d67);
    Lz v0 = lz_add(s01, s23), v2 = lz_sub(s01, s23);
    Lz v1 = lz_sub(d01, t23), v3 = lz_add(d01, t23);
    Lz v4 = lz_add(s45, s67), v6 = lz_sub(s45, s67);
    Lz v5 = lz_sub(d45, t67), v7 = lz_add(d45, t67);
    Lz t5 = lz_shl<72>(v5), t6 = lz_shl<48>(v6), t7 = lz_shl24_wide(v7);
    v[0] = fold(lz_add(v0, v4));
    v[4 * STEP] = fold(lz_sub(v0, v4));
    v[1 * STEP] = fold(lz_sub(v1, t5));
    v[5 * STEP] = fold(lz_add(v1, t5));
    v[2 * STEP] = fold(lz_sub(v2, t6));
    v[6 * STEP] = fold(lz_add(v2, t6));
    v[3 * STEP] = fold(lz_sub(v3, t7));
    v[7 * STEP] = fold(lz_add(v3, t7));
  }
}

// First stage of a 2^B-point decimation in frequency, elements M ..: x_M +
// x_(M+H) and (x_M - x_(M+H)) w^M, w = 2^(192 / 2^B) (INV: (x_(M+H) - x_M)
// 2^(96 - s) for w^-M = 2^-s = -2^(96-s)).  UPPER0: x_(M+H) is zero.
template <int B, bool INV, bool UPPER0 = false, int M = 1>
__device__ __forceinline__ void dif_stage(gl::Lz* x) {
  using namespace gl;
  constexpr int H = 1 << (B - 1), W = 192 >> B;
  if constexpr (M < H) {
    if constexpr (UPPER0) {
      static_assert(!INV, "zero upper halves only come in forward");
      x[M + H] = lz_shl<W * M>(x[M]);
    } else {
      const Lz a = lz_add(x[M], x[M + H]);
      if constexpr (!INV)
        x[M + H] = lz_shl<W * M>(lz_sub(x[M], x[M + H]));
      else
        x[M + H] = lz_shl<96 - W * M>(lz_sub(x[M + H], x[M]));
      x[M] = a;
    }
    dif_stage<B, INV, UPPER0, M + 1>(x);
  }
}

// DFT of 2^B lazy values (B = 2 .. 5; INV: its unscaled inverse) with w =
// 2^(192 / 2^B), the 2^B-th root of unity: all internal twiddles are constant
// shifts.  Natural-order folded outputs at v[STEP k].  x[0] carries the bias
// of lz_bias; |k| <= 1 in the other inputs (e.g. products from lz_mul); x is
// overwritten.  UPPER0 (forward): inputs 2^(B-1) .. are zero (not read).
template <int B, bool INV, bool UPPER0 = false, int STEP = 1>
__device__ __forceinline__ void dft_lz(gl::Lz* x, uint64_t* v) {
  static_assert(!UPPER0 || B > 3, "a zero upper half needs 16 points or more");
  if constexpr (B == 2) {
    using namespace gl;
    const Lz a = lz_add(x[0], x[2]), c = lz_sub(x[0], x[2]);
    const Lz b = lz_add(x[1], x[3]);
    const Lz d = lz_shl<48>(INV ? lz_sub(x[3], x[1]) : lz_sub(x[1], x[3]));
    v[0] = fold(lz_add(a, b));
    v[1 * STEP] = fold(lz_add(c, d));
    v[2 * STEP] = fold(lz_sub(a, b));
    v[3 * STEP] = fold(lz_sub(c, d));
  } else if constexpr (B == 3) {
    dft8_lz<INV, STEP>(x, v);
  } else {
    constexpr int H = 1 << (B - 1);
    if constexpr (UPPER0) {
      x[H] = x[0];
    } else {
      const gl::Lz a = gl::lz_add(x[0], x[H]);
      x[H] = gl::lz_sub(x[0], x[H]);
      x[0] = a;
    }
    dif_stage<B, INV, UPPER0>(x);
    dft_lz<B - 1, INV, false, 2 * STEP>(x, v);
    dft_lz<B - 1, INV, false, 2 * STEP>(x + H, v + STEP);
  }
}

// 3-point DFT (INV: its inverse) with the cube root of unity w = 2^64: with
// 1 + w + w^2 = 0 both other outputs need only w (x1 - x2).
template <bool INV>
__device__ __forceinline__ void dft3_lz(gl::Lz x0, gl::Lz x1, gl::Lz x2, gl::Lz* y) {
  using namespace gl;
  const Lz t = lz_shl<64>(lz_sub(x1, x2));
  y[0] = lz_add(x0, lz_add(x1, x2));
  y[INV ? 2 : 1] = lz_add(lz_sub(x0, x2), t);
  y[INV ? 1 : 2] = lz_sub(lz_sub(x0, x1), t);
}

// 12-point DFT (INV: its unscaled inverse) with w = 2^16: n = 4a + b, k = c +
// 3d, a 3-point DFT over a, the twiddles w^(b c) = 2^(16 b c), a 4-point DFT
// over b.  (w^-s = -2^(96 - s); w^6 = 2^96 = -1.)  As dft_lz otherwise.
template <bool INV>
__device__ __forceinline__ void dft12_lz(const gl::Lz* x, uint64_t* v) {
  using namespace gl;
  Lz y[4][3];
#pragma unroll
  for (int b = 0; b < 4; b++) dft3_lz<INV>(x[b], x[4 + b], x[8 + b], y[b]);
#pragma unroll
  for (int c = 0; c < 3; c++) {
    Lz z1 = y[1][c], z2 = y[2][c], z3 = y[3][c];
    // the inverse's twiddles are those of 96 - s with the sign of z_b turned
    constexpr bool NEG = INV;
    if (c == 1) z1 = lz_shl<INV ? 80 : 16>(z1), z2 = lz_shl<INV ? 64 : 32>(z2), z3 = lz_shl<48>(z3);
    if (c == 2) z1 = lz_shl<INV ? 64 : 32>(z1), z2 = lz_shl<INV ? 32 : 64>(z2);
    const bool n1 = c > 0 && NEG, n2 = c > 0 && NEG;
    const bool n3 = c == 2 || (c == 1 && NEG);  // 2^96 = 2^-96 = -1 for c = 2
    const Lz a = n2 ? lz_sub(y[0][c], z2) : lz_add(y[0][c], z2);
    const Lz e = n2 ? lz_add(y[0][c], z2) : lz_sub(y[0][c], z2);
    // b = z1 + z3 and z1 - z3 with their signs
    const Lz s = n1 == n3 ? lz_add(z1, z3) : lz_sub(z1, z3);
    const Lz d = n1 == n3 ? lz_sub(z1, z3) : lz_add(z1, z3);
    const Lz t = lz_shl<48>(d);
    v[c] = fold(n1 ? lz_sub(a, s) : lz_add(a, s));
    v[c + 6] = fold(n1 ? lz_add(a, s) : lz_sub(a, s));
    v[c + 3] = fold((n1 != INV) ? lz_sub(e, t) : lz_add(e, t));
    v[c + 9] = fold((n1 != INV) ? lz_add(e, t) : lz_sub(e, t));
  }
}

// ----------------------------------------------------------- two-round passes
// An HBM pass of radix 2^R (R = 5 .. 9) is two rounds in registers, radix
// 2^B1 over rows 2^B2 apart and radix 2^B2 over the 2^B2 rows of each result,
// with one exchange through shared memory between them: a length-512 DFT
// costs one general twiddle product per element (w_512^(k1 m)) instead of the
// two of an 8 x 8 x 8 split, its other twiddles being shifts (the 32nd root
// of unity is 2^6), and the first round reads and the second one writes HBM
// directly.  The integer pipes bind (ALU 60 %, IMAD 72 % busy before), so the
// split that needs the fewest instructions per element is taken; against three
// shared-memory rounds of radix 8 a 2^25-point pass of radix 2^9 went from 203
// to 154 us (columns, 3.5 TB/s) and 156 to 114 us (contiguous, 4.7 TB/s), the
// 2^30 x 2^30-bit product from 7.46 to 5.62 ms.  Forward: output index k1 of
// round 1 and k2 of round 2 (row k1 2^B2 + k2) hold frequency k1 + 2^B1 k2.
__host__ __device__ constexpr int pass_b1(int r) { return r <= 6 ? 3 : r <= 8 ? 4 : 5; }
__host__ __device__ constexpr int pass_b2(int r) { return r - pass_b1(r); }

// Frequency index held at row `row` after a pass of radix 2^R.  (A bit
// permutation: pass_freq(a | b) = pass_freq(a) | pass_freq(b) for disjoint
// bit sets.)
template <int R>
__host__ __device__ __forceinline__ constexpr uint32_t pass_freq(uint32_t row) {
  return (row >> pass_b2(R)) | ((row & ((1u << pass_b2(R)) - 1)) << pass_b1(R));
}

// Column passes: a CTA of 128 threads takes 2^R rows x 2^T columns, T = 3 for
// R = 8, 9 and 4 for R = 6, 7 (64- and 128-byte row segments; every thread has
// one item in the round of radix 2^B1 and one or two in the other).  Exchange
// element (k1, m, column) at k1 KS + (m << T | column); for T = 3 the eight
// pad words put the two k1 of a half-warp on different banks.
constexpr int PASS_THREADS = 128;
template <int R>
struct ColGeom {
  static constexpr int B1 = pass_b1(R), B2 = pass_b2(R);
  static constexpr int T = R >= 8 ? 3 : 4;
  static constexpr int TILE = R + T;                          // log2 words per CTA
  static constexpr uint32_t TM = (1u << T) - 1;
  static constexpr uint32_t KS = (1u << (B2 + T)) + (T == 3 ? 8 : 0);
  static constexpr uint32_t XWORDS = (1u << B1) * KS;         // exchange area
  static constexpr int ITERS2 = (1 << (B1 + T)) / PASS_THREADS;  // items per thread of the (k1, column) round
  static_assert((1 << (B2 + T)) == PASS_THREADS, "one (m, column) item per thread");
};

// Contiguous passes: each warp owns 32 2^B1 words (whole blocks of 2^R), so
// only __syncwarp separates its rounds.  Exchange element (block, k1, m) at
// (block 2^B1 + k1) (2^B2 + 1) + m, plus 8 words per block for R = 7 (blocks
// 144 words apart would share banks).
template <int R>
struct RowGeom {
  static constexpr int B1 = pass_b1(R), B2 = pass_b2(R);
  static constexpr uint32_t WWORDS = 32u << B1;               // words per warp
  static constexpr int TILE = 7 + B1;                         // log2 words per CTA (four warps)
  static constexpr uint32_t KS = (1u << B2) + 1;
  static constexpr uint32_t BPAD = R == 7 ? 8 : 0;
  static constexpr uint32_t XWORDS = (WWORDS >> B2) * KS + (WWORDS >> R) * BPAD;  // exchange words per warp
  static constexpr int ITERS2 = (int)(WWORDS >> B2) / 32;
};

// Round twiddles of a pass, in exchange order: forward w_(2^R)^(k1 m) at
// [m 2^B1 + k1], inverse w_(2^R)^-(k1 m) at [k1 2^B2 + m] (L1-resident: 4 KB
// per direction for R = 9).
constexpr uint32_t RT_WORDS = 2 * ((1u << 10) - (1u << 5));
__host__ __device__ constexpr uint32_t rt_offset(int r, bool inverse) {
  return 2 * ((1u << r) - (1u << 5)) + (inverse ? 1u << r : 0);
}

// First passes of 192 = 16 x 12 rows, for transforms of 3 2^k points: output k1
// of the radix-16 round and k2 of the radix-12 round (row 12 k1 + k2) hold
// frequency k1 + 16 k2.  2 is the 192nd root of unity: the round twiddles are
// 2^(k1 m) at [m 16 + k1] and 2^-(k1 m) at [k1 12 + m], behind the others.
constexpr uint32_t RT3_WORDS = 2 * 192;
struct ThreeGeom {
  static constexpr int T = 3;                       // eight columns
  static constexpr uint32_t ROWS = 192, KS = 12 * 8 + 8;
  static constexpr uint32_t XWORDS = 16 * KS;
  static constexpr uint32_t CWORDS = ROWS * 9;      // coefficients, one pad word per row
};

// Forward round 2 / inverse round 1 share the exchange layout (k1 fixed, m
// over the inputs); forward round 1 / inverse round 2 have m fixed.
// Forward round 2's inputs: exchange words times their round twiddles.
template <int R>
__device__ __forceinline__ void pass_fwd2(const uint64_t* sx, uint32_t stride, const uint64_t* __restrict__ rt, uint32_t k1,
                                          uint64_t* v) {
  constexpr int B1 = pass_b1(R), B2 = pass_b2(R);
  gl::Lz x[1 << B2];
#pragma unroll
  for (int m = 0; m < (1 << B2); m++) v[m] = sx[m * stride];
  x[0] = gl::lz_bias(gl::lz(v[0]));  // w^0 = 1
#pragma unroll
  for (int m = 1; m < (1 << B2); m++) x[m] = gl::lz_mul(v[m], __ldg(rt + (m << B1) + k1));
  dft_lz<B2, false>(x, v);
}

// Inverse round 2: over k1, inputs times their round twiddles.
template <int R>
__device__ __forceinline__ void pass_inv2(const uint64_t* sx, uint32_t stride, const uint64_t* __restrict__ rt, uint32_t m,
                                          uint64_t* v) {
  constexpr int B1 = pass_b1(R), B2 = pass_b2(R);
  gl::Lz x[1 << B1];
#pragma unroll
  for (int k = 0; k < (1 << B1); k++) v[k] = sx[k * stride];
  x[0] = gl::lz_bias(gl::lz(v[0]));
#pragma unroll
  for (int k = 1; k < (1 << B1); k++) x[k] = gl::lz_mul(v[k], __ldg(rt + (k << B2) + m));
  dft_lz<B1, true>(x, v);
}

}  // namespace pimul
