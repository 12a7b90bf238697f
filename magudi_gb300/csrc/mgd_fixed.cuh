// mgd_fixed.cuh -- interior stencil sums in exact integer arithmetic.
//
// GB300's FP64 pipe takes 64 cycles per warp instruction and SM sub-partition
// (76 for an addition); 32-bit integer instructions take 1 to 2 and IMAD.WIDE
// about 5. The interior coefficients of the SBP first derivatives and of the
// composite dissipation are integers over a common denominator (672, -168,
// 32, -3 over 840; 56, -28, 8, -1 and -70 over 256), so an interior stencil
// is an integer sum once its taps share an exponent:
//   - the largest exponent E among the taps gives the unit 2^(E - 61); each
//     tap's 53-bit significand becomes a signed integer below 2^62 of that
//     unit. Taps of up to 9 binary places below the largest stay exact, the
//     others lose less than one unit, 2^-61 of the largest tap;
//   - differences (or sums) of opposite taps and their products with the
//     integer coefficients are exact in 96 bits;
//   - the sum is normalised to 64 bits, multiplied by 1/denominator to 64 bits
//     and rounded once to a double.
// So the result carries one rounding of its own and at most a few units of
// 2^-61 of the largest tap, against one rounding per operation in FP64
// arithmetic. FP64 does better in one case: large opposite taps cancel and the
// others are so much smaller that the integers lose bits of them. That case,
// taps that are infinite or not numbers, and stencils whose largest tap is
// near the ends of the exponent range take the FP64 sum; so zeros stay zeros
// on a symmetry line, whatever the sign of the field's zeros.
//
// Measured over L1-resident data with 16 warps per SM: 572 cycles per warp and
// sub-partition for the eight-tap FP64 sum, 206 in integers (before the test
// for cancelling taps); and the FP64 pipe is left to the pointwise arithmetic,
// which runs at the same time. Stage kernels, FP64 sums -> integer sums,
// microseconds a launch: 128^3 periodic, composite dissipation 623 -> 270 (74%
// of the integer pipe), gradient/flux 681 -> 425, divergence 701 -> 476,
// adjoint diffusion 404 -> 246; 201^2, 12.3 -> 8.2, 20.5 -> 16.4, 16.4 -> 12.4
// and 10.4 -> 8.3. (By this change alone; the kernels' comments have what
// followed.) The test for cancelling taps costs 2D and 3D runs about 1% and the
// persistent batch 4%: after the sum, with the taps loaded again in a function
// of its own; keeping them for it cost the 128^3 forward stage 27%, the
// smallest and largest of all taps 15%.
#pragma once

#include <cstdint>

namespace mgd {

// Interior stencil c_0 x_0 + sum_j c_j (x_j -+ x_-j) over integers:
// c_j = s (-1)^(j+1) a[j] / den with a[j] >= 0 and s = +1 or -1; symmetric
// operators have c_0 = -s a[0] / den. Skew: rcp = 2^(64 + shift) / den rounded,
// with 1/2 <= 2^shift / den < 1. Symmetric: den = 2^shift. valid: the
// operator has this form.
struct FixedOp {
  int a[5];
  int half;                // taps beyond it have coefficient 0 (padding)
  int shift;
  unsigned flip;           // 0x80000000 when s = -1
  int valid;
  unsigned long long rcp;
};

__device__ __forceinline__ uint32_t hiWord(double x) { return (uint32_t)__double2hiint(x); }

// The tap x in units of 2^(E - 1023 - 61): its significand with the leading
// bit at bit 61, shifted right by its distance from the largest exponent.
// top = (E << 21) | 0x1fffff. Negative taps are one's complements, i.e. one
// unit lower than their value (opposite taps of equal sign cancel it). The
// distance joins `below` from bit 21 on.
__device__ __forceinline__ long long alignTap(double x, uint32_t top, uint32_t& below) {
  const uint32_t h = hiWord(x), l = (uint32_t)__double2loint(x);
  const uint32_t t = top - (h + h), s = t >> 21;
  below |= t;
  const uint32_t m = (uint32_t)((int)h >> 31);
  const uint32_t hi = (__funnelshift_l(l, h, 9) & 0x1fffffffu) ^ (m ^ 0x20000000u);
  const uint32_t lo = (l << 9) ^ m;
  long long r;  // shr clamps shifts beyond 63
  asm("shr.s64 %0, %1, %2;" : "=l"(r) : "l"((long long)(((unsigned long long)hi << 32) | lo)), "r"(s));
  return r;
}

__device__ __forceinline__ long long alignTap(double x, uint32_t top) {
  uint32_t below = 0;
  return alignTap(x, top, below);
}

// (T 2^32 + r) 2^(E - 1023 - 61) / den as a double, rounded once.
template <bool POW2>
__device__ __forceinline__ double packFixed(long long T, uint32_t r, uint32_t E, const FixedOp& F) {
  const uint32_t t1 = (uint32_t)((unsigned long long)T >> 32), t0 = (uint32_t)T;
  const uint32_t s = (uint32_t)((int)t1 >> 31);
  uint32_t u0 = r ^ s, u1 = t0 ^ s, u2 = t1 ^ s;
  asm("sub.cc.u32 %0, %0, %3;\n\tsubc.cc.u32 %1, %1, %3;\n\tsubc.u32 %2, %2, %3;"
      : "+r"(u0), "+r"(u1), "+r"(u2)
      : "r"(s));
  int e = (int)E + 34 - F.shift;  // biased exponent of a leading bit at bit 95, over 2^shift
  if (u2 == 0) { u2 = u1; u1 = u0; u0 = 0; e -= 32; }
  if (u2 == 0) { u2 = u1; u1 = 0; e -= 32; }
  const int n = __clz((int)u2);
  uint32_t hi = __funnelshift_l(u1, u2, n), lo = __funnelshift_l(u0, u1, n);
  e -= n + 1;  // the significand's implicit bit adds one to the exponent field
  uint32_t sh = 11;
  if constexpr (!POW2) {
    const uint32_t rh = (uint32_t)(F.rcp >> 32), rl = (uint32_t)F.rcp;
    const unsigned long long y = (unsigned long long)hi * rh + __umulhi(hi, rl) + __umulhi(lo, rh);
    hi = (uint32_t)(y >> 32);
    lo = (uint32_t)y;
    const uint32_t b = hi >> 31;  // leading bit at bit 63 or 62
    sh = 10u + b;
    e += (int)b - 1;
  }
  uint32_t ml = __funnelshift_r(lo, hi, sh), mh = hi >> sh;
  mh += (uint32_t)e << 20;
  const uint32_t half = (lo >> (sh - 1)) & 1u;
  asm("add.cc.u32 %0, %0, %2;\n\taddc.u32 %1, %1, 0;" : "+r"(ml), "+r"(mh) : "r"(half));
  mh |= (s ^ F.flip) & 0x80000000u;
  if (u2 == 0) mh = ml = 0;
  return __hiloint2double((int)mh, (int)ml);
}

// Whether n taps are all zero.
__device__ __forceinline__ bool allZero(const double* t, int n) {
  unsigned long long any = 0;
#pragma unroll
  for (int j = 0; j < n; ++j) any |= (unsigned long long)__double_as_longlong(t[j]);
  return (any << 1) == 0;
}

// Twice the largest high word (sign dropped) of the taps.
__device__ __forceinline__ uint32_t largestTap(const double* p, const double* m) {
  uint32_t top = 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint32_t hp = hiWord(p[j]), hm = hiWord(m[j]);
    top = max(top, max(hp + hp, hm + hm));
  }
  return top;
}

// Whether the largest tap's exponent lies in the range of the integer form.
__device__ __forceinline__ bool inFixedRange(uint32_t top) { return (top >> 21) - 128u < 1900u; }

// Finite taps beyond a narrow stencil's half width, whose coefficients are 0,
// give way to its nearest ones, so that they do not set the unit. Infinities
// and NaN stay and take the FP64 sum.
__device__ __forceinline__ void dropPadding(double* p, double* m, int half) {
#pragma unroll
  for (int j = 1; j < 4; ++j)
    if (j >= half) {
      if ((hiWord(p[j]) & 0x7ff00000u) != 0x7ff00000u) p[j] = p[0];
      if ((hiWord(m[j]) & 0x7ff00000u) != 0x7ff00000u) m[j] = m[0];
    }
}

// Skew stencil over the taps p[j] = x_{j+1}, m[j] = x_{-(j+1)}, whose largest
// is in range. cancel: the taps are spread (one of p is zero or 8 or more
// binary places below the largest; 10 lose bits) and every pair cancels to
// below 2^-11 of the largest, those of m being as small as their p then. The
// FP64 sum's roundings are below the bits that the integers lose (2^-61 of the
// largest tap), and it keeps what the small taps give; zeros on a symmetry
// line among that.
__device__ __forceinline__ bool pairsCancel(long long d1, long long d2, long long d3, long long d4) {
  // upper words: the leading bit of the largest tap is bit 29 there
  auto bits = [](long long d) { return (uint32_t)(d >> 32) + (1u << 18); };
  return (bits(d1) | bits(d2) | bits(d3) | bits(d4)) < 1u << 19;
}
__device__ __forceinline__ double skewFixed(const double* p, const double* m, uint32_t top, const FixedOp& F,
                                            bool& cancel) {
  const uint32_t E = top >> 21;
  top |= 0x1fffffu;
  uint32_t below = 0;
  const long long d1 = alignTap(p[0], top, below) - alignTap(m[0], top);
  const long long d2 = alignTap(m[1], top) - alignTap(p[1], top, below);
  const long long d3 = alignTap(p[2], top, below) - alignTap(m[2], top);
  const long long d4 = alignTap(m[3], top) - alignTap(p[3], top, below);
  cancel = below >= 8u << 21 && pairsCancel(d1, d2, d3, d4);
  unsigned long long lo = (unsigned long long)(uint32_t)d1 * (uint32_t)F.a[1];
  lo += (unsigned long long)(uint32_t)d2 * (uint32_t)F.a[2];
  lo += (unsigned long long)(uint32_t)d3 * (uint32_t)F.a[3];
  lo += (unsigned long long)(uint32_t)d4 * (uint32_t)F.a[4];
  long long T = (long long)(lo >> 32);
  T += (long long)(int)(d1 >> 32) * F.a[1];
  T += (long long)(int)(d2 >> 32) * F.a[2];
  T += (long long)(int)(d3 >> 32) * F.a[3];
  T += (long long)(int)(d4 >> 32) * F.a[4];
  return packFixed<false>(T, (uint32_t)lo, E, F);
}

// The same test before the sum, for the kernel that keeps the taps for it.
__device__ __forceinline__ bool skewCancels(const double* p, const double* m, uint32_t top) {
  top |= 0x1fffffu;
  uint32_t below = 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) below |= top - (hiWord(p[j]) + hiWord(p[j]));
  if (below < 8u << 21) return false;
  return pairsCancel(alignTap(p[0], top) - alignTap(m[0], top), alignTap(m[1], top) - alignTap(p[1], top),
                     alignTap(p[2], top) - alignTap(m[2], top), alignTap(m[3], top) - alignTap(p[3], top));
}

// K skew stencils at once; the bits of the fields that need the FP64 sum (a
// field's result does not depend on the others'). A field at rest (all taps
// zero) needs none. One branch for all K leaves their sums in one block of
// code, which the compiler interleaves. KEEP: decided before the sum, with the
// taps still at hand.
template <int K, bool KEEP = false>
__device__ __forceinline__ unsigned fixedSkew(double (*p)[4], double (*m)[4], const FixedOp& F, double* out) {
  if (F.half < 4)
#pragma unroll
    for (int k = 0; k < K; ++k) dropPadding(p[k], m[k], F.half);
  bool cancel;
  if constexpr (K == 1) {
    const uint32_t t = largestTap(p[0], m[0]);
    if (!inFixedRange(t) || (KEEP && skewCancels(p[0], m[0], t))) {
      out[0] = 0.0;
      return allZero(p[0], 4) && allZero(m[0], 4) ? 0u : 1u;
    }
    out[0] = skewFixed(p[0], m[0], t, F, cancel);
    return !KEEP && cancel ? 1u : 0u;
  }
  uint32_t top[K];
  unsigned zero = 0, redo = 0;
  bool ok = true;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    top[k] = largestTap(p[k], m[k]);
    ok = ok && inFixedRange(top[k]);
  }
  if (!ok) {
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (!inFixedRange(top[k])) (allZero(p[k], 4) && allZero(m[k], 4) ? zero : redo) |= 1u << k;
  }
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const double s = skewFixed(p[k], m[k], top[k], F, cancel);
    const bool rest = zero >> k & 1u;
    out[k] = rest ? 0.0 : s;
    if (cancel && !rest) redo |= 1u << k;
  }
  return redo;
}

// Symmetric stencils of the axes through a point summed, x0 the centre tap of
// each (denominator a power of two); closed: bits of the axes that are left
// out, whose taps are 0. False when the sum needs FP64.
template <int ND>
__device__ __forceinline__ bool fixedSymmetric(double (*p)[4], double (*m)[4], double x0, unsigned closed,
                                               const FixedOp& F, double& out) {
  if (F.half < 4)
#pragma unroll
    for (int d = 0; d < ND; ++d) dropPadding(p[d], m[d], F.half);
  const uint32_t h0 = hiWord(x0) + hiWord(x0);
  uint32_t top = h0;
#pragma unroll
  for (int d = 0; d < ND; ++d) top = max(top, largestTap(p[d], m[d]));
  const uint32_t E = top >> 21, limit = (E - 11u) << 21;
  if (!inFixedRange(top) || h0 < limit) {
    // out of range; or a centre below 2^-11 of the largest tap, about which
    // every pair may cancel to that too: as with skew stencils, the FP64 sum
    // then keeps what the integers lose. 2D is often here, on the fronts of
    // waves, and compares words; in 3D their registers spill (128^3: 279 us
    // against 268 with FP64 sums)
    bool fp64 = true;
#pragma unroll
    for (int d = 0; d < ND; ++d)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if constexpr (ND == 2) {
          // both small, or of opposite sign and alike in 11 places
          const uint32_t hp = hiWord(p[d][j]), hm = hiWord(m[d][j]) ^ 0x80000000u;
          fp64 = fp64 && (max(hp + hp, hm + hm) < limit || hp - hm + 510u < 1021u);
        } else {
          const uint32_t h = hiWord(p[d][j] + m[d][j]);
          fp64 = fp64 && h + h < limit;
        }
      }
    if (fp64 || !inFixedRange(top)) {
      bool zero = allZero(&x0, 1);
#pragma unroll
      for (int d = 0; d < ND; ++d) zero = allZero(p[d], 4) && allZero(m[d], 4) && zero;
      out = 0.0;
      return zero;
    }
  }
  top |= 0x1fffffu;
  const long long d0 = alignTap(x0, top);
  const uint32_t a0 = (uint32_t)(F.a[0] * (ND - __popc(closed)));
  unsigned long long lp = 0, ln = (unsigned long long)(uint32_t)d0 * a0;
  long long T = -((long long)(int)(d0 >> 32) * (int)a0);
  // opposite taps of up to three axes: |sums| < 3 * 2^63, so each axis has its own products
#pragma unroll
  for (int d = 0; d < ND; ++d) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const long long t = alignTap(p[d][j], top) + alignTap(m[d][j], top);
      unsigned long long& l = j % 2 ? ln : lp;
      l += (unsigned long long)(uint32_t)t * (uint32_t)F.a[j + 1];
      T += (long long)(int)(t >> 32) * (j % 2 ? -F.a[j + 1] : F.a[j + 1]);
    }
  }
  const long long l = (long long)(lp - ln);
  T += l >> 32;
  out = packFixed<true>(T, (uint32_t)l, E, F);
  return true;
}

// ---------------------------------------------------------------------------
// 1/x and x^n in 64-bit fixed point, for the primitive variables: about 100
// and 300 cycles of the integer pipes instead of 8 and 27 FP64 instructions
// (64 cycles each). Q_k: an integer in units of 2^-k.
// ---------------------------------------------------------------------------

// The significand of a normal x with its leading bit at bit 63.
__device__ __forceinline__ unsigned long long significand(uint32_t h, uint32_t l) {
  const uint32_t m = (h & 0xfffffu) | 0x100000u;
  return ((unsigned long long)__funnelshift_l(l, m, 11) << 32) | (l << 11);
}

// Y 2^(e - 63), Y with its leading bit at bit 63 (or one unit of rounding
// below it), rounded half up to a positive double; biased is e + 1023.
__device__ __forceinline__ double packSignificand(unsigned long long Y, int biased) {
  unsigned long long r = (Y >> 11) + ((Y >> 10) & 1u);  // the leading bit adds one to the exponent field
  r += (unsigned long long)(unsigned)(biased - 1) << 52;
  return __longlong_as_double((long long)r);
}

// 1/x, rounded to nearest: a 32-bit seed Y0 of 1/m from the FP32 reciprocal,
// e0 = 1 - m Y0 (below 2^-21), and Y0 (1 + e0 + e0^2), whose next term is below
// 2^-63, rounded to 53 bits Q; its residual 2^105 - Q M, exact in 64 bits, then
// tells whether a neighbour is nearer (it is for one in a thousand, never by
// more than one unit). Values whose reciprocal is not normal take the division.
__device__ __forceinline__ double fixedReciprocal(double x) {
  const uint32_t h = hiWord(x), l = (uint32_t)__double2loint(x);
  const int be = (int)((h >> 20) & 0x7ffu);
  if ((unsigned)(be - 2) > 2042u) return 1.0 / x;
  const unsigned long long M = significand(h, l);  // Q63 of m in [1, 2)
  float seed;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(seed) : "f"(__uint_as_float(0x3f800000u | (uint32_t)(M >> 40 & 0x7fffffu))));
  const uint32_t y0 = __float2uint_rd(seed * 4294967296.0f);  // Q32, saturates at 1
  const unsigned long long p0 = (unsigned long long)(uint32_t)M * y0;
  const unsigned long long p1 = (M >> 32) * y0 + (p0 >> 32);  // (p1 : low word of p0) is Q95 of m Y0
  // e0 in Q75: 2^95 - p, shifted right by 20
  const long long d = (long long)(0x8000000000000000ull - p1);  // in units of 2^-63, |d| < 2^43
  const long long e0 = d * 4096 - (long long)((uint32_t)p0 >> 20);
  const int eh = (int)(e0 >> 24);                             // Q51
  const long long c = e0 + (((long long)eh * eh) >> 27);      // Q75
  const unsigned long long Y =
      ((unsigned long long)y0 << 32) + (unsigned long long)(__mul64hi((long long)y0 << 31, c) >> 10) - 2;  // Q64
  const long long M53 = (long long)(M >> 11);
  long long Q = (long long)((Y >> 11) + ((Y >> 10) & 1u));
  const long long R2 = -2 * (long long)((unsigned long long)Q * (unsigned long long)M53);
  Q += (R2 > M53 ? 1 : 0) - (R2 < -M53 ? 1 : 0);
  const double r = __longlong_as_double(Q + ((long long)(2044 - be) << 52));
  return __hiloint2double((int)((uint32_t)__double2hiint(r) | (h & 0x80000000u)), __double2loint(r));
}

// x^n = 2^(n log2 x), x = 2^e m: log2 m = T_j + log2(1 + r) with G_j a 32-bit
// 1/F_j, F_j = 1 + (j + 1/2)/512, r = m G_j - 1 exactly and T_j = -log2 G_j;
// 2^f = E_k 2^z with E_k = 2^((k + 1/2)/512). |r| and |z| stay below 2^-9.9,
// so five terms of log2(1 + r) and four of 2^z leave less than 2^-59. The
// table-driven split follows P. T. P. Tang (ACM TOMS 15(2), 1989; 16(4), 1990).
struct FixedPowTables {
  uint32_t g[512];            // Q32
  unsigned long long t[512];  // Q62
  unsigned long long e[512];  // Q63
};

// n in Q62, 2^-8 <= n < 2. False when x is outside [2^-400, 2^400).
__device__ __forceinline__ bool fixedPow(double x, unsigned long long n, const FixedPowTables* __restrict__ tab,
                                         double& out) {
  const uint32_t h = hiWord(x), l = (uint32_t)__double2loint(x);
  const int e = (int)(h >> 20) - 1023;  // the sign bit takes negative x out of range
  if ((unsigned)(e + 400) >= 800u) return false;
  const unsigned long long M = significand(h, l);
  const uint32_t j = (h >> 11) & 0x1ffu, g = __ldg(&tab->g[j]);
  const unsigned long long p0 = (unsigned long long)(uint32_t)M * g;
  const unsigned long long p1 = (M >> 32) * g + (p0 >> 32);
  const long long r = (long long)((p1 - 0x8000000000000000ull) << 9) + ((uint32_t)p0 >> 23);  // Q72
  const int rq = (int)(r >> 32);                                                             // Q40
  // log2(1 + r) = r (c1 + r (c2 + r (c3 + r (c4 + r c5)))), c_i = (-1)^(i+1) log2(e) / i
  constexpr int c3 = 2065442673, c4 = -1549082005, c5 = 1239265604;  // Q32
  constexpr long long c1 = 6653256548922161246ll, c2 = -3326628274461080623ll;  // Q62
  const int q3 = c3 + (__mulhi(c4 + (__mulhi(c5, rq) >> 8), rq) >> 8);
  const long long s2 = c2 + (((long long)q3 * rq) >> 10);
  const long long s1 = c1 + (__mul64hi(r, s2) >> 8);
  const long long log2m = (long long)__ldg(&tab->t[j]) + (__mul64hi(r, s1) >> 8);
  // n log2 x: the part of e exactly (Q62, two words), the part of m in Q60
  const unsigned long long lo = n * (unsigned long long)(long long)e;
  const long long hi = __mul64hi((long long)n, (long long)e);
  const unsigned long long w =
      ((lo & 0x3fffffffffffffffull) >> 2) + (unsigned long long)__mul64hi(log2m, (long long)n);  // Q60
  const int whole = (int)((hi << 2) | (long long)(lo >> 62)) + (int)((long long)w >> 60);
  const unsigned long long f = w << 4;  // Q64 fraction
  const uint32_t k = (uint32_t)(f >> 55);
  const long long z = (long long)((f & 0x7fffffffffffffull) - 0x40000000000000ull) << 8;  // Q72
  const int zq = (int)(z >> 32);
  // 2^z - 1 = z (d1 + z (d2 + z (d3 + z d4))), d_i = ln(2)^i / i!
  constexpr int d3 = 238388332, d4 = 41309550;  // Q32
  constexpr long long d1 = 3196577161300663915ll, d2 = 1107849223398934356ll;  // Q62
  const int q = d3 + (__mulhi(d4, zq) >> 8);
  const long long u2 = d2 + (((long long)q * zq) >> 10);
  const long long u1 = d1 + (__mul64hi(z, u2) >> 8);
  const long long p = __mul64hi(z, u1) << 2;  // Q72
  const unsigned long long E = __ldg(&tab->e[k]);
  const unsigned long long Y = E + (unsigned long long)(__mul64hi((long long)(E >> 1), p) >> 7) - 4;
  out = packSignificand(Y, whole + 1023);
  return true;
}

}  // namespace mgd
