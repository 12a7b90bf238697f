// mgd_device.cuh -- device-side building blocks: SBP operator application
// from constant-memory tables and the pointwise gas dynamics of magudi's
// CNSHelper (src/CNSHelperImpl.f90), with FP64 operands and results.
//
// Design note: on GB300 FP64 arithmetic runs on a narrow pipe (64 cycles a
// warp instruction and sub-partition). So the interior stencils, the
// reciprocals and the power law run in integers (mgd_fixed.cuh), and the
// pointwise algebra shares its products before it forms them. With that, the
// 3D kernels are near the FP64 and the integer pipe at once, and the code's
// size and the index arithmetic count too: loops over axes and fields that
// keep one copy of the stencil code are faster than unrolled ones.
#pragma once

#include <cstdint>

#include "mgd_fixed.cuh"

namespace mgd {

enum OpId { OP_D1 = 0, OP_D1ADJ = 1, OP_DISS = 2, OP_DISST = 3, OP_DCOMP = 4, OP_COUNT = 5 };

// Compile-time shape of each operator's boundary block.
template <int OP> struct OpShape;
template <> struct OpShape<OP_D1> { static constexpr int depth = 8, width = 12, half = 4; static constexpr bool skew = true; };
template <> struct OpShape<OP_D1ADJ> { static constexpr int depth = 12, width = 16, half = 4; static constexpr bool skew = true; };
template <> struct OpShape<OP_DISS> { static constexpr int depth = 2, width = 5, half = 2; static constexpr bool skew = false; };
template <> struct OpShape<OP_DISST> { static constexpr int depth = 8, width = 10, half = 2; static constexpr bool skew = false; };
template <> struct OpShape<OP_DCOMP> { static constexpr int depth = 8, width = 12, half = 4; static constexpr bool skew = false; };

// SBP schemes (defaults/discretization_scheme): index = MGD_SBP_* (4-8, 1-2,
// 2-4, 3-6). Every scheme's operators are stored in the fixed shapes of
// OpShape (the 4-8 shapes, the largest): lower-order closures are padded
// with interior rows and their interiors with zero coefficients.
constexpr int kSchemes = 4;

struct OpTables {
  double interior[kSchemes][OP_COUNT][9];  // offsets -half..half
  int asym[kSchemes][OP_COUNT];            // general interior sum and explicit right block
  FixedOp fixed[kSchemes][OP_COUNT];       // integer interiors (OP_D1, OP_D1ADJ, OP_DCOMP)
};

// One copy per translation unit; only mgd_kernels.cu launches kernels and
// fills them. Interior coefficients are uniform across a warp and live in
// constant memory; boundary-closure rows differ between lanes and are read
// from global memory through L1, which serves divergent addresses at once.
static __constant__ OpTables c_ops;
static __device__ double g_opLeft[kSchemes][OP_COUNT][16 * 12];
static __device__ double g_opRight[kSchemes][OP_COUNT][16 * 12];  // explicit right blocks (asym only)

// One direction of a block: n points along it, memory stride, periodicity,
// and the block's SBP scheme.
struct Axis {
  int n;
  int per;          // 0 none, 1 plane, 2 overlap
  long long stride;
  int scheme;       // MGD_SBP_*
};

// Index of point i + j along a periodic line (fillGhostPoints for one
// process, src/MPIHelperImpl.f90:113-390): PLANE wraps with period n;
// OVERLAP skips the duplicated end point.
__device__ __forceinline__ int wrapIndex(int i, int n, int per) {
  if (i < 0) return per == 2 ? i + n - 1 : i + n;
  if (i >= n) return per == 2 ? i - n + 1 : i - n;
  return i;
}

// y_i = (Op x)_i along one axis; `line` points at element 0 of the pencil.
// Follows applyOperator_{1,2,3} (src/StencilOperatorImpl.f90:35-457):
// sum over taps left to right, boundary rows from the left block and its
// (skew-)reflection on the right.
// Load of a stencil tap: through the read-only data path (NC), or as an
// ordinary cached load (ld.global.ca) for data that the same kernel launch
// writes elsewhere (the persistent batched kernel). The read-only path lies
// outside the memory model and may serve such data stale; ordinary loads
// after the acquiring fence of a grid barrier see the other CTAs' writes and
// still share L1 lines between neighbouring points within a phase.
template <bool NC>
__device__ __forceinline__ double tap(const double* p) {
  if constexpr (NC) return __ldg(p);
  else return __ldca(p);
}

// Interior stencil of OP in FP64 over the taps p[j] = x_{j+1}, m[j] =
// x_{-(j+1)} and the centre x0 (unused by skew operators), left to right;
// spelled out, so that every kernel that holds it rounds alike.
template <int OP>
__device__ __forceinline__ double interiorSumFp64(const double* p, const double* m, double x0, int scheme) {
  using S = OpShape<OP>;
  const double* __restrict__ cin = c_ops.interior[scheme][OP];
  double s = __dmul_rn(cin[S::half + 1], S::skew ? p[0] - m[0] : p[0] + m[0]);
#pragma unroll
  for (int j = 2; j <= S::half; ++j)
    s = fma(cin[S::half + j], S::skew ? p[j - 1] - m[j - 1] : p[j - 1] + m[j - 1], s);
  return S::skew ? s : fma(cin[S::half], x0, s);
}

// The interior taps of point i again, for the rare sums in FP64: volatile
// loads, so that the taps of the integer sum need not be kept for them.
__device__ __forceinline__ void interiorTapsAgain(const double* c, int i, const Axis& ax, double* p, double* m) {
  const double* line = c - i * ax.stride;
#pragma unroll
  for (int j = 1; j <= 4; ++j) {
    p[j - 1] = *(const volatile double*)(line + (long long)wrapIndex(i + j, ax.n, ax.per) * ax.stride);
    m[j - 1] = *(const volatile double*)(line + (long long)wrapIndex(i - j, ax.n, ax.per) * ax.stride);
  }
}
template <int OP>
__device__ __noinline__ double interiorSumAgain(const double* c, int i, Axis ax) {
  double p[4], m[4];
  interiorTapsAgain(c, i, ax, p, m);
  return interiorSumFp64<OP>(p, m, 0.0, ax.scheme);
}

// Interior stencils of OP of K fields, c + off(k): the first derivatives in
// integers where the taps allow it, field by field. The persistent batched
// kernel (NC = false) has one field at a time and keeps its taps for the FP64
// sum: a call inside it costs registers in all its phases, 16 runs 21.6 ms
// against 20.3 without.
template <int OP, int K, bool NC, class Off>
__device__ __forceinline__ void interiorSums(double (*p)[4], double (*m)[4], const double* __restrict__ c, Off off,
                                             int i, const Axis& ax, double* out) {
  static_assert(OP == OP_D1 || OP == OP_D1ADJ, "skew operators");
  const FixedOp& F = c_ops.fixed[ax.scheme][OP];
  unsigned redo = (1u << K) - 1u;
  if (F.valid) redo = fixedSkew<K, !NC>(p, m, F, out);
  if (redo == 0) return;
  if constexpr (!NC) {
    static_assert(K == 1, "one field");
    out[0] = interiorSumFp64<OP>(p[0], m[0], 0.0, ax.scheme);
    return;
  }
#pragma unroll
  for (int k = 0; k < K; ++k)
    if (redo >> k & 1u) out[k] = interiorSumAgain<OP>(c + off(k), i, ax);
}

// Boundary closure row of point i (i < depth or i >= n - depth) of a
// non-periodic line: CU taps' loads in flight at a time; the sum keeps its
// order either way. c points at the line's point i.
template <int OP, bool NC, int CU>
__device__ __forceinline__ double closureSum(const double* __restrict__ c, int i, long long st, const Axis& ax) {
  using S = OpShape<OP>;
  const double* __restrict__ line = c - i * st;
  if (i < S::depth) {
    const double* __restrict__ row = &g_opLeft[ax.scheme][OP][i * S::width];
    double s = __dmul_rn(__ldg(row), tap<NC>(line));
#pragma unroll CU
    for (int k = 1; k < S::width; ++k) s = fma(__ldg(row + k), tap<NC>(line + k * st), s);
    return s;
  }
  const int m = ax.n - 1 - i;
  const double* __restrict__ end = line + (long long)(ax.n - S::width) * st;
  // only the non-composite dissipation pair of SBP 3-6 is asymmetric
  if (!S::skew && (OP == OP_DISS || OP == OP_DISST) && c_ops.asym[ax.scheme][OP]) {
    // explicit right block, columns left to right
    const double* __restrict__ row = &g_opRight[ax.scheme][OP][m * S::width];
    double s = __dmul_rn(__ldg(row), tap<NC>(end));
#pragma unroll CU
    for (int k = 1; k < S::width; ++k) s = fma(__ldg(row + k), tap<NC>(end + k * st), s);
    return s;
  }
  const double* __restrict__ row = &g_opLeft[ax.scheme][OP][m * S::width];
  // right block = reflection of the left block, negated for skew operators
  double s = __dmul_rn(__ldg(row + S::width - 1), tap<NC>(end));
#pragma unroll CU
  for (int k = 1; k < S::width; ++k) s = fma(__ldg(row + S::width - 1 - k), tap<NC>(end + k * st), s);
  return S::skew ? -s : s;
}

template <int OP>
__device__ __forceinline__ bool inClosure(int i, const Axis& ax) {
  return ax.per == 0 && (i < OpShape<OP>::depth || i >= ax.n - OpShape<OP>::depth);
}

// Taps p[j] = x_{i+j+1}, m[j] = x_{i-j-1} of the interior stencil; a periodic
// line wraps near its ends only.
template <int HALF, bool NC>
__device__ __forceinline__ void interiorTaps(const double* __restrict__ c, int i, long long st, const Axis& ax,
                                             double* p, double* m) {
  if (i >= HALF && i < ax.n - HALF) {
#pragma unroll
    for (int j = 1; j <= HALF; ++j) {
      p[j - 1] = tap<NC>(c + j * st);
      m[j - 1] = tap<NC>(c - j * st);
    }
  } else {
    const double* __restrict__ line = c - i * st;
#pragma unroll
    for (int j = 1; j <= HALF; ++j) {
      p[j - 1] = tap<NC>(line + (long long)wrapIndex(i + j, ax.n, ax.per) * st);
      m[j - 1] = tap<NC>(line + (long long)wrapIndex(i - j, ax.n, ax.per) * st);
    }
  }
}

// (Op x)_i along one axis; c points at the point itself, X: the axis of unit
// stride.
template <int OP, bool NC = true, int CU = 1, bool X = false>
__device__ __forceinline__ double applyOp(const double* __restrict__ c, int i, const Axis& ax) {
  using S = OpShape<OP>;
  const long long st = X ? 1 : ax.stride;
  if (inClosure<OP>(i, ax)) return closureSum<OP, NC, CU>(c, i, st, ax);
  double p[S::half], m[S::half];
  interiorTaps<S::half, NC>(c, i, st, ax, p, m);
  if (!S::skew && (OP == OP_DISS || OP == OP_DISST) && c_ops.asym[ax.scheme][OP]) {
    const double* __restrict__ cin = c_ops.interior[ax.scheme][OP];
    double s = cin[0] * m[S::half - 1];
#pragma unroll
    for (int j = 1 - S::half; j <= S::half; ++j)
      s += cin[S::half + j] * (j < 0 ? m[-j - 1] : (j > 0 ? p[j - 1] : tap<NC>(c)));
    return s;
  }
  if constexpr (OP == OP_D1 || OP == OP_D1ADJ) {
    double s;
    interiorSums<OP, 1, NC>(&p, &m, c, [](int) { return 0LL; }, i, ax, &s);
    return s;
  } else {
    return interiorSumFp64<OP>(p, m, S::skew ? 0.0 : tap<NC>(c), ax.scheme);
  }
}

// The first derivative OP of the K fields c + off[k] along one axis, all taps
// loaded before the first sum (interior) or all fields' closure rows summed
// side by side: one round of load latency for the axis instead of K.
template <int OP, int K, bool NC>
__device__ __forceinline__ void applyOpFields(const double* __restrict__ c, const long long* off, int i, const Axis& ax,
                                              double* out) {
  using S = OpShape<OP>;
  const long long st = ax.stride;
  if (inClosure<OP>(i, ax)) {
    const bool left = i < S::depth;
    const double* __restrict__ row = &g_opLeft[ax.scheme][OP][(left ? i : ax.n - 1 - i) * S::width];
    const double* __restrict__ first = c - i * st + (left ? 0LL : (long long)(ax.n - S::width) * st);
#pragma unroll
    for (int w = 0; w < S::width; ++w) {
      const double r = __ldg(row + (left ? w : S::width - 1 - w));
#pragma unroll
      for (int k = 0; k < K; ++k) {
        const double x = tap<NC>(first + off[k] + w * st);
        out[k] = w == 0 ? __dmul_rn(r, x) : fma(r, x, out[k]);
      }
    }
    if (!left)
#pragma unroll
      for (int k = 0; k < K; ++k) out[k] = -out[k];
    return;
  }
  double p[K][4], m[K][4];
#pragma unroll
  for (int k = 0; k < K; ++k) interiorTaps<4, NC>(c + off[k], i, st, ax, p[k], m[k]);
  interiorSums<OP, K, NC>(p, m, c, [&](int k) { return off[k]; }, i, ax, out);
}

// The composite dissipation's interior stencils of the axes summed, in
// integers where the taps allow it; closed: bits of the axes left out, whose
// taps are 0.
template <int ND>
__device__ __forceinline__ double compositeInteriorSum(double (*p)[4], double (*m)[4], double x0, unsigned closed,
                                                       int scheme) {
  double s;
  const FixedOp& F = c_ops.fixed[scheme][OP_DCOMP];
  if (F.valid && fixedSymmetric<ND>(p, m, x0, closed, F, s)) return s;
  const double* __restrict__ cin = c_ops.interior[scheme][OP_DCOMP];
  s = __dmul_rn((ND - __popc(closed)) * cin[4], x0);
#pragma unroll
  for (int d = 0; d < ND; ++d)
#pragma unroll
    for (int j = 0; j < 4; ++j) s = fma(cin[5 + j], p[d][j] + m[d][j], s);
  return s;
}

// Composite dissipation sum_d Dc_d x at a point, all axes' interior stencils
// as one integer sum (they act on the same field, so one unit serves them):
// one normalisation instead of one per axis. An axis whose closure holds the
// point adds its FP64 row.
template <int ND, bool NC, int CU>
__device__ __forceinline__ double compositeDissipationSum(const double* __restrict__ c, const int* idx,
                                                          const Axis* ax) {
  double p[ND][4], m[ND][4], closure = 0.0;
  const double x0 = tap<NC>(c);
  unsigned closed = 0;
#pragma unroll
  for (int d = 0; d < ND; ++d) {
    const long long st = d == 0 ? 1 : ax[d].stride;
    if (inClosure<OP_DCOMP>(idx[d], ax[d])) {
      closure += closureSum<OP_DCOMP, NC, CU>(c, idx[d], st, ax[d]);
#pragma unroll
      for (int j = 0; j < 4; ++j) p[d][j] = m[d][j] = 0.0;
      closed |= 1u << d;
    } else {
      interiorTaps<4, NC>(c, idx[d], st, ax[d], p[d], m[d]);
    }
  }
  if (closed == (1u << ND) - 1u) return closure;
  const double s = compositeInteriorSum<ND>(p, m, x0, closed, ax[0].scheme);
  return closed ? s + closure : s;
}

// x != 0.0 with integer operations: false for +0 and -0 only, as the
// comparison is (NaN and every other value compare unequal to zero). GB300
// runs double-precision compares on the FP64 pipe, which the stage kernels
// keep busy; integer tests leave it to the arithmetic.
__device__ __forceinline__ bool nonzero(double x) { return (__double_as_longlong(x) << 1) != 0; }

// ---------------------------------------------------------------------------
// x^n for x > 0 in FP64 with few FP64 operations, after P. T. P. Tang's
// table-driven logarithm and exponential (ACM TOMS 15(2), 1989; 16(4), 1990):
//   log x = e ln2 + log(F) + log1p(m/F - 1), F from a 128-entry table
//   exp y = 2^(k/64) exp(r), |r| <= ln2/128, 2^(j/64) from a 64-entry table.
// Exponent and mantissa are split with integer operations, which do not
// occupy the FP64 pipe. Non-positive or non-finite x falls back to pow().
// ---------------------------------------------------------------------------
struct PowTables {
  double invF[128];   // G_j = 1 / F_j rounded, F_j = 1 + (j + 1/2)/128
  double logFhi[128]; // -log G_j, high part
  double logFlo[128]; // -log G_j, low part
  double exp2j[64];   // 2^(j/64)
};

__device__ __forceinline__ double fastPowPositive(double x, double n, const PowTables* __restrict__ tab) {
  const long long bits = __double_as_longlong(x);
  const int be = (int)((bits >> 52) & 0x7FF);
  // bits <= 0: x is -0, +0 or negative (the NaNs and infinities have be == 0x7FF)
  if (bits <= 0 || be == 0 || be == 0x7FF) return pow(x, n);
  const int e = be - 1023;
  const int j = (int)((bits >> 45) & 0x7F);
  const double m = __longlong_as_double((bits & 0x000FFFFFFFFFFFFFLL) | 0x3FF0000000000000LL);
  const double t = fma(m, __ldg(&tab->invF[j]), -1.0);  // |t| < 2^-8
  // log1p(t) - t = t^2 (-1/2 + t/3 - t^2/4 + ... - t^6/8)
  double q = -1.0 / 8.0;
  q = fma(q, t, 1.0 / 7.0);
  q = fma(q, t, -1.0 / 6.0);
  q = fma(q, t, 1.0 / 5.0);
  q = fma(q, t, -1.0 / 4.0);
  q = fma(q, t, 1.0 / 3.0);
  q = fma(q, t, -0.5);
  const double t2 = t * t;
  const double ln2hi = 6.93147180369123816490e-01, ln2lo = 1.90821492927058770002e-10;
  const double ed = (double)e;
  const double lo = fma(t2, q, fma(ed, ln2lo, __ldg(&tab->logFlo[j])));
  const double hi = fma(ed, ln2hi, __ldg(&tab->logFhi[j]));
  const double logx = hi + (t + lo);
  const double y = n * logx;
  // exp(y): y = k ln2/64 + r
  const double inv = 92.332482616893656877;  // 64 / ln 2
  const double shifter = 6755399441055744.0;   // 1.5 * 2^52: rounds to an integer
  const double kd_s = fma(y, inv, shifter);
  const long long kbits = __double_as_longlong(kd_s);
  const double kd = kd_s - shifter;
  const double l64hi = 0.01083042469326756, l64lo = 2.9815858269852933e-12;  // ln2/64 = hi + lo, hi*k exact
  double r = fma(-kd, l64hi, y);
  r = fma(-kd, l64lo, r);
  double pe = 1.0 / 720.0;
  pe = fma(pe, r, 1.0 / 120.0);
  pe = fma(pe, r, 1.0 / 24.0);
  pe = fma(pe, r, 1.0 / 6.0);
  pe = fma(pe, r, 0.5);
  pe = fma(pe * r, r, r);                      // exp(r) - 1
  const int k = (int)(kbits & 0xFFFFFFFFLL);
  const int jj = k & 63, kk = k >> 6;
  const double tj = __ldg(&tab->exp2j[jj]);
  const double res = fma(tj, pe, tj);
  // scale by 2^kk through the exponent field (result stays normal here)
  return __longlong_as_double(__double_as_longlong(res) + ((long long)kk << 52));
}

// ---------------------------------------------------------------------------
// Pointwise gas dynamics (FP64). Layouts follow the reference: metrics of
// direction i are m[nD*i + 0..nD-1]; stress tau[nD*c + d] = tau_{c,d}.
// ---------------------------------------------------------------------------

// Incoming Jacobian A+ of the inviscid flux along `metrics` for a state of
// conserved variables cv (computeIncomingJacobianOfInviscidFlux{2D,3D},
// src/CNSHelperImpl.f90:1669-2343). out(i,j) at out[i + nU*j].
// Forward-mode dual number with K directional derivatives. Evaluating the
// incoming Jacobian of a Roe-averaged state on duals seeded with the left
// state gives its exact variation with respect to that state, which the
// block-interface adjoint needs (src/CNSHelperImpl.f90:1669-2343 with
// deltaRoeAverage, src/BlockInterfacePatchImpl.f90:337-420).
template <int K>
struct DualN {
  double v;
  double d[K];
  __host__ __device__ DualN() : v(0.0) {
    for (int k = 0; k < K; ++k) d[k] = 0.0;
  }
  __host__ __device__ DualN(double x) : v(x) {
    for (int k = 0; k < K; ++k) d[k] = 0.0;
  }
};
__host__ __device__ inline double valueOf(double x) { return x; }

// a / b rounded to nearest from the rounded reciprocal of b: the product's
// residual is exact (P. Markstein, IBM J. Res. Dev. 34(1), 1990). Three
// operations where several quotients share a divisor, instead of ten.
__host__ __device__ inline double quotient(double a, double b, double inv) {
  const double r = a * inv;
  return fma(fma(-b, r, a), inv, r);
}
template <int K> __host__ __device__ inline double valueOf(const DualN<K>& x) { return x.v; }
template <int K> __host__ __device__ inline DualN<K> operator+(const DualN<K>& a, const DualN<K>& b) {
  DualN<K> r(a.v + b.v);
  for (int k = 0; k < K; ++k) r.d[k] = a.d[k] + b.d[k];
  return r;
}
template <int K> __host__ __device__ inline DualN<K> operator-(const DualN<K>& a, const DualN<K>& b) {
  DualN<K> r(a.v - b.v);
  for (int k = 0; k < K; ++k) r.d[k] = a.d[k] - b.d[k];
  return r;
}
template <int K> __host__ __device__ inline DualN<K> operator-(const DualN<K>& a) {
  DualN<K> r(-a.v);
  for (int k = 0; k < K; ++k) r.d[k] = -a.d[k];
  return r;
}
template <int K> __host__ __device__ inline DualN<K> operator*(const DualN<K>& a, const DualN<K>& b) {
  DualN<K> r(a.v * b.v);
  for (int k = 0; k < K; ++k) r.d[k] = a.d[k] * b.v + a.v * b.d[k];
  return r;
}
template <int K> __host__ __device__ inline DualN<K> operator/(const DualN<K>& a, const DualN<K>& b) {
  const double inv = 1.0 / b.v;  // about ten instructions
  DualN<K> r(quotient(a.v, b.v, inv));
  for (int k = 0; k < K; ++k) r.d[k] = (a.d[k] - r.v * b.d[k]) * inv;
  return r;
}
template <int K> __host__ __device__ inline DualN<K> operator+(const DualN<K>& a, double b) {
  DualN<K> r(a);
  r.v += b;
  return r;
}
template <int K> __host__ __device__ inline DualN<K> operator+(double a, const DualN<K>& b) { return b + a; }
template <int K> __host__ __device__ inline DualN<K> operator-(const DualN<K>& a, double b) { return a + (-b); }
template <int K> __host__ __device__ inline DualN<K> operator-(double a, const DualN<K>& b) { return (-b) + a; }
template <int K> __host__ __device__ inline DualN<K> operator*(const DualN<K>& a, double b) {
  DualN<K> r(a.v * b);
  for (int k = 0; k < K; ++k) r.d[k] = a.d[k] * b;
  return r;
}
template <int K> __host__ __device__ inline DualN<K> operator*(double a, const DualN<K>& b) { return b * a; }
template <int K> __host__ __device__ inline DualN<K> operator/(const DualN<K>& a, double b) {
  const double inv = 1.0 / b;
  DualN<K> r(quotient(a.v, b, inv));
  for (int k = 0; k < K; ++k) r.d[k] = a.d[k] * inv;
  return r;
}
template <int K> __host__ __device__ inline DualN<K> operator/(double a, const DualN<K>& b) {
  const double inv = 1.0 / b.v;
  DualN<K> r(quotient(a, b.v, inv));
  for (int k = 0; k < K; ++k) r.d[k] = -(r.v * b.d[k]) * inv;
  return r;
}
template <int K> __host__ __device__ inline DualN<K>& operator+=(DualN<K>& a, const DualN<K>& b) {
  a = a + b;
  return a;
}
__host__ __device__ inline double sqrtOf(double x) { return sqrt(x); }
template <int K> __host__ __device__ inline DualN<K> sqrtOf(const DualN<K>& a) {
  DualN<K> r(::sqrt(a.v));
  const double h = 0.5 / r.v;
  for (int k = 0; k < K; ++k) r.d[k] = a.d[k] * h;
  return r;
}

// Roe average of two conserved states (computeRoeAverage,
// src/CNSHelperImpl.f90:179-351, without the variations). Of dual numbers, the
// right state may be plain (not differentiated). Every quotient is rounded
// once: products with rounded reciprocals made the average's error 5 to 8%
// larger (random states, against 40 digits).
template <int ND, class S, class SR>
__host__ __device__ inline void roeAverage(const S* qL, const SR* qR, double g, S* roe) {
  const S sL = sqrtOf(qL[0]);
  const SR sR = sqrtOf(qR[0]);
  const S vL = 1.0 / qL[0], w = sL + sR;
  const SR vR = 1.0 / qR[0];
  S mL2 = qL[1] * qL[1];
  SR mR2 = qR[1] * qR[1];
  for (int d = 1; d < ND; ++d) {
    mL2 = mL2 + qL[1 + d] * qL[1 + d];
    mR2 = mR2 + qR[1 + d] * qR[1 + d];
  }
  const S hL = g * qL[ND + 1] - 0.5 * (g - 1.0) * vL * mL2;
  const SR hR = g * qR[ND + 1] - 0.5 * (g - 1.0) * vR * mR2;
  roe[0] = sL * sR;
  for (int d = 0; d < ND; ++d) roe[1 + d] = (sR * qL[1 + d] + sL * qR[1 + d]) / w;
  roe[ND + 1] = (sR * hL + sL * hR) / w;
  S m2 = roe[1] * roe[1];
  for (int d = 1; d < ND; ++d) m2 = m2 + roe[1 + d] * roe[1 + d];
  roe[ND + 1] = (roe[ND + 1] + 0.5 * (g - 1.0) / roe[0] * m2) / g;
}

// The incoming Jacobian A+ of incomingJacobian below without its matrix. With
// n the unit normal, k = |u|^2/2, eigenvalues a (entropy and shear) and b+, b-
// (acoustic; those of the other direction are zero), and for a vector x
//   y = x_m - u x_0,  X = (k x_0 - u . x_m + x_E) / T,  w+- = (X +- n.y / c) / 2,
// its eigenvector expansion sums to
//   A+ x = a (x_0 - X, u (x_0 - X) + y - n (n.y), k (x_0 - X) + u.y - U (n.y))
//          + sum+- b+- w+- (1, u +- n c, T + k +- c U).
template <int ND, class S>
struct Incoming {
  S u[ND], T, iT, k, U, c, ic, a, bp, bm;
  double n[ND];
};

template <int ND, class S>
__host__ __device__ inline Incoming<ND, S> incomingState(const S* cv, const double* metrics, double g, int direction) {
  Incoming<ND, S> I;
  double arc = 0.0;
  for (int d = 0; d < ND; ++d) arc += metrics[d] * metrics[d];
  arc = sqrt(arc);
  const double arcInv = 1.0 / arc;
  for (int d = 0; d < ND; ++d) I.n[d] = quotient(metrics[d], arc, arcInv);
  const S v = 1.0 / cv[0];
  for (int d = 0; d < ND; ++d) I.u[d] = v * cv[1 + d];
  S u2 = I.u[0] * I.u[0];
  I.U = I.n[0] * I.u[0];
  for (int d = 1; d < ND; ++d) {
    u2 = u2 + I.u[d] * I.u[d];
    I.U = I.U + I.n[d] * I.u[d];
  }
  I.k = 0.5 * u2;
  I.T = g * (v * cv[ND + 1] - I.k);
  I.c = sqrtOf((g - 1.0) * I.T);
  I.ic = 1.0 / I.c;
  I.iT = (g - 1.0) * I.ic * I.ic;
  I.a = arc * I.U;
  I.bp = arc * (I.U + I.c);
  I.bm = arc * (I.U - I.c);
  if (direction * valueOf(I.a) < 0.0) I.a = S(0.0);
  if (direction * valueOf(I.bp) < 0.0) I.bp = S(0.0);
  if (direction * valueOf(I.bm) < 0.0) I.bm = S(0.0);
  return I;
}

// out = A+ x.
template <int ND, class S>
__host__ __device__ inline void incomingProduct(const Incoming<ND, S>& I, const double* x, S* out) {
  constexpr int E = ND + 1;
  S um = I.u[0] * x[1];
  for (int d = 1; d < ND; ++d) um = um + I.u[d] * x[1 + d];
  const S X = I.iT * (I.k * x[0] - um + x[E]);
  S y[ND], ny = S(0.0), uy = S(0.0);
  for (int d = 0; d < ND; ++d) {
    y[d] = x[1 + d] - I.u[d] * x[0];
    ny = d ? ny + I.n[d] * y[d] : I.n[0] * y[0];
    uy = d ? uy + I.u[d] * y[d] : I.u[0] * y[0];
  }
  const S s = x[0] - X, wp = 0.5 * I.bp * (X + I.ic * ny), wm = 0.5 * I.bm * (X - I.ic * ny);
  const S sum = wp + wm, dif = I.c * (wp - wm), as = I.a * s;
  out[0] = as + sum;
  for (int d = 0; d < ND; ++d) out[1 + d] = I.u[d] * out[0] + I.a * (y[d] - I.n[d] * ny) + I.n[d] * dif;
  out[E] = I.k * out[0] + I.a * (uy - I.U * ny) + I.T * sum + I.U * dif;
}

// lam^T A+ x, and with grad != nullptr its gradient A+^T lam with respect to
// x (values only):
//   a [C (x_0 - X) + q.y - (n.q)(n.y)] + sum+- b+- (A +- c n.q) w+-,
//   q = lam_m + u lam_E, C = lam_0 + u . lam_m + k lam_E, A = C + T lam_E.
template <int ND, class S>
__host__ __device__ inline S incomingForm(const Incoming<ND, S>& I, const double* lam, const double* x, double* grad) {
  constexpr int E = ND + 1;
  S q[ND], y[ND], nq = S(0.0), ny = S(0.0), qy = S(0.0), um = S(0.0), C = I.k * lam[E] + lam[0];
  for (int d = 0; d < ND; ++d) {
    q[d] = I.u[d] * lam[E] + lam[1 + d];
    y[d] = x[1 + d] - I.u[d] * x[0];
    C = C + I.u[d] * lam[1 + d];
    um = d ? um + I.u[d] * x[1 + d] : I.u[0] * x[1];
    nq = d ? nq + I.n[d] * q[d] : I.n[0] * q[0];
    ny = d ? ny + I.n[d] * y[d] : I.n[0] * y[0];
    qy = d ? qy + q[d] * y[d] : q[0] * y[0];
  }
  const S X = I.iT * (I.k * x[0] - um + x[E]), A = C + I.T * lam[E], cq = I.c * nq, cy = I.ic * ny;
  const S hp = 0.5 * I.bp * (A + cq), hm = 0.5 * I.bm * (A - cq);
  if (grad) {
    const double gX = valueOf(hp) + valueOf(hm) - valueOf(I.a) * valueOf(C);
    const double gn = (valueOf(hp) - valueOf(hm)) * valueOf(I.ic) - valueOf(I.a) * valueOf(nq);
    const double gi = valueOf(I.iT) * gX;
    double ug = 0.0;
    for (int d = 0; d < ND; ++d) {
      const double gy = valueOf(I.a) * valueOf(q[d]) + I.n[d] * gn;
      grad[1 + d] = gy - gi * valueOf(I.u[d]);
      ug += valueOf(I.u[d]) * gy;
    }
    grad[0] = valueOf(I.a) * valueOf(C) + gi * valueOf(I.k) - ug;
    grad[E] = gi;
  }
  return I.a * (C * (x[0] - X) + qy - nq * ny) + hp * (X + cy) + hm * (X - cy);
}

template <int ND, class S = double>
__host__ __device__ inline void incomingJacobian(const S* cv, const double* metrics, double g,
                                                 int incomingDirection, S* out) {
  constexpr int nU = ND + 2;
  double arc = 0.0;
  for (int d = 0; d < ND; ++d) arc += metrics[d] * metrics[d];
  arc = sqrt(arc);
  double nm[3];
  for (int d = 0; d < ND; ++d) nm[d] = metrics[d] / arc;
  const S v = 1.0 / cv[0];
  S u[3], u2 = 0.0;
  for (int d = 0; d < ND; ++d) u[d] = v * cv[d + 1];
  for (int d = 0; d < ND; ++d) u2 += u[d] * u[d];
  const S T = g * (v * cv[ND + 1] - 0.5 * u2);
  S U = 0.0;
  for (int d = 0; d < ND; ++d) U += nm[d] * u[d];
  const S c = sqrtOf((g - 1.0) * T);
  const S phi2 = 0.5 * (g - 1.0) * u2;
  const S rho = cv[0];
  S R[nU][nU], L[nU][nU], lam[nU];
  if constexpr (ND == 2) {
    lam[0] = U; lam[1] = U; lam[2] = U + c; lam[3] = U - c;
    R[0][0] = 1.0; R[1][0] = u[0]; R[2][0] = u[1]; R[3][0] = phi2 / (g - 1.0);
    R[0][1] = 0.0; R[1][1] = nm[1] * rho; R[2][1] = -nm[0] * rho;
    R[3][1] = rho * (nm[1] * u[0] - nm[0] * u[1]);
    R[0][2] = 1.0; R[1][2] = u[0] + nm[0] * c; R[2][2] = u[1] + nm[1] * c;
    R[3][2] = T + phi2 / (g - 1.0) + c * U;
    R[0][3] = 1.0; R[1][3] = u[0] - nm[0] * c; R[2][3] = u[1] - nm[1] * c;
    R[3][3] = T + phi2 / (g - 1.0) - c * U;
    L[0][0] = 1.0 - phi2 / (c * c);
    L[1][0] = -v * (nm[1] * u[0] - nm[0] * u[1]);
    L[2][0] = 0.5 * (phi2 / (c * c) - U / c);
    L[3][0] = 0.5 * (phi2 / (c * c) + U / c);
    L[0][1] = u[0] / T; L[1][1] = v * nm[1];
    L[2][1] = -0.5 * (u[0] / T - nm[0] / c); L[3][1] = -0.5 * (u[0] / T + nm[0] / c);
    L[0][2] = u[1] / T; L[1][2] = -v * nm[0];
    L[2][2] = -0.5 * (u[1] / T - nm[1] / c); L[3][2] = -0.5 * (u[1] / T + nm[1] / c);
    L[0][3] = -1.0 / T; L[1][3] = 0.0; L[2][3] = 0.5 / T; L[3][3] = 0.5 / T;
  } else {
    lam[0] = U; lam[1] = U; lam[2] = U; lam[3] = U + c; lam[4] = U - c;
    const S h0 = phi2 / (g - 1.0);
    const S q = 1.0 - phi2 / (c * c);
    S (*r)[nU] = R;
    r[0][0] = nm[0]; r[1][0] = nm[0] * u[0]; r[2][0] = nm[0] * u[1] + rho * nm[2];
    r[3][0] = nm[0] * u[2] - rho * nm[1];
    r[4][0] = rho * (nm[2] * u[1] - nm[1] * u[2]) + h0 * nm[0];
    r[0][1] = nm[1]; r[1][1] = nm[1] * u[0] - rho * nm[2]; r[2][1] = nm[1] * u[1];
    r[3][1] = nm[1] * u[2] + rho * nm[0];
    r[4][1] = rho * (nm[0] * u[2] - nm[2] * u[0]) + h0 * nm[1];
    r[0][2] = nm[2]; r[1][2] = nm[2] * u[0] + rho * nm[1]; r[2][2] = nm[2] * u[1] - rho * nm[0];
    r[3][2] = nm[2] * u[2];
    r[4][2] = rho * (nm[1] * u[0] - nm[0] * u[1]) + h0 * nm[2];
    r[0][3] = 1.0; r[1][3] = u[0] + nm[0] * c; r[2][3] = u[1] + nm[1] * c;
    r[3][3] = u[2] + nm[2] * c; r[4][3] = T + h0 + c * U;
    r[0][4] = 1.0; r[1][4] = u[0] - nm[0] * c; r[2][4] = u[1] - nm[1] * c;
    r[3][4] = u[2] - nm[2] * c; r[4][4] = T + h0 - c * U;
    S (*l)[nU] = L;
    l[0][0] = nm[0] * q - v * (nm[2] * u[1] - nm[1] * u[2]);
    l[1][0] = nm[1] * q - v * (nm[0] * u[2] - nm[2] * u[0]);
    l[2][0] = nm[2] * q - v * (nm[1] * u[0] - nm[0] * u[1]);
    l[3][0] = 0.5 * (phi2 / (c * c) - U / c);
    l[4][0] = 0.5 * (phi2 / (c * c) + U / c);
    l[0][1] = nm[0] * u[0] / T; l[1][1] = nm[1] * u[0] / T - v * nm[2];
    l[2][1] = nm[2] * u[0] / T + v * nm[1];
    l[3][1] = -0.5 * (u[0] / T - nm[0] / c); l[4][1] = -0.5 * (u[0] / T + nm[0] / c);
    l[0][2] = nm[0] * u[1] / T + v * nm[2]; l[1][2] = nm[1] * u[1] / T;
    l[2][2] = nm[2] * u[1] / T - v * nm[0];
    l[3][2] = -0.5 * (u[1] / T - nm[1] / c); l[4][2] = -0.5 * (u[1] / T + nm[1] / c);
    l[0][3] = nm[0] * u[2] / T - v * nm[1]; l[1][3] = nm[1] * u[2] / T + v * nm[0];
    l[2][3] = nm[2] * u[2] / T;
    l[3][3] = -0.5 * (u[2] / T - nm[2] / c); l[4][3] = -0.5 * (u[2] / T + nm[2] / c);
    l[0][4] = -nm[0] / T; l[1][4] = -nm[1] / T; l[2][4] = -nm[2] / T;
    l[3][4] = 0.5 / T; l[4][4] = 0.5 / T;
  }
  for (int k = 0; k < nU; ++k) {
    lam[k] = arc * lam[k];
    if (incomingDirection * valueOf(lam[k]) < 0.0) lam[k] = 0.0;
  }
  for (int j = 0; j < nU; ++j)
    for (int i = 0; i < nU; ++i) {
      S s = R[i][0] * lam[0] * L[0][j];
      for (int k = 1; k < nU; ++k) s += R[i][k] * lam[k] * L[k][j];
      out[i + nU * j] = s;
    }
}

// y += A^T w for the inviscid flux Jacobian A along metric m
// (computeJacobianOfInviscidFlux{2D,3D}, src/CNSHelperImpl.f90:1098-1445),
// formed column by column and contracted immediately (wall SATs).
template <int ND, class Phys>
__device__ __forceinline__ void addFluxJacobianTransposeProduct(const double* m, const double* u, double T,
                                                                const Phys& P, const double* w, double* y) {
  const double g = P.g;
  constexpr int E = ND + 1;
  double U = m[0] * u[0];
  for (int d = 1; d < ND; ++d) U += m[d] * u[d];
  double u2 = u[0] * u[0];
  for (int d = 1; d < ND; ++d) u2 += u[d] * u[d];
  const double phi2 = 0.5 * (g - 1.0) * u2;
  {
    // column 0 of A: (0, phi2 m_d - U u_d, U((g-2)/(g-1) phi2 - T))
    double s = 0.0;
    for (int d = 0; d < ND; ++d) s += (phi2 * m[d] - U * u[d]) * w[1 + d];
    s += U * (P.gm2OverGm1 * phi2 - T) * w[E];
    y[0] += s;
  }
  for (int c = 0; c < ND; ++c) {
    double s = m[c] * w[0];
    for (int d = 0; d < ND; ++d) {
      const double a = d == c ? U - (g - 2.0) * u[c] * m[c] : u[d] * m[c] - (g - 1.0) * u[c] * m[d];
      s += a * w[1 + d];
    }
    s += ((T + phi2 * P.invGm1) * m[c] - (g - 1.0) * U * u[c]) * w[E];
    y[1 + c] += s;
  }
  {
    double s = 0.0;
    for (int d = 0; d < ND; ++d) s += (g - 1.0) * m[d] * w[1 + d];
    s += g * U * w[E];
    y[E] += s;
  }
}

// y += B1^T w alone (first partial viscous Jacobian transpose product), used
// by the far-field adjoint viscous penalty (src/FarFieldPatchImpl.f90:237-257).
template <int ND>
__device__ __forceinline__ void firstPartialViscousTransposeProduct(
    const double* m, const double* u, double T, double v, double g, double n,
    const double* tau, const double* hf, const double* w, double* y) {
  constexpr int E = ND + 1;
  double u2 = u[0] * u[0];
  for (int d = 1; d < ND; ++d) u2 += u[d] * u[d];
  const double phi2 = 0.5 * (g - 1.0) * u2;
  double ct[3];
  for (int a = 0; a < ND; ++a) {
    double s = m[0] * tau[ND * a];
    for (int d = 1; d < ND; ++d) s += m[d] * tau[ND * a + d];
    ct[a] = s;
  }
  double cq = m[0] * hf[0];
  for (int d = 1; d < ND; ++d) cq += m[d] * hf[d];
  double uct = u[0] * ct[0];
  for (int d = 1; d < ND; ++d) uct += u[d] * ct[d];
  const double t1 = uct - cq, nTv = n * g * v / T;
  {
    const double t2 = nTv * (phi2 / (g - 1.0) - T / g);
    double s = 0.0;
    for (int d = 0; d < ND; ++d) s += t2 * ct[d] * w[1 + d];
    y[0] += s + (t2 * t1 - v * uct) * w[E];
  }
  for (int c = 0; c < ND; ++c) {
    const double t2 = -nTv * u[c];
    double s = 0.0;
    for (int d = 0; d < ND; ++d) s += t2 * ct[d] * w[1 + d];
    y[1 + c] += s + (t2 * t1 + v * ct[c]) * w[E];
  }
  {
    double s = 0.0;
    for (int d = 0; d < ND; ++d) s += nTv * ct[d] * w[1 + d];
    y[E] += s + nTv * t1 * w[E];
  }
}

// y += B2(m1, m2)^T w for the second partial viscous Jacobian
// (computeSecondPartialViscousJacobian{2D,3D}, src/CNSHelperImpl.f90:2636-2757);
// w and y have nD+1 entries (momentum, energy).
template <int ND>
__device__ __forceinline__ void secondPartialViscousTransposeProduct(
    const double* u, double mu, double la, double k, double jac, const double* m1,
    const double* m2, const double* w, double* y) {
  double t1 = m1[0] * m2[0], t2 = m2[0] * u[0], t3 = m1[0] * u[0];
  for (int d = 1; d < ND; ++d) {
    t1 += m1[d] * m2[d];
    t2 += m2[d] * u[d];
    t3 += m1[d] * u[d];
  }
  t2 = mu * t2;
  t3 = la * t3;
  // column c of B2 (c < ND): rows r < ND and energy row ND
  for (int c = 0; c < ND; ++c) {
    double s = 0.0;
    for (int r = 0; r < ND; ++r) {
      const double b = r == c ? mu * t1 + (mu + la) * m1[c] * m2[c]
                              : mu * m1[c] * m2[r] + la * m1[r] * m2[c];
      s += b * w[r];
    }
    s += (mu * t1 * u[c] + m1[c] * t2 + m2[c] * t3) * w[ND];
    y[c] += jac * s;
  }
  y[ND] += jac * (k * t1) * w[ND];
}

// The inviscid linearized flux A(m) x along a metric row (rows of
// computeJacobianOfInviscidFlux{2D,3D}, src/CNSHelperImpl.f90:1098-1445,
// contracted with x).
template <int ND>
__device__ __forceinline__ void fluxJacobianProduct(const double* m, const double* u, double T, double g,
                                                    const double* x, double* Ax) {
  constexpr int E = ND + 1;
  double U = m[0] * u[0], u2 = u[0] * u[0], mx = m[0] * x[1], ux = u[0] * x[1];
  for (int d = 1; d < ND; ++d) {
    U += m[d] * u[d];
    u2 += u[d] * u[d];
    mx += m[d] * x[1 + d];
    ux += u[d] * x[1 + d];
  }
  const double phi2 = 0.5 * (g - 1.0) * u2;
  Ax[0] = mx;
  for (int d = 0; d < ND; ++d)
    Ax[1 + d] = (phi2 * m[d] - U * u[d]) * x[0] + U * x[1 + d] + u[d] * mx - (g - 1.0) * m[d] * ux +
                (g - 1.0) * m[d] * x[E];
  Ax[E] = U * ((g - 2.0) / (g - 1.0) * phi2 - T) * x[0] + (T + phi2 / (g - 1.0)) * mx - (g - 1.0) * U * ux +
          g * U * x[E];
}

// The linearized fluxes of every axis at a point (computeRhsLinearized,
// src/RhsHelperImpl.f90:655-775): F[i] = A_i x - V[i] and the viscous part
// V[i] = B1_i x + (0, sum_j B2(m_i, m_j) dt_j), dt[j] the derivative along axis
// j of (delta u, the temperature perturbation). All are linear in the metric
// rows, so the Cartesian directions' fluxes are written out first, with
// D_y = sum_j m_{j,y} dt_j, y_c = x_1+c - u_c x_0, dp the pressure perturbation
// and H = T + |u|^2/2:
//   A_x x = (w, u_c w + u_x y_c + [c = x] dp, u_x (dp + x_E - H x_0) + H w), w = x_1+x,
//   V_x   = (0, t_c = tau_cx sg + J (mu (D_x[c] + D_c[x]) + [c = x] lambda tr D),
//            (u . tau_x - q_x) sg + v tau_x . y + J (u . S_x + k D_x[E])),
//   sg = n gamma v / T ((|u|^2/2 - T/gamma) x_0 - u . x_m + x_E),
// S_x the second half of t. The axes then combine them with their rows.
template <int ND, bool CURV, bool VISC, class Phys>
__device__ __forceinline__ void linearizedPointwise(const double* m, const double* u, double T, double v,
                                                    const Phys& P, const double* tau, const double* hf, double mu,
                                                    double la, double kd, double jac, const double* x,
                                                    const double (*dt)[ND + 1], double (*F)[ND + 2],
                                                    double (*V)[ND + 2]) {
  constexpr int nU = ND + 2, E = ND + 1;
  double k = u[0] * u[0], um = u[0] * x[1];
#pragma unroll
  for (int d = 1; d < ND; ++d) {
    k += u[d] * u[d];
    um += u[d] * x[1 + d];
  }
  k *= 0.5;
  const double H = T + k, b = k * x[0] - um + x[E];  // dp / (gamma - 1)
  const double dp = P.gm1 * b, he = dp + x[E] - H * x[0];
  double y[ND], cF[ND][nU], cV[ND][nU];
#pragma unroll
  for (int c = 0; c < ND; ++c) y[c] = x[1 + c] - u[c] * x[0];
#pragma unroll
  for (int d = 0; d < ND; ++d) {
    const double w = x[1 + d];
    cF[d][0] = w;
#pragma unroll
    for (int c = 0; c < ND; ++c) cF[d][1 + c] = u[c] * w + u[d] * y[c];
    cF[d][1 + d] += dp;
    cF[d][E] = u[d] * he + H * w;
    cV[d][0] = 0.0;
  }
  if (VISC) {
    const double sg = P.powerLawExponent * P.g * v * fixedReciprocal(T) * (b - T * P.invG * x[0]);
    double D[ND][ND + 1], tr = 0.0;
#pragma unroll
    for (int d = 0; d < ND; ++d) {
#pragma unroll
      for (int c = 0; c <= ND; ++c) {
        if (CURV) {
          double s = m[d] * dt[0][c];
#pragma unroll
          for (int j = 1; j < ND; ++j) s += m[ND * j + d] * dt[j][c];
          D[d][c] = s;
        } else {
          D[d][c] = m[ND * d + d] * dt[d][c];
        }
      }
      tr = d ? tr + D[d][d] : D[0][0];
    }
    const double jm = jac * mu, jl = jac * la * tr, jk = jac * kd;
    double S[ND][ND];
#pragma unroll
    for (int d = 0; d < ND; ++d) {
      S[d][d] = 2.0 * jm * D[d][d] + jl;
#pragma unroll
      for (int c = d + 1; c < ND; ++c) S[d][c] = S[c][d] = jm * (D[d][c] + D[c][d]);
    }
#pragma unroll
    for (int d = 0; d < ND; ++d) {
      double e = jk * D[d][ND], t1 = -hf[d], ty = 0.0;
#pragma unroll
      for (int c = 0; c < ND; ++c) {
        const double t = tau[ND * c + d];
        cV[d][1 + c] = t * sg + S[d][c];
        t1 += u[c] * t;
        ty = c ? ty + t * y[c] : t * y[0];
        e += u[c] * S[d][c];
      }
      cV[d][E] = t1 * sg + v * ty + e;
    }
  }
#pragma unroll
  for (int i = 0; i < ND; ++i)
#pragma unroll
    for (int c = 0; c < nU; ++c) {
      double f, g = 0.0;
      if (CURV) {
        f = m[ND * i] * cF[0][c];
        if (VISC) g = m[ND * i] * cV[0][c];
#pragma unroll
        for (int d = 1; d < ND; ++d) {
          f += m[ND * i + d] * cF[d][c];
          if (VISC) g += m[ND * i + d] * cV[d][c];
        }
      } else {
        f = m[ND * i + i] * cF[i][c];
        if (VISC) g = m[ND * i + i] * cV[i][c];
      }
      F[i][c] = VISC ? f - g : f;
      V[i][c] = g;
    }
}

// The pointwise part of the adjoint core over all directions at once:
//   y     = sum_i (A_i - B1_i)^T w_i,
//   ad[j] = sum_i B2(m_i, m_j)^T w_i,
// with w[i] the adjoint derivative of lambda along axis i. A_i, B1_i and B2
// are linear in the metric rows, so the axes' w are first combined into
// Cartesian directions, W_x = sum_i m_{i,x} w_i (a scaling on Cartesian
// grids), and the unit-direction products are written out and summed before
// the factors they share are applied. With e_x = W_x,E,
//   P_xc = W_x,1+c + u_c e_x,   Z = sum_x P_xx,   r_x = sum_d u_d W_x,1+d + (T + |u|^2/2) e_x,
//   A_x^T W_x : (gamma-1)(|u|^2/2) P_xx - u_x r_x  (density)
//               u_x W_x,1+c - (gamma-1) u_c P_xx + [c = x] (W_x,0 + r_x)  (momentum c)
//               (gamma-1) P_xx + u_x e_x  (energy)
//   B1: X = sum_xc tau_xc P_xc - sum_x q_x e_x and g_c = sum_x tau_cx e_x enter as
//       N X (|u|^2/2 - T/gamma) - v u.g, -N X u_c + v g_c, N X with N = n gamma v / T,
//   B2: AD_yc = J mu (P_yc + P_cy) (c != y), J (2 mu P_yy + lambda Z) (c = y), J k e_y
//       (energy), and ad[j] = sum_y m_{j,y} AD_y.
// boundary(W) adds the far-field viscous penalties' share to W's momentum and
// energy entries, for ad only, and says whether the point has any.
// The core is bound by the FP64 pipe (88% busy at 128^3 with each direction's
// products formed separately: about 440 FP64 instructions a warp, 1735 us);
// this form takes about 130 (772 us; 543 with MinBlocks' registers and
// derivatives()' single copy of the stencil code: FP64 pipe 70% busy before
// the latter); 201^2 39.6 -> 28.7 us, 20.6 with the latter two.
template <int ND, bool CURV, bool VISC, class Phys, class Boundary>
__device__ __forceinline__ void adjointPointwise(const double (*w)[ND + 2], const double* m, const double* u,
                                                 double T, double v, const Phys& P, const double* tau,
                                                 const double* hf, double mu, double la, double kd, double jac,
                                                 Boundary boundary, double* y, double (*ad)[ND + 1]) {
  constexpr int nU = ND + 2, E = ND + 1;
  double W[ND][nU];
#pragma unroll
  for (int x = 0; x < ND; ++x)
#pragma unroll
    for (int c = 0; c < nU; ++c) {
      if (CURV) {
        double s = m[x] * w[0][c];
#pragma unroll
        for (int i = 1; i < ND; ++i) s += m[ND * i + x] * w[i][c];
        W[x][c] = s;
      } else {
        W[x][c] = m[ND * x + x] * w[x][c];
      }
    }
  double k = u[0] * u[0];
#pragma unroll
  for (int d = 1; d < ND; ++d) k += u[d] * u[d];
  k *= 0.5;
  const double H = T + k;
  double Pm[ND][ND], Z = 0.0, ur = 0.0, ue = 0.0, r[ND];
#pragma unroll
  for (int x = 0; x < ND; ++x) {
    double s = u[0] * W[x][1];
#pragma unroll
    for (int c = 0; c < ND; ++c) {
      Pm[x][c] = W[x][1 + c] + u[c] * W[x][E];
      if (c) s += u[c] * W[x][1 + c];
    }
    Z = x ? Z + Pm[x][x] : Pm[x][x];
    r[x] = s + H * W[x][E];
    ur = x ? ur + u[x] * r[x] : u[x] * r[x];
    ue = x ? ue + u[x] * W[x][E] : u[x] * W[x][E];
  }
#pragma unroll
  for (int c = 0; c < ND; ++c) {
    double s = W[c][0] + r[c];
#pragma unroll
    for (int x = 0; x < ND; ++x) s += u[x] * W[x][1 + c];
    y[1 + c] = s;
  }
  double S1 = -P.gm1 * Z;
  y[0] = -ur;
  y[E] = ue;
  if (VISC) {
    double X = 0.0, ug = 0.0;
#pragma unroll
    for (int c = 0; c < ND; ++c) {
      // tau is symmetric: its upper triangle is read
      double g = tau[c] * W[0][E];
#pragma unroll
      for (int x = 1; x < ND; ++x) g += tau[x < c ? ND * x + c : ND * c + x] * W[x][E];
      ug = c ? ug + u[c] * g : u[c] * g;
      y[1 + c] -= v * g;
      X = c ? X + tau[ND * c + c] * Pm[c][c] : tau[0] * Pm[0][0];
      X -= hf[c] * W[c][E];
    }
    double S[ND][ND];
#pragma unroll
    for (int x = 0; x < ND; ++x)
#pragma unroll
      for (int c = x + 1; c < ND; ++c) {
        S[x][c] = Pm[x][c] + Pm[c][x];
        X += tau[ND * x + c] * S[x][c];
      }
    const double NX = P.powerLawExponent * P.g * v * fixedReciprocal(T) * X;
    S1 += NX;
    y[0] += T * P.invG * NX + v * ug;
    if (boundary(W)) {
      Z = 0.0;
#pragma unroll
      for (int x = 0; x < ND; ++x) {
#pragma unroll
        for (int c = 0; c < ND; ++c) Pm[x][c] = W[x][1 + c] + u[c] * W[x][E];
        Z += Pm[x][x];
      }
#pragma unroll
      for (int x = 0; x < ND; ++x)
#pragma unroll
        for (int c = x + 1; c < ND; ++c) S[x][c] = Pm[x][c] + Pm[c][x];
    }
    const double jm = jac * mu, lz = jac * la * Z, jk = jac * kd;
#pragma unroll
    for (int x = 0; x < ND; ++x) {
      ad[x][ND] = jk * W[x][E];
      ad[x][x] = 2.0 * jm * Pm[x][x] + lz;
#pragma unroll
      for (int c = x + 1; c < ND; ++c) ad[x][c] = ad[c][x] = jm * S[x][c];
    }
    // Cartesian directions to the axes
    if (CURV) {
#pragma unroll
      for (int c = 0; c <= ND; ++c) {
        double t[ND];
#pragma unroll
        for (int j = 0; j < ND; ++j) {
          t[j] = m[ND * j] * ad[0][c];
#pragma unroll
          for (int x = 1; x < ND; ++x) t[j] += m[ND * j + x] * ad[x][c];
        }
#pragma unroll
        for (int j = 0; j < ND; ++j) ad[j][c] = t[j];
      }
    } else {
#pragma unroll
      for (int j = 0; j < ND; ++j)
#pragma unroll
        for (int c = 0; c <= ND; ++c) ad[j][c] *= m[ND * j + j];
    }
  }
  y[0] -= k * S1;
#pragma unroll
  for (int c = 0; c < ND; ++c) y[1 + c] += u[c] * S1;
  y[E] -= S1;
}

}  // namespace mgd
