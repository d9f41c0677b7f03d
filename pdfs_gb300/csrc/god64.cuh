// god64.cuh -- the FP64 local solvers with few FP64-pipe operations.
//
// GB300 runs an FP64 instruction of a warp in 64 cycles of its scheduler's
// pipe (76 with all four schedulers at it; measured), while 64 integer or FP32
// instructions issue beside it.  The solvers of godunov.cuh take about 104
// (god_ref64) and 67 (god_fast64) of them an update, compares, minima, square
// roots (10 each) and divisions (9 each) included.  Here the compares and minima
// are integer compares of the bit patterns, everything that depends on the
// spacings alone comes from a table by the sorted order of the axes, a division
// by such a constant is its correctly rounded reciprocal and one correction
// (P. W. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", IBM J. Res. Dev. 34, 1990: with y = RN(1/b), q within
// an ulp of a/b and r = a - b q exact, RN(q + r y) = RN(a/b)), and a square root
// starts from an FP32 reciprocal root refined to 45 bits in FP32 (the series of
// (1 - e)^(-1/2) to second order, e the exact residual): 61 and 29 FP64 operations an
// update.  A node with three terms is mostly known to have them without its two-term
// solution: 44 and 18.  Rounding by rounding, god64_ref is god_ref64 and god64_fast is
// god_fast64: bricks give the bits of columns, pencils and batches.
// A 384^3 sweep, 8 x 8 x 16 bricks: 8.9 ms reference and 4.4 fast, on pencils with the
// plain solvers 18.7 and 10.4; with the two-term solution always first 10.1
// (reference).  The fast one takes 4.5 with three_terms as its test too; 4.0 with roots
// to within an ulp and products with reciprocals instead of divisions, but then its
// bits are not the other tiles'.  64^3: 0.54 and 0.34 (pencils 1.35 and 0.82).
//
// They take finite or +inf non-negative values; anything else (negative
// values, NaN) goes to the plain solvers.
#pragma once
#include "godunov.cuh"

namespace pdfs {

__device__ __forceinline__ unsigned d_hi(double v) { return (unsigned)__double2hiint(v); }
__device__ __forceinline__ unsigned d_lo(double v) { return (unsigned)__double2loint(v); }
// a < b for values >= 0 (or NaN above both)
__device__ __forceinline__ bool d_less(double a, double b) { return __double_as_longlong(a) < __double_as_longlong(b); }

// a < b ? a : b, a != b, a < b (b a cap bound) and the running max of changes
// (NaN left out, as fmax does), off the FP64 pipe where the values are plain.
__device__ __forceinline__ bool d_plain(double a, double b) { return max(d_hi(a), d_hi(b)) <= 0x7ff00000u; }
__device__ __forceinline__ double d_min(double a, double b) {
  return (d_plain(a, b) ? d_less(a, b) : a < b) ? a : b;
}
__device__ __forceinline__ bool d_differ(double a, double b) {
  return d_plain(a, b) ? __double_as_longlong(a) != __double_as_longlong(b) : a != b;
}
__device__ __forceinline__ bool d_below(double a, double b) { return d_plain(a, b) ? d_less(a, b) : a < b; }
__device__ __forceinline__ double d_max(double a, double d) {  // a, d >= 0, d may be NaN
  return d_hi(d) <= 0x7ff00000u && d_less(a, d) ? d : a;
}
__device__ __forceinline__ float d_min(float a, float) { return a; }  // (never called: the FP32 kernels' types)
__device__ __forceinline__ bool d_differ(float, float) { return false; }
__device__ __forceinline__ float d_max(float a, float) { return a; }

// sqrt(m) for m in [1, 4): FP32 reciprocal root r0, one step in FP32 on the
// exact residual 1 - m r0^2 (c, so that r0 + c is good to 45 bits), the root
// from it, and one correction in FP64: within 2^-66 of the root before its
// last rounding.
__device__ __forceinline__ double sqrt_core(double m) {
  const unsigned hi = d_hi(m), lo = d_lo(m);
  // m = mh + ml, the leading 24 bits and the rest
  const float mh = __uint_as_float(((hi - 0x38000000u) << 3) | (lo >> 29));
  const float ml = __fmul_rn(__uint2float_rn(lo & 0x1fffffffu), hi >= 0x40000000u ? 0x1p-51f : 0x1p-52f);
  float r0;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r0) : "f"(mh));
  const float th = __fmul_rn(r0, r0), tl = __fmaf_rn(r0, r0, -th);
  float e = __fmaf_rn(-mh, th, 1.0f);
  e = __fmaf_rn(-mh, tl, e);
  e = __fmaf_rn(-ml, th, e);
  const float c = __fmul_rn(__fmul_rn(r0, e), __fmaf_rn(0.375f, e, 0.5f));
  // r0 in [1/2, 1] and c (below 2^-21, 0 included) as doubles, by their bits
  const unsigned rb = __float_as_uint(r0), cb = __float_as_uint(c);
  const double r0d = __hiloint2double((int)((rb >> 3) + 0x38000000u), (int)(rb << 29));
  const unsigned cm = cb & 0x7fffffffu;
  const double cd = cm < 0x00800000u
                        ? 0.0
                        : __hiloint2double((int)((cb & 0x80000000u) | ((cm >> 3) + 0x38000000u)), (int)(cm << 29));
  const double hr = __hiloint2double((int)(d_hi(r0d) - 0x00100000u), (int)d_lo(r0d));  // r0 / 2
  const double s = __fma_rn(m, cd, __dmul_rn(m, r0d));
  return __fma_rn(__fma_rn(-s, s, m), hr, s);
}

// The square root of a positive normal number (anything else: ok false), correctly
// rounded, and the rounding is checked -- s is RN(sqrt(m)) if |m - s^2| < s ulp(s);
// m - s^2 is a multiple of ulp(s)^2 below 2^54 of them, so the multiply-add gives it
// exactly -- with ok false for the rare root too close to a midpoint.
__device__ __forceinline__ double sqrt64(double x, bool &ok) {
  const unsigned hi = d_hi(x);
  ok = ok && hi - 0x00100000u < 0x7fe00000u;
  // x = m 4^k, m in [1, 4)
  const unsigned odd = (hi >> 20) & 1u;  // biased exponent: odd, m in [1, 2); even, m in [2, 4)
  const double m = __hiloint2double((int)((hi & 0x000fffffu) | (odd ? 0x3ff00000u : 0x40000000u)), (int)d_lo(x));
  const int k = ((int)(hi >> 20) - (odd ? 1023 : 1024)) >> 1;
  const double s = sqrt_core(m);
  const double r = __fma_rn(-s, s, m);
  // s in [1, 2]: s ulp(s) = s 2^-52 (2^-51 for s = 2, which only makes the test stricter)
  const double t = __hiloint2double((int)(d_hi(s) - (52u << 20)), (int)d_lo(s));
  ok = ok && d_less(__hiloint2double((int)(d_hi(r) & 0x7fffffffu), (int)d_lo(r)), t);
  return __hiloint2double((int)d_hi(s) + (k << 20), (int)d_lo(s));
}

// a / b, correctly rounded, for a constant b with ib = RN(1/b); a away from the
// ends of the exponent range (else ok false).
__device__ __forceinline__ double div64(double a, double b, double ib, bool &ok) {
  ok = ok && (d_hi(a) & 0x7fffffffu) - 0x10000000u < 0x60000000u;
  const double q = __dmul_rn(a, ib);
  return __fma_rn(__fma_rn(-q, b, a), ib, q);
}

// Minima sorted ascending, ties in axis order (the strict compare-exchanges
// of god_ref64); the order's index in GodConst64::p.
__device__ __forceinline__ int sort64(double &m0, double &m1, double &m2) {
  int a0 = 0, a1 = 1, a2 = 2;
  if (d_less(m1, m0)) { cswap(m0, m1); cswap(a0, a1); }
  if (d_less(m2, m1)) { cswap(m1, m2); cswap(a1, a2); }
  if (d_less(m1, m0)) { cswap(m0, m1); cswap(a0, a1); }
  return 2 * a0 + (a1 > a2 ? 1 : 0);  // a0, then whether the other two are swapped
}

// v >= 0 as a float, cut off (0 below the normal floats, +inf above)
__device__ __forceinline__ float d_float(double v) {
  const unsigned h = d_hi(v);
  const float f = __uint_as_float(((h - 0x38000000u) << 3) | (d_lo(v) >> 29));
  return h < 0x38100000u ? 0.0f : h >= 0x47f00000u ? INFINITY : f;
}

// Does the two-term solution of god_ref64 surely exceed m2, whatever its rounding?
// It does in exact arithmetic where T = w0 (m2 - m0)^2 + w1 (m2 - m1)^2 < 1, and by
// at least (1 - T) / (2 sqrt(w0 + w1)).  With M = m1 + d0 + d1, dm = min(d0, d1) and
// R = M / dm, its rounding error is below 16 u M^2 / dm, u = 2^-53 (the
// discriminant's terms are products of the minima, 8 u M^2 in all, and its root is
// at least d1), so 1 - T > 1e-14 R^2 is enough; T itself, from the minima cut to
// floats, is good to 4 times 2^-22 R and some 2^-20.  1e-5 + 2e-6 R covers both (it
// is below 1, so that anything is sure at all, only for R < 5e5).  True spares the
// two-term solution: 17 FP64 operations of 61.
__device__ __forceinline__ bool three_terms(double m0, double m1, double m2, const GodPerm64 &k) {
  const float f0 = d_float(m0), f1 = d_float(m1), f2 = d_float(m2);
  const float b = __fmul_rn(__fsub_rn(f2, f0), k.r0), c = __fmul_rn(__fsub_rn(f2, f1), k.r1);
  const float T = __fmaf_rn(b, b, __fmul_rn(c, c));
  return T < 1.0f - __fmaf_rn(__fmaf_rn(f1, k.rm, k.rd), 2e-6f, 1e-5f);  // (false for infinities and NaN)
}

// god_ref64 on sorted minima: the same roundings.  A doubled product is a
// multiply-add with 2 (exact), -x - x is -2 x.
__device__ __forceinline__ double god64_ref(double m0, double m1, double m2, const GodPerm64 &k, bool &ok) {
  double u = __dadd_rn(m0, k.d0);
  if (d_less(m1, u)) {
    const double m00 = __dmul_rn(m0, m0), m11 = __dmul_rn(m1, m1), p01 = __dmul_rn(m0, m1);
    const double m1q0 = __dmul_rn(m1, k.q0), m0q1 = __dmul_rn(m0, k.q1);
    const unsigned lanes = __activemask();
    bool three = d_less(m2, u) && three_terms(m0, m1, m2, k);
    if (!three) {
      double t = __fma_rn(2.0, p01, -m00);
      t = __dadd_rn(__dadd_rn(__dsub_rn(t, m11), k.q0), k.q1);
      u = div64(__dadd_rn(__dadd_rn(m1q0, m0q1), __dmul_rn(k.d01, sqrt64(t, ok))), k.s, k.is, ok);
      three = d_less(m2, u);
    }
    __syncwarp(lanes);  // one pass over the third term for all (see god64_node)
    if (three) {
      const double m22 = __dmul_rn(m2, m2), p02 = __dmul_rn(m0, m2), p12 = __dmul_rn(m1, m2);
      double r = __dsub_rn(__dmul_rn(-m00, k.q1), __dmul_rn(m00, k.q2));
      r = __fma_rn(2.0, __dmul_rn(p01, k.q2), r);
      r = __dsub_rn(r, __dmul_rn(m11, k.q0));
      r = __dsub_rn(r, __dmul_rn(m11, k.q2));
      r = __fma_rn(2.0, __dmul_rn(p02, k.q1), r);
      r = __dsub_rn(r, __dmul_rn(m22, k.q0));
      r = __dsub_rn(r, __dmul_rn(m22, k.q1));
      r = __fma_rn(2.0, __dmul_rn(p12, k.q0), r);
      r = __dadd_rn(__dadd_rn(__dadd_rn(r, k.q01), k.q02), k.q12);
      double n = __dadd_rn(__dmul_rn(__dmul_rn(m2, k.q0), k.q1), __dmul_rn(m1q0, k.q2));
      n = __dadd_rn(n, __dmul_rn(m0q1, k.q2));
      n = __dadd_rn(n, __dmul_rn(k.d012, sqrt64(r, ok)));
      u = div64(n, k.den, k.iden, ok);
    }
  }
  return u;
}

// god_fast64 on sorted minima: the same roundings (its sum and product of the
// two-term numerator and of the three-term result round once, as its expressions
// contract), but with the three-term solution v first.  Where v exceeds m2 by more
// than k.sure units of the last place, the two-term one does too, whatever its
// rounding, and is spared: in exact arithmetic it is the larger of the two, and with
// r = the largest spacing over the smallest and u = 2^-53 the error of v is below
// (63 r^3 + 93 r^2 + 50) u v and that of the two-term solution below 20 r u v (the
// discriminants are at least the square of the inverse of the largest spacing where v
// is a solution at all, and where it is not, r <= 1000 keeps v below m2).
__device__ __forceinline__ double god64_fast(double m0, double m1, double m2, const GodPerm64 &k, bool &ok) {
  double u = __dadd_rn(m0, k.d0);
  if (d_less(m1, u)) {
    const double a = __dsub_rn(m1, m0), aa = __dmul_rn(a, a);
    const unsigned lanes = __activemask();
    bool three = false, solved = d_less(m2, u);
    double v = 0.0;
    if (solved) {
      const double b = __dsub_rn(m2, m0);
      const double B = __fma_rn(a, k.w1, __dmul_rn(b, k.w2));
      const double C = __fma_rn(aa, k.w1, __fma_rn(__dmul_rn(b, b), k.w2, -1.0));
      bool real = true;
      v = __fma_rn(__dadd_rn(B, sqrt64(__fma_rn(B, B, __dmul_rn(-k.wsum, C)), real)), k.iwsum, m0);
      three = real && __double_as_longlong(v) - __double_as_longlong(m2) > k.sure;
      solved = real;
      if (three) u = v;
    }
    __syncwarp(lanes);  // one pass over the two-term solution for all (see god64_node)
    if (!three) {
      u = __dadd_rn(m0, div64(__fma_rn(a, k.w1, sqrt64(__fma_rn(-aa, k.w01, k.ws), ok)), k.ws, k.iws, ok));
      if (d_less(m2, u)) {
        ok = ok && solved;
        u = v;
      }
    }
  }
  return u;
}

// Everything else: negative values, NaN, roots of negative, subnormal or
// infinite discriminants, roots next to a rounding midpoint.  One copy, out of
// the hot code.
template <int ARITH>
__device__ __noinline__ double god64_plain(double x0, double x1, double y0, double y1, double z0, double z1,
                                           const GodConst64 &k) {
  const double m0 = x0 < x1 ? x0 : x1, m1 = y0 < y1 ? y0 : y1, m2 = z0 < z1 ? z0 : z1;
  return ARITH == 0 ? god_ref64(m0, m1, m2, k) : god_fast64(m0, m1, m2, k);
}

// The update of a node from its six neighbours, in grid orientation.
template <int ARITH>
__device__ __forceinline__ double god64_node(double x0, double x1, double y0, double y1, double z0, double z1,
                                             const GodConst64 &k, const GodPerm64 *perm) {
  // the largest high word: below +inf's, every value is finite and >= 0
  const unsigned hx = max(d_hi(x0), d_hi(x1)), hy = max(d_hi(y0), d_hi(y1)), hz = max(d_hi(z0), d_hi(z1));
  const unsigned h = max(max(hx, hy), hz);
  bool ok = perm && h <= 0x7ff00000u;
  if (h == 0x7ff00000u) {  // +inf among them (the halo's), or a NaN with a low word only
    auto odd = [](double v) { return d_hi(v) == 0x7ff00000u && d_lo(v) != 0u; };
    ok = ok && !(odd(x0) || odd(x1) || odd(y0) || odd(y1) || odd(z0) || odd(z1));
  }
  const unsigned lanes = __activemask();
  double u = 0.0;
  if (ok) {
    double m0 = d_less(x0, x1) ? x0 : x1, m1 = d_less(y0, y1) ? y0 : y1, m2 = d_less(z0, z1) ? z0 : z1;
    const GodPerm64 &kp = perm[sort64(m0, m1, m2)];
    u = ARITH == 0 ? god64_ref(m0, m1, m2, kp, ok) : god64_fast(m0, m1, m2, kp, ok);
  }
  // Lanes with one, two and three terms meet again here: with a branch on ok as
  // the next thing the compiler carries them apart to the end of the update, and
  // whatever FP64 operations follow run once for each (a 64^3 sweep: 930 -> 541 us
  // reference, 464 -> 292 us fast).
  __syncwarp(lanes);
  if (!ok) u = god64_plain<ARITH>(x0, x1, y0, y1, z0, z1, k);
  return u;
}

}  // namespace pdfs
