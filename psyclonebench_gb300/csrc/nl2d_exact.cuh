// Exact FP64 building blocks for the fused NEMOLite2D step.
//
// On GB300 the FP64 pipe issues 2 thread-operations per clock per SM, ~60x
// fewer than the integer and FP32 pipes, and an IEEE FP64 divide costs ~15
// FP64 instructions.  Each helper below returns the SAME bits as the plain
// IEEE expression it replaces, for every input, but spends fewer FP64
// instructions:
//
//  * div_rn(x, d, r): x / d rounded to nearest for a divisor d > 0 whose
//    reciprocal r = RN(1/d) was computed beforehand.  q0 = RN(x * r) is
//    within 1.5 ulp of x / d; the exact remainder q0 * d - x, formed from
//    the significands in 64-bit integers and compared with half an ulp of q0
//    times d, picks the correctly rounded quotient among q0 and its two
//    neighbours.  1 DMUL and about 20 integer instructions (the remainder by
//    FMA cost one DFMA more, 64 issue slots of a scheduler against ~10).
//    When q0 is a power of two (the spacing changes below it) the quotient
//    takes Markstein's two refinements instead (Markstein, "Computation of
//    elementary functions on the IBM RISC System/6000 processor", IBM J.
//    Res. Dev. 34(1), 1990; Muller et al., Handbook of Floating-Point
//    Arithmetic, 2nd ed., Sec. 4.7), 1 DMUL + 4 DFMA.
//    x = +-0 returns x.  Dividends whose magnitude is tiny (below 2^-899,
//    other than zero), huge (2^900 and above) or not finite use the IEEE
//    divide, so no intermediate underflows or overflows; divisors are
//    checked on the host to lie in [2^-100, 2^100].
//  * mul_const(x, f, c): x * c for a step constant c of at most 32
//    significant bits, in integers.
//  * half(x): 0.5 * x.  For normal x with a biased exponent >= 2 this is
//    exact, i.e. the exponent minus one, done in integer arithmetic; zero
//    keeps its bits; subnormal, smallest-normal and non-finite x use DMUL.
//  * upwind(w, p, q): (0.5 - copysign(0.5, w)) * p + (0.5 + copysign(0.5, w)) * q,
//    the first-order upwind pick of momentum_{u,v}_kern.c.  One weight is
//    1 and the other +0, so the value is the picked operand plus a zero
//    carrying the sign of the other operand; that is the picked operand,
//    or a zero whose sign is the AND of both signs.  Integer select; a
//    non-finite partner takes the IEEE expression.
#pragma once
#include <cuda_runtime.h>

namespace nl2d {

// A double's bit pattern and back.  Moved through inline PTX so the
// compiler treats the integer work on the bits as integer work: through a
// plain bitcast it may rewrite bits(x) & 0x7fff... as fabs(x), a sign-bit
// merge as copysign and a zero test as an FP64 compare, and on GB300 those
// run on the FP64 pipe the helpers are there to spare.  (The move itself
// costs nothing: both sides live in the same 64-bit register pair.)
__device__ __forceinline__ long long bits(double x) {
  long long b;
  asm("mov.b64 %0, %1;" : "=l"(b) : "d"(x));
  return b;
}
__device__ __forceinline__ double from_bits(long long b) {
  double x;
  asm("mov.b64 %0, %1;" : "=d"(x) : "l"(b));
  return x;
}
// The IEEE expressions the helpers fall back to, kept out of line: inlined,
// the compiler may predicate them and issue their FP64 instructions on every
// call, taken or not; as calls behind a branch they cost nothing when not
// taken.
static __device__ __noinline__ double div_ieee(double x, double d) { return x / d; }
static __device__ __noinline__ double half_ieee(double x) { return 0.5 * x; }
static __device__ __noinline__ double pick_ieee(double a, double z) { return a + 0.0 * z; }

// Markstein's two refinements: a faithful quotient, then the correctly
// rounded one.  Out of line: taken only when x * r lands on a power of two.
static __device__ __noinline__ double div_markstein(double x, double d, double r) {
  const double q0 = x * r;
  const double e0 = fma(q0, d, -x);
  const double q1 = fma(-e0, r, q0);
  const double e1 = fma(q1, d, -x);
  return fma(-e1, r, q1);
}

__device__ __forceinline__ double div_rn(double x, double d, double r) {
  const unsigned long long xb = (unsigned long long)bits(x);
  const unsigned xh = (unsigned)(xb >> 32);
  const int ex = (int)((xh >> 20) & 0x7ff);
  if (ex < 124 || ex > 1922) {
    if ((xb & 0x7fffffffffffffffULL) == 0) return x;  // +-0 / d keeps the sign for d > 0
    return div_ieee(x, d);
  }
  const double q0 = x * r;
  const unsigned long long qb = (unsigned long long)bits(q0), db = (unsigned long long)bits(d);
  constexpr unsigned long long kFrac = 0xfffffffffffffULL, kOne = 1ULL << 52;
  if ((qb & kFrac) == 0) return div_markstein(x, d, r);
  // q0 is not a power of two, so q = x / d lies in q0's binade and within
  // 1.5 ulp of it: RN(q) is q0 - ulp, q0 or q0 + ulp.  With the significands
  // mq, md, mx as integers, q0 * d - x = 2^t (mq md - mx 2^s) for the s of
  // the three exponents (52 or 53 here), and RN(q) moves off q0 exactly when
  // |mq md - mx 2^s| > md / 2 (a quotient is never a midpoint).  That
  // difference is below 1.5 md + 1 < 2^55 in size, so its low 64 bits are
  // all of it: of mx 2^s only the low bits of x count.
  const unsigned long long mq = (qb & kFrac) | kOne, md = (db & kFrac) | kOne;
  const unsigned sh = ((xh >> 20) - ((unsigned)(qb >> 32) >> 20) - (unsigned)(db >> 52) +
                       (1075u - 32u)) & 31u;  // s - 32
  const unsigned long long rem =
      mq * md - ((unsigned long long)((unsigned)xb << sh) << 32);
  // +1: one ulp up in magnitude (the remainder is negative), -1: one down
  long long k = 0;
  if (rem + (md >> 1) > (md & ~1ULL)) k = (long long)rem < 0 ? 1 : -1;
  return from_bits((long long)qb + k);
}

// A constant factor c > 0 in [2^-100, 2^100] of at most 32 significant bits
// (grid spacings and time steps in whole or simply fractional units), as
// mul_const takes it: co 2^e with co in [2^31, 2^32), and what the product's
// exponent field gains.  co = 0: c is not of that kind.
struct IntFactor {
  unsigned co, add;
};

// RN(x * c) in integers: the product of the significands (85 bits) is exact
// in three words, normalised by its leading bit and rounded to nearest even.
// Magnitudes of x below 2^-899 or from 2^900 take the IEEE product, +-0
// itself.  About 20 instructions on the integer pipes, where the DMUL holds
// a scheduler's share of the FP64 pipe for 64 issue slots.
static __device__ __noinline__ double mul_ieee(double x, double c) { return x * c; }
__device__ __forceinline__ double mul_const(double x, IntFactor f, double c) {
  const unsigned long long b = (unsigned long long)bits(x);
  const unsigned xl = (unsigned)b, xh = (unsigned)(b >> 32);
  if (((xh >> 20) & 0x7ffu) - 124u > 1798u) {
    if ((b & 0x7fffffffffffffffULL) == 0) return x;
    return mul_ieee(x, c);
  }
  const unsigned long long p = (unsigned long long)xl * f.co;
  const unsigned long long t =
      (unsigned long long)((xh & 0xfffffu) | 0x100000u) * f.co + (p >> 32);
  const unsigned w0 = (unsigned)p, w1 = (unsigned)t, w2 = (unsigned)(t >> 32);
  const unsigned top = w2 >> 20, s = top ^ 1u;  // the leading bit is bit 84 or 83
  const unsigned qh = __funnelshift_l(w1, w2, s), ql = __funnelshift_l(w0, w1, s);
  const unsigned frac = w0 << s;
  unsigned long long q = ((unsigned long long)qh << 32) | ql;
  if (frac > 0x80000000u - (ql & 1u)) q++;  // above half, or half and odd
  const unsigned eh = (xh & 0xfff00000u) + f.add + (top << 20);
  return from_bits((long long)(q + ((unsigned long long)eh << 32)));
}

__device__ __forceinline__ double half(double x) {
  const long long b = bits(x);
  const int ex = (int)((b >> 52) & 0x7ff);
  if (ex >= 2 && ex <= 2046) return from_bits(b - (1LL << 52));
  if ((b & 0x7fffffffffffffffLL) == 0) return x;
  return half_ieee(x);
}

// a + (+0 * z): the operand with weight 1 plus the zero-weighted partner.
__device__ __forceinline__ double pick(double a, double z) {
  const long long ab = bits(a), zb = bits(z);
  if (((zb >> 52) & 0x7ff) == 0x7ff) return pick_ieee(a, z);
  if ((ab & 0x7fffffffffffffffLL) != 0) return a;
  return from_bits(ab & (zb | 0x7fffffffffffffffLL));
}

__device__ __forceinline__ double upwind(double w, double p, double q) {
  return (bits(w) < 0) ? pick(p, q) : pick(q, p);
}

}  // namespace nl2d
