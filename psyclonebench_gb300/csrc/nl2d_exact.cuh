// Exact FP64 building blocks for the fused NEMOLite2D step.
//
// On GB300 the FP64 pipe issues 2 thread-operations per clock per SM, ~60x
// fewer than the integer and FP32 pipes, and an IEEE FP64 divide costs ~15
// FP64 instructions.  Each helper below returns the SAME bits as the plain
// IEEE expression it replaces, for every input, but spends fewer FP64
// instructions:
//
//  * div_core / div_const / div_depth: x / d rounded to nearest for a divisor
//    d in [2^-100, 2^100] whose 64-bit reciprocal was computed beforehand,
//    entirely in integers (about 32 instructions, no FP64): the quotient's
//    leading 53 bits by a multiply with the reciprocal, never above the true
//    quotient and less than 1.01 units below it, then the exact remainder
//    decides whether it rounds up.  (An FP64 multiply by RN(1/d) with the
//    remainder by FMA held the FP64 pipe for two instructions, with the
//    remainder in integers for one; IEEE division takes ~15.)
//    x = +-0 returns x.  Dividends of tiny magnitude (below 2^-899) take the
//    same quotient and round it once more where it is subnormal (div_other);
//    huge ones (2^900 and above) and non-finite ones use the IEEE divide.
//  * mul_bounded, div_bounded, upwind_bounded: the operations of the tiles'
//    straight-line code, on operands whose range has been tested.
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

#include <cstring>

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

// floor((2^116 - 1) / md) for md in [2^52, 2^53): the 64-bit reciprocal of
// the divisor whose significand md is.
__host__ __device__ __forceinline__ unsigned long long recip64(unsigned long long md) {
  const unsigned __int128 n = ((unsigned __int128)1 << 116) - 1;
  return (unsigned long long)(n / md);
}

__host__ __device__ __forceinline__ unsigned long long recip64_of(double d) {
  if (!(d >= 0x1p-100 && d <= 0x1p100)) return 0;
  unsigned long long b;
  memcpy(&b, &d, sizeof b);
  return recip64((b & 0xfffffffffffffULL) | (1ULL << 52));
}

// The significand q in [2^52, 2^53] of x / d rounded to nearest, for a
// normal x (bits xb), the divisor's significand md and its reciprocal rc; top
// = 1 where x's significand is at least d's.  With mx the dividend's
// significand, t = hi64(2^11 mx rc) is mx / md 2^63 to within 4 units below
// (the low partial product is left out): its leading bit says whether mx >=
// md, and its top 53 bits are less than 1.01 below the quotient mx 2^s / md
// (s = 52 or 53).  The remainder mx 2^s - q md is below 2^54, so its low 64
// bits are all of it, and q rounds up exactly when it is above md / 2 (a
// quotient of two significands is never a midpoint).
__device__ __forceinline__ unsigned long long div_significand(unsigned long long xb,
                                                              unsigned long long md,
                                                              unsigned long long rc,
                                                              unsigned& top) {
  const unsigned xl = (unsigned)xb, xh = (unsigned)(xb >> 32);
  const unsigned rl = (unsigned)rc, rh = (unsigned)(rc >> 32);
  const unsigned ah = __funnelshift_l(xl, xh, 11) | 0x80000000u, al = xl << 11;
  const unsigned long long t = (unsigned long long)ah * rh + __umulhi(ah, rl) + __umulhi(al, rh);
  top = (unsigned)(t >> 32) >> 31;
  unsigned long long q = t >> (10 + top);
  const unsigned long long rem = ((unsigned long long)(xl << (21 - top)) << 32) - q * md;
  if ((long long)rem > (long long)(md >> 1)) q++;
  return q;
}
// The quotient for a dividend of biased exponent 124 .. 1922; add = (1023 -
// the divisor's biased exponent - 2) << 20 is what its exponent field gains.
__device__ __forceinline__ double div_core(unsigned long long xb, unsigned long long md,
                                           unsigned long long rc, unsigned add) {
  unsigned top;
  const unsigned long long q = div_significand(xb, md, rc, top);
  const unsigned eh = ((unsigned)(xb >> 32) & 0xfff00000u) + add + (top << 20);
  return from_bits((long long)(q + ((unsigned long long)eh << 32)));
}

// The quotient for a nonzero dividend outside div_core's exponents.  Below
// them it is the 53-bit quotient of the normalised significand and, where the
// result is subnormal (q 2^-s units of 2^-1074), q shifted to those units and
// rounded to nearest even.  q itself is rounded, so where its discarded bits
// are exactly half the remainder's sign says on which side the true quotient
// lies.  One call, out of line: where a wave's front spreads from rest, values
// from 1e-270 down to the smallest subnormal fill whole tiles and every one of
// a cell's 19 divisions comes here; by the IEEE divide (about 600 clocks for
// such operands) a step of 128^2 took 25 us there, and takes 15.6.
static __device__ __noinline__ double div_other(double x, double d, unsigned long long rc) {
  const unsigned long long xb = (unsigned long long)bits(x), db = (unsigned long long)bits(d);
  if (xb & (1ULL << 62)) return x / d;  // 2^900 and above, or not finite
  const unsigned long long md = (db & 0xfffffffffffffULL) | (1ULL << 52);
  const unsigned long long sign = xb & (1ULL << 63);
  unsigned long long mx = xb & 0xfffffffffffffULL;
  int ex = (int)(xb >> 52) & 0x7ff;
  if (ex == 0) {
    const int n = __clzll((long long)mx) - 11;
    mx <<= n;
    ex = 1 - n;
  } else {
    mx |= 1ULL << 52;
  }
  unsigned top;
  const unsigned long long q = div_significand(mx, md, rc, top);
  // the result's exponent field less q's leading bit
  const int e = ex + 1021 - ((int)(db >> 52) & 0x7ff) + (int)top;
  if (e >= 0) return from_bits((long long)(sign | (q + ((unsigned long long)e << 52))));
  const int s = -e;
  if (s > 53) return from_bits((long long)sign);  // q is at most 2^53, then less than half a unit
  const long long rem = (long long)((mx << (53 - top)) - q * md);
  const unsigned long long low = q & ((1ULL << s) - 1), mid = 1ULL << (s - 1);
  unsigned long long c = q >> s;
  if (low > mid || (low == mid && (rem > 0 || (rem == 0 && (c & 1))))) c++;
  return from_bits((long long)(sign | c));
}

// A step constant as a divisor.
struct IntDivisor {
  double d;
  unsigned long long md, rc;
  unsigned add;
};
__device__ __forceinline__ double div_const(double x, const IntDivisor& v) {
  const unsigned long long xb = (unsigned long long)bits(x);
  if (((unsigned)(xb >> 52) & 0x7ffu) - 124u > 1798u) {
    if ((xb & 0x7fffffffffffffffULL) == 0) return x;  // +-0 / d keeps the sign for d > 0
    return div_other(x, v.d, v.rc);
  }
  return div_core(xb, v.md, v.rc, v.add);
}
// The same for a divisor from an array, with its reciprocal rc (not 0).
__device__ __forceinline__ double div_depth(double x, double d, unsigned long long rc) {
  const unsigned long long xb = (unsigned long long)bits(x), db = (unsigned long long)bits(d);
  if (((unsigned)(xb >> 52) & 0x7ffu) - 124u > 1798u) {
    if ((xb & 0x7fffffffffffffffULL) == 0) return x;
    return div_other(x, d, rc);
  }
  return div_core(xb, (db & 0xfffffffffffffULL) | (1ULL << 52), rc,
                  (1021u << 20) - ((unsigned)(db >> 32) & 0x7ff00000u));
}

// A constant factor c > 0 in [2^-100, 2^100] of at most 32 significant bits
// (grid spacings and time steps in whole or simply fractional units), as
// mul_bounded takes it: co 2^e with co in [2^31, 2^32), and what the product's
// exponent field gains.  co = 0: c is not of that kind.
struct IntFactor {
  unsigned co, add;
};

// The bounded forms, for straight-line code (a range branch per operation
// would keep the compiler from interleaving independent chains): operands are
// +-0 or normal, results too.
//
// The result with exponent field e (less q's leading bit), sign bit sign,
// significand q in [2^52, 2^53].
__device__ __forceinline__ double bounded_result(bool zero, unsigned sign, unsigned e,
                                                 unsigned long long q) {
  const unsigned long long r = q + ((unsigned long long)(e + sign) << 32);
  return from_bits((long long)(zero ? (unsigned long long)sign << 32 : r));
}

// RN(x * c): the product of the significands (85 bits) is exact in three
// words, normalised by its leading bit and rounded to nearest even.  About 25
// instructions on the integer pipes, where a DMUL holds its scheduler's FP64
// unit for 64 clocks.
__device__ __forceinline__ double mul_bounded(double x, IntFactor f) {
  const unsigned long long xb = (unsigned long long)bits(x);
  const unsigned xl = (unsigned)xb, xh = (unsigned)(xb >> 32);
  const unsigned long long p = (unsigned long long)xl * f.co;
  const unsigned long long t =
      (unsigned long long)((xh & 0xfffffu) | 0x100000u) * f.co + (p >> 32);
  const unsigned w0 = (unsigned)p, w1 = (unsigned)t, w2 = (unsigned)(t >> 32);
  const unsigned top = w2 >> 20, s = top ^ 1u;  // the leading bit is bit 84 or 83
  const unsigned qh = __funnelshift_l(w1, w2, s), ql = __funnelshift_l(w0, w1, s);
  const unsigned frac = w0 << s;
  unsigned long long q = ((unsigned long long)qh << 32) | ql;
  if (frac > 0x80000000u - (ql & 1u)) q++;  // above half, or half and odd
  const unsigned ex = xh & 0x7ff00000u;
  return bounded_result(ex == 0, xh & 0x80000000u, ex + f.add + (top << 20), q);
}

// RN(x * y): the 106-bit product of the significands in four words (x's
// aligned so that the leading bit is bit 116 or 115), rounded to nearest
// even; about 35 instructions.
__device__ __forceinline__ double mul_bounded(double x, double y) {
  const unsigned long long xb = (unsigned long long)bits(x), yb = (unsigned long long)bits(y);
  const unsigned xl = (unsigned)xb, xh = (unsigned)(xb >> 32);
  const unsigned yl = (unsigned)yb, yh = (unsigned)(yb >> 32);
  const unsigned ah = __funnelshift_l(xl, xh, 11) | 0x80000000u, al = xl << 11;
  const unsigned bh = (yh & 0xfffffu) | 0x100000u, bl = yl;
  const unsigned long long p0 = (unsigned long long)al * bl;
  const unsigned long long p1 = (unsigned long long)ah * bl + (p0 >> 32);
  const unsigned long long p2 = (unsigned long long)al * bh + (unsigned)p1;
  const unsigned long long hi = (unsigned long long)ah * bh + (p1 >> 32) + (p2 >> 32);
  const unsigned w3 = (unsigned)(hi >> 32), w2 = (unsigned)hi, w1 = (unsigned)p2,
                 w0 = (unsigned)p0;
  const unsigned top = w3 >> 20, s = top ^ 1u;
  const unsigned qh = __funnelshift_l(w2, w3, s), ql = __funnelshift_l(w1, w2, s);
  const unsigned f1 = __funnelshift_l(w0, w1, s), f0 = w0 << s;
  unsigned long long q = ((unsigned long long)qh << 32) | ql;
  const unsigned most = (f0 | (ql & 1u)) ? 0x7fffffffu : 0x80000000u;
  if (f1 > most) q++;  // above half, or half and odd
  const unsigned ex = xh & 0x7ff00000u, ey = yh & 0x7ff00000u;
  return bounded_result(ex == 0 || ey == 0, (xh ^ yh) & 0x80000000u,
                        ex + ey + (top << 20) - (1024u << 20), q);
}

// RN(x / d), see div_core.
__device__ __forceinline__ double div_bounded(double x, unsigned long long md,
                                              unsigned long long rc, unsigned add) {
  const unsigned long long xb = (unsigned long long)bits(x);
  const unsigned xh = (unsigned)(xb >> 32);
  const unsigned ex = xh & 0x7ff00000u;
  unsigned top;
  const unsigned long long q = div_significand(xb, md, rc, top);
  return bounded_result(ex == 0, xh & 0x80000000u, ex + add + (top << 20), q);
}
__device__ __forceinline__ double div_bounded(double x, const IntDivisor& v) {
  return div_bounded(x, v.md, v.rc, v.add);
}
__device__ __forceinline__ double div_bounded(double x, double d, unsigned long long rc) {
  const unsigned long long db = (unsigned long long)bits(d);
  return div_bounded(x, (db & 0xfffffffffffffULL) | (1ULL << 52), rc,
                     (1021u << 20) - ((unsigned)(db >> 32) & 0x7ff00000u));
}
// upwind() for operands that are +-0 or normal: the picked one, or, where
// that is a zero, a zero with the AND of both signs.
__device__ __forceinline__ double upwind_bounded(double w, double p, double q) {
  const bool neg = bits(w) < 0;
  const unsigned long long a = (unsigned long long)bits(neg ? p : q),
                           z = (unsigned long long)bits(neg ? q : p);
  const unsigned ah = (unsigned)(a >> 32), zh = (unsigned)(z >> 32);
  const unsigned h = (ah & 0x7ff00000u) == 0 ? ah & zh : ah;
  return from_bits((long long)(((unsigned long long)h << 32) | (unsigned)a));
}
// Whether x is neither +-0 nor of magnitude in [2^-lo, 2^hi).
__device__ __forceinline__ bool beyond(double x, unsigned lo, unsigned hi) {
  const unsigned h = (unsigned)((unsigned long long)bits(x) >> 32);
  const bool zero = ((unsigned)bits(x) | (h << 1)) == 0;
  return !zero && ((h >> 20) & 0x7ffu) - (1023u - lo) >= lo + hi;
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
