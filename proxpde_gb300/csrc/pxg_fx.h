// 64-bit fixed-point arithmetic for the element kernels.
//
// GB300 issues an FP64 operation every 64 cycles per SM sub-partition (2 per clock and
// SM), but a 32 x 32 + 64-bit integer multiply-add every 2 cycles and a 64-bit addition
// every 3 (measured).  A product of two 64-bit fixed-point numbers, rounded to its upper
// 64 bits, is three to four such multiply-adds: about 8 cycles where a double's product
// takes 64, with a 62-bit significand instead of 53 as long as the operands share a
// common exponent.  An element's values do: every length is at most the element's size,
// so one power of two per element (and per reference direction) normalises them.  The
// elements whose values do not fit such a format (strongly degenerate or stretched ones,
// zero, non-finite or out-of-range inputs) are computed in FP64 instead.
//
// "F = k" in the comments: the integer is the value times 2^k.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define PXG_HD __host__ __device__ __forceinline__
#else
#define PXG_HD inline __attribute__((always_inline))
#endif

namespace pxg
{
namespace fx
{

PXG_HD int32_t hi32(int64_t x) { return (int32_t)(x >> 32); }
PXG_HD uint32_t lo32(int64_t x) { return (uint32_t)x; }

PXG_HD int clz32(uint32_t x)
{
#ifdef __CUDA_ARCH__
  return __clz((int)x);
#else
  return x ? __builtin_clz(x) : 32;
#endif
}

PXG_HD float rcpApprox(float x)
{
#ifdef __CUDA_ARCH__
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
#else
  return 1.0f / x;
#endif
}

PXG_HD int64_t doubleBits(double x)
{
#ifdef __CUDA_ARCH__
  return __double_as_longlong(x);
#else
  union
  {
    double d;
    int64_t i;
  } u;
  u.d = x;
  return u.i;
#endif
}
PXG_HD double bitsDouble(int64_t x)
{
#ifdef __CUDA_ARCH__
  return __longlong_as_double(x);
#else
  union
  {
    double d;
    int64_t i;
  } u;
  u.i = x;
  return u.d;
#endif
}

// biased exponent field of a double
PXG_HD int expoField(double x) { return (hi32(doubleBits(x)) >> 20) & 0x7ff; }
// x 2^k by an addition to the exponent field; the caller keeps the result normal (an
// unchecked sum wraps into the sign).  Zeros (and subnormals) stay zero.
PXG_HD double scaleExp(double x, int k)
{
  int64_t const b = doubleBits(x);
  int32_t const h = hi32(b);
  return (h & 0x7ff00000) ? bitsDouble((int64_t)(((uint64_t)((uint32_t)h + ((uint32_t)k << 20)) << 32) | lo32(b))) : 0.0;
}
PXG_HD int64_t roundToInt(double x)
{
#ifdef __CUDA_ARCH__
  return __double2ll_rn(x);
#else
  return (int64_t)__builtin_nearbyint(x);
#endif
}

// a b + c: one IMAD.WIDE (the multiplication and the addition written in C++ become a
// product and a separate 64-bit addition)
PXG_HD int64_t madw(int32_t a, int32_t b, int64_t c)
{
#ifdef __CUDA_ARCH__
  int64_t d;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
  return d;
#else
  return (int64_t)a * b + c;
#endif
}
PXG_HD int64_t madwu(uint32_t a, uint32_t b, int64_t c)
{
#ifdef __CUDA_ARCH__
  int64_t d;
  asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
  return d;
#else
  return (int64_t)((uint64_t)a * b + (uint64_t)c);
#endif
}

// x as hi 2^32 + lo with both words signed, so that the partial products of a product
// are signed 32 x 32 multiplications
struct Sp
{
  int32_t h, l;
};
PXG_HD Sp split(int64_t x)
{
  return {(int32_t)((uint32_t)hi32(x) + (lo32(x) >> 31)), (int32_t)lo32(x)};
}
// as split, with an odd low word: -2^31 does not occur, so both words can be negated
PXG_HD Sp splitOdd(int64_t x) { return split(x | 1); }
PXG_HD Sp neg(Sp x) { return {-x.h, -x.l}; }

constexpr int64_t kHalf = 0x80000000ll; // rounds the words shifted out

// x y / 2^64, rounded (the product of the low words, below one unit, is dropped), plus c
PXG_HD int64_t mulAdd(Sp x, Sp y, int64_t c)
{
  int64_t const b = madw(x.l, y.h, madw(x.h, y.l, kHalf));
  return madw(x.h, y.h, c) + hi32(b);
}
PXG_HD int64_t mul(Sp x, Sp y)
{
  int64_t const b = madw(x.l, y.h, madw(x.h, y.l, kHalf));
  return madw(x.h, y.h, hi32(b));
}
// x y + z w
PXG_HD int64_t dot2(Sp x, Sp y, Sp z, Sp w)
{
  int64_t const b = madw(z.l, w.h, madw(z.h, w.l, madw(x.l, y.h, madw(x.h, y.l, kHalf))));
  return madw(z.h, w.h, madw(x.h, y.h, hi32(b)));
}
PXG_HD int64_t dot3(Sp const (&x)[3], Sp const (&y)[3])
{
  int64_t b = kHalf;
#pragma unroll
  for (int r = 0; r < 3; ++r)
    b = madw(x[r].l, y[r].h, madw(x[r].h, y[r].l, b));
  int64_t s = hi32(b);
#pragma unroll
  for (int r = 0; r < 3; ++r)
    s = madw(x[r].h, y[r].h, s);
  return s;
}

// a compile-time constant 0 < c < 0.36 at F = 64, split like Sp
struct Cst
{
  int32_t h, l;
};
constexpr Cst cst(int64_t c64)
{
  int64_t const h = (c64 + 0x80000000ll) >> 32;
  return {(int32_t)h, (int32_t)(c64 - h * 4294967296ll)};
}
// c x, rounded; |x| < 2^62
PXG_HD int64_t mulc(Cst c, int64_t x)
{
  int64_t const b = madw(hi32(x), c.l, madwu(lo32(x), (uint32_t)c.h, kHalf));
  return madw(hi32(x), c.h, hi32(b));
}

// an integer times 2^k as a double, correctly rounded (k keeps it normal)
PXG_HD double toDouble(int64_t x, int k) { return scaleExp((double)x, k); }
// the same for any k whose result is below 2^1023; zero below the normal range (a check that
// costs 2 % of the hexahedra's kernels where every entry makes it)
PXG_HD double toDoubleFlush(int64_t x, int k)
{
  double const d = (double)x;
  return expoField(d) + k > 0 ? scaleExp(d, k) : 0.0;
}
// the factor m 2^e (F = 62) of values whose last bit is 2^(e - bits), made smaller where that
// is below the normal range, so that they end at 2^-1022
PXG_HD void limitFactor(int64_t & m, int & e, int bits)
{
  int const low = bits - 1022 - e;
  if (low > 0)
  {
    m >>= low < 63 ? low : 63;
    e += low;
  }
}

// 1 / d for d at F = 60 in [1/2, 1): F = 56, relative error below 2^-55.  A float
// estimate y0 (relative error e below 2^-21), then y0 (1 + e + e^2), e = 1 - d y0.
PXG_HD int64_t recip(int64_t d)
{
  uint32_t const w = (uint32_t)(d >> 30);                                        // F = 30
  int32_t const y0 = (int32_t)(rcpApprox((float)w) * 18014398509481984.0f + 0.5f); // F = 24
  // 1 at F = 84 is 0 modulo 2^64: e is the wrapped product, negated
  int64_t const e = (int64_t)(0ull - ((uint64_t)madwu(lo32(d), (uint32_t)y0, 0) +
                                      ((uint64_t)((uint32_t)hi32(d) * (uint32_t)y0) << 32)));
  int64_t const t = e + (madw(hi32(e), hi32(e), 0) >> 20);
  int64_t const c = madw(hi32(t), y0, (int64_t)(uint32_t)hi32(madwu(lo32(t), (uint32_t)y0, 0))); // F = 76
  return (int64_t)((uint64_t)(uint32_t)y0 << 32) + ((c + (1 << 19)) >> 20);
}

// mantissa (F = 62, in [0.5, 1), signed) and exponent of a double: x = m 2^-62 2^e;
// false for zeros, subnormals, infinities and NaN
PXG_HD bool decompose(double x, int64_t & m, int & e)
{
  int64_t const b = doubleBits(x);
  int const f = (hi32(b) >> 20) & 0x7ff;
  int64_t const a = ((b & 0xfffffffffffffll) | 0x10000000000000ll) << 9;
  m = b < 0 ? -a : a;
  e = f - 1022;
  return f != 0 && f != 0x7ff;
}
// the same of an operator's coefficient: zero is 0 2^0 (its elements' values are zero in
// fixed point too); false also beyond 2^+-300
PXG_HD bool coefParts(double x, int64_t & m, int & e)
{
  if (x == 0.)
  {
    m = 0, e = 0;
    return true;
  }
  return decompose(x, m, e) && e > -300 && e < 300;
}

} // namespace fx
} // namespace pxg
