// The load sin(pi x) sin(pi y) sin(pi z) of a tetrahedron in 64-bit fixed point (pxg_fx.h):
// the Taylor series of each factor about vertex 0 in the offsets of the quadrature points
// (the machinery of pxg_q1x.h), their products, and the weighted sums to the nodes.
#pragma once

#include "pxg_q1x.h"

namespace pxg
{
namespace tetx
{
using namespace fx;

// the series for offsets in units of 2^sc: (4 pi)^k / k! = m 2^j
#ifdef __CUDACC__
__constant__
#endif
  q1x::SerC const kSeries[16] = {
    {cst(0), 0}, // coefficient 0 is S itself
    {cst(0x3243f6a8885a308dll), 6},
    {cst(0x4ef4f326f9177969ll), 8},
    {cst(0x52aef39896f94afbll), 10},
    {cst(0x40f07c206d6b0ecdll), 12},
    {cst(0x519af19dd6ab8749ll), 13},
    {cst(0x5574f1f8f2ffe7f1ll), 14},
    {cst(0x4cb4b3398af616fall), 15},
    {cst(0x3c3ea0d1237575e9ll), 16},
    {cst(0x541e0d21fb9e06e4ll), 16},
    {cst(0x34da3e5440951753ll), 17},
    {cst(0x3c60e9fbd10e3ec4ll), 17},
    {cst(0x3f3a7146ec79851cll), 17},
    {cst(0x3d1e869a031ac665ll), 17},
    {cst(0x36dc49e896251e5bll), 17},
    {cst(0x5beb6e7c555d0e45ll), 16},
};
// exponent of the coefficients, as q1x::seriesExponent: (8 pi 2^sc)^i / i! 2^-e below 0.36
PXG_HD int seriesExponent(int es, int sc)
{
  int const k = sc + (sc == -2 ? 9 : 6);
  return 1 + (es > k ? es : k);
}

// The three factors at the points, interleaved (their chains of products hide each other's
// latency): d[r][a] = differences of coordinate r of vertices 1..3 to vertex 0 (units
// 2^sc[r], F = 62), xi(q, a) the points (F = 62), S[r], C[r] = sin, cos of pi times vertex
// 0's coordinate, |pi offset| below 2^et[r]; f[r] at F = 62; returns the sum of their exponents
template <int NQ, class XI>
PXG_HD int factors(Sp const (&d)[3][3], int const (&sc)[3], int const (&et)[3], int deg, double const (&S)[3],
                   double const (&C)[3], XI const & xi, int64_t (&f)[3][NQ])
{
  int64_t ms[3], mc[3];
  int es[3], ec[3], e[3];
  Sp u[3][NQ];
#pragma unroll
  for (int r = 0; r < 3; ++r)
  {
    q1x::sineParts(S[r], ms[r], es[r]);
    q1x::sineParts(C[r], mc[r], ec[r]);
    e[r] = seriesExponent(es[r], sc[r]);
    int64_t const top = q1x::seriesCoef(kSeries[deg], e[r], sc[r], deg, (deg & 1) ? mc[r] : ms[r], (deg & 1) ? ec[r] : es[r]);
#pragma unroll
    for (int q = 0; q < NQ; ++q)
    {
      Sp const x[3] = {xi(q, 0), xi(q, 1), xi(q, 2)};
      u[r][q] = split(q1x::shl(dot3(d[r], x), 1)); // the offset at F = 61
      f[r][q] = top;
    }
  }
#pragma unroll 1
  for (int i = deg - 1; i >= 0; --i)
  {
    bool const odd = i & 1;
#pragma unroll
    for (int r = 0; r < 3; ++r)
    {
      int64_t const c = q1x::seriesCoef(kSeries[i], e[r], sc[r], i, odd ? mc[r] : ms[r], odd ? ec[r] : es[r]);
#pragma unroll
      for (int q = 0; q < NQ; ++q)
        f[r][q] = mulAdd(split(f[r][q]), u[r][q], c);
    }
  }
  int ex = 0;
#pragma unroll
  for (int r = 0; r < 3; ++r)
  {
    int const n = q1x::seriesShift(e[r], es[r], et[r]);
    ex += e[r] - n;
#pragma unroll
    for (int q = 0; q < NQ; ++q)
      f[r][q] = q1x::shl(f[r][q], n);
  }
  return ex;
}
} // namespace tetx
} // namespace pxg
