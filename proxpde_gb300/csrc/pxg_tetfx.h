// Tetrahedron geometry in 64-bit fixed point (pxg_q1x.h, whose point functions take the edge
// vectors as columns).
#pragma once

#include "pxg_internal.h"
#include "pxg_q1x.h"

namespace pxg
{
// G = km 2^ke C_a . C_b / |det J| (xx yy zz xy xz yz; C the cofactor vectors of J[r][a], the
// difference of coordinate r of vertex a + 1 to vertex 0; km at F = 62) times 2^-eG, and
// |det J|.  False for an element the format refuses, or with ok false.
__device__ __forceinline__ bool tetTensor(double const (&J)[3][3], bool ok, int64_t km, int ke, int64_t (&G)[6],
                                          int & eG, double & adet)
{
  using q1x::Sp;
  int32_t m[3];
#pragma unroll
  for (int r = 0; r < 3; ++r)
  {
    m[r] = 0;
#pragma unroll
    for (int k = 0; k < 3; ++k)
      m[r] = max(m[r], fx::hi32(fx::doubleBits(J[r][k])) & 0x7fffffff);
  }
  int sc[3];
  ok = q1x::coordScales(m[0], m[1], m[2], sc) && ok;
  int const scMin = min(sc[0], min(sc[1], sc[2]));
  int64_t D[3][3]; // [column][coordinate] at F = 60
  uint32_t cm[9];
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int k = 0; k < 3; ++k)
    {
      D[k][r] = fx::roundToInt(fx::scaleExp(J[r][k], 60 - sc[r]));
      cm[3 * k + r] = (uint32_t)abs(fx::hi32(D[k][r])) + 1u;
    }
  q1x::Shifts s;
  ok = q1x::columnShifts(cm, s) && ok;
  Sp c[3][3];
#pragma unroll
  for (int k = 0; k < 3; ++k)
#pragma unroll
    for (int r = 0; r < 3; ++r)
      c[k][r] = fx::splitOdd(q1x::shl(D[k][r], s.n[k]));
  int const wt[3] = {sc[0] - scMin, sc[1] - scMin, sc[2] - scMin};
  int64_t const det =
      q1x::pointProducts(c[0], c[1], c[2], __any_sync(__activemask(), (wt[0] | wt[1] | wt[2]) != 0) != 0, wt, G);
  uint32_t const h = (uint32_t)fx::hi32(det);
  int nd, k;
  ok = q1x::detShifts(h, h, nd, k) && ok;
  if (!ok)
    return false;
  int const sg = q1x::productShift(q1x::productSize(G, s));
  q1x::pointInverse(det, k, sg, fx::split(km), s, G);
  eG = q1x::tensorExponent(sc, scMin, s, k, sg) + ke - 58;
  adet = fx::toDouble(q1x::shl(det, nd), q1x::detExponent(sc, s, nd) - 60);
  return true;
}
} // namespace pxg
