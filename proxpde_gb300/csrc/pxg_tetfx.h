// Tetrahedron geometry in 64-bit fixed point (pxg_fx.h).  Compiles for the host too, where its
// accuracy is tested.
//
// The edge vectors and their cofactor vectors (the cross products) each have an exponent of
// their own, and a cross product is formed to 2^-92 before it is normalised and rounded: a
// small face or a short edge beside large ones keeps its bits, as it does in FP64, whose form
// (adj3, gram) this replaces and whose errors it stays at or below.  Refused, for that form:
// edges whose components need more bits than the common exponent of the edge leaves (below
// 2^-8 of the largest) in an element whose faces or volume are small enough to show it, an
// element whose volume cancels against every face, and non-finite, zero and extreme values.
// About 450 integer instructions and 16 conversions take the place of 75 FP64 operations of 64
// cycles each: P1 96^3 x 6 in 0.75 ms, 1.14 ms in FP64; elements flat along an axis are told by
// their coordinates' extents before most of it (96^3 x 6 flattened by 1e-3 1.04 ms; refused after
// the attempt 1.60).  Not kept: one exponent for all six products (0.79 ms), which loses the small
// entries (2^-45 of themselves at a shear of 0.1, 2^-18 beside an edge of 1e-3); weights of the
// coordinates for the flat ones (0.84 ms flattened, but 0.81 for all others: 128 registers).  P2's
// group kernel takes longer with this form (K + M and a load at 64^3 x 6 1.05 to 1.3 ms by shape,
// FP64 1.01).
#pragma once

#include "pxg_fx.h"

namespace pxg
{
namespace tetx
{
using namespace fx;

// hi 2^32 + lo
struct Wide
{
  int64_t hi;
  uint32_t lo;
};
PXG_HD int32_t mulHi(int32_t a, int32_t b)
{
#ifdef __CUDA_ARCH__
  return __mulhi(a, b);
#else
  return (int32_t)(((int64_t)a * b) >> 32);
#endif
}
PXG_HD Wide wide(int64_t h, int64_t m)
{
  return {h + (m >> 32), lo32(m)};
}
// (x y - z w) / 2^32; all below 2^61
PXG_HD Wide wideDiff(Sp x, Sp y, Sp z, Sp w)
{
  int64_t const m = madw(x.h, y.l, madw(y.h, x.l, madw(-z.h, w.l, madw(-w.h, z.l, 0))));
  return wide(madw(x.h, y.h, madw(-z.h, w.h, 0)), m + (mulHi(x.l, y.l) - (int64_t)mulHi(z.l, w.l)));
}
PXG_HD Wide wideDot(Sp const (&x)[3], Sp const (&y)[3])
{
  int64_t h = 0, m = 0, l = 0;
#pragma unroll
  for (int r = 0; r < 3; ++r)
  {
    h = madw(x[r].h, y[r].h, h);
    m = madw(x[r].h, y[r].l, madw(x[r].l, y[r].h, m));
    l += mulHi(x[r].l, y[r].l);
  }
  return wide(h, m + l);
}
// w 2^n / 2^32, 0 < n < 32
PXG_HD int64_t wideShl(Wide w, int n) { return (int64_t)((uint64_t)w.hi << n) | (int64_t)(w.lo >> (32 - n)); }
PXG_HD uint32_t absHi(int64_t x)
{
  int32_t const h = hi32(x);
  return (uint32_t)(h < 0 ? -h : h);
}

// G = km 2^ke C_a . C_b / |det J| (xx yy zz xy xz yz; C the cofactor vectors of J[r][a], the
// difference of coordinate r of vertex a + 1 to vertex 0; km at F = 62, or zero) and |det J|, each
// within a few 2^-54 (the mixed ones of |C_a| |C_b|) of the given J's.  False for an element the
// form refuses, or with ok false.
PXG_HD bool tetGram(double const (&J)[3][3], bool ok, int64_t km, int ke, double (&G)[6], double & adet)
{
  // edges at F = 61 - e, their largest component in [1/2, 1) 2^e
  Sp x[3][3];
  int e[3];
  bool exact = true;
#pragma unroll
  for (int k = 0; k < 3; ++k)
  {
    int const f0 = expoField(J[0][k]), f1 = expoField(J[1][k]), f2 = expoField(J[2][k]);
    int f = f0 > f1 ? f0 : f1;
    f = f > f2 ? f : f2;
    e[k] = f - 1022;
    ok = ok && e[k] >= -300 && e[k] <= 59;
    // (a double has 53 bits; its exponent field is 0 for zero)
    exact = exact && (f0 == 0 || f0 >= f - 8) && (f1 == 0 || f1 >= f - 8) && (f2 == 0 || f2 >= f - 8);
#pragma unroll
    for (int r = 0; r < 3; ++r)
      x[k][r] = split(roundToInt(scaleExp(J[r][k], 61 - e[k])));
  }
  // an element flat along an axis by more than 2^6: nearly all of these would be refused below
  // (here, not before the conversions: there the kernel takes 100 registers instead of 96, a fifth of
  // its warps)
  {
    int m[3];
#pragma unroll
    for (int r = 0; r < 3; ++r)
    {
      int const a = hi32(doubleBits(J[r][0])) & 0x7fffffff, b = hi32(doubleBits(J[r][1])) & 0x7fffffff,
                c = hi32(doubleBits(J[r][2])) & 0x7fffffff;
      m[r] = a > b ? a : b;
      m[r] = m[r] > c ? m[r] : c;
    }
    int const hi = m[0] > m[1] ? (m[0] > m[2] ? m[0] : m[2]) : (m[1] > m[2] ? m[1] : m[2]),
              lo = m[0] < m[1] ? (m[0] < m[2] ? m[0] : m[2]) : (m[1] < m[2] ? m[1] : m[2]);
    if (hi - lo > (6 << 20))
      return false;
  }
  // cofactor vectors, the largest component in [1/4, 1/2) at F = 62: times 2^E
  Sp c[3][3];
  int n[3], E[3];
#pragma unroll
  for (int k = 0; k < 3; ++k)
  {
    int const a = (k + 1) % 3, b = (k + 2) % 3;
    Wide w[3];
    uint32_t z = 0;
#pragma unroll
    for (int r = 0; r < 3; ++r)
    {
      int const s = (r + 1) % 3, t = (r + 2) % 3;
      w[r] = wideDiff(x[a][s], x[b][t], x[a][t], x[b][s]);
      uint32_t const h = absHi(w[r].hi);
      z = h > z ? h : z;
    }
    ok = ok && z >= 8u;
    n[k] = clz32(z) - 3;
    E[k] = e[a] + e[b] - 58 - n[k];
#pragma unroll
    for (int r = 0; r < 3; ++r)
      c[k][r] = split(wideShl(w[r], n[k]));
  }
  // the determinant from the edge with the smallest cofactors
  int const k = n[0] >= n[1] && n[0] >= n[2] ? 0 : (n[1] >= n[2] ? 1 : 2);
  int const nk = k == 0 ? n[0] : (k == 1 ? n[1] : n[2]);
  Sp xk[3], ck[3];
#pragma unroll
  for (int r = 0; r < 3; ++r)
  {
    xk[r] = k == 0 ? x[0][r] : (k == 1 ? x[1][r] : x[2][r]);
    ck[r] = k == 0 ? c[0][r] : (k == 1 ? c[1][r] : c[2][r]);
  }
  Wide d = wideDot(xk, ck);
  if (d.hi < 0)
    d.hi = ~d.hi, d.lo = ~d.lo;
  uint32_t const z = (uint32_t)hi32(d.hi);
  int const nd = clz32(z) - 4;
  // nd: up to 8 the volume is 2^-5 of its edge times its face or more; nk + nd: the volume, and
  // nk the smallest face, against the edges' product
  ok = ok && nd >= 0 && nd <= 8 && (exact || (nk + nd <= 12 && nk <= 10));
  if (!ok)
    return false;
  int64_t const det = nd ? wideShl(d, nd) : d.hi; // F = 60, in [1/2, 1): |det J| = det 2^-60 2^eD
  int const eD = e[0] + e[1] + e[2] + 5 - nk - nd;
  // km / det at F = 61
  Sp const y = split((int64_t)((uint64_t)mul(split((int64_t)((uint64_t)recip(det) << 5)), split(km)) << 2));
#pragma unroll
  for (int i = 0; i < 6; ++i)
  {
    int const a = i < 3 ? i : (i == 5 ? 1 : 0), b = i < 3 ? i : (i == 3 ? 1 : 2);
    G[i] = toDouble(mul(split(dot3(c[a], c[b]) * 4), y), 65 + E[a] + E[b] - eD + ke);
  }
  adet = toDouble(det, eD - 60);
  return true;
}
} // namespace tetx
} // namespace pxg
