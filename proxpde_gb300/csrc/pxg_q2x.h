// Q2 hexahedron element in 64-bit fixed point (pxg_fx.h): the one-axis contractions of
// the sum factorisation in the notation of pxg_q2f64.h.  A line is three values v0, v1, v2
// at the 1D Gauss points -t, 0, t; with s = v0 + v2 and d = v2 - v0 the even parts of the
// class functions multiply s, the odd ones d, most vanish at 0, and the classes come in
// mirrored pairs: five products (two for the D and A classes) give six values where the
// three-term sums take eighteen.  Geometry as in pxg_q1x.h, whose functions it shares.
#pragma once

#include "pxg_q1x.h"

namespace pxg
{
namespace q2x
{
using namespace fx;

// t = 0.774596669241483 (src/qr.cpp:38); constants at F = 64, for arguments below 2^61
constexpr Cst kPa = cst(0x3d70a3d70a3d570cll); // t^2 (1 + t^2) / 4
constexpr Cst kPb = cst(0x3b7d30b098455dfall); // t^3 / 2
constexpr Cst kPe = cst(0x28f5c28f5c291afdll); // (1 - t^2)^2
constexpr Cst kPp = cst(0x0f5c28f5c28f5e7dll); // t^2 (1 - t^2) / 4
constexpr Cst kPh = cst(0x27a8cb206583b206ll); // t (1 - t^2) / 2
constexpr Cst kT2h = cst(0x4cccccccccccb589ll); // t^2 / 2
constexpr Cst kTh = cst(0x6325fbd0fdc91000ll); // t / 2
constexpr Cst kSu = cst(0x4f519640cb07640bll); // t (1 - t^2)
constexpr Cst kSw = cst(0x09ea32c81960d5fall); // (2 t^3 - t) / 4
constexpr Cst kSz = cst(0x6d102e991729e5fall); // (2 t^3 + t) / 4
constexpr Cst kSx = cst(0x3999999999998826ll); // 3 t^2 / 8
constexpr Cst kSy = cst(0x333333333333104dll); // (3 t^2 - 1) / 4
constexpr Cst kLc = cst(0x66666666666694efll); // 1 - t^2

// P_ab = l_a l_b in the classes (0,0) (1,1) (2,2) (0,1) (0,2) (1,2), with l_0 = x(x-1)/2,
// l_1 = x(x+1)/2, l_2 = 1 - x^2
PXG_HD void lineP(int64_t v0, int64_t v1, int64_t v2, int64_t (&o)[6])
{
  int64_t const s = v0 + v2, d = v2 - v0;
  int64_t const a = mulc(kPa, s), b = mulc(kPb, d), p = mulc(kPp, s), h = mulc(kPh, d);
  o[0] = a - b, o[1] = a + b;
  o[2] = v1 + mulc(kPe, s);
  o[3] = -p;
  o[4] = 2 * p - h, o[5] = 2 * p + h;
}
// D_ab = l'_a l'_b
PXG_HD void lineD(int64_t v0, int64_t v1, int64_t v2, int64_t (&o)[6])
{
  int64_t const s = v0 + v2, d = v2 - v0;
  int64_t const a = 2 * mulc(kT2h, s), b = 2 * mulc(kTh, d), q = (v1 + s + 2) >> 2;
  o[0] = q + a - b, o[1] = q + a + b;
  o[2] = 4 * a;
  o[3] = a - q;
  o[4] = b - 2 * a, o[5] = -b - 2 * a;
}
// S_ab = (l_a l_b)' / 2
PXG_HD void lineS(int64_t v0, int64_t v1, int64_t v2, int64_t (&o)[6])
{
  int64_t const s = v0 + v2, d = v2 - v0;
  int64_t const x = 2 * mulc(kSx, s), z = mulc(kSz, d), w = mulc(kSw, d), y = mulc(kSy, s) - ((v1 + 2) >> 2);
  o[0] = z - x, o[1] = z + x;
  o[2] = -2 * mulc(kSu, d);
  o[3] = w;
  o[4] = y - 2 * w, o[5] = -y - 2 * w;
}
// A_ab = (l'_a l_b - l'_b l_a) / 2 in the classes (0,1) (0,2) (1,2)
PXG_HD void lineA(int64_t v0, int64_t v1, int64_t v2, int64_t (&o)[3])
{
  int64_t const s = v0 + v2, d = v2 - v0;
  int64_t const a = 2 * mulc(kT2h, s), b = mulc(kTh, d), q = (v1 + s + a + 2) >> 2;
  o[0] = (a + 2) >> 2;
  o[1] = b - q, o[2] = b + q;
}
// l_a
PXG_HD void lineL(int64_t v0, int64_t v1, int64_t v2, int64_t (&o)[3])
{
  int64_t const s = v0 + v2, d = v2 - v0;
  int64_t const a = mulc(kT2h, s), b = mulc(kTh, d);
  o[0] = a - b, o[1] = a + b;
  o[2] = v1 + mulc(kLc, s);
}

// the sine series of pxg_q1x.h for offsets d = t (signed column sums): (4 pi t)^k / k! = m 2^j
#ifdef __CUDACC__
__constant__
#endif
  q1x::SerC const kSeries[16] = {
    {cst(0), 0}, // coefficient 0 is S itself
    {cst(0x4ddef69dfbeb86d1ll), 5},
    {cst(0x2f5fc51762413a7fll), 8},
    {cst(0x4cdb052bcdbe2572ll), 9},
    {cst(0x2ec1a10d1b94a6a6ll), 11},
    {cst(0x5b0628f027924bd6ll), 11},
    {cst(0x49d5ae3f8a4549e7ll), 12},
    {cst(0x3355e434d67bab81ll), 13},
    {cst(0x3e762e50074577e0ll), 13},
    {cst(0x438e0933001f7254ll), 13},
    {cst(0x41c1c9a7fbced01bll), 13},
    {cst(0x3a302bc94dcf0651ll), 13},
    {cst(0x2f331d5494ef7932ll), 13},
    {cst(0x46aeaf5936c4e0ball), 12},
    {cst(0x3124ce70db7c12acll), 12},
    {cst(0x3fc7fd3e91e670b1ll), 11},
};
// pi t / (pi g), rounded up: the bound of the offsets against q1x::offsetBound's
constexpr float kBoundRatio = 1.3417f;

} // namespace q2x
} // namespace pxg
