// Q1 hexahedron element in 64-bit fixed point (pxg_fx.h): the steps of an element's
// geometry, stiffness and mass tables, entries and sine load, as functions of one
// coordinate, one quadrature point or one table, which the kernel deals to its warps.  The
// same quantities as the FP64 form computes (pxg_q1f64.h, whose notation this keeps), in
// a shape that suits the format: determinants from the Jacobian's cofactors (the Gram
// determinant, their square, would double the lost bits) and contractions on moments,
// sums and differences of the points' values, as additions cost little and products much.
// Compiles for the host too, where its accuracy is tested.
//
// Magnitudes.  Each coordinate is taken as differences to vertex 0 in units of a power of
// two above the largest (one unit for the three where they differ by at most 4: only
// elements flat along an axis need more), so that a thin extent keeps its bits; in these
// units the Jacobian columns (half edges) are shifted left by n_a until a bound of their
// 1-norm over the points is in [1/2, 1), and cofactors, their products and the
// determinants all stay below one.  The determinants' reciprocals and the products are
// normalised once more, per point and per element.  Every step rounds at 2^-60 of its largest
// value, so that cancellation loses bits from there: a rotated thin element of aspect a has
// entries within about a 2^-53 of their bounds, one sheared until its edges meet at 1 / a
// a 2^-52.  The FP64 form (pxg_q1f64.h), whose Gram determinant squares the condition, is 5 to
// 10^5 times further off in every shape (tests/test_fixed_point_host.py); FP64 cofactors of an
// axis-aligned shear would lose less than either.  Refused are non-finite coordinates and
// coefficients, elements whose determinant is below 2^-28 of their edges' product at some
// point, and sizes whose exponents the results could not hold.
#pragma once

#include "pxg_fx.h"

namespace pxg
{
namespace q1x
{
using namespace fx;

// Constants at F = 64: g = 0.5773502691896258 (src/qr.cpp:27) and the moments' factors of
// the 1D weights.  With m0 = v(-g) + v(g) and m1 = v(g) - v(-g): sum l_a v = (m0 + e_a g
// m1) / 2, sum l_a l_a v = a m0 + e_a b m1, sum l_0 l_1 v = c m0, where a = (1 + g^2) / 4,
// b = g / 2, c = (1 - g^2) / 4, e_0 = -1, e_1 = 1.
constexpr Cst kB = cst(0x49e69d1640cc7400ll); // g / 2
constexpr Cst kGG = cst(0x5555555555555bcall); // g^2
// 2 W W of the two-axis tables
constexpr Cst kAA = cst(0x38e38e38e38e3b0all); // 2 a a
constexpr Cst kAC = cst(0x1c71c71c71c71be8ll); // 2 a c
constexpr Cst kCC = cst(0x0e38e38e38e38d26ll); // 2 c c
constexpr Cst kAB = cst(0x314468b980884e44ll); // 2 a b
constexpr Cst kCB = cst(0x18a2345cc04425bcll); // 2 c b
constexpr Cst kBB = cst(0x2aaaaaaaaaaaade5ll); // 2 b b
// 2 l l W of the mixed tables: l = (1 + e g m1 / m0) / 2
constexpr Cst kUA = cst(0x2aaaaaaaaaaaab79ll); // a / 2
constexpr Cst kUC = cst(0x1555555555555487ll); // c / 2
constexpr Cst kUB = cst(0x24f34e8b20663a00ll); // b / 2
constexpr Cst kUAg = cst(0x18a2345cc0442722ll); // a g / 2
constexpr Cst kUCg = cst(0x0c511a2e602212dell); // c g / 2
constexpr Cst kUBg = cst(0x15555555555556f2ll); // b g / 2
constexpr Cst kUAgg = cst(0x0e38e38e38e38f91ll); // a g^2 / 2
constexpr Cst kUCgg = cst(0x071c71c71c71c761ll); // c g^2 / 2
constexpr Cst kUBgg = cst(0x0c511a2e60221444ll); // b g^2 / 2
// 8 W W W of the mass table
constexpr Cst kAAA = cst(0x4bda12f684bda57dll); // 8 a a a
constexpr Cst kAAC = cst(0x25ed097b425ed098ll); // 8 a a c
constexpr Cst kACC = cst(0x12f684bda12f6738ll); // 8 a c c
constexpr Cst kCCC = cst(0x097b425ed097b313ll); // 8 c c c
constexpr Cst kAAB = cst(0x41b08ba200b5beeell); // 8 a a b
constexpr Cst kACB = cst(0x20d845d1005add9all); // 8 a c b
constexpr Cst kCCB = cst(0x106c22e8802d6ddell); // 8 c c b
constexpr Cst kABB = cst(0x38e38e38e38e3e44ll); // 8 a b b
constexpr Cst kCBB = cst(0x1c71c71c71c71d85ll); // 8 c b b
constexpr Cst kBBB = cst(0x314468b98088510fll); // 8 b b b
// 2 l l l of the load
constexpr Cst kL0 = cst(0x4000000000000000ll); // 1 / 4
constexpr Cst kL1 = cst(0x24f34e8b20663a00ll); // g / 4
constexpr Cst kL2 = cst(0x15555555555556f2ll); // g^2 / 4
constexpr Cst kL3 = cst(0x0c511a2e60221444ll); // g^3 / 4

// sum and difference
PXG_HD void pairSum(int64_t & a, int64_t & b)
{
  int64_t const s = a + b, d = b - a;
  a = s, b = d;
}
// a -+ b: the values of classes 0 and 1 from the even and odd moments
PXG_HD void pairExpand(int64_t & a, int64_t & b)
{
  int64_t const s = a - b, d = a + b;
  a = s, b = d;
}
// moments over the three bits of the index (a set bit: difference), and back
PXG_HD void moments(int64_t (&v)[8])
{
#pragma unroll
  for (int s = 1; s < 8; s *= 2)
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (!(q & s))
        pairSum(v[q], v[q | s]);
}
PXG_HD void expand(int64_t (&v)[8])
{
#pragma unroll
  for (int s = 1; s < 8; s *= 2)
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (!(q & s))
        pairExpand(v[q], v[q | s]);
}
PXG_HD void expand2(int64_t & v0, int64_t & v1, int64_t & v2, int64_t & v3)
{
  pairExpand(v0, v1), pairExpand(v2, v3);
  pairExpand(v0, v2), pairExpand(v1, v3);
}
PXG_HD int64_t shl(int64_t x, int k) { return (int64_t)((uint64_t)x << k); }
PXG_HD uint32_t shr32(uint32_t x, int k) { return k < 32 ? x >> k : 0u; }
PXG_HD int64_t join(Sp x) { return shl((int64_t)x.h, 32) + x.l; }

// ------------------------------------------------------------------- geometry
// Columns of one coordinate r from its eight vertex values' differences to vertex 0 (d,
// index bits x, y, z; d[0] = 0) in units of 2^sc: col[a][p] at F = 60 for the column a at
// the points p = (qy, qz), (qx, qz), (qx, qy) (first bit lowest), and their largest high
// words per column; and the points' offsets J xi / g, their signed sums, at F = 61.
PXG_HD void coordColumns(double const (&d)[8], int sc, int64_t (&col)[3][4], uint32_t (&cmax)[3], int64_t (&off)[8])
{
  int64_t H[8];
  H[0] = 0;
#pragma unroll
  for (int v = 1; v < 8; ++v)
    H[v] = roundToInt(scaleExp(d[v], 57 - sc));
  // the Walsh-Hadamard transform, at most 7 2^57, is eight times the mean: F = 60
  moments(H);
  int64_t const a110 = 2 * mulc(kB, H[3]), a101 = 2 * mulc(kB, H[5]), a011 = 2 * mulc(kB, H[6]),
                a111 = mulc(kGG, H[7]);
#pragma unroll
  for (int p = 0; p < 2; ++p)
  {
    int64_t const u1 = p ? H[1] + a110 : H[1] - a110, u2 = p ? H[2] + a110 : H[2] - a110,
                  u3 = p ? H[4] + a101 : H[4] - a101;
    int64_t const w1 = p ? a101 + a111 : a101 - a111, w2 = p ? a011 + a111 : a011 - a111;
    col[0][p] = u1 - w1, col[0][p + 2] = u1 + w1; // (qy = p, qz)
    col[1][p] = u2 - w2, col[1][p + 2] = u2 + w2; // (qx = p, qz)
    col[2][p] = u3 - w2, col[2][p + 2] = u3 + w2; // (qx = p, qy)
  }
#pragma unroll
  for (int q = 0; q < 8; ++q)
  {
    int64_t const x = col[0][q >> 1], y = col[1][(q & 1) + 2 * (q >> 2)], z = col[2][q & 3];
    int64_t t = (q & 4) ? z : -z;
    t = (q & 2) ? t + y : t - y;
    off[q] = 2 * ((q & 1) ? t + x : t - x);
  }
#pragma unroll
  for (int a = 0; a < 3; ++a)
  {
    uint32_t m = 0;
#pragma unroll
    for (int p = 0; p < 4; ++p)
    {
      int32_t const h = hi32(col[a][p]);
      uint32_t const t = (uint32_t)(h < 0 ? -h : h);
      m = t > m ? t : m;
    }
    cmax[a] = m;
  }
}
// exponents sc[r] of the units from the largest differences' high words; false where the
// format does not take them (non-finite, or the conversions' exponents out of range)
PXG_HD bool coordScales(int32_t m0, int32_t m1, int32_t m2, int (&sc)[3])
{
  sc[0] = (m0 >> 20) - 1022, sc[1] = (m1 >> 20) - 1022, sc[2] = (m2 >> 20) - 1022;
  int const t = sc[0] > sc[1] ? sc[0] : sc[1], hi = t > sc[2] ? t : sc[2];
  int lo = hi;
#pragma unroll
  for (int r = 0; r < 3; ++r)
  {
    sc[r] = sc[r] >= hi - 2 ? hi : sc[r];
    lo = sc[r] < lo ? sc[r] : lo;
  }
  return lo >= -300 && hi <= 57; // (57: the conversion to F = 57 does not lower an exponent)
}

// Column shifts from the largest high words cmax[a * 3 + r]: the columns at F = 62 are then
// the half edges times 2^(n - 2) in units of 2^sc[r]
struct Shifts
{
  int n[3], nmin, nmax;
};
PXG_HD bool columnShifts(uint32_t const (&cmax)[9], Shifts & s)
{
  bool ok = true;
#pragma unroll
  for (int a = 0; a < 3; ++a)
  {
    s.n[a] = clz32(cmax[3 * a] + cmax[3 * a + 1] + cmax[3 * a + 2]) - 2;
    ok = ok && s.n[a] >= 0 && s.n[a] <= 40;
  }
  s.nmax = s.n[0] > s.n[1] ? s.n[0] : s.n[1];
  s.nmax = s.nmax > s.n[2] ? s.nmax : s.n[2];
  s.nmin = s.n[0] < s.n[1] ? s.n[0] : s.n[1];
  s.nmin = s.nmin < s.n[2] ? s.nmin : s.n[2];
  return ok;
}

// One point: the cofactors A, B, C of its shifted columns a, b, d, |det| and the products
// xx yy zz xy xz yz, all at F = 60; w[r]: the bits by which coordinate r's unit exceeds
// the smallest one (flat: some are not zero)
PXG_HD int64_t pointProducts(Sp const (&a)[3], Sp const (&b)[3], Sp const (&d)[3], bool flat, int const (&w)[3],
                             int64_t (&G)[6])
{
  Sp A[3], B[3], C[3];
#pragma unroll
  for (int r = 0; r < 3; ++r)
  {
    int const s = (r + 1) % 3, t = (r + 2) % 3;
    A[r] = split(shl(dot2(b[s], d[t], neg(b[t]), d[s]), 2)); // F = 62
    B[r] = split(shl(dot2(d[s], a[t], d[t], neg(a[s])), 2));
    C[r] = split(shl(dot2(a[s], b[t], a[t], neg(b[s])), 2));
  }
  int64_t const v = dot3(a, A);
  if (flat)
  {
#pragma unroll
    for (int r = 0; r < 3; ++r)
    {
      int const k = w[r] < 63 ? w[r] : 63;
      A[r] = split(join(A[r]) >> k), B[r] = split(join(B[r]) >> k), C[r] = split(join(C[r]) >> k);
    }
  }
  G[0] = dot3(A, A), G[1] = dot3(B, B), G[2] = dot3(C, C);
  G[3] = dot3(A, B), G[4] = dot3(A, C), G[5] = dot3(B, C);
  return v < 0 ? -v : v;
}

// Shifts from the high words of |det| at the eight points, the smallest lo and the largest
// hi: nd and k take the largest and the smallest to [1/2, 1) at F = 60
PXG_HD bool detShifts(uint32_t lo, uint32_t hi, int & nd, int & k)
{
  nd = clz32(hi) - 4, k = clz32(lo) - 4;
  return lo != 0 && nd >= 0;
}
// The largest diagonal product of a point, aligned to the common exponent (high word),
// and the shift to the left its maximum over the points leaves
PXG_HD uint32_t productSize(int64_t const (&G)[6], Shifts const & s)
{
  uint32_t const a = shr32((uint32_t)hi32(G[0]), 2 * (s.nmax - s.n[0])),
                 b = shr32((uint32_t)hi32(G[1]), 2 * (s.nmax - s.n[1])),
                 c = shr32((uint32_t)hi32(G[2]), 2 * (s.nmax - s.n[2]));
  uint32_t const m = a > b ? a : b;
  return m > c ? m : c;
}
PXG_HD int productShift(uint32_t size)
{
  int const k = clz32(size) - 4;
  return k < 0 ? 0 : k;
}
// exponents: det = det' 2^-60 2^eD (after the shift nd), G = G' 2^-58 2^eG
PXG_HD int detExponent(int const (&sc)[3], Shifts const & s, int nd)
{
  return sc[0] + sc[1] + sc[2] + 6 - (s.n[0] + s.n[1] + s.n[2]) - nd;
}
PXG_HD int tensorExponent(int const (&sc)[3], int scMin, Shifts const & s, int k, int sg)
{
  return k + 3 + sc[0] + sc[1] + sc[2] - 2 * scMin - (s.n[0] + s.n[1] + s.n[2]) + 2 * s.nmax - sg;
}
// G = km |J| (J^T J)^-1 at one point (F = 58) from its products and unshifted |det|: times
// 2^-(k+1) km / |det|, the components aligned to one exponent
PXG_HD void pointInverse(int64_t det, int k, int sg, Sp km, Shifts const & s, int64_t (&G)[6])
{
  int const n = clz32((uint32_t)hi32(det)) - 4;
  Sp const y = split(shl(mul(split(shl(recip(shl(det, n)), 5) >> (k - n)), km), 2));
#pragma unroll
  for (int c = 0; c < 6; ++c)
  {
    int const a = c < 3 ? c : (c == 5 ? 1 : 0), b = c < 3 ? c : (c == 3 ? 1 : 2);
    int const t = sg - (2 * s.nmax - s.n[a] - s.n[b]);
    G[c] = mul(split(shl(G[c], t > 0 ? t : 0)), y) >> (t > 0 ? 0 : (t > -63 ? -t : 63));
  }
}

// --------------------------------------------------------------------- tables
// Class tables of the stiffness, twice the sums over the points at the scale of G: class
// 0 / 1 of two equal 1D indices, 2 of a mixed pair.  S_x[cy][cz], S_y[cx][cz], S_z[cx][cy]
// (S[c][ce][cf]) and U_xy[jx][iy][cz], U_xz[jx][iz][cy], U_yz[jy][iz][cx] (U[c][a][b][w]),
// numbered one after the other.
constexpr int kTables = 63;
PXG_HD constexpr int idxS(int c, int ce, int cf) { return c * 9 + ce * 3 + cf; }
PXG_HD constexpr int idxU(int c, int a, int b, int w) { return 27 + c * 12 + (a * 2 + b) * 3 + w; }
// S of one component from its points v: bit 0 the axis summed out, W over bits 1 and 2
PXG_HD void tableS(int64_t const (&v)[8], int64_t (&S)[9])
{
  int64_t n00 = v[0] + v[1], n10 = v[2] + v[3], n01 = v[4] + v[5], n11 = v[6] + v[7];
  pairSum(n00, n10), pairSum(n01, n11);
  pairSum(n00, n01), pairSum(n10, n11);
  S[0] = mulc(kAA, n00), S[3] = mulc(kAB, n10), S[1] = mulc(kAB, n01), S[4] = mulc(kBB, n11);
  expand2(S[0], S[3], S[1], S[4]);
  S[2] = mulc(kAC, n00), S[5] = mulc(kCB, n10);
  S[6] = S[2], S[7] = mulc(kCB, n01);
  pairExpand(S[2], S[5]), pairExpand(S[6], S[7]);
  S[8] = mulc(kCC, n00);
}
// U of one component: l over bits 0 (a) and 1 (b), W over bit 2
PXG_HD void tableU(int64_t (&m)[8], int64_t (&U)[12])
{
  moments(m);
  int64_t A[4], B[4], C[4]; // index a + 2 b
  A[0] = mulc(kUA, m[0]), A[1] = mulc(kUAg, m[1]), A[2] = mulc(kUAg, m[2]), A[3] = mulc(kUAgg, m[3]);
  B[0] = mulc(kUB, m[4]), B[1] = mulc(kUBg, m[5]), B[2] = mulc(kUBg, m[6]), B[3] = mulc(kUBgg, m[7]);
  C[0] = mulc(kUC, m[0]), C[1] = mulc(kUCg, m[1]), C[2] = mulc(kUCg, m[2]), C[3] = mulc(kUCgg, m[3]);
  expand2(A[0], A[1], A[2], A[3]), expand2(B[0], B[1], B[2], B[3]), expand2(C[0], C[1], C[2], C[3]);
#pragma unroll
  for (int k = 0; k < 4; ++k)
  {
    int const u = ((k & 1) * 2 + (k >> 1)) * 3;
    U[u] = A[k] - B[k], U[u + 1] = A[k] + B[k], U[u + 2] = C[k];
  }
}

PXG_HD constexpr int cls(int a, int b) { return a == b ? a : 2; }
template <bool PLUS>
PXG_HD int64_t acc(int64_t a, int64_t b)
{
  return PLUS ? a + b : a - b;
}

// The entries of the y/z block (iy, iz), (jy, jz) and its x pairs, eight times K_ij at
// the scale of G: K(ix, jx) = e_ix e_jx Sx + e_ix F[jx] + e_jx F'[ix] + T[c(ix, jx)].
// t(k) is table value k.
template <int iy, int iz, int jy, int jz, class T>
PXG_HD void entryBlock(T const & t, int64_t (&K)[2][2])
{
  constexpr int cy = cls(iy, jy), cz = cls(iz, jz);
  constexpr bool yy = iy == jy, zz = iz == jz, yz = iy == jz, zy = jy == iz; // e e > 0
  constexpr bool diag = yy && zz;
  int64_t X[3];
#pragma unroll
  for (int cx = 0; cx < 3; ++cx)
  {
    // e_iy e_jy Sy + e_iz e_jz Sz + e_iy e_jz U(jy, iz) + e_jy e_iz U(iy, jz)
    int64_t const sy = t(idxS(1, cx, cz)), s = acc<zz>(yy ? sy : -sy, t(idxS(2, cx, cy)));
    if constexpr (diag)
      X[cx] = acc<yz>(s, 2 * t(idxU(2, jy, iz, cx)));
    else
      X[cx] = acc<yz>(acc<zy>(s, t(idxU(2, iy, jz, cx))), t(idxU(2, jy, iz, cx)));
  }
  int64_t F[2], Fp[2];
#pragma unroll
  for (int x = 0; x < 2; ++x)
  {
    int64_t const f = t(idxU(0, x, iy, cz));
    F[x] = acc<jz == 1>(jy ? f : -f, t(idxU(1, x, iz, cy)));
    if constexpr (diag)
      Fp[x] = F[x];
    else
    {
      int64_t const fp = t(idxU(0, x, jy, cz));
      Fp[x] = acc<iz == 1>(iy ? fp : -fp, t(idxU(1, x, jz, cy)));
    }
  }
  int64_t const sx = t(idxS(0, cy, cz));
#pragma unroll
  for (int ix = 0; ix < 2; ++ix)
#pragma unroll
    for (int jx = 0; jx < 2; ++jx)
    {
      if (diag && jx < ix)
        continue;
      int64_t k = X[cls(ix, jx)];
      k = jx ? k + Fp[ix] : k - Fp[ix];
      k = ix ? k + F[jx] : k - F[jx];
      K[ix][jx] = ix == jx ? k + sx : k - sx;
    }
}

// Mass class table, eight times Mt[cx][cy][cz] = sum_q v_q W W W at the scale of the
// points' values v (below one at F = 58)
PXG_HD void massTable(int64_t (&v)[8], int64_t (&M)[3][3][3])
{
  moments(v);
  int64_t w[8];
  w[0] = mulc(kAAA, v[0]);
  w[1] = mulc(kAAB, v[1]), w[2] = mulc(kAAB, v[2]), w[4] = mulc(kAAB, v[4]);
  w[3] = mulc(kABB, v[3]), w[5] = mulc(kABB, v[5]), w[6] = mulc(kABB, v[6]);
  w[7] = mulc(kBBB, v[7]);
  expand(w);
#pragma unroll
  for (int q = 0; q < 8; ++q)
    M[q & 1][(q >> 1) & 1][q >> 2] = w[q];
  // one mixed axis, two mixed axes
  int64_t const aac = mulc(kAAC, v[0]), x = mulc(kACB, v[1]), y = mulc(kACB, v[2]), z = mulc(kACB, v[4]);
  M[2][0][0] = aac, M[2][1][0] = y, M[2][0][1] = z, M[2][1][1] = mulc(kCBB, v[6]);
  expand2(M[2][0][0], M[2][1][0], M[2][0][1], M[2][1][1]);
  M[0][2][0] = aac, M[1][2][0] = x, M[0][2][1] = z, M[1][2][1] = mulc(kCBB, v[5]);
  expand2(M[0][2][0], M[1][2][0], M[0][2][1], M[1][2][1]);
  M[0][0][2] = aac, M[1][0][2] = x, M[0][1][2] = y, M[1][1][2] = mulc(kCBB, v[3]);
  expand2(M[0][0][2], M[1][0][2], M[0][1][2], M[1][1][2]);
  int64_t const acc0 = mulc(kACC, v[0]);
  M[0][2][2] = acc0, M[1][2][2] = mulc(kCCB, v[1]);
  M[2][0][2] = acc0, M[2][1][2] = mulc(kCCB, v[2]);
  M[2][2][0] = acc0, M[2][2][1] = mulc(kCCB, v[4]);
  pairExpand(M[0][2][2], M[1][2][2]), pairExpand(M[2][0][2], M[2][1][2]), pairExpand(M[2][2][0], M[2][2][1]);
  M[2][2][2] = mulc(kCCC, v[0]);
}

// ------------------------------------------------------------------ sine load
// sin(pi (o + d)) at the points, d = J xi: with u the signed column sums at F = 63 of
// their quarter (coordColumns), pi d = 4 pi g 2^sc u, and the Taylor series about o in u,
// Horner from the top.  A step multiplies by u at F = 63 and so loses one bit:
// coefficient k is kept at F = 62 + k, scaled by 2^-e so that it holds for sc <= -2.
struct SerC
{
  Cst m; // (4 pi g)^k / k! = m 2^j, k = 1..15
  int j;
};
#ifdef __CUDACC__
__constant__
#endif
  SerC const kSeries[16] = {
      {cst(0), 0}, // coefficient 0 is S itself
      {cst(0x3a0aa4f6dc87a652ll), 5},
      {cst(0x34a34cc4a60faa41ll), 7},
      {cst(0x3fa653af99556461ll), 8},
      {cst(0x39b951e3ef7ba41dll), 9},
      {cst(0x53c27987d5f2ba05ll), 9},
      {cst(0x32a41d9d01c719aell), 10},
      {cst(0x347cbede9f4066dfll), 10},
      {cst(0x2f99c7c1b08f6eball), 10},
      {cst(0x4cbeb872823ea0c4ll), 9},
      {cst(0x37ae156aab47d0ecll), 9},
      {cst(0x4972f1a42e34445cll), 8},
      {cst(0x58d08305dcd934c0ll), 7},
      {cst(0x31911161a51cebd5ll), 7},
      {cst(0x335faba26fce95fall), 6},
      {cst(0x31b2653d29e4b398ll), 5},
};
constexpr int kLoadMaxScale = -2;   // largest sc
constexpr float kLoadMaxT = 0.5f; // largest |pi d|
// a bound x 2^k of |pi d| as a float (zero below 2^-100: for the degree) and its exponent
struct Bound
{
  float f;
  int e; // below 2^e
};
PXG_HD Bound makeBound(float x, int k)
{
  Bound b;
#ifdef __CUDA_ARCH__
  int const i = __float_as_int(x);
  b.e = (i >> 23) - 126 + k;
  b.f = b.e < -100 ? 0.f : __int_as_float(i + (k << 23));
#else
  b.e = __builtin_ilogbf(x) + 1 + k;
  b.f = b.e < -100 ? 0.f : __builtin_ldexpf(x, k);
#endif
  return b;
}
// the bound for one coordinate from its columns' largest high words: pi g 2^(sc - 28) sum cmax
PXG_HD Bound offsetBound(uint32_t const (&cmax)[3], int sc, float ratio = 1.f)
{
  return makeBound((float)(cmax[0] + cmax[1] + cmax[2] + 1u) * (ratio * 1.8138f), sc - 28);
}
// mantissa (F = 62, signed) and exponent (at most 0) of a sine or cosine; zero: 0, -400
PXG_HD void sineParts(double x, int64_t & m, int & e)
{
  if (!decompose(x, m, e))
    m = 0, e = -400;
  if (e > 0) // +-1
    m *= 2, e = 0;
  e = e < -400 ? -400 : e;
}
// exponent of the coefficients of a series about o with sin(pi o) = m 2^es: they stay
// below 0.72 at F = 62 + i, that is (8 pi t 2^sc)^i / i! 2^-e < 0.72 for every i, t = g
// (Q2: the larger t of the three-point rule)
template <bool Q2 = false>
PXG_HD int seriesExponent(int es, int sc)
{
  int const k = sc + (Q2 ? (sc == -2 ? 8 : (sc == -3 ? 6 : 5)) : (sc == -2 ? 6 : 5));
  return 1 + (es > k ? es : k);
}
// the shift that normalises the series' sum, |pi d| below 2^et: sin = sum 2^-62
// 2^(e - shift) after it
PXG_HD int seriesShift(int e, int es, int et)
{
  int const n = e - 1 - (es > et ? es : et);
  return n < 0 ? 0 : (n > 40 ? 40 : n);
}
// coefficient i at F = 62 + i (t: entry i of the constants); m 2^em = S (i even) or C (odd)
PXG_HD int64_t seriesCoef(SerC const & t, int e, int sc, int i, int64_t m, int em)
{
  int const sr = e - em - t.j - i * (sc + 1);
  int64_t const v = (i ? mulc(t.m, m) : m) >> (sr < 63 ? sr : 63);
  return (i & 2) ? -v : v;
}
// degree for a bound of |pi d|: truncation below 8e-19
PXG_HD int seriesDegree(float bound) { return bound <= 0.0205f ? 7 : (bound <= 0.07f ? 9 : (bound <= 0.16f ? 11 : 15)); }
// |det| sin sin sin from the three normalised values: F = 59
PXG_HD int64_t pointLoad(int64_t f0, int64_t f1, int64_t f2, int64_t det)
{
  int64_t const f = shl(mul(split(f0), split(f1)), 2), g = shl(mul(split(f2), split(shl(det, 2))), 2);
  return mul(split(f), split(g)) >> 1;
}
// twice sum_q r_q l l l at the eight nodes (index bits x, y, z)
PXG_HD void nodeSums(int64_t (&r)[8])
{
  moments(r);
  r[0] = mulc(kL0, r[0]);
  r[1] = mulc(kL1, r[1]), r[2] = mulc(kL1, r[2]), r[4] = mulc(kL1, r[4]);
  r[3] = mulc(kL2, r[3]), r[5] = mulc(kL2, r[5]), r[6] = mulc(kL2, r[6]);
  r[7] = mulc(kL3, r[7]);
  expand(r);
}

} // namespace q1x
} // namespace pxg
