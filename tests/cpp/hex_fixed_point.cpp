// Host accuracy of the Q1 hexahedron in fixed point (csrc/pxg_q1x.h) against 128-bit arithmetic: the
// element's stiffness and mass, over shapes from cubes to strongly sheared, thin and needle-like ones,
// beside the FP64 form that takes the refused elements (J by a Walsh-Hadamard transform of the vertices,
// the Gram determinant of J).  Prints one line per shape: name, parameter, elements taken, refused, the
// largest errors of the stiffness (against the geometric mean of two diagonal entries) and of the mass
// (of itself) in fixed point and in FP64.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>

#include "pxg_q1x.h"

using namespace pxg::q1x;
typedef __float128 Quad;

static Quad root(Quad x)
{
  Quad y = (Quad)std::sqrt((double)x);
  for (int i = 0; i < 4; ++i)
    y = (y + x / y) / 2;
  return y;
}
static double root(double x) { return std::sqrt(x); }

// vertices and nodes by lattice index x + 2 y + 4 z
template <class T>
static void byQuadrature(double const (&X)[8][3], T k, T (&K)[8][8], T (&M)[8][8])
{
  T const g = 0.5773502691896258;
  for (int i = 0; i < 8; ++i)
    for (int j = 0; j < 8; ++j)
      K[i][j] = M[i][j] = 0;
  for (int q = 0; q < 8; ++q)
  {
    T const xi[3] = {(q & 1) ? g : -g, (q & 2) ? g : -g, (q & 4) ? g : -g};
    T phi[8], d[8][3], J[3][3];
    for (int v = 0; v < 8; ++v)
    {
      T l[3], e[3];
      for (int a = 0; a < 3; ++a)
        l[a] = (1 + ((v >> a) & 1 ? xi[a] : -xi[a])) / 2, e[a] = (v >> a) & 1 ? (T)0.5 : (T)-0.5;
      phi[v] = l[0] * l[1] * l[2];
      d[v][0] = e[0] * l[1] * l[2], d[v][1] = l[0] * e[1] * l[2], d[v][2] = l[0] * l[1] * e[2];
    }
    for (int r = 0; r < 3; ++r)
    {
      T H[8];
      for (int v = 0; v < 8; ++v)
        H[v] = X[v][r];
      for (int s = 1; s < 8; s *= 2)
        for (int v = 0; v < 8; ++v)
          if (!(v & s))
          {
            T const a = H[v], b = H[v | s];
            H[v] = a + b, H[v | s] = b - a;
          }
      J[r][0] = ((H[1] + xi[1] * H[3]) + xi[2] * (H[5] + xi[1] * H[7])) / 8;
      J[r][1] = ((H[2] + xi[0] * H[3]) + xi[2] * (H[6] + xi[0] * H[7])) / 8;
      J[r][2] = ((H[4] + xi[0] * H[5]) + xi[1] * (H[6] + xi[0] * H[7])) / 8;
    }
    T G[3][3], A[3][3];
    for (int a = 0; a < 3; ++a)
      for (int b = 0; b < 3; ++b)
        G[a][b] = J[0][a] * J[0][b] + J[1][a] * J[1][b] + J[2][a] * J[2][b];
    for (int a = 0; a < 3; ++a)
      for (int b = 0; b < 3; ++b)
      {
        int const a1 = (a + 1) % 3, a2 = (a + 2) % 3, b1 = (b + 1) % 3, b2 = (b + 2) % 3;
        A[a][b] = G[a1][b1] * G[a2][b2] - G[a1][b2] * G[a2][b1];
      }
    T const det = root(G[0][0] * A[0][0] + G[0][1] * A[0][1] + G[0][2] * A[0][2]);
    for (int i = 0; i < 8; ++i)
      for (int j = 0; j < 8; ++j)
      {
        T s = 0;
        for (int a = 0; a < 3; ++a)
          for (int b = 0; b < 3; ++b)
            s += d[i][a] * A[a][b] * d[j][b];
        K[i][j] += k * s / det;
        M[i][j] += det * phi[i] * phi[j];
      }
  }
}

struct Tables
{
  int64_t v[kTables];
  int64_t operator()(int k) const { return v[k]; }
};
template <int iy, int iz, int jy, int jz>
static void block(Tables const & t, int e, double (&K)[8][8])
{
  int64_t k[2][2] = {};
  entryBlock<iy, iz, jy, jz>(t, k);
  for (int ix = 0; ix < 2; ++ix)
    for (int jx = 0; jx < 2; ++jx)
    {
      if (iy == jy && iz == jz && jx < ix)
        continue;
      int const i = ix + 2 * iy + 4 * iz, j = jx + 2 * jy + 4 * jz;
      K[i][j] = K[j][i] = toDouble(k[ix][jx], e);
    }
}

static bool byFixedPoint(double const (&X)[8][3], double k, double (&K)[8][8], double (&M)[8][8])
{
  double d[3][8];
  int32_t m[3] = {};
  for (int r = 0; r < 3; ++r)
    for (int v = 0; v < 8; ++v)
    {
      d[r][v] = X[v][r] - X[0][r];
      m[r] = std::max(m[r], hi32(doubleBits(d[r][v])) & 0x7fffffff);
    }
  int sc[3];
  if (!coordScales(m[0], m[1], m[2], sc))
    return false;
  int const low = std::min(sc[0], std::min(sc[1], sc[2])), w[3] = {sc[0] - low, sc[1] - low, sc[2] - low};
  int64_t col[3][3][4];
  uint32_t cm[9];
  for (int r = 0; r < 3; ++r)
  {
    int64_t c[3][4], off[8];
    uint32_t z[3];
    coordColumns(d[r], sc[r], c, z, off);
    for (int a = 0; a < 3; ++a)
    {
      cm[a * 3 + r] = z[a];
      std::memcpy(col[a][r], c[a], sizeof(c[a]));
    }
  }
  Shifts s;
  if (!columnShifts(cm, s))
    return false;
  int64_t G[8][6], det[8];
  uint32_t lo = 0xffffffffu, hi = 0, size = 0;
  for (int q = 0; q < 8; ++q)
  {
    int const x = q & 1, y = (q >> 1) & 1, z = q >> 2;
    Sp c[3][3];
    for (int r = 0; r < 3; ++r)
    {
      c[0][r] = splitOdd(shl(col[0][r][y + 2 * z], s.n[0]));
      c[1][r] = splitOdd(shl(col[1][r][x + 2 * z], s.n[1]));
      c[2][r] = splitOdd(shl(col[2][r][x + 2 * y], s.n[2]));
    }
    det[q] = pointProducts(c[0], c[1], c[2], (w[0] | w[1] | w[2]) != 0, w, G[q]);
    uint32_t const h = (uint32_t)hi32(det[q]);
    lo = std::min(lo, h), hi = std::max(hi, h), size = std::max(size, productSize(G[q], s));
  }
  int nd, kd, ke, me;
  int64_t km, mm;
  if (!detShifts(lo, hi, nd, kd) || !coefParts(k, km, ke) || !coefParts(1., mm, me))
    return false;
  int const sg = productShift(size), eD = detExponent(sc, s, nd), eK = tensorExponent(sc, low, s, kd, sg) + ke - 61;
  limitFactor(mm, me, 61 - eD);
  for (int q = 0; q < 8; ++q)
  {
    pointInverse(det[q], kd, sg, split(km), s, G[q]);
    det[q] = mul(split(shl(det[q], nd)), split(mm));
  }
  Tables t;
  for (int c = 0; c < 3; ++c)
  {
    int64_t v[8], S[9], U[12];
    int const D = 1 << c, E = c == 0 ? 2 : 1, F = c == 2 ? 2 : 4;
    for (int i = 0; i < 8; ++i)
      v[i] = G[(i & 1) * D + ((i >> 1) & 1) * E + (i >> 2) * F][c];
    tableS(v, S);
    std::memcpy(t.v + 9 * c, S, sizeof(S));
    int const D2 = c == 2 ? 2 : 1, E2 = c == 0 ? 2 : 4, F2 = c == 0 ? 4 : (c == 1 ? 2 : 1);
    for (int i = 0; i < 8; ++i)
      v[i] = G[(i & 1) * D2 + ((i >> 1) & 1) * E2 + (i >> 2) * F2][3 + c];
    tableU(v, U);
    std::memcpy(t.v + 27 + 12 * c, U, sizeof(U));
  }
  int64_t Mt[3][3][3];
  massTable(det, Mt);
  for (int i = 0; i < 8; ++i)
    for (int j = 0; j < 8; ++j)
      M[i][j] = toDouble(Mt[cls(i & 1, j & 1)][cls((i >> 1) & 1, (j >> 1) & 1)][cls(i >> 2, j >> 2)], eD + me - 61);
  block<0, 0, 0, 0>(t, eK, K), block<1, 0, 1, 0>(t, eK, K), block<0, 1, 0, 1>(t, eK, K), block<1, 1, 1, 1>(t, eK, K);
  block<0, 0, 1, 0>(t, eK, K), block<0, 0, 0, 1>(t, eK, K), block<0, 0, 1, 1>(t, eK, K), block<1, 0, 0, 1>(t, eK, K);
  block<1, 0, 1, 1>(t, eK, K), block<0, 1, 1, 1>(t, eK, K);
  return true;
}

int main()
{
  std::mt19937_64 rng(3);
  auto U = [&] { return (double)(rng() >> 11) * 0x1p-53; };
  char const * const names[] = {"cube", "shear", "thin", "thin_rotated", "shear_rotated", "needle_rotated", "small"};
  for (int kind = 0; kind < 7; ++kind)
    for (double eps : {1., 0.1, 1e-2, 1e-3, 1e-4})
    {
      if (kind == 0 && eps < 1.)
        continue;
      int taken = 0, refused = 0;
      double fx[2] = {}, fp[2] = {};
      for (int it = 0; it < 200; ++it)
      {
        double A[3][3] = {{0.5 + U(), 0., 0.}, {0., 0.5 + U(), 0.}, {0., 0., 0.5 + U()}}, R[3][3] = {{1, 0, 0}, {0, 1, 0}, {0, 0, 1}};
        if (kind == 1 || kind == 4)
          A[0][1] = 0.3 + U(), A[1][1] *= eps, A[0][2] = U(), A[1][2] = U();
        if (kind == 2 || kind == 3 || kind == 5)
          A[2][2] *= eps;
        if (kind == 5)
          A[1][1] *= eps;
        if (kind >= 3 && kind <= 5)
        {
          double q[4], n = 0.;
          for (double & x : q)
            x = U() - 0.5, n += x * x;
          for (double & x : q)
            x /= std::sqrt(n);
          double const T[3][3] = {{1 - 2 * (q[2] * q[2] + q[3] * q[3]), 2 * (q[1] * q[2] - q[0] * q[3]), 2 * (q[1] * q[3] + q[0] * q[2])},
                                  {2 * (q[1] * q[2] + q[0] * q[3]), 1 - 2 * (q[1] * q[1] + q[3] * q[3]), 2 * (q[2] * q[3] - q[0] * q[1])},
                                  {2 * (q[1] * q[3] - q[0] * q[2]), 2 * (q[2] * q[3] + q[0] * q[1]), 1 - 2 * (q[1] * q[1] + q[2] * q[2])}};
          std::memcpy(R, T, sizeof(R));
        }
        double const h = kind == 6 ? std::pow(eps, 12.) : 1. / 16., base = kind == 6 ? 0. : 0.4;
        double X[8][3], o[3] = {base * U(), base * U(), base * U()};
        for (int v = 0; v < 8; ++v)
        {
          double p[3], t[3] = {};
          for (int a = 0; a < 3; ++a)
            p[a] = ((v >> a) & 1) + 0.1 * (2 * U() - 1);
          for (int r = 0; r < 3; ++r)
            for (int a = 0; a < 3; ++a)
              t[r] += A[r][a] * p[a];
          for (int r = 0; r < 3; ++r)
            X[v][r] = o[r] + h * (R[r][0] * t[0] + R[r][1] * t[1] + R[r][2] * t[2]);
        }
        double const k = std::exp(4. * (U() - 0.5));
        double K[8][8], M[8][8], Kd[8][8], Md[8][8];
        if (!byFixedPoint(X, k, K, M))
        {
          ++refused;
          continue;
        }
        ++taken;
        Quad Kq[8][8], Mq[8][8];
        byQuadrature<Quad>(X, k, Kq, Mq);
        byQuadrature<double>(X, k, Kd, Md);
        for (int i = 0; i < 8; ++i)
          for (int j = 0; j < 8; ++j)
          {
            double const s = std::sqrt((double)(Kq[i][i] * Kq[j][j]));
            fx[0] = std::max(fx[0], std::fabs((double)(Kq[i][j] - K[i][j])) / s);
            fx[1] = std::max(fx[1], std::fabs((double)((Mq[i][j] - M[i][j]) / Mq[i][j])));
            // (NaN where the Gram form breaks down)
            double const ek = std::fabs((double)(Kq[i][j] - Kd[i][j])) / s, em = std::fabs((double)((Mq[i][j] - Md[i][j]) / Mq[i][j]));
            fp[0] = ek <= fp[0] ? fp[0] : ek, fp[1] = em <= fp[1] ? fp[1] : em;
          }
      }
      std::printf("%s %g %d %d %.3e %.3e %.3e %.3e\n", names[kind], eps, taken, refused, fx[0], fx[1], fp[0], fp[1]);
    }
}
