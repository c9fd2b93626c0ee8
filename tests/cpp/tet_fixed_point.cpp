// Host accuracy of the tetrahedron geometry in fixed point (csrc/pxg_tetfx.h) against 128-bit
// arithmetic, over shapes from regular to strongly sheared, thin and flat ones.  Prints one line
// per shape: name, elements taken, refused, largest errors of |det J|, of the Gram entries (the
// diagonal ones of themselves, the mixed ones of the geometric mean of the two diagonal ones), and
// those of the plain FP64 formulas on the same elements.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <random>

#include "pxg_tetfx.h"

typedef __float128 Quad;

template <class T>
static void plain(double const (&J)[3][3], T k, T (&G)[6], T & det)
{
  T C[3][3];
  for (int a = 0; a < 3; ++a)
    for (int r = 0; r < 3; ++r)
    {
      int const b = (a + 1) % 3, c = (a + 2) % 3, s = (r + 1) % 3, t = (r + 2) % 3;
      C[a][r] = (T)J[s][b] * J[t][c] - (T)J[t][b] * J[s][c];
    }
  det = 0;
  for (int r = 0; r < 3; ++r)
    det += J[r][0] * C[0][r];
  det = det < 0 ? -det : det;
  int const A[6] = {0, 1, 2, 0, 0, 1}, B[6] = {0, 1, 2, 1, 2, 2};
  for (int i = 0; i < 6; ++i)
  {
    T s = 0;
    for (int r = 0; r < 3; ++r)
      s += C[A[i]][r] * C[B[i]][r];
    G[i] = k * s / det;
  }
}

static void error(Quad const (&R)[6], Quad rd, double const (&G)[6], double d, double (&worst)[2])
{
  int const A[6] = {0, 1, 2, 0, 0, 1}, B[6] = {0, 1, 2, 1, 2, 2};
  worst[0] = std::max(worst[0], std::fabs((double)((rd - d) / rd)));
  for (int i = 0; i < 6; ++i)
    worst[1] = std::max(worst[1], std::fabs((double)(R[i] - G[i])) / std::sqrt((double)(R[A[i]] * R[B[i]])));
}

int main()
{
  using namespace pxg;
  std::mt19937_64 rng(5);
  auto U = [&] { return (double)(rng() >> 11) * 0x1p-53; };
  char const * const names[] = {"kuhn", "random", "shear", "thin", "short", "face", "flat", "scaled"};
  double const shapes[] = {1., 0.1, 1e-2, 1e-4};
  for (int kind = 0; kind < 8; ++kind)
    for (double eps : shapes)
    {
      if (kind < 2 && eps < 1.)
        continue;
      int taken = 0, refused = 0;
      double fx[2] = {0., 0.}, fp[2] = {0., 0.};
      for (int it = 0; it < (kind < 2 ? 40000 : 4000); ++it)
      {
        double J[3][3] = {}; // [coordinate][edge]
        for (int r = 0; r < 3; ++r)
          for (int k = 0; k < 3; ++k)
            J[r][k] = kind == 0 ? (r <= k ? 1. : 0.) + 0.4 * (U() - U()) : (kind == 1 || kind > 3 ? U() - 0.5 : 0.);
        if (kind == 2 || kind == 3)
        {
          J[0][0] = 0.5 + U(), J[1][1] = 0.5 + U(), J[2][2] = 0.5 + U(), J[0][2] = U() - 0.5, J[1][2] = U() - 0.5;
          if (kind == 2)
            J[0][1] = 0.5 + U(), J[1][1] *= eps;
          else
            J[2][2] *= eps;
        }
        double scale = 1.;
        for (int r = 0; r < 3; ++r)
        {
          if (kind == 4)
            J[r][1] *= eps;
          if (kind == 5)
            J[r][1] = 0.7 * J[r][0] + eps * J[r][1];
          if (kind == 6)
            J[r][2] = 0.3 * J[r][0] + 0.7 * J[r][1] + eps * J[r][2];
          if (kind == 7) // sizes far from one
            scale = std::pow(eps, 15.);
        }
        for (auto & row : J)
          for (double & x : row)
            x *= scale;
        double const k = std::exp(4. * (U() - 0.5));
        int64_t km;
        int ke;
        fx::decompose(k, km, ke);
        double G[6], d, Gd[6], dd;
        if (!tetx::tetGram(J, true, km, ke, G, d))
        {
          ++refused;
          continue;
        }
        ++taken;
        Quad R[6], rd;
        plain<Quad>(J, k, R, rd);
        plain<double>(J, k, Gd, dd);
        error(R, rd, G, d, fx);
        error(R, rd, Gd, dd, fp);
      }
      printf("%s %g %d %d %.3e %.3e %.3e %.3e\n", names[kind], eps, taken, refused, fx[0], fx[1], fp[0], fp[1]);
    }
}
