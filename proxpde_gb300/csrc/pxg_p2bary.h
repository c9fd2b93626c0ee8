// Affine geometry and the P2 tetrahedron's stiffness in barycentric form, shared by the
// one-thread kernel (pxg_assemble.cu) and the group kernel (pxg_p2group.cu).
#pragma once

#include <type_traits>

#include "pxg_internal.h"

namespace pxg
{
// adjugate and determinant of a 3x3 matrix
__device__ __forceinline__ double adj3(double const (&J)[3][3], double (&A)[3][3])
{
  A[0][0] = J[1][1] * J[2][2] - J[1][2] * J[2][1];
  A[0][1] = J[0][2] * J[2][1] - J[0][1] * J[2][2];
  A[0][2] = J[0][1] * J[1][2] - J[0][2] * J[1][1];
  A[1][0] = J[1][2] * J[2][0] - J[1][0] * J[2][2];
  A[1][1] = J[0][0] * J[2][2] - J[0][2] * J[2][0];
  A[1][2] = J[0][2] * J[1][0] - J[0][0] * J[1][2];
  A[2][0] = J[1][0] * J[2][1] - J[1][1] * J[2][0];
  A[2][1] = J[0][1] * J[2][0] - J[0][0] * J[2][1];
  A[2][2] = J[0][0] * J[1][1] - J[0][1] * J[1][0];
  return J[0][0] * A[0][0] + J[0][1] * A[1][0] + J[0][2] * A[2][0];
}

// G = s * A A^T (symmetric, packed 00 11 22 01 02 12)
__device__ __forceinline__ void gram(double const (&A)[3][3], double s, double * G)
{
  G[0] = s * (A[0][0] * A[0][0] + A[0][1] * A[0][1] + A[0][2] * A[0][2]);
  G[1] = s * (A[1][0] * A[1][0] + A[1][1] * A[1][1] + A[1][2] * A[1][2]);
  G[2] = s * (A[2][0] * A[2][0] + A[2][1] * A[2][1] + A[2][2] * A[2][2]);
  G[3] = s * (A[0][0] * A[1][0] + A[0][1] * A[1][1] + A[0][2] * A[1][2]);
  G[4] = s * (A[0][0] * A[2][0] + A[0][1] * A[2][1] + A[0][2] * A[2][2]);
  G[5] = s * (A[1][0] * A[2][0] + A[1][1] * A[2][1] + A[1][2] * A[2][2]);
}

// P2 in barycentric form.  With lambda_0 = 1 - x - y - z, lambda_1..3 = x, y, z, the
// vertex and edge functions are phi_i = lambda_i (2 lambda_i - 1) and
// phi_(ab) = 4 lambda_a lambda_b, whose gradients are linear in the lambdas, so with
// s_kl = k |T| grad lambda_k . grad lambda_l and the exact moments
// (1/|T|) int lambda_k lambda_l = (1 + delta_kl) / 20 the stiffness entries are short
// integer combinations of s' = s / 5:
//   vertex-vertex        K_ii = 3 s'_ii,  K_ij = -s'_ij
//   vertex i, edge (ab)  i = a: 3 s'_ib - s'_ii;  i not in (ab): -(s'_ia + s'_ib)
//   edge-edge            the same edge: 8 (s'_aa + s'_bb + s'_ab); sharing vertex v with
//                        other ends p, q: 4 (s'_vv + s'_vq + s'_pv + 2 s'_pq); disjoint
//                        (ab), (cd): 4 (s'_ac + s'_ad + s'_bc + s'_bd)
// The gradients of the lambdas sum to zero, so every row of s sums to zero and so does
// all of s.  With E_ab = s'_aa + s'_bb + s'_ab and r the vertex outside v, p, q the
// edge-edge entries become 8 E_ab, 4 (2 s'_pq - s'_vr) (six distinct values over the
// twelve pairs: the pairs sharing r with the same p, q give the same) and
// -4 (E_ab + s'_ab): 36 FP64 operations for the 21 entries instead of 78.
// The reference's 11-point rule integrates these degree-2 integrands exactly, so the
// values agree with its per-quadrature-point sums to round-off (64 FP64 operations per
// element for the 55 entries, instead of 177 for the reference-tensor products without
// their zero terms).
// exact negation: the sign bit flipped on the integer pipe
__device__ __forceinline__ double negx(double x)
{
  return __hiloint2double(__double2hiint(x) ^ (int)0x80000000, __double2loint(x));
}
template <int I, int J>
__device__ __forceinline__ double p2Stiff(double const (&s)[4][4], double const (&E)[6])
{
  if constexpr (J < 4)
    return I == J ? 3.0 * s[I][I] : negx(s[I][J]);
  else
  {
    constexpr int c = p2EdgeEnd(J, 0), d = p2EdgeEnd(J, 1);
    if constexpr (I < 4)
    {
      if constexpr (I == c)
        return fma(3.0, s[I][d], -s[I][I]);
      else if constexpr (I == d)
        return fma(3.0, s[I][c], -s[I][I]);
      else
        return -s[I][c] - s[I][d];
    }
    else
    {
      constexpr int a = p2EdgeEnd(I, 0), b = p2EdgeEnd(I, 1);
      if constexpr (I == J)
        return 8.0 * E[I - 4];
      else if constexpr (a == c || a == d || b == c || b == d)
      {
        constexpr int v = (a == c || a == d) ? a : b, p = v == a ? b : a, q = c == v ? d : c;
        constexpr int r = 6 - v - p - q;
        return 4.0 * fma(2.0, s[p < q ? p : q][p < q ? q : p], -s[v < r ? v : r][v < r ? r : v]);
      }
      else
        return -4.0 * (E[I - 4] + s[a][b]);
    }
  }
}
// a representative entry of each P2 mass class
__host__ __device__ constexpr int p2MassRepI(int c) { return c < 4 ? 0 : 4; }
__host__ __device__ constexpr int p2MassRepJ(int c)
{
  return c == 0 ? 0 : c == 1 ? 1 : c == 2 ? 4 : c == 3 ? 5 : c == 4 ? 4 : c == 5 ? 5 : 9;
}
// f(I, J) for the 55 pairs I <= J of the P2 element, as compile-time constants
template <int I, int J, class F>
__device__ __forceinline__ void p2ForPairs(F && f)
{
  f(std::integral_constant<int, I>{}, std::integral_constant<int, J>{});
  if constexpr (J + 1 < 10)
    p2ForPairs<I, J + 1>(f);
  else if constexpr (I + 1 < 10)
    p2ForPairs<I + 1, I + 1>(f);
}

} // namespace pxg
