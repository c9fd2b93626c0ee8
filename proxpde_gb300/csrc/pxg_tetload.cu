// The load sin(pi x) sin(pi y) sin(pi z) on P1 and P2 tetrahedra (AssemblyRhsAnalytic,
// include/assembly_rhs.hpp:34-91, with f at CurFE::qpoint and the Tet4 / Tet11 rule), one
// thread per element in 64-bit fixed point (pxg_tetx.h).  As part of the FP64 element
// kernel it took 33 sines and 330 further FP64 operations per P2 element, 64 cycles each on
// this part: more than the matrices (30^3 x 6, K + M with this load 0.63 ms, without it
// 0.24).  Elements too large for the series are evaluated in FP64.
#include <vector>

#include "pxg_internal.h"
#include "pxg_sinpi.h"
#include "pxg_tetx.h"

namespace pxg
{
namespace
{
using fx::Sp;

// the rule's points and the weights w_q phi_i(q) at F = 62, the weights times 2^shiftOf
struct TetRule
{
  Sp xi[11][3];
  Sp w[10][11];
  double xid[11][3], wd[10][11];
};
__constant__ TetRule cRule[2];
__host__ __device__ constexpr int shiftOf(int t) { return t == P1TET ? 4 : 3; } // sum_q |w_q phi_i| 2^shift below one

template <int T>
__global__ void __launch_bounds__(64) kTetSineLoad(AsmArgs const __grid_constant__ a)
{
  constexpr int N = Elem<T>::N, NQ = Elem<T>::NQ;
  int64_t const i0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i0 >= a.nelem)
    return;
  int64_t const e = elemOf(a, i0);
  TetRule const & R = cRule[T];
  double X[4][3];
  {
    uint4 const c = reinterpret_cast<uint4 const *>(a.conn)[e];
    uint32_t const v[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int r = 0; r < 3; ++r)
        X[n][r] = a.xyz[3 * (int64_t)v[n] + r];
  }
  double D[3][3]; // [r][a]
  int32_t m[3];
#pragma unroll
  for (int r = 0; r < 3; ++r)
  {
    m[r] = 0;
#pragma unroll
    for (int k = 0; k < 3; ++k)
    {
      D[r][k] = X[k + 1][r] - X[0][r];
      m[r] = max(m[r], fx::hi32(fx::doubleBits(D[r][k])) & 0x7fffffff);
    }
  }
  double const adet = fabs(D[0][0] * (D[1][1] * D[2][2] - D[1][2] * D[2][1]) -
                           D[0][1] * (D[1][0] * D[2][2] - D[1][2] * D[2][0]) +
                           D[0][2] * (D[1][0] * D[2][1] - D[1][1] * D[2][0]));
  int sc[3];
  bool ok = q1x::coordScales(m[0], m[1], m[2], sc);
  Sp d[3][3];
  float bm = 0.f;
  int et[3];
#pragma unroll
  for (int r = 0; r < 3; ++r)
  {
    uint32_t t = 0;
#pragma unroll
    for (int k = 0; k < 3; ++k)
    {
      int64_t const x = fx::roundToInt(fx::scaleExp(D[r][k], 62 - sc[r]));
      t = max(t, (uint32_t)abs(fx::hi32(x)) + 1u);
      d[r][k] = fx::split(x);
    }
    // |pi sum xi_a d_a| <= pi 2^(sc - 30) max |d|
    q1x::Bound const b = q1x::makeBound((float)t * 3.1416f, sc[r] - 30);
    et[r] = b.e;
    bm = fmaxf(bm, b.f);
  }
  ok = ok && max(sc[0], max(sc[1], sc[2])) <= q1x::kLoadMaxScale && bm <= q1x::kLoadMaxT;
  uint32_t dof[N];
#pragma unroll
  for (int i = 0; i < N; ++i)
    dof[i] = a.emap[e * N + i];
  uint32_t cons = 0;
  if (a.rbc && a.bcMask)
  {
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (a.bcMask[dof[i]])
        cons |= 1u << i;
  }
  double const f0 = a.rc * adet;
  pdlWait(); // the writes start here
  if (ok)
  {
    // the degree of the warp's elements (uniform control flow)
    int const deg = q1x::seriesDegree(__uint_as_float(__reduce_max_sync(__activemask(), __float_as_uint(bm))));
    auto const xi = [&](int q, int k) { return R.xi[q][k]; };
    int64_t f[3][NQ];
    double S[3], C[3];
#pragma unroll
    for (int r = 0; r < 3; ++r)
      sinCosPiTab(X[0][r], S[r], C[r]);
    int const ex = tetx::factors<NQ>(d, sc, et, deg, S, C, xi, f);
    Sp r[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q)
    {
      int64_t const t = q1x::shl(fx::mul(fx::split(f[0][q]), fx::split(f[1][q])), 2);
      r[q] = fx::split(fx::mul(fx::split(t), fx::split(f[2][q])) >> 1); // F = 59
    }
#pragma unroll
    for (int i = 0; i < N; ++i)
    {
      int64_t b = fx::kHalf, s;
#pragma unroll
      for (int q = 0; q < NQ; ++q)
        b = fx::madw(r[q].l, R.w[i][q].h, fx::madw(r[q].h, R.w[i][q].l, b));
      s = fx::hi32(b);
#pragma unroll
      for (int q = 0; q < NQ; ++q)
        s = fx::madw(r[q].h, R.w[i][q].h, s);
      if (!((cons >> i) & 1u))
        atomicAdd(a.b + dof[i], f0 * fx::toDoubleFlush(s, ex - 57 - shiftOf(T)));
    }
    return;
  }
  double fq[NQ];
#pragma unroll 1
  for (int q = 0; q < NQ; ++q)
  {
    double x[3];
#pragma unroll
    for (int r = 0; r < 3; ++r)
      x[r] = X[0][r] + (D[r][0] * R.xid[q][0] + D[r][1] * R.xid[q][1] + D[r][2] * R.xid[q][2]);
    fq[q] = f0 * (sinPiTab(x[0]) * sinPiTab(x[1]) * sinPiTab(x[2]));
  }
#pragma unroll 1
  for (int i = 0; i < N; ++i)
  {
    if ((cons >> i) & 1u)
      continue;
    double fe = 0.;
    for (int q = 0; q < NQ; ++q)
      fe = fma(R.wd[i][q], fq[q], fe);
    atomicAdd(a.b + a.emap[e * N + i], fe);
  }
}

Sp splitHost(double x)
{
  int64_t const v = (int64_t)(x * 4611686018427387904.0); // |x| < 1
  return fx::split(v);
}
} // namespace

pxg_status initTetLoad(pxg_ctx * c)
{
  std::vector<TetRule> R(2);
  for (int t = 0; t < 2; ++t)
  {
    std::vector<double> xi, w;
    hostRule(t, xi, w);
    int const nq = (int)w.size(), N = numDofs(t);
    std::vector<double> phi(N), dphi(3 * N), sum(N, 0.);
    for (int q = 0; q < nq; ++q)
    {
      hostShape(t, &xi[3 * q], phi.data(), dphi.data());
      for (int k = 0; k < 3; ++k)
        R[t].xi[q][k] = splitHost(xi[3 * q + k]), R[t].xid[q][k] = xi[3 * q + k];
      for (int i = 0; i < N; ++i)
      {
        double const v = w[q] * phi[i];
        R[t].wd[i][q] = v;
        R[t].w[i][q] = splitHost(v * (1 << shiftOf(t)));
        sum[i] += v < 0 ? -v : v;
      }
    }
    for (double s : sum)
      if (s * (1 << shiftOf(t)) >= 1.)
        return fail(c, PXG_ERR_UNSUPPORTED, "tetrahedron load weights");
  }
  PXG_CUDA(c, cudaMemcpyToSymbol(cRule, R.data(), sizeof(TetRule) * 2));
  return PXG_OK;
}

void launchTetSineLoad(int etype, AsmArgs const & a, cudaStream_t s)
{
  if (a.nelem <= 0)
    return;
  unsigned const blocks = (unsigned)((a.nelem + 63) / 64);
  if (etype == P1TET)
    launchElemKernel(kTetSineLoad<P1TET>, blocks, 64, 0, s, a);
  else
    launchElemKernel(kTetSineLoad<P2TET>, blocks, 64, 0, s, a);
}
} // namespace pxg
