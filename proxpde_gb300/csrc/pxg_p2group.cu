// P2 tetrahedra with the warp-group scatter (pxg_group.cu), a block of two warps per group of 32
// elements.  Warp 0 forms the elements' values, one element per lane, from the geometry in fixed
// point (pxg_tetfx.h) and in barycentric form (pxg_p2bary.h), and leaves them in shared memory, while warp 1 copies the
// group's contribution codes there; then both sum the group's distinct positions and add
// each sum once.  Shared memory (22.5 KB per group) limits an SM to ten groups: with one warp
// per group its ten warps left the map's loads and the additions' latency exposed
// (13^3 x 6, less than one group per SM sub-partition: 45 us).
// Loads that need the points (a function but the sine, a DOF field) are warp 1's too, beside the
// values (K + M with the Poisson right hand side: 57 us at 6^3 x 6 and 0.40 ms at 30^3 x 6; by the
// one-thread kernel in a second launch 80 us and 0.49 ms), or a kernel's of their own without
// operators (19 us and 0.095 ms a DOF field at 13^3 x 6 and 30^3 x 6, 37 and 0.199 by the other).
// Dirichlet conditions: a mask per element leaves its constrained pairs out of the sums, and
// its lane adds the constrained diagonals and the free rows' lifts (builder.hpp:76-124).
#include <vector>

#include "pxg_internal.h"
#include "pxg_p2bary.h"
#include "pxg_tetfx.h"

namespace pxg
{
namespace
{
// mass values of the seven classes and sum_q w_q phi_i(q), for |det J| = 1
__constant__ double cMass[7];
__constant__ double cInt[10];
// the rule's points, weights and basis values
__constant__ double cXi[11][3], cW[11], cPhi[11][10];

struct GroupShared
{
  double val[kP2GroupValues * 32];
  uint4 item[kP2GroupItems / 8];
  unsigned long long cons[32];
};

__device__ __forceinline__ void red(double * p, double v) { atomicAdd(p, v); }

// s (4 x 4, zero row sums) and E_ab = s_aa + s_bb + s_ab of the six edges from the Gram
// entries of vertices 1..3
__device__ __forceinline__ void gramRows(double const (&G)[6], double (&s)[4][4], double (&E)[6])
{
  s[1][1] = G[0], s[2][2] = G[1], s[3][3] = G[2];
  s[1][2] = s[2][1] = G[3];
  s[1][3] = s[3][1] = G[4];
  s[2][3] = s[3][2] = G[5];
  double const c1 = G[0] + (G[3] + G[4]), c2 = G[3] + (G[1] + G[5]), c3 = G[4] + (G[5] + G[2]);
  s[0][1] = s[1][0] = -c1;
  s[0][2] = s[2][0] = -c2;
  s[0][3] = s[3][0] = -c3;
  s[0][0] = c1 + (c2 + c3);
#pragma unroll
  for (int n = 0; n < 6; ++n)
    E[n] = (s[p2EdgeEnd(4 + n, 0)][p2EdgeEnd(4 + n, 0)] + s[p2EdgeEnd(4 + n, 1)][p2EdgeEnd(4 + n, 1)]) +
           s[p2EdgeEnd(4 + n, 0)][p2EdgeEnd(4 + n, 1)];
}

// whether a load is one that the element's own points are needed for (the sine has a kernel of its
// own, pxg_tetload.cu)
__host__ __device__ __forceinline__ bool pointLoad(AsmArgs const & a)
{
  return a.rkind == 2 || (a.rkind == 1 && a.fn != PXG_FN_CONST);
}
// such a load of element e in FP64: a function or a DOF field at the points of the rule.  Out of
// line, its registers are not the other calls'.
__device__ __noinline__ void elementLoad(AsmArgs const & a, int64_t e)
{
  double X[4][3], J[3][3], A[3][3];
  uint4 const c = reinterpret_cast<uint4 const *>(a.conn)[e];
  uint32_t const v[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
  for (int n = 0; n < 4; ++n)
#pragma unroll
    for (int d = 0; d < 3; ++d)
      X[n][d] = a.xyz[3 * (int64_t)v[n] + d];
  uint32_t dof[10];
#pragma unroll
  for (int i = 0; i < 10; ++i)
    dof[i] = a.emap[e * 10 + i];
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int k = 0; k < 3; ++k)
      J[r][k] = X[k + 1][r] - X[0][r];
  double const f0 = a.rc * fabs(adj3(J, A));
  double rq[11];
  if (a.rkind == 1)
  {
#pragma unroll
    for (int q = 0; q < 11; ++q)
    {
      double x[3];
#pragma unroll
      for (int r = 0; r < 3; ++r)
        x[r] = X[0][r] + (J[r][0] * cXi[q][0] + J[r][1] * cXi[q][1] + J[r][2] * cXi[q][2]);
      rq[q] = (f0 * cW[q]) * evalFn(a.fn, 1.0, x[0], x[1], x[2]);
    }
  }
  else
  {
    double loc[10];
#pragma unroll
    for (int n = 0; n < 10; ++n)
      loc[n] = a.field[dof[n]];
#pragma unroll
    for (int q = 0; q < 11; ++q)
    {
      double s = 0.;
#pragma unroll
      for (int n = 0; n < 10; ++n)
        s = fma(cPhi[q][n], loc[n], s);
      rq[q] = (f0 * cW[q]) * s;
    }
  }
#pragma unroll
  for (int i = 0; i < 10; ++i)
  {
    if (a.rbc && a.bcMask && a.bcMask[dof[i]])
      continue;
    double fe = 0.;
#pragma unroll
    for (int q = 0; q < 11; ++q)
      fe = fma(cPhi[q][i], rq[q], fe);
    red(a.b + dof[i], fe);
  }
}

// such a load by itself
__global__ void __launch_bounds__(64) kP2PointLoad(AsmArgs const __grid_constant__ a)
{
  int64_t const i = blockIdx.x * 64ll + threadIdx.x;
  if (i >= a.nelem)
    return;
  pdlWait();
  elementLoad(a, elemOf(a, i));
}

// PLAIN: one operator's stiffness and the other's mass, no Dirichlet conditions
template <bool PLAIN>
__global__ void __launch_bounds__(64, PLAIN ? 10 : 7) kAssembleP2Group(AsmArgs const __grid_constant__ a)
{
  __shared__ GroupShared sh;
  int const lane = threadIdx.x & 31;
  bool const first = threadIdx.x < 32;
  int64_t const g = blockIdx.x, e = g * 32 + lane;
  int const W = (int)min((int64_t)32, a.nelem - g * 32); // elements of the group
  bool const needK = PLAIN || a.fold.needK, needM = PLAIN || a.fold.needM;
  // value v of lane l at v * 32 + (l ^ (v & 15)): the flush reads, in one instruction,
  // values of the same few elements (lanes) for different entries, which this swizzle
  // spreads over the banks
  auto at = [&](uint32_t v, uint32_t l) -> double & { return sh.val[v * 32 + (l ^ (v & 15u))]; };
  int const nItems = W * 100;
  int32_t const dBeg = a.grpOff[g], dEnd = a.grpOff[g + 1];
  // the map of the next batch of positions is loaded while this one is summed and reduced
  constexpr int U = 4;
  int32_t npos[U];
  int nb0[U], nb1[U];
  auto loadBatch = [&](int32_t d0) {
#pragma unroll
    for (int u = 0; u < U; ++u)
    {
      int32_t const d = d0 + u * 64 + (int)threadIdx.x;
      npos[u] = d < dEnd ? a.grpPos[d] : 0;
      nb0[u] = d < dEnd ? a.grpBeg[d] : 0;
      nb1[u] = d + 1 < dEnd ? a.grpBeg[d + 1] : nItems;
    }
  };
  uint32_t dof[10];
  uint32_t cons = 0;
  double adet = 0.;
  double hv[10];     // Dirichlet values and diagonal positions of the constrained nodes
  int32_t pii[10];
  if (first)
  {
    if (lane < W)
    {
      double X[4][3];
      uint4 const c = reinterpret_cast<uint4 const *>(a.conn)[e];
      uint32_t const v[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
      for (int n = 0; n < 4; ++n)
#pragma unroll
        for (int d = 0; d < 3; ++d)
          X[n][d] = a.xyz[3 * (int64_t)v[n] + d];
      double const kfac = a.fold.coef ? a.kE[e] : 1.0;
      if (!PLAIN || a.b)
      {
#pragma unroll
        for (int i = 0; i < 10; ++i)
          dof[i] = a.emap[e * 10 + i];
      }
      if (!PLAIN && a.bcMask)
      {
#pragma unroll
        for (int i = 0; i < 10; ++i)
          if (a.bcMask[dof[i]])
            cons |= 1u << i;
        if (a.fold.bc && cons)
        {
#pragma unroll
          for (int i = 0; i < 10; ++i)
          {
            bool const c = (cons >> i) & 1u;
            hv[i] = c ? a.bcVal[dof[i]] : 0.;
            pii[i] = c ? a.rowPtr[dof[i]] + a.rank[e * 100 + i * 11] : 0;
          }
        }
      }
      double J[3][3];
#pragma unroll
      for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int k = 0; k < 3; ++k)
          J[r][k] = X[k + 1][r] - X[0][r];
      double const ks = a.fold.coefK ? a.fold.sK * kfac : a.fold.sK;
      // s'_(a+1)(b+1) = G_ab, the Gram matrix of the cofactors times k / (30 |det J|), in fixed
      // point (16 conversions for about 75 FP64 operations): km carries 16 / 30
      double G[6];
      int64_t km;
      int ke;
      bool const okK = fx::coefParts(ks, km, ke);
      km = (int64_t)((uint64_t)fx::mulc(fx::cst(0x4444444444444444ll), km) << 1);
      if (!tetx::tetGram(J, okK, km, ke - 4, G, adet))
      {
        double A[3][3];
        adet = fabs(adj3(J, A));
        // 1/|det J|: hardware estimate and one third-order Newton step (y (1 + t + t^2),
        // t = 1 - x y), instead of a full-precision division with its special cases
        double ra;
        asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(ra) : "d"(adet));
        double const t = fma(-adet, ra, 1.0);
        ra = fma(ra, fma(t, t, t), ra);
        gram(A, ks * ra * (1.0 / 30.0), G);
      }
      if (needK)
      {
        double s[4][4], E[6];
        gramRows(G, s, E);
        p2ForPairs<0, 0>([&](auto I, auto Jj) {
          constexpr int i = decltype(I)::value, j = decltype(Jj)::value;
          at(p2UpperIdx(i, j), lane) = p2Stiff<i, j>(s, E);
        });
      }
      if (needM)
      {
        double const am = (a.fold.coefM ? a.fold.sM * kfac : a.fold.sM) * adet;
#pragma unroll
        for (int c7 = 0; c7 < 7; ++c7)
          at(55 + c7, lane) = am * cMass[c7];
      }
    }
    if (!PLAIN)
    {
      unsigned long long m = 0;
      if (lane < W && a.fold.bc && cons)
        p2ForPairs<0, 0>([&](auto I, auto Jj) {
          constexpr int i = decltype(I)::value, j = decltype(Jj)::value;
          if ((cons & (1u << i)) || (cons & (1u << j)))
            m |= 1ull << p2UpperIdx(i, j);
        });
      sh.cons[lane] = m;
    }
    loadBatch(dBeg);
  }
  else
  {
    loadBatch(dBeg);
    // the group's codes, 16 bytes (8 codes) per load, seven loads in flight; the map pads
    // the last group's codes to a multiple of 8
    uint4 const * const gi = reinterpret_cast<uint4 const *>(a.grpItem + g * kP2GroupItems);
    int const n8 = (nItems + 7) / 8;
    for (int k0 = lane; k0 < n8; k0 += 7 * 32)
    {
      uint4 t[7];
#pragma unroll
      for (int r = 0; r < 7; ++r)
        if (k0 + 32 * r < n8)
          t[r] = gi[k0 + 32 * r];
#pragma unroll
      for (int r = 0; r < 7; ++r)
        if (k0 + 32 * r < n8)
          sh.item[k0 + 32 * r] = t[r];
    }
    if (!PLAIN && pointLoad(a) && lane < W)
    {
      pdlWait(); // its writes start here
      elementLoad(a, e);
    }
  }
  __syncthreads();
  pdlWait(); // the writes start here
  bool const bc = !PLAIN && a.fold.bc && a.bcMask && __any_sync(0xffffffffu, sh.cons[lane] != 0ull);
  uint16_t const * const si = reinterpret_cast<uint16_t const *>(sh.item);
  for (int32_t d0 = dBeg; d0 < dEnd; d0 += U * 64)
  {
    int32_t pos[U];
    int b0[U], b1[U];
#pragma unroll
    for (int u = 0; u < U; ++u)
      pos[u] = npos[u], b0[u] = nb0[u], b1[u] = nb1[u];
    loadBatch(d0 + U * 64);
#pragma unroll
    for (int u = 0; u < U; ++u)
    {
      if (d0 + u * 64 + (int)threadIdx.x >= dEnd)
        break;
      // the position's contributions in element order.  Few contributions: one reduction
      // each (the L2 atomic unit has room, the FP64 pipe has not); more: summed here, no
      // addition for the first
      if (PLAIN)
      {
        if (b1[u] - b0[u] <= a.grpRedMax)
        {
          for (int k = b0[u]; k < b1[u]; ++k)
          {
            uint32_t const code = si[k];
            red(a.fold.K + pos[u], at((code >> 5) & 63u, code & 31u));
            red(a.fold.M + pos[u], at(55 + (code >> 11), code & 31u));
          }
          continue;
        }
        uint32_t code = si[b0[u]];
        double kk = at((code >> 5) & 63u, code & 31u);
        double mm = at(55 + (code >> 11), code & 31u);
        for (int k = b0[u] + 1; k < b1[u]; ++k)
        {
          code = si[k];
          kk += at((code >> 5) & 63u, code & 31u);
          mm += at(55 + (code >> 11), code & 31u);
        }
        red(a.fold.K + pos[u], kk);
        red(a.fold.M + pos[u], mm);
        continue;
      }
      bool const each = b1[u] - b0[u] <= a.grpRedMax;
      double kk = 0., mm = 0.;
      for (int k = b0[u]; k < b1[u]; ++k)
      {
        uint32_t const code = si[k], v = (code >> 5) & 63u, l = code & 31u;
        // constrained pairs are left out of the matrices of operators with BCs
        bool const c = bc && ((sh.cons[l] >> v) & 1ull);
        double ka = needK && !(c && a.fold.bcK) ? at(v, l) : 0.;
        double const ma = needM && !(c && a.fold.bcM) ? at(55 + (code >> 11), l) : 0.;
        if (a.fold.same)
          ka += ma;
        if (each)
        {
          if (needK)
            red(a.fold.K + pos[u], ka);
          if (needM && !a.fold.same)
            red(a.fold.M + pos[u], ma);
        }
        else if (k == b0[u])
          kk = ka, mm = ma;
        else
        {
          if (needK)
            kk += ka;
          if (needM && !a.fold.same)
            mm += ma;
        }
      }
      if (!each)
      {
        if (needK)
          red(a.fold.K + pos[u], kk);
        if (needM && !a.fold.same)
          red(a.fold.M + pos[u], mm);
      }
    }
  }
  if (!first || lane >= W)
    return;
  if (!PLAIN && a.fold.bc && cons)
  {
    AsmArgs::Fold const & f = a.fold;
    bool lift = false;
#pragma unroll
    for (int i = 0; i < 10; ++i)
    {
      if (!((cons >> i) & 1u))
        continue;
      if (needK && f.bcK)
        red(f.K + pii[i], a.bcDiag);
      if (needM && !f.same && f.bcM)
        red(f.M + pii[i], a.bcDiag);
      if (hv[i] != 0. && a.b)
      {
        lift = true;
        // buildLhs' Dirichlet values, once per operator with BCs
#pragma unroll
        for (int m = 0; m < 2; ++m)
          if (a.op[m].on && a.op[m].bc)
            red(a.b + dof[i], hv[i]);
      }
    }
    if (lift)
    {
      // the free rows' lifts -K_ij h_j
      double z[10];
#pragma unroll
      for (int i = 0; i < 10; ++i)
        z[i] = 0.;
      p2ForPairs<0, 0>([&](auto I, auto Jj) {
        constexpr int i = decltype(I)::value, j = decltype(Jj)::value;
        if constexpr (i != j)
        {
          bool const ci = (cons >> i) & 1u, cj = (cons >> j) & 1u;
          if (ci == cj)
            return;
          double v = needK && f.bcK ? at(p2UpperIdx(i, j), lane) : 0.;
          if (needM && f.bcM)
            v += at(55 + p2MassClass(i, j), lane);
          if (cj)
            z[i] = fma(v, hv[j], z[i]);
          else
            z[j] = fma(v, hv[i], z[j]);
        }
      });
#pragma unroll
      for (int i = 0; i < 10; ++i)
        if (z[i] != 0.)
          red(a.b + dof[i], -z[i]);
    }
  }
  if (a.rkind && (PLAIN || !pointLoad(a))) // a constant load
  {
    double const f = a.rc * adet;
#pragma unroll
    for (int i = 0; i < 10; ++i)
      if (!(a.rbc && ((cons >> i) & 1u)))
        red(a.b + dof[i], f * cInt[i]);
  }
}
} // namespace

pxg_status initP2Group(pxg_ctx * c)
{
  std::vector<double> xi, w;
  hostRule(P2TET, xi, w);
  double M[100] = {}, I[10] = {}, P[110], dphi[30];
  for (size_t q = 0; q < w.size(); ++q)
  {
    double * const phi = P + 10 * q;
    hostShape(P2TET, &xi[3 * q], phi, dphi);
    for (int i = 0; i < 10; ++i)
    {
      I[i] += w[q] * phi[i];
      for (int j = 0; j < 10; ++j)
        M[10 * i + j] += w[q] * phi[i] * phi[j];
    }
  }
  double m7[7];
  for (int k = 0; k < 7; ++k)
    m7[k] = M[10 * p2MassRepI(k) + p2MassRepJ(k)];
  PXG_CUDA(c, cudaMemcpyToSymbol(cMass, m7, sizeof(m7)));
  PXG_CUDA(c, cudaMemcpyToSymbol(cInt, I, sizeof(I)));
  PXG_CUDA(c, cudaMemcpyToSymbol(cXi, xi.data(), sizeof(cXi)));
  PXG_CUDA(c, cudaMemcpyToSymbol(cW, w.data(), sizeof(cW)));
  PXG_CUDA(c, cudaMemcpyToSymbol(cPhi, P, sizeof(P)));
  return PXG_OK;
}

void launchAssembleP2Group(AsmArgs const & a, cudaStream_t s, int)
{
  unsigned const blocks = (unsigned)((a.nelem + 31) / 32);
  if (blocks == 0)
    return;
  // the usual pair without Dirichlet conditions has its own instance: the others' branches
  // cost its loops
  bool const plain = a.fold.needK && a.fold.needM && !a.fold.same &&
                     !(a.bcMask && (a.fold.bc || (a.rkind && a.rbc))) && !pointLoad(a);
  if (plain)
    launchElemKernel(kAssembleP2Group<true>, blocks, 64, 0, s, a);
  else
    launchElemKernel(kAssembleP2Group<false>, blocks, 64, 0, s, a);
}

bool launchP2PointLoad(AsmArgs const & a, cudaStream_t s)
{
  if (a.op[0].on || a.op[1].on || !pointLoad(a))
    return false;
  if (a.nelem > 0)
    launchElemKernel(kP2PointLoad, (unsigned)((a.nelem + 63) / 64), 64, 0, s, a);
  return true;
}
} // namespace pxg
