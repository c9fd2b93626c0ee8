// P2 tetrahedra with the warp-group scatter (pxg_group.cu), a block of two warps per group of 32
// elements.  Warp 0 forms the elements' geometry in FP64, one element per lane, and their entries
// in barycentric form (pxg_p2bary.h), or both warps those by the rule's tensors, while warp 1
// copies the group's contribution codes to shared memory, where the entries go too; then both sum
// the group's distinct positions and add each sum once.  Shared memory (22.3 KB per group) limits
// an SM to ten groups: with one warp per group its ten warps left the map's loads and the
// additions' latency exposed (13^3 x 6, less than one group per SM sub-partition: 45 us).
// Loads that need the points (a function but the sine, a DOF field) are warp 1's too where there
// are no conditions (K + M with the Poisson right hand side at 6^3, 30^3 and 64^3 x 6: 51, 339 and
// 2,865 us; in a launch of their own 57, 391 and 3,200), and a launch of their own elsewhere (with
// conditions 85, 519 and 4,450 us, together 88, 643 and 7,147).
// Dirichlet conditions: a mask per element leaves its constrained pairs out of the sums, and
// its lane adds the constrained diagonals and the free rows' lifts (builder.hpp:76-124).
#include <vector>

#include "pxg_internal.h"
#include "pxg_p2bary.h"

namespace pxg
{
namespace
{
// the rule: for |det J| = 1 the mass values of the seven classes and of all 55 pairs and sum_q
// w_q phi_i(q); the points, weights and basis values; the reference tensors of the pairs (xx yy zz
// xy xz yz, the mixed ones summed over both orders)
struct P2Rule
{
  double mass7[7], mass[kP2Pairs], integral[10];
  double xi[11][3], w[11], phi[11][10];
  double T[6][kP2Pairs];
};
__constant__ P2Rule cR;

struct GroupShared
{
  double val[kP2GroupValues * 32];
  uint4 item[kP2GroupItems / 8];
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

// whether the gradient of P2 function i has a component along reference direction d
__host__ __device__ constexpr bool hasDir(int i, int d)
{
  return i < 4 ? (i == 0 || i == d + 1)
               : p2EdgeEnd(i, 0) == 0 || p2EdgeEnd(i, 1) == 0 || p2EdgeEnd(i, 0) == d + 1 || p2EdgeEnd(i, 1) == d + 1;
}
// entry (I, J) of the stiffness by the rule's tensor, without the 129 terms of 330 that are zero
template <int I, int J>
__device__ __forceinline__ double tensorEntry(double const (&G)[6])
{
  constexpr int A[6] = {0, 1, 2, 0, 0, 1}, B[6] = {0, 1, 2, 1, 2, 2};
  double k = 0.;
#pragma unroll
  for (int c = 0; c < 6; ++c)
    if ((hasDir(I, A[c]) && hasDir(J, B[c])) || (hasDir(I, B[c]) && hasDir(J, A[c])))
      k = fma(cR.T[c][p2UpperIdx(I, J)], G[c], k);
  return k;
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
        x[r] = X[0][r] + (J[r][0] * cR.xi[q][0] + J[r][1] * cR.xi[q][1] + J[r][2] * cR.xi[q][2]);
      rq[q] = (f0 * cR.w[q]) * evalFn(a.fn, 1.0, x[0], x[1], x[2]);
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
        s = fma(cR.phi[q][n], loc[n], s);
      rq[q] = (f0 * cR.w[q]) * s;
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
      fe = fma(cR.phi[q][i], rq[q], fe);
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

// PLAIN: the first operator's stiffness and the second's mass, no Dirichlet conditions, in the
// barycentric form and with one mass value per class of pairs.  The others by the rule's own
// tensors: its points and weights have 13 to 16 digits, so that they differ by 2e-15 from the exact
// moments of the barycentric form (the mass by 8e-16 within a class).
// LOAD (PLAIN only): with a load that needs the points.
template <bool PLAIN, bool LOAD>
__global__ void __launch_bounds__(64, PLAIN ? 10 : 7) kAssembleP2Group(AsmArgs const __grid_constant__ a)
{
  __shared__ GroupShared sh;
  __shared__ unsigned long long conMask[32]; // not PLAIN: without it ten groups fit an SM
  int const lane = threadIdx.x & 31;
  bool const first = threadIdx.x < 32;
  int64_t const g = blockIdx.x, e = g * 32 + lane;
  int const W = (int)min((int64_t)32, a.nelem - g * 32); // elements of the group
  bool const needK = PLAIN || a.fold.needK, needM = PLAIN || a.fold.needM;
  // value v of lane l at v * 32 + (l ^ (v & 15)): the flush reads, in one instruction,
  // values of the same few elements (lanes) for different entries, which this swizzle
  // spreads over the banks
  auto at = [&](uint32_t v, uint32_t l) -> double & { return sh.val[v * 32 + (l ^ (v & 15u))]; };
  // not PLAIN: the lanes' mass factors are value 55, and cR.mass for the flush's scattered reads follows
  double * const mass = sh.val + 56 * 32;
  static_assert(56 * 32 + kP2Pairs <= kP2GroupValues * 32, "mass values in the place of the classes'");
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
      // lengths beyond 2^+-200, whose cofactors' squares leave the range, in units of their size
      int size = 0;
#pragma unroll
      for (int k = 0; k < 9; ++k)
        size = max(size, __double2hiint(J[k / 3][k % 3]) & 0x7fffffff);
      size = (size >> 20) - 1023;
      bool const scaled = abs(size) > 200 && abs(size) < 1000;
      if (scaled)
#pragma unroll
        for (int k = 0; k < 9; ++k)
          J[k / 3][k % 3] = ldexp(J[k / 3][k % 3], -size);
      double A[3][3];
      adet = fabs(adj3(J, A));
      // 1/|det J|: hardware estimate and one third-order Newton step (y (1 + t + t^2),
      // t = 1 - x y), instead of a full-precision division with its special cases
      double ra;
      asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(ra) : "d"(adet));
      double const t = fma(-adet, ra, 1.0);
      ra = fma(ra, fma(t, t, t), ra);
      // the Gram matrix of the cofactors times k / |det J|; PLAIN: over 30, s'_(a+1)(b+1) = G_ab
      double G[6];
      gram(A, PLAIN ? ks * ra * (1.0 / 30.0) : ks * ra, G);
      if (scaled)
      {
        adet = ldexp(adet, 3 * size);
#pragma unroll
        for (int k = 0; k < 6; ++k)
          G[k] = ldexp(G[k], size);
      }
      if (!PLAIN && needK)
#pragma unroll
        for (int k = 0; k < 6; ++k)
          at(k, lane) = G[k];
      if (PLAIN)
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
        if (!PLAIN)
          at(55, lane) = am;
        else
#pragma unroll
          for (int c7 = 0; c7 < 7; ++c7)
            at(55 + c7, lane) = am * cR.mass7[c7];
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
      conMask[lane] = m;
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
    if (!PLAIN && needM)
      for (int k = lane; k < kP2Pairs; k += 32)
        mass[k] = cR.mass[k];
    if (LOAD && lane < W)
    {
      pdlWait(); // its writes start here
      elementLoad(a, e);
    }
  }
  if (!PLAIN && needK)
  {
    // the tensors' 201 products are dealt to the two warps (13^3 x 6 with conditions and the sine
    // load: 65.6 us, by the first alone 67.6; K alone at 6^3 x 6 23.5 and 27.3)
    __syncthreads();
    double G[6];
#pragma unroll
    for (int k = 0; k < 6; ++k)
      G[k] = at(k, lane);
    __syncthreads();
    auto half = [&](auto odd) {
      p2ForPairs<0, 0>([&](auto I, auto Jj) {
        constexpr int i = decltype(I)::value, j = decltype(Jj)::value;
        if constexpr ((p2UpperIdx(i, j) & 1) == decltype(odd)::value)
          at(p2UpperIdx(i, j), lane) = tensorEntry<i, j>(G);
      });
    };
    if (first)
      half(std::integral_constant<int, 0>{});
    else
      half(std::integral_constant<int, 1>{});
  }
  __syncthreads();
  pdlWait(); // the writes start here
  bool bc = false;
  if constexpr (!PLAIN)
    bc = a.fold.bc && a.bcMask && __any_sync(0xffffffffu, conMask[lane] != 0ull);
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
        bool const c = bc && ((conMask[l] >> v) & 1ull);
        double ka = needK && !(c && a.fold.bcK) ? at(v, l) : 0.;
        double const ma = needM && !(c && a.fold.bcM) ? at(55, l) * mass[v] : 0.;
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
            v = fma(at(55, lane), cR.mass[p2UpperIdx(i, j)], v);
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
  if (!LOAD && a.rkind) // a constant load
  {
    double const f = a.rc * adet;
#pragma unroll
    for (int i = 0; i < 10; ++i)
      if (!(a.rbc && ((cons >> i) & 1u)))
        red(a.b + dof[i], f * cR.integral[i]);
  }
}
} // namespace

pxg_status initP2Group(pxg_ctx * c)
{
  std::vector<double> xi, w;
  hostRule(P2TET, xi, w);
  P2Rule R{};
  for (size_t q = 0; q < w.size(); ++q)
  {
    double dphi[30], * const phi = R.phi[q];
    hostShape(P2TET, &xi[3 * q], phi, dphi);
    R.w[q] = w[q];
    for (int d = 0; d < 3; ++d)
      R.xi[q][d] = xi[3 * q + d];
    for (int i = 0; i < 10; ++i)
    {
      R.integral[i] += w[q] * phi[i];
      for (int j = i; j < 10; ++j)
      {
        int const u = p2UpperIdx(i, j);
        double const *gi = dphi + 3 * i, *gj = dphi + 3 * j;
        R.mass[u] += w[q] * phi[i] * phi[j];
        for (int d = 0; d < 3; ++d)
          R.T[d][u] += w[q] * gi[d] * gj[d];
        R.T[3][u] += w[q] * (gi[0] * gj[1] + gi[1] * gj[0]);
        R.T[4][u] += w[q] * (gi[0] * gj[2] + gi[2] * gj[0]);
        R.T[5][u] += w[q] * (gi[1] * gj[2] + gi[2] * gj[1]);
      }
    }
  }
  for (int k = 0; k < 7; ++k)
    R.mass7[k] = R.mass[p2UpperIdx(p2MassRepI(k), p2MassRepJ(k))];
  PXG_CUDA(c, cudaMemcpyToSymbol(cR, &R, sizeof(R)));
  return PXG_OK;
}

void launchAssembleP2Group(AsmArgs const & a, cudaStream_t s)
{
  unsigned const blocks = (unsigned)((a.nelem + 31) / 32);
  if (blocks == 0)
    return;
  // the usual pair without Dirichlet conditions (a load that needs the points has its own) has an
  // instance of its own: the others' branches cost its loops
  bool const load = pointLoad(a);
  bool const plain = a.fold.needK && a.fold.needM && !a.fold.same && a.op[0].stiff &&
                     !(a.bcMask && (a.fold.bc || (a.rkind && a.rbc && !load)));
  if (plain)
  {
    launchElemKernel(load ? kAssembleP2Group<true, true> : kAssembleP2Group<true, false>, blocks, 64, 0, s, a);
    return;
  }
  AsmArgs l = a;
  if (load)
    l.rkind = 0;
  launchElemKernel(kAssembleP2Group<false, false>, blocks, 64, 0, s, l);
  if (load)
  {
    l = a;
    l.op[0].on = l.op[1].on = 0;
    l.pdl = 0;
    launchP2PointLoad(l, s);
  }
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
