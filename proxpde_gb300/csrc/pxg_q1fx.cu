// Q1 hexahedra in 64-bit fixed point (pxg_q1x.h): a block of eight warps computes 32
// elements, lane = element throughout, and deals the steps of an element to its warps:
//  0. warps 0-2 take one coordinate each (differences to vertex 0, Walsh-Hadamard
//     transform, Jacobian columns), warps 3-5 the sine and cosine of the element origin;
//  1. each warp takes one quadrature point: cofactors, determinant, products, the load
//     offset, and after the block-wide scale of the determinants the tensor G and the
//     load value (warps 3-5 first form the sine series' coefficients);
//  2. six warps contract one component of G each to its class tables, one warp the mass
//     table, one the load, which it adds to b;
//  3. the 36 entries from the tables, four or six per warp, to doubles;
//  4. the scatter: eight consecutive lanes add one row of one element, so that the two
//     x neighbours of a row share a 32-byte sector (the L2 unit adds 2.0e11 values/s
//     with one lane per sector, 3.1e11 with two).
// Why so: the whole element in one thread is 12,000 instructions of straight-line code at
// 255 registers, which two warps per scheduler cannot hide and the instruction caches do
// not hold (0.20 instructions per cycle, 2.8 of 10 cycles per instruction waiting for
// code, 3.4 ms at 128^3).  Dealt over warps, each executes a tenth of it, 64 registers
// suffice and 32 warps are resident: 2.16 ms (in FP64, one thread per element, 4.97 ms:
// 1,233 operations at 64 issue cycles a warp).  What is left is latency: the barriers
// between the steps, instruction fetches and the reductions' queue.
// Elements the format refuses (pxg_q1x.h) are computed in FP64 by a thread of their own.
#include "pxg_q1f64.h"
#include "pxg_q1x.h"

namespace pxg
{
namespace
{
using q1x::Sp;

struct Q1Shared
{
  union
  {
    struct
    {
      int64_t col[36][32];     // column a, coordinate r, point p at (a * 3 + r) * 4 + p
      int64_t coef[3][16][32]; // sine series of each coordinate
    };
    int64_t tab[q1x::kTables][32];
  };
  union
  {
    int64_t G[48][32];    // component c at point q: c * 8 + q
    double kval[32][37];  // entries of the stiffness (an odd stride: no bank conflicts)
    int64_t off[3][8][32]; // offsets of the points, before G
  };
  union
  {
    int64_t rq[8][32]; // load values of the points
    double rqd[8][32]; // the same in FP64
    int64_t sm[6][32]; // sine, cosine of pi times the origin: mantissas
  };
  int se[6][32]; // and exponents
  double org[3][32];
  int64_t det[8][32];
  union
  {
    int64_t mtab[32][27]; // the mass table, then as doubles
    double mval[32][27];
    uint32_t psize[8][32];
    int32_t dmax[3][32]; // high word of the largest difference per coordinate
  };
  uint32_t cmax[9][32];
  uint32_t dof[8][32];
  int32_t rp[32][8];
  int32_t ee[3][32];            // exponents of the sine series
  float bound[3][32];           // bounds of its argument, and their exponents
  int32_t et[3][32];
  int32_t el[32];               // exponent of the load values
  uint32_t flags[32]; // bits 0-7 constrained nodes, 8 in the mesh, 9 fixed point holds it
};

// position of the pair (li, lj) of lattice nodes among the 36 entries: the four diagonal
// y/z blocks with three each, then the pairs of blocks with four each
__device__ __forceinline__ int entryIndex(int li, int lj)
{
  int a = li >> 1, b = lj >> 1, ix = li & 1, jx = lj & 1;
  if (a == b)
    return 3 * a + ix + jx;
  if (a > b)
  {
    int const t = a;
    a = b, b = t;
    int const u = ix;
    ix = jx, jx = u;
  }
  return 12 + 4 * (a == 0 ? b - 1 : (a == 1 ? b + 1 : 5)) + 2 * ix + jx;
}
// lattice index (bits x, y, z) of node n
__device__ __forceinline__ int latticeOf(int n) { return (((n >> 1) ^ n) & 1) | (n & 6); }

// one y/z block of entries to doubles
template <int a, int b>
__device__ __forceinline__ void entriesOut(Q1Shared & sh, int l, int eK)
{
  int64_t K[2][2];
  auto const t = [&](int k) { return sh.tab[k][l]; };
  q1x::entryBlock<(a & 1), (a >> 1), (b & 1), (b >> 1)>(t, K);
  constexpr int base = a == b ? 3 * a : 12 + 4 * (a == 0 ? b - 1 : (a == 1 ? b + 1 : 5));
#pragma unroll
  for (int ix = 0; ix < 2; ++ix)
#pragma unroll
    for (int jx = 0; jx < 2; ++jx)
      if (!(a == b && jx < ix))
        sh.kval[l][base + (a == b ? ix + jx : 2 * ix + jx)] = q1x::toDouble(K[ix][jx], eK);
}

// an analytic function at a point, out of line
__device__ __noinline__ double evalPoint(int fn, double x, double y, double z) { return evalFn(fn, 1.0, x, y, z); }
// sum_n phi_n field_n at point q: one axis at a time, l_a = A on the node's side, B on the other
__device__ __noinline__ double fieldPoint(double const * field, Q1Shared const & sh, int l, int q)
{
  double f[8];
#pragma unroll
  for (int k = 0; k < 8; ++k)
    f[k] = field[sh.dof[q1f::node((k ^ q) & 1, ((k ^ q) >> 1) & 1, (k ^ q) >> 2)][l]];
#pragma unroll
  for (int t = 1; t < 8; t *= 2)
#pragma unroll
    for (int k = 0; k < 8; k += 2 * t)
      f[k] = fma(q1f::A, f[k], q1f::B * f[k | t]);
  return f[0];
}

// Dirichlet condensation (builder.hpp:76-124) of entry (i, j) of element el under the
// operator of K (with k) and of M (with m): the diagonal of a constrained DOF, the lift
// -K_ij h_j of a free row
__device__ __forceinline__ void condense(AsmArgs const & a, Q1Shared const & sh, int el, int i, int j, bool k, bool m,
                                         bool ci, int32_t pij, double kv, double mv)
{
  if (i == j)
  {
    if (k)
      atomicAdd(a.fold.K + pij, a.bcDiag);
    if (m)
      atomicAdd(a.fold.M + pij, a.bcDiag);
  }
  else if (!ci && a.b && (k || m))
  {
    double const z = ((k ? kv : 0.) + (m ? mv : 0.)) * a.bcVal[sh.dof[j][el]];
    if (z != 0.)
      atomicAdd(a.b + sh.dof[i][el], -z);
  }
}

// Entry (i, j) of the block's element el for any operators and with the Dirichlet
// condensation (builder.hpp:76-124): the diagonal of a constrained DOF, the lift -K_ij h_j
// of a free row.  kx, mx: its places in the stiffness and mass values.
__device__ __noinline__ void scatterGeneral(AsmArgs const & a, Q1Shared const & sh, int el, int i, int j, int kx, int mx)
{
  int64_t const e = elemOf(a, blockIdx.x * 32ll + el);
  int32_t const pij = sh.rp[el][i] + a.rank[e * 64 + i * 8 + j];
  uint32_t const cons = sh.flags[el] & 0xffu;
  bool const ci = (cons >> i) & 1u, cj = (cons >> j) & 1u;
  double const kfac = a.fold.coef ? a.kE[e] : 1.0;
#pragma unroll
  for (int m = 0; m < 2; ++m)
  {
    LhsDev const & op = a.op[m];
    if (!op.on)
      continue;
    // a single operator's coefficient is folded into the values
    double const kf = a.fold.foldK ? 1. : (op.stiff == 2 ? op.sc * kfac : op.sc),
                 mf = a.fold.foldM ? 1. : massCoef(op, kfac);
    double val = op.stiff ? kf * sh.kval[el][kx] : mf * sh.mval[el][mx];
    if (op.stiff && op.mass)
      val = fma(mf, sh.mval[el][mx], val);
    if (!(op.bc && (ci || cj)))
      atomicAdd(op.vals + pij, val);
    else if (i == j)
      atomicAdd(op.vals + pij, a.bcDiag);
    else if (!ci && a.b)
    {
      double const z = val * a.bcVal[sh.dof[j][el]];
      if (z != 0.)
        atomicAdd(a.b + sh.dof[i][el], -z);
    }
  }
}

// out of line: the few elements the fixed-point form refuses
__device__ __noinline__ void elementF64Rare(AsmArgs const & a, int64_t e) { elementF64(a, e); }

} // namespace

// MINB blocks of 256 threads per SM: 4 -> 64 registers per thread, 3 -> 80
template <int MINB>
__global__ void __launch_bounds__(256, MINB) kAssembleQ1Fx(AsmArgs const __grid_constant__ a)
{
  __shared__ Q1Shared sh;
  int const w = threadIdx.x >> 5, l = threadIdx.x & 31;
  int64_t const i0 = blockIdx.x * 32ll + l;
  bool const inMesh = i0 < a.nelem;
  int64_t const e = elemOf(a, inMesh ? i0 : a.nelem - 1);
  bool const needK = a.fold.needK, needM = a.fold.needM;
  // loads: sin sin sin by its series, a constant, and anything else (another function, the
  // projection of a DOF field, elements too large for the series) point by point in FP64
  bool const analytic = a.rkind == 1 && a.fn != PXG_FN_CONST, sine = a.rkind == 1 && a.fn == PXG_FN_SIN3;

  // ---- 0. inputs
  double const kfac = a.fold.coef ? a.kE[e] : 1.0;
  double d[8];
  if (w < 6)
  {
    if (w < 3 || analytic)
    {
      int const r = w < 3 ? w : w - 3;
      uint4 const c0 = reinterpret_cast<uint4 const *>(a.conn)[2 * e];
      uint4 const c1 = reinterpret_cast<uint4 const *>(a.conn)[2 * e + 1];
      // lattice order: nodes 0 1 3 2 4 5 7 6
      d[0] = a.xyz[3 * (int64_t)c0.x + r], d[1] = a.xyz[3 * (int64_t)c0.y + r];
      d[2] = a.xyz[3 * (int64_t)c0.w + r], d[3] = a.xyz[3 * (int64_t)c0.z + r];
      d[4] = a.xyz[3 * (int64_t)c1.x + r], d[5] = a.xyz[3 * (int64_t)c1.y + r];
      d[6] = a.xyz[3 * (int64_t)c1.w + r], d[7] = a.xyz[3 * (int64_t)c1.z + r];
      if (w < 3)
      {
        int32_t m = 0;
#pragma unroll
        for (int v = 7; v >= 0; --v)
        {
          d[v] -= d[0];
          int32_t const h = q1x::hi32(q1x::doubleBits(d[v])) & 0x7fffffff;
          m = h > m ? h : m;
        }
        sh.dmax[r][l] = m;
      }
    }
  }
  else if (w == 6)
  {
    uint4 const d0 = reinterpret_cast<uint4 const *>(a.emap)[2 * e];
    uint4 const d1 = reinterpret_cast<uint4 const *>(a.emap)[2 * e + 1];
    uint32_t const dof[8] = {d0.x, d0.y, d0.z, d0.w, d1.x, d1.y, d1.z, d1.w};
    uint32_t cons = 0;
#pragma unroll
    for (int n = 0; n < 8; ++n)
    {
      sh.dof[n][l] = dof[n];
      sh.rp[l][n] = a.rowPtr[dof[n]];
      if (a.bcMask && a.bcMask[dof[n]])
        cons |= 1u << n;
    }
    sh.flags[l] = cons;
  }
  __syncthreads();
  int sc[3];
  bool ok = q1x::coordScales(sh.dmax[0][l], sh.dmax[1][l], sh.dmax[2][l], sc);
  int const scMin = min(sc[0], min(sc[1], sc[2]));
  if (w < 3)
  {
    int const scw = w == 0 ? sc[0] : (w == 1 ? sc[1] : sc[2]);
    int64_t col[3][4];
    uint32_t cm[3];
    int64_t off[8];
    q1x::coordColumns(d, scw, col, cm, off);
    if (analytic)
    {
#pragma unroll
      for (int q = 0; q < 8; ++q)
        sh.off[w][q][l] = off[q];
      q1x::Bound const b = q1x::offsetBound(cm, scw);
      sh.bound[w][l] = b.f, sh.et[w][l] = b.e;
    }
#pragma unroll
    for (int c = 0; c < 3; ++c)
    {
#pragma unroll
      for (int p = 0; p < 4; ++p)
        sh.col[(c * 3 + w) * 4 + p][l] = col[c][p];
      sh.cmax[c * 3 + w][l] = cm[c];
    }
  }
  else if (w < 6 && analytic)
  {
    // element origin = vertex average (geo.hpp:721-728)
    double const o = 0.125 * (((d[0] + d[1]) + (d[2] + d[3])) + ((d[4] + d[5]) + (d[6] + d[7])));
    sh.org[w - 3][l] = o;
    double t[2] = {0., 0.};
    if (sine)
      sinCosPiTab(o, t[0], t[1]);
#pragma unroll
    for (int i = 0; i < 2; ++i)
    {
      int64_t m;
      int x;
      q1x::sineParts(t[i], m, x);
      sh.sm[2 * (w - 3) + i][l] = m, sh.se[2 * (w - 3) + i][l] = x;
      if (i == 0)
        sh.ee[w - 3][l] = q1x::seriesExponent(x, w == 3 ? sc[0] : (w == 4 ? sc[1] : sc[2]));
    }
  }
  __syncthreads();

  // ---- 1. scales, and one point per warp
  q1x::Shifts s;
  int deg = 0;
  bool series = false;
  {
    uint32_t cm[9];
#pragma unroll
    for (int k = 0; k < 9; ++k)
      cm[k] = sh.cmax[k][l];
    ok = q1x::columnShifts(cm, s) && ok;
    if (sine)
    {
      float const bm = fmaxf(sh.bound[0][l], fmaxf(sh.bound[1][l], sh.bound[2][l]));
      series = ok && max(sc[0], max(sc[1], sc[2])) <= q1x::kLoadMaxScale && bm <= q1x::kLoadMaxT;
      // one degree for the block (every warp sees the same elements); a warp forms the
      // coefficients w, w + 8 of each coordinate
      deg = q1x::seriesDegree(__uint_as_float(__reduce_max_sync(0xffffffffu, series ? __float_as_uint(bm) : 0u)));
      for (int i = w; i <= deg; i += 8)
#pragma unroll
        for (int r = 0; r < 3; ++r)
          sh.coef[r][i][l] =
              q1x::seriesCoef(q1x::kSeries[i], sh.ee[r][l], sc[r], i, sh.sm[2 * r + (i & 1)][l], sh.se[2 * r + (i & 1)][l]);
    }
  }
  int64_t G[6];
  int64_t det;
  int64_t u[3];
  {
    Sp c1[3], c2[3], c3[3];
    int const p1 = w >> 1, p2 = (w & 1) | ((w >> 2) << 1), p3 = w & 3;
#pragma unroll
    for (int r = 0; r < 3; ++r)
    {
      int64_t const x = sh.col[r * 4 + p1][l], y = sh.col[(3 + r) * 4 + p2][l], z = sh.col[(6 + r) * 4 + p3][l];
      c1[r] = q1x::splitOdd(q1x::shl(x, s.n[0]));
      c2[r] = q1x::splitOdd(q1x::shl(y, s.n[1]));
      c3[r] = q1x::splitOdd(q1x::shl(z, s.n[2]));
      u[r] = analytic ? sh.off[r][w][l] : 0;
    }
    int const wt[3] = {sc[0] - scMin, sc[1] - scMin, sc[2] - scMin};
    det = q1x::pointProducts(c1, c2, c3, __any_sync(0xffffffffu, (wt[0] | wt[1] | wt[2]) != 0) != 0, wt, G);
    sh.det[w][l] = det;
    sh.psize[w][l] = q1x::productSize(G, s);
  }
  __syncthreads();
  int64_t km, mm;
  int ke, me, nd, k, eK, eD;
  {
    uint32_t lo = 0xffffffffu, hi = 0, ps = 0;
#pragma unroll
    for (int q = 0; q < 8; ++q)
    {
      uint32_t const t = (uint32_t)q1x::hi32(sh.det[q][l]);
      lo = t < lo ? t : lo, hi = t > hi ? t : hi;
      uint32_t const z = sh.psize[q][l];
      ps = z > ps ? z : ps;
    }
    ok = q1x::detShifts(lo, hi, nd, k) && ok;
    // the coefficient of a single stiffness (mass) operator is folded into its values
    // (their range keeps the products below 2^1023)
    ok = q1x::coefParts(a.fold.coefK ? a.fold.sK * kfac : a.fold.sK, km, ke) && ok;
    ok = q1x::coefParts(a.fold.coefM ? a.fold.sM * kfac : a.fold.sM, mm, me) && ok;
    int const sg = q1x::productShift(ps);
    eD = q1x::detExponent(sc, s, nd);
    q1x::limitFactor(mm, me, 61 - eD);
    eK = q1x::tensorExponent(sc, scMin, s, k, sg) + ke - 61;
    if (needK)
    {
      q1x::pointInverse(det, k, sg, q1x::split(km), s, G);
#pragma unroll
      for (int c = 0; c < 6; ++c)
        sh.G[c * 8 + w][l] = G[c];
    }
    det = q1x::shl(det, nd);
  }
  if (series)
  {
    Sp const u0 = q1x::split(u[0]), u1 = q1x::split(u[1]), u2 = q1x::split(u[2]);
    int64_t f0 = sh.coef[0][deg][l], f1 = sh.coef[1][deg][l], f2 = sh.coef[2][deg][l];
    for (int i = deg - 1; i >= 0; --i)
    {
      f0 = q1x::mulAdd(q1x::split(f0), u0, sh.coef[0][i][l]);
      f1 = q1x::mulAdd(q1x::split(f1), u1, sh.coef[1][i][l]);
      f2 = q1x::mulAdd(q1x::split(f2), u2, sh.coef[2][i][l]);
    }
    int const n0 = q1x::seriesShift(sh.ee[0][l], sh.se[0][l], sh.et[0][l]),
              n1 = q1x::seriesShift(sh.ee[1][l], sh.se[2][l], sh.et[1][l]),
              n2 = q1x::seriesShift(sh.ee[2][l], sh.se[4][l], sh.et[2][l]);
    sh.rq[w][l] = q1x::pointLoad(q1x::shl(f0, n0), q1x::shl(f1, n1), q1x::shl(f2, n2), det);
    if (w == 7)
      sh.el[l] = sh.ee[0][l] + sh.ee[1][l] + sh.ee[2][l] - (n0 + n1 + n2);
  }
  else if (a.rkind == 1 && !analytic)
    sh.rq[w][l] = det >> 2;
  else if (a.rkind && ok)
  {
    double f;
    if (a.rkind == 1)
    {
      // u = J xi / g at F = 61
      double x[3];
#pragma unroll
      for (int r = 0; r < 3; ++r)
        x[r] = fma(q1f::g, q1x::toDouble(u[r], sc[r] - 61), sh.org[r][l]);
      f = evalPoint(a.fn, x[0], x[1], x[2]);
    }
    else
      f = fieldPoint(a.field, sh, l, w);
    sh.rqd[w][l] = a.rc * (q1x::toDoubleFlush(det, eD - 60) * f);
  }
  __syncthreads();
  pdlWait(); // the writes start below

  // ---- 2. tables; load vector (buildLhs' BC values and buildRhs)
  if (w < 3)
  {
    if (needK)
    {
      int const D = 1 << w, E = w == 0 ? 2 : 1, F = w == 2 ? 2 : 4;
      int64_t v[8], S[9];
#pragma unroll
      for (int i = 0; i < 8; ++i)
        v[i] = sh.G[w * 8 + (i & 1) * D + ((i >> 1) & 1) * E + (i >> 2) * F][l];
      q1x::tableS(v, S);
#pragma unroll
      for (int i = 0; i < 9; ++i)
        sh.tab[w * 9 + i][l] = S[i];
    }
  }
  else if (w < 6)
  {
    if (needK)
    {
      int const c = w - 3, D = c == 2 ? 2 : 1, E = c == 0 ? 2 : 4, F = c == 0 ? 4 : (c == 1 ? 2 : 1);
      int64_t v[8], U[12];
#pragma unroll
      for (int i = 0; i < 8; ++i)
        v[i] = sh.G[(3 + c) * 8 + (i & 1) * D + ((i >> 1) & 1) * E + (i >> 2) * F][l];
      q1x::tableU(v, U);
#pragma unroll
      for (int i = 0; i < 12; ++i)
        sh.tab[27 + c * 12 + i][l] = U[i];
    }
  }
  else if (w == 6)
  {
    if (needM)
    {
      int64_t v[8], M[3][3][3];
      Sp const ms = q1x::split(mm);
#pragma unroll
      for (int q = 0; q < 8; ++q)
        v[q] = q1x::mul(q1x::split(q1x::shl(sh.det[q][l], nd)), ms);
      q1x::massTable(v, M);
#pragma unroll
      for (int i = 0; i < 27; ++i)
        sh.mtab[l][i] = M[i / 9][(i / 3) % 3][i % 3];
    }
  }
  else
  {
    uint32_t const cons = sh.flags[l];
    if (ok && inMesh)
    {
      uint32_t dof[8];
#pragma unroll
      for (int n = 0; n < 8; ++n)
        dof[n] = sh.dof[n][l];
      if (a.b && cons && a.fold.bc)
        q1f::addBcValues(a, dof, cons);
      if (a.rkind)
      {
        double fe[8];
        if (series || (a.rkind == 1 && !analytic))
        {
          int64_t r[8];
#pragma unroll
          for (int q = 0; q < 8; ++q)
            r[q] = sh.rq[q][l];
          int const el = sine ? eD + sh.el[l] - 60 : eD - 59;
          q1x::nodeSums(r);
#pragma unroll
          for (int q = 0; q < 8; ++q)
            fe[q] = a.rc * q1x::toDoubleFlush(r[q], el);
        }
        else
        {
          // sum_q r_q l l l, one axis at a time
#pragma unroll
          for (int q = 0; q < 8; ++q)
            fe[q] = sh.rqd[q][l];
#pragma unroll
          for (int t = 1; t < 8; t *= 2)
#pragma unroll
            for (int q = 0; q < 8; ++q)
              if (!(q & t))
              {
                double const v0 = fe[q], v1 = fe[q | t];
                fe[q] = fma(q1f::A, v0, q1f::B * v1), fe[q | t] = fma(q1f::B, v0, q1f::A * v1);
              }
        }
#pragma unroll
        for (int q = 0; q < 8; ++q)
        {
          int const n = q1f::node(q & 1, (q >> 1) & 1, q >> 2);
          if (!(a.rbc && ((cons >> n) & 1u)))
            atomicAdd(a.b + dof[n], fe[q]);
        }
      }
    }
    sh.flags[l] = cons | (inMesh ? 0x100u : 0u) | (ok ? 0x200u : 0u);
  }
  __syncthreads();

  // ---- 3. entries; the scatter's ranks are fetched ahead of them
  int kx[2], mx[2];
  uint16_t rank[8];
  if (a.fold.simple)
  {
    // (row, column) of the lane in its element's 8 x 8 ranks: 32 (t & 1) + l
#pragma unroll
    for (int t = 0; t < 8; ++t)
    {
      int64_t const i = blockIdx.x * 32ll + 4 * w + (t >> 1);
      rank[t] = a.rank[elemOf(a, i < a.nelem ? i : a.nelem - 1) * 64 + 32 * (t & 1) + l];
    }
  }
#pragma unroll
  for (int h = 0; h < 2; ++h)
  {
    int const li = latticeOf(4 * h + (l >> 3)), lj = latticeOf(l & 7), q = li ^ lj;
    kx[h] = entryIndex(li, lj);
    mx[h] = ((q & 1) ? 2 : (li & 1)) * 9 + ((q & 2) ? 2 : ((li >> 1) & 1)) * 3 + ((q & 4) ? 2 : (li >> 2));
  }
  if (needK)
  {
    switch (w)
    {
    case 0:
      entriesOut<0, 1>(sh, l, eK);
      break;
    case 1:
      entriesOut<0, 2>(sh, l, eK);
      break;
    case 2:
      entriesOut<0, 3>(sh, l, eK);
      break;
    case 3:
      entriesOut<1, 2>(sh, l, eK);
      break;
    case 4:
      entriesOut<1, 3>(sh, l, eK);
      break;
    case 5:
      entriesOut<2, 3>(sh, l, eK);
      break;
    case 6:
      entriesOut<0, 0>(sh, l, eK);
      entriesOut<1, 1>(sh, l, eK);
      break;
    default:
      entriesOut<2, 2>(sh, l, eK);
      entriesOut<3, 3>(sh, l, eK);
    }
  }
  if (needM)
    for (int i = w; i < 27; i += 8)
      sh.mval[l][i] = q1x::toDouble(sh.mtab[l][i], eD + me - 61);
  __syncthreads();

  // ---- 4. scatter: lane = (row i, column j) of four rows, warp w the elements 4w..4w+3
  if (needK || needM)
  {
    if (a.fold.simple)
    {
#pragma unroll
      for (int t = 0; t < 8; ++t)
      {
        int const el = 4 * w + (t >> 1), i = 4 * (t & 1) + (l >> 3);
        uint32_t const fl = sh.flags[el];
        if ((fl & 0x300u) != 0x300u)
          continue;
        int32_t const pij = sh.rp[el][i] + rank[t];
        double kv = sh.kval[el][kx[t & 1]], mv = sh.mval[el][mx[t & 1]];
        if (a.fold.same)
          kv += mv;
        bool addK = needK, addM = needM && !a.fold.same;
        if (a.fold.bc && (fl & 0xffu))
        {
          bool const ci = (fl >> i) & 1u, cj = (fl >> (l & 7)) & 1u, c = ci || cj;
          condense(a, sh, el, i, l & 7, c && addK && a.fold.bcK, c && addM && a.fold.bcM, ci, pij, kv, mv);
          addK = addK && !(c && a.fold.bcK), addM = addM && !(c && a.fold.bcM);
        }
        if (addK)
          atomicAdd(a.fold.K + pij, kv);
        if (addM)
          atomicAdd(a.fold.M + pij, mv);
      }
    }
    else
    {
#pragma unroll 1
      for (int t = 0; t < 8; ++t)
      {
        int const el = 4 * w + (t >> 1);
        if ((sh.flags[el] & 0x300u) == 0x300u)
          scatterGeneral(a, sh, el, 4 * (t & 1) + (l >> 3), l & 7, kx[t & 1], mx[t & 1]);
      }
    }
  }
  if (w == 0 && inMesh && !ok)
    elementF64Rare(a, e);
}

void launchAssembleQ1F64(AsmArgs const & args, cudaStream_t s, int threads)
{
  if (args.nelem <= 0)
    return;
  AsmArgs a = args;
  foldOps(a);
  unsigned const blocks = (unsigned)((a.nelem + 31) / 32);
  if (threads == 64)
    launchElemKernel(kAssembleQ1Fx<3>, blocks, 256, 0, s, a);
  else
    launchElemKernel(kAssembleQ1Fx<4>, blocks, 256, 0, s, a);
}

} // namespace pxg
