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
// suffice and 32 warps are resident.
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
    int64_t G[48][32];  // component c at point q: c * 8 + q
    double kval[32][37]; // entries of the stiffness (an odd stride: no bank conflicts)
  };
  union
  {
    int64_t rq[8][32];     // load values of the points
    double sc[6][32];      // sine, cosine of pi times the origin
  };
  union
  {
    int64_t det[8][32];
    int32_t dmax[3][32]; // high word of the largest difference per coordinate
  };
  union
  {
    double mval[32][27]; // the mass table
    uint32_t psize[8][32];
  };
  uint32_t cmax[9][32];
  uint32_t dof[8][32];
  int32_t rp[8][32];
  int32_t ee[3][32], nf[3][32]; // exponents and shifts of the sine series
  int32_t scale[32];
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
  LhsDev const & op0 = a.op[0];
  LhsDev const & op1 = a.op[1];
  bool const k0 = op0.on && op0.stiff, k1 = op1.on && op1.stiff;
  bool const m0 = op0.on && op0.mass, m1 = op1.on && op1.mass;
  bool const needK = k0 || k1, needM = m0 || m1;
  bool const sine = a.rkind && a.fn == PXG_FN_SIN3;

  // ---- 0. inputs
  double d[8];
  if (w < 6)
  {
    if (w < 3 || sine)
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
      else
      {
        // element origin = vertex average (geo.hpp:721-728)
        double const o = 0.125 * (((d[0] + d[1]) + (d[2] + d[3])) + ((d[4] + d[5]) + (d[6] + d[7])));
        double S, C;
        sinCosPiTab(o, S, C);
        sh.sc[r][l] = S, sh.sc[3 + r][l] = C;
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
      sh.rp[n][l] = a.rowPtr[dof[n]];
      if (a.bcMask && a.bcMask[dof[n]])
        cons |= 1u << n;
    }
    sh.flags[l] = cons;
  }
  __syncthreads();
  if (w < 3)
  {
    int32_t m = sh.dmax[0][l] > sh.dmax[1][l] ? sh.dmax[0][l] : sh.dmax[1][l];
    m = m > sh.dmax[2][l] ? m : sh.dmax[2][l];
    int const sc = q1x::coordScale(m);
    int64_t col[3][4];
    uint32_t cm[3];
    q1x::coordColumns(d, sc, col, cm);
#pragma unroll
    for (int c = 0; c < 3; ++c)
    {
#pragma unroll
      for (int p = 0; p < 4; ++p)
        sh.col[(c * 3 + w) * 4 + p][l] = col[c][p];
      sh.cmax[c * 3 + w][l] = cm[c];
    }
    if (w == 0)
      sh.scale[l] = sc;
  }
  __syncthreads();

  // ---- 1. scales, and one point per warp
  int const sc = sh.scale[l];
  q1x::Shifts s;
  int deg = 0;
  bool ok;
  {
    uint32_t cm[9];
#pragma unroll
    for (int k = 0; k < 9; ++k)
      cm[k] = sh.cmax[k][l];
    ok = q1x::columnShifts(cm, s) && q1x::coordScaleOk(sc);
    if (sine)
    {
      float const b0 = q1x::offsetBound(cm, 0, sc), b1 = q1x::offsetBound(cm, 1, sc), b2 = q1x::offsetBound(cm, 2, sc);
      float const bm = fmaxf(b0, fmaxf(b1, b2));
      int const p = sc - s.nmin;
      ok = ok && p <= q1x::kLoadMaxP && bm <= q1x::kLoadMaxT;
      // one degree for the block (every warp sees the same elements)
      uint32_t const t = __reduce_max_sync(0xffffffffu, ok ? __float_as_uint(bm) : 0u);
      deg = t <= __float_as_uint(0.0205f) ? 7 : (t <= __float_as_uint(0.07f) ? 9 : 15);
      if (w >= 3 && w < 6)
      {
        int const r = w - 3;
        float const b = r == 0 ? b0 : (r == 1 ? b1 : b2);
        double const S = sh.sc[r][l], C = sh.sc[3 + r][l];
        int64_t k[16];
        int nf, es;
        if (deg == 7)
          es = q1x::seriesCoefs<7>(S, C, p, b, reinterpret_cast<int64_t(&)[8]>(k), nf);
        else if (deg == 9)
          es = q1x::seriesCoefs<9>(S, C, p, b, reinterpret_cast<int64_t(&)[10]>(k), nf);
        else
          es = q1x::seriesCoefs<15>(S, C, p, b, k, nf);
#pragma unroll
        for (int i = 0; i < 16; ++i)
          if (i <= deg)
            sh.coef[r][i][l] = k[i];
        sh.ee[r][l] = es;
        sh.nf[r][l] = nf;
      }
    }
  }
  int64_t G[6];
  int64_t det;
  Sp u[3];
  {
    Sp c1[3], c2[3], c3[3];
    int const p1 = w >> 1, p2 = (w & 1) | ((w >> 2) << 1), p3 = w & 3;
#pragma unroll
    for (int r = 0; r < 3; ++r)
    {
      c1[r] = q1x::splitOdd(q1x::shl(sh.col[r * 4 + p1][l], s.n[0]));
      c2[r] = q1x::splitOdd(q1x::shl(sh.col[(3 + r) * 4 + p2][l], s.n[1]));
      c3[r] = q1x::splitOdd(q1x::shl(sh.col[(6 + r) * 4 + p3][l], s.n[2]));
      if (sine)
        u[r] = q1x::pointOffset(c1[r], c2[r], c3[r], w, s);
    }
    det = q1x::pointProducts(c1, c2, c3, G);
    sh.det[w][l] = det;
    sh.psize[w][l] = q1x::productSize(G, s);
  }
  __syncthreads();
  double const kfac = ((usesCoef(op0) || usesCoef(op1)) && a.kE) ? a.kE[e] : 1.0;
  // the coefficient of a single stiffness (mass) operator is folded into its values
  bool const foldK = k0 != k1, foldM = m0 != m1;
  double const ks0 = k0 ? (op0.stiff == 2 ? op0.sc * kfac : op0.sc) : 0.;
  double const ks1 = k1 ? (op1.stiff == 2 ? op1.sc * kfac : op1.sc) : 0.;
  double const ms0 = m0 ? massCoef(op0, kfac) : 0., ms1 = m1 ? massCoef(op1, kfac) : 0.;
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
    ok = q1x::decompose(foldK ? (k0 ? ks0 : ks1) : 1.0, km, ke) && ok;
    ok = q1x::decompose(foldM ? (m0 ? ms0 : ms1) : 1.0, mm, me) && ok;
    ok = ok && abs(ke) < 300 && abs(me) < 300; // every value stays normal
    int const sg = q1x::productShift(ps);
    eD = q1x::detExponent(sc, s, nd);
    eK = q1x::tensorExponent(sc, s, nd, k, sg) + ke - 61;
    det = q1x::shl(det, nd);
    if (needK)
    {
      q1x::pointInverse(det, k, sg, q1x::split(km), s, G);
#pragma unroll
      for (int c = 0; c < 6; ++c)
        sh.G[c * 8 + w][l] = G[c];
    }
  }
  if (sine)
  {
    int64_t f0 = sh.coef[0][deg][l], f1 = sh.coef[1][deg][l], f2 = sh.coef[2][deg][l];
    for (int i = deg - 1; i >= 0; --i)
    {
      f0 = q1x::mulAdd(q1x::split(f0), u[0], sh.coef[0][i][l]);
      f1 = q1x::mulAdd(q1x::split(f1), u[1], sh.coef[1][i][l]);
      f2 = q1x::mulAdd(q1x::split(f2), u[2], sh.coef[2][i][l]);
    }
    sh.rq[w][l] = q1x::pointLoad(q1x::shl(f0, sh.nf[0][l]), q1x::shl(f1, sh.nf[1][l]), q1x::shl(f2, sh.nf[2][l]), det);
  }
  else if (a.rkind)
    sh.rq[w][l] = det >> 2;
  __syncthreads();
  pdlWait(); // the writes start below

  // ---- 2. tables; load vector (buildLhs' BC values and buildRhs)
  bool const bcOps = (op0.on && op0.bc) || (op1.on && op1.bc);
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
        sh.mval[l][i] = q1x::toDouble(M[i / 9][(i / 3) % 3][i % 3], eD + me - 61);
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
      if (a.b && cons && bcOps)
        q1f::addBcValues(a, dof, cons);
      if (a.rkind)
      {
        int64_t r[8];
#pragma unroll
        for (int q = 0; q < 8; ++q)
          r[q] = sh.rq[q][l];
        int const el = sine ? eD + sh.ee[0][l] + sh.ee[1][l] + sh.ee[2][l] - 60 : eD - 59;
        q1x::nodeSums(r);
#pragma unroll
        for (int q = 0; q < 8; ++q)
        {
          int const n = q1f::node(q & 1, (q >> 1) & 1, q >> 2);
          if (!(a.rbc && ((cons >> n) & 1u)))
            atomicAdd(a.b + dof[n], a.rc * q1x::toDouble(r[q], el));
        }
      }
    }
    sh.flags[l] = cons | (inMesh ? 0x100u : 0u) | (ok ? 0x200u : 0u);
  }
  __syncthreads();

  // ---- 3. entries
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
  __syncthreads();

  // ---- 4. scatter: lane = (row i, column j) of four rows, warp w the elements 4w..4w+3
  if (needK || needM)
  {
    int const j = l & 7;
    int kx[2], mx[2];
#pragma unroll
    for (int h = 0; h < 2; ++h)
    {
      int const li = latticeOf(4 * h + (l >> 3)), lj = latticeOf(j), q = li ^ lj;
      kx[h] = entryIndex(li, lj);
      mx[h] = ((q & 1) ? 2 : (li & 1)) * 9 + ((q & 2) ? 2 : ((li >> 1) & 1)) * 3 + ((q & 4) ? 2 : (li >> 2));
    }
    // the usual pair: one operator's stiffness, the other's mass
    bool const pair = foldK && foldM && ((k0 && !m0 && m1 && !k1) || (k1 && !m1 && m0 && !k0));
#pragma unroll
    for (int t = 0; t < 4; ++t)
    {
      int const el = 4 * w + t;
      uint32_t const fl = sh.flags[el];
      if ((fl & 0x300u) != 0x300u)
        continue;
      int64_t const ee = elemOf(a, blockIdx.x * 32ll + el);
      uint32_t const cons = fl & 0xffu;
      bool const anyBc = cons && bcOps;
#pragma unroll
      for (int h = 0; h < 2; ++h)
      {
        int const i = 4 * h + (l >> 3);
        int32_t const pij = sh.rp[i][el] + a.rank[ee * 64 + i * 8 + j];
        double const kv = needK ? sh.kval[el][kx[h]] : 0., mv = needM ? sh.mval[el][mx[h]] : 0.;
        if (pair && !anyBc)
        {
          atomicAdd((k0 ? op0.vals : op1.vals) + pij, kv);
          atomicAdd((k0 ? op1.vals : op0.vals) + pij, mv);
          continue;
        }
        double kf = 1., mf = 1., kg = 1., mg = 1.; // coefficients of op0 and op1 not folded
        if (!foldK || !foldM)
        {
          double const kfe = ((usesCoef(op0) || usesCoef(op1)) && a.kE) ? a.kE[ee] : 1.0;
          if (!foldK)
            kf = op0.stiff == 2 ? op0.sc * kfe : op0.sc, kg = op1.stiff == 2 ? op1.sc * kfe : op1.sc;
          if (!foldM)
            mf = massCoef(op0, kfe), mg = massCoef(op1, kfe);
        }
        bool const ci = (cons >> i) & 1u, cj = (cons >> j) & 1u;
#pragma unroll
        for (int m = 0; m < 2; ++m)
        {
          LhsDev const & op = a.op[m];
          if (!op.on)
            continue;
          double const ksm = m ? kg : kf, msm = m ? mg : mf;
          double val = op.stiff ? ksm * kv : msm * mv;
          if (op.stiff && op.mass)
            val = fma(msm, mv, val);
          if (anyBc && op.bc && (ci || cj))
          {
            // condensation (builder.hpp:76-124): the diagonal of a constrained DOF, the
            // lift -K_ij h_j of a free row
            if (i == j)
              atomicAdd(op.vals + pij, a.bcDiag);
            else if (!ci && a.b)
            {
              double const z = val * a.bcVal[sh.dof[j][el]];
              if (z != 0.)
                atomicAdd(a.b + sh.dof[i][el], -z);
            }
            continue;
          }
          atomicAdd(op.vals + pij, val);
        }
      }
    }
  }
  if (w == 0 && inMesh && !ok)
    elementF64Rare(a, e);
}

void launchAssembleQ1Fx(AsmArgs const & a, cudaStream_t s, int threads)
{
  unsigned const blocks = (unsigned)((a.nelem + 31) / 32);
  if (threads == 64)
    launchElemKernel(kAssembleQ1Fx<4>, blocks, 256, 0, s, a);
  else
    launchElemKernel(kAssembleQ1Fx<3>, blocks, 256, 0, s, a);
}

} // namespace pxg
