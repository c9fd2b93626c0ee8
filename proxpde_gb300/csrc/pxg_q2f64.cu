// Q2 hexahedron elements with sum factorisation, in 64-bit fixed point (the kernel, at the
// end) and, for the few elements that format refuses, in FP64 by one warp.  An element
// computes what proxpde's element loop computes for a Q2 hexahedron with
// the 3x3x3 Gauss rule (include/builder.hpp:53-153): CurFE::reinit (include/curfe.hpp:
// 50-103), AssemblyStiffness(FE) / AssemblyScalarMass / AssemblyMassFE
// (include/assembly_lhs.hpp:52-109, 207-221, 262-277), AssemblyRhsAnalytic and
// AssemblyS2SProjection (include/assembly_rhs.hpp:61-88, 130-159) and the Dirichlet
// condensation (builder.hpp:76-124), with FP64 reductions into the CSR values and the
// load vector.
//
// The Q2 basis is a tensor product of the 1D functions l_0 = x(x-1)/2, l_1 = x(x+1)/2,
// l_2 = 1 - x^2 (src/reffe.cpp:374-383), and the rule a tensor product of the 3-point
// Gauss rule, so every sum over the 27 points factors into three 3-term sums:
//  - per point (lane q): J of the trilinear map from the Walsh-Hadamard transform of
//    the vertices (the 27 mapping points lie on the trilinear image, so this is the
//    reference's J), J^T J, its adjugate and determinant D, 1/|det J| = rsqrt(D) (one
//    third-order Newton step), w_q |det J_q|, G_q = k w_q |det J| (J^T J)^-1;
//  - stiffness tables, each three one-axis contractions of one G component with the
//    1D products D_ab = l'_a l'_b, P_ab = l_a l_b (6 symmetric classes): S_x = sum
//    G_xx D P P, S_y, S_z (216 values each).  The mixed terms of K_ij,
//    sum G_xy (E_ix,jx E_jy,iy + E_jx,ix E_iy,jy) P with E_ab = l'_a l_b, split E into
//    its symmetric part S_ab = (l_a l_b)'/2 (6 classes) and antisymmetric part
//    A_ab = (l'_a l_b - l'_b l_a)/2 (3 classes, a < b, and its sign): the sum is
//    2 sum G S S P - 2 s_x s_y sum G A A P, so each of G_xy, G_xz, G_yz gives a table SS
//    (216 values) and a table AA (54), sharing their first stage (the 6-class P axis),
//    instead of the 486 values of sum G E E P;
//    the stiffness stages use each class's three coefficients divided by the first, so
//    that an output costs two FP64 operations, and an entry K_ij, a sum of nine table
//    values (three S, an SS and an AA per mixed component), multiplies each by its
//    deferred scale (the product of the three classes' first coefficients, with the
//    factor 2 and the sign) in the FMA that adds it;
//  - mass table sum |det J| w P P P (216), M_ij one value of it;
//  - the load r_q = w_q |det J_q| f(qpoint_q), contracted to the nodes with l_a.
// About 16k FP64 operations per element against about 100k for the per-point form.
// A contraction stage maps [3][m] (point axis first) to [m][C] (C classes last), so
// three stages turn [qx][qy][qz] into [cx][cy][cz]; the lanes take the stage's outputs
// in turn.
#include <vector>

#include "pxg_internal.h"
#include "pxg_q2x.h"
#include "pxg_sinpi.h"

namespace pxg
{
namespace q2f
{
constexpr int NQ = 27, N = 27, NP = N * (N + 1) / 2;

// 1D tables at the three Gauss points t_0 < t_1 = 0 < t_2 (from initQ2F64Tables):
// [0, 9) l_a(t_k) at 3a + k; [9, 27) P classes; [27, 45) D classes; [45, 63) S classes;
// [63, 72) A classes.  Symmetric classes: (0,0) (1,1) (2,2) (0,1) (0,2) (1,2);
// antisymmetric: (0,1) (0,2) (1,2).
__device__ double gCoef[72];
__device__ double gCoefN[72];      // P, D, S, A classes divided by their first coefficient
// the deferred scales: S_x S_y S_z (216 each), then per mixed component its SS table
// (216) and its AA table (128: index a for a positive orientation, 64 + a for a
// negative one, 54 for the pairs without an AA term, whose scale is 0)
constexpr int kAA = 128;
constexpr int kScales = 3 * 216 + 3 * (216 + kAA);
__device__ double gScale[kScales];
__device__ double gT[3];           // t_k
__device__ double gWl[NQ];         // weights in lattice order qx * 9 + qy * 3 + qz
__device__ uint8_t gRuleOfLat[NQ]; // the rule's point index of each lattice point
__device__ uint8_t gLatOfNode[N];  // node n -> ax * 9 + ay * 3 + az (1D function indices)
__device__ uint8_t gNodeOfLat[N];
__device__ uint16_t gPairsF[NP];   // (i << 8 | j), i <= j
// per pair, its index into each table (the layouts of the contractions below): the S
// tables' (shared by the mass and S_x, S_y, S_z), then SS_xy, AA_xy, SS_xz, AA_xz,
// SS_yz, AA_yz (an AA index with the orientation, as gScale lays them out); 8 per pair
// (one padding)
__device__ uint16_t gPairIdx[NP * 8];
constexpr int kPairsPerLane = (NP + 31) / 32; // 12
// for the fixed-point kernel: the weights at F = 62 in lattice order; the places of each
// pair's terms in the tables of the two rounds (S_x, S_y, S_z, mass; SS and AA of xy, xz,
// yz, 16 bits each), and of each entry (row, column) its row and pair (i | pair << 8)
__device__ int64_t gWx[NQ];
__device__ ushort4 gPairA[NP];
__device__ uint4 gPairB[NP];
__device__ uint32_t gEntry[N * N];
// The tables' rows, one array: 7 x 54 after the first axis, then 4 x 6 x 36 of a round, a
// plane of 36 every 37 rows (a row is 32 bytes: eight planes written at once at a stride
// of 36 would share their banks).  In
// the second round AA and -AA (54 each) of xy and xz take the first-axis rows of the
// first four tables, those of yz and a zero follow SS.
constexpr int kPlane = 37, kTab = 7 * 54, kRows = kTab + 24 * kPlane, kZero = kTab + 18 * kPlane + 108;
__host__ __device__ constexpr int rowAA(int m) { return m < 2 ? 108 * m : kTab + 18 * kPlane; }
// table T of a round, classes a (of its first axis), b and c
__host__ __device__ constexpr int rowOf(int T, int a, int b, int c) { return kTab + (T * 6 + a) * kPlane + b * 6 + c; }


__host__ __device__ constexpr int symCls(int a, int b)
{
  return a == b ? a : (a + b == 1 ? 3 : (a + b == 2 ? 4 : 5));
}

// 1/sqrt(x) by the hardware estimate and one third-order Newton step
__device__ __forceinline__ double rsqrtN(double x)
{
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  double const e = fma(-(x * y), y, 1.0);
  return fma(y * e, fma(0.375, e, 0.5), y);
}

// out[r * C + c] = sum_k coef[3c + k] in[k * m + r] (r < m, c < C), lanes in turn
__device__ __forceinline__ void stage(double const * in, int m, int C, double const * coef, double * out, int lane)
{
  for (int o = lane; o < m * C; o += 32)
  {
    int const r = o / C, c = o - r * C;
    double const * k = coef + 3 * c;
    out[o] = fma(k[2], in[2 * m + r], fma(k[1], in[m + r], k[0] * in[r]));
  }
  __syncwarp();
}
// the same with normalised coefficients (coef[3c] = 1): two operations per output
__device__ __forceinline__ void stageN(double const * in, int m, int C, double const * coef, double * out, int lane)
{
  for (int o = lane; o < m * C; o += 32)
  {
    int const r = o / C, c = o - r * C;
    double const * k = coef + 3 * c;
    out[o] = fma(k[2], in[2 * m + r], fma(k[1], in[m + r], in[r]));
  }
  __syncwarp();
}
__device__ __forceinline__ void contract3N(double const * in, int c0, double const * k0, int c1, double const * k1,
                                           int c2, double const * k2, double * out, double * scr0, double * scr1,
                                           int lane)
{
  stageN(in, 9, c0, k0, scr0, lane);
  stageN(scr0, 3 * c0, c1, k1, scr1, lane);
  stageN(scr1, c0 * c1, c2, k2, out, lane);
}
// three stages of a [3][3][3] array with the coefficient tables of the three axes
__device__ __forceinline__ void contract3(double const * in, int c0, double const * k0, int c1, double const * k1,
                                          int c2, double const * k2, double * out, double * scr0, double * scr1,
                                          int lane)
{
  stage(in, 9, c0, k0, scr0, lane);       // [3][3][c0]
  stage(scr0, 3 * c0, c1, k1, scr1, lane); // [3][c0][c1]
  stage(scr1, c0 * c1, c2, k2, out, lane); // [c0][c1][c2]
}

__device__ __noinline__ void condenseF(double * pij, double bcDiag, double * b, uint32_t dofi, uint32_t dofj,
                                       double bvi, double bvj, bool ci, bool cj, bool isDiag, double val)
{
  if (isDiag)
  {
    atomicAdd(pij, bcDiag);
    return;
  }
  if (!b)
    return;
  if (!ci)
  {
    double const t = val * bvj;
    if (t != 0.)
      atomicAdd(b + dofi, -t);
  }
  if (!cj)
  {
    double const t = val * bvi;
    if (t != 0.)
      atomicAdd(b + dofj, -t);
  }
}

// f at the point, out of line (its FP64 code is only run for the load)
__device__ __noinline__ double evalPoint(int fn, double rc, double x, double y, double z)
{
  return evalFn(fn, rc, x, y, z);
}

struct Smem
{
  double coef[72];
  double coefN[72];
  double w[NQ];
  double X[8][3];
  double H[8][3]; // Walsh-Hadamard transform of the vertices, [kx + 2 ky + 4 kz][r]
  double G[6][NQ];
  double ad[NQ];
  double tab[272]; // one table at a time: the mass, S_x, S_y, S_z, then SS [0, 216) and
                   // AA [216, 270) of each mixed component, tab[270] = 0
  double scr[2][243];
  double bv[N];
  uint32_t dof[N];
  int32_t rp[N];
  uint8_t latOfNode[N];
  uint8_t nodeOfLat[N];
  uint8_t ruleOfLat[NQ];
};
} // namespace q2f

// One element in FP64 by a warp
__device__ __noinline__ void elementQ2F64(AsmArgs const & a, int64_t e, q2f::Smem & S)
{
  using namespace q2f;
  int const lane = threadIdx.x & 31;
  for (int k = lane; k < 72; k += 32)
    S.coef[k] = gCoef[k], S.coefN[k] = gCoefN[k];
  if (lane < NQ)
  {
    S.w[lane] = gWl[lane];
    S.latOfNode[lane] = gLatOfNode[lane];
    S.nodeOfLat[lane] = gNodeOfLat[lane];
    S.ruleOfLat[lane] = gRuleOfLat[lane];
  }
  // ---- inputs
  if (lane < 24)
  {
    uint32_t const id = a.conn[e * 8 + lane / 3];
    S.X[lane / 3][lane % 3] = a.xyz[3 * (int64_t)id + lane % 3];
  }
  bool mine = false;
  if (lane < N)
  {
    uint32_t const d = a.emap[e * N + lane];
    S.dof[lane] = d;
    S.rp[lane] = a.rowPtr[d];
    mine = a.bcMask && a.bcMask[d];
    S.bv[lane] = mine ? a.bcVal[d] : 0.;
  }
  uint32_t const cons = __ballot_sync(0xffffffffu, mine);
  __syncwarp();
  LhsDev const & op0 = a.op[0];
  LhsDev const & op1 = a.op[1];
  bool const k0 = op0.on && op0.stiff, k1 = op1.on && op1.stiff;
  bool const m0 = op0.on && op0.mass, m1 = op1.on && op1.mass;
  bool const needK = k0 || k1, needM = m0 || m1;
  double const kfac = ((usesCoef(op0) || usesCoef(op1)) && a.kE) ? a.kE[e] : 1.0;
  bool const foldK = k0 != k1, foldM = m0 != m1;
  double const ks0 = k0 ? (op0.stiff == 2 ? op0.sc * kfac : op0.sc) : 0.;
  double const ks1 = k1 ? (op1.stiff == 2 ? op1.sc * kfac : op1.sc) : 0.;
  double const ms0 = m0 ? massCoef(op0, kfac) : 0., ms1 = m1 ? massCoef(op1, kfac) : 0.;

  // ---- the Walsh-Hadamard transform of the vertices, x(xi) = 1/8 sum_k H_k xi^kx
  // eta^ky zeta^kz: lane 3 lat + r holds coordinate r of the vertex at lattice point
  // lat = vx + 2 vy + 4 vz (proxpde's Q1 vertex order, src/reffe.cpp:684-759), and
  // each stage pairs the lanes whose lattice points differ along one axis
  {
    int const lat = lane / 3, r = lane % 3;
    int const vx = lat & 1, vy = (lat >> 1) & 1, vz = lat >> 2;
    int const v = vz * 4 + (vy ? (vx ? 2 : 3) : (vx ? 1 : 0));
    double h = lane < 24 ? S.X[v][r] : 0.;
#pragma unroll
    for (int ax = 0; ax < 3; ++ax)
    {
      int const bit = (lat >> ax) & 1, step = 3 << ax;
      double const o = __shfl_sync(0xffffffffu, h, lane < 24 ? (bit ? lane - step : lane + step) : lane);
      h = bit ? h - o : h + o;
    }
    if (lane < 24)
      S.H[lat][r] = h;
  }
  __syncwarp();
  // ---- per point: lane q = qx * 9 + qy * 3 + qz; the Jacobian columns (x8)
  // c1 = H100 + eta H110 + zeta H101 + eta zeta H111, ...
  if (lane < NQ)
  {
    int const qx = lane / 9, qy = (lane / 3) % 3, qz = lane % 3;
    double const xi = gT[qx], eta = gT[qy], zeta = gT[qz];
    double c[3][3]; // c[col][r]
    double o[3];    // the element origin, the vertex average (geo.hpp:721-728)
#pragma unroll
    for (int r = 0; r < 3; ++r)
    {
      // H[kx + 2 ky + 4 kz]
      double const H000 = S.H[0][r], H100 = S.H[1][r], H010 = S.H[2][r], H110 = S.H[3][r];
      double const H001 = S.H[4][r], H101 = S.H[5][r], H011 = S.H[6][r], H111 = S.H[7][r];
      c[0][r] = fma(zeta, fma(eta, H111, H101), fma(eta, H110, H100));
      c[1][r] = fma(zeta, fma(xi, H111, H011), fma(xi, H110, H010));
      c[2][r] = fma(eta, fma(xi, H111, H011), fma(xi, H101, H001));
      o[r] = 0.125 * H000;
    }
    double const g11 = fma(c[0][0], c[0][0], fma(c[0][1], c[0][1], c[0][2] * c[0][2]));
    double const g22 = fma(c[1][0], c[1][0], fma(c[1][1], c[1][1], c[1][2] * c[1][2]));
    double const g33 = fma(c[2][0], c[2][0], fma(c[2][1], c[2][1], c[2][2] * c[2][2]));
    double const g12 = fma(c[0][0], c[1][0], fma(c[0][1], c[1][1], c[0][2] * c[1][2]));
    double const g13 = fma(c[0][0], c[2][0], fma(c[0][1], c[2][1], c[0][2] * c[2][2]));
    double const g23 = fma(c[1][0], c[2][0], fma(c[1][1], c[2][1], c[1][2] * c[2][2]));
    double const A11 = fma(-g23, g23, g22 * g33);
    double const A22 = fma(-g13, g13, g11 * g33);
    double const A33 = fma(-g12, g12, g11 * g22);
    double const A12 = fma(g13, g23, -(g12 * g33));
    double const A13 = fma(g12, g23, -(g13 * g22));
    double const A23 = fma(g12, g13, -(g11 * g23));
    double const D = fma(g11, A11, fma(g12, A12, g13 * A13));
    double const rs = rsqrtN(D);
    double const wq = S.w[lane];
    S.ad[lane] = (D * rs) * wq; // w |det J| x 512
    // k w |det J| (J^T J)^-1 = k w adj rsqrt(D) / 8 (the columns carry x8)
    double const sG = ((foldK ? (k0 ? ks0 : ks1) : 1.0) * 0.125) * (wq * rs);
    S.G[0][lane] = sG * A11, S.G[1][lane] = sG * A22, S.G[2][lane] = sG * A33;
    // G_xy as [qz][qx][qy] and G_xz as [qy][qx][qz]: their tables contract the P axis first
    S.G[3][qz * 9 + qx * 3 + qy] = sG * A12, S.G[4][qy * 9 + qx * 3 + qz] = sG * A13, S.G[5][lane] = sG * A23;
    // the qpoint origin + J xi (curfe.hpp:80), for the analytic load
    if (a.rkind == 1)
    {
      double const x = fma(0.125, fma(xi, c[0][0], fma(eta, c[1][0], zeta * c[2][0])), o[0]);
      double const y = fma(0.125, fma(xi, c[0][1], fma(eta, c[1][1], zeta * c[2][1])), o[1]);
      double const z = fma(0.125, fma(xi, c[0][2], fma(eta, c[1][2], zeta * c[2][2])), o[2]);
      S.scr[0][lane] = x, S.scr[0][32 + lane] = y, S.scr[0][64 + lane] = z;
    }
  }
  __syncwarp();
  double const * const cL = S.coef;
  double const * const cP = S.coef + 9;

  // ---- load vector (buildLhs' BC values, buildRhs)
  bool const bcOps = (op0.on && op0.bc) || (op1.on && op1.bc);
  if (a.b && cons && bcOps && lane < N && ((cons >> lane) & 1u))
  {
#pragma unroll
    for (int m = 0; m < 2; ++m)
      if (a.op[m].on && a.op[m].bc && S.bv[lane] != 0.)
        atomicAdd(a.b + S.dof[lane], S.bv[lane]);
  }
  if (a.rkind)
  {
    // r_q = w_q |det J_q| f_q (x512: the 1/512 is in rc), then Fe = sum_q r_q l l l
    double const rc = a.rc * (1. / 512.);
    double * const rq = S.scr[1];
    if (lane < NQ)
    {
      double f;
      if (a.rkind == 1 && a.fn == PXG_FN_SIN3)
        f = rc * (sinPiTab(S.scr[0][lane]) * sinPiTab(S.scr[0][32 + lane]) * sinPiTab(S.scr[0][64 + lane]));
      else if (a.rkind == 1)
        f = evalPoint(a.fn, rc, S.scr[0][lane], S.scr[0][32 + lane], S.scr[0][64 + lane]);
      else if (a.rkind == 3)
        f = rc * a.field[e * NQ + S.ruleOfLat[lane]];
      else
      {
        // projection: the field at the point, sum_n phi_n(q) field_n with phi_n = l l l
        int const qx = lane / 9, qy = (lane / 3) % 3, qz = lane % 3;
        double s = 0.;
        for (int n = 0; n < N; ++n)
        {
          int const L = S.latOfNode[n];
          s = fma(cL[3 * (L / 9) + qx] * cL[3 * ((L / 3) % 3) + qy] * cL[3 * (L % 3) + qz], a.field[S.dof[n]], s);
        }
        f = rc * s;
      }
      rq[lane] = S.ad[lane] * f;
    }
    __syncwarp();
    double * const bn = S.scr[0] + 96; // [ax][ay][az]
    stage(rq, 9, 3, cL, S.scr[0], lane);
    stage(S.scr[0], 9, 3, cL, S.scr[0] + 128, lane);
    stage(S.scr[0] + 128, 9, 3, cL, bn, lane);
    if (lane < N)
    {
      int const n = S.nodeOfLat[lane];
      if (!(a.rbc && ((cons >> n) & 1u)))
        atomicAdd(a.b + S.dof[n], bn[lane]);
    }
    __syncwarp();
  }

  // ---- the tables one at a time into S.tab, each lane adding them into the entries
  // of its pairs p = lane + 32 k (kv, mv in registers): the mass table w |det J| (times
  // a single mass operator's coefficient, and the 1/512) contracted with P over the
  // three axes, then the six stiffness tables (normalised stages; each value times its
  // deferred scale, gScale in the tables' concatenated layout)
  double kv[kPairsPerLane], mv[kPairsPerLane];
#pragma unroll
  for (int k = 0; k < kPairsPerLane; ++k)
    kv[k] = 0., mv[k] = 0.;
  auto addTable = [&](int slot0, int slot1, int scaleBase, bool toMass) {
#pragma unroll
    for (int k = 0; k < kPairsPerLane; ++k)
    {
      int const p = lane + 32 * k;
      if (p >= NP)
        break;
      int const t0 = gPairIdx[8 * p + slot0];
      if (toMass)
        mv[k] = S.tab[t0];
      else
      {
        kv[k] = fma(S.tab[t0], __ldg(gScale + scaleBase + t0), kv[k]);
        if (slot1 >= 0)
        {
          // the AA value of the pair's orientation (index mod 64) and its signed scale
          int const t1 = gPairIdx[8 * p + slot1];
          kv[k] = fma(S.tab[216 + (t1 & 63)], __ldg(gScale + scaleBase + 216 + t1), kv[k]);
        }
      }
    }
    __syncwarp(); // before the next table overwrites S.tab
  };
  if (needM)
  {
    double const mcf = (foldM ? (m0 ? ms0 : ms1) : 1.0) * (1. / 512.);
    if (lane < NQ)
      S.scr[1][lane] = mcf * S.ad[lane];
    __syncwarp();
    contract3(S.scr[1], 6, cP, 6, cP, 6, cP, S.tab, S.scr[0], S.scr[1], lane);
    addTable(0, -1, 0, true);
  }
  if (needK)
  {
    double const * const nP = S.coefN + 9;
    double const * const nD = S.coefN + 27;
    double const * const nS = S.coefN + 45;
    double const * const nA = S.coefN + 63;
    contract3N(S.G[0], 6, nD, 6, nP, 6, nP, S.tab, S.scr[0], S.scr[1], lane); // [px][py][pz]
    addTable(0, -1, 0, false);
    contract3N(S.G[1], 6, nP, 6, nD, 6, nP, S.tab, S.scr[0], S.scr[1], lane);
    addTable(0, -1, 216, false);
    contract3N(S.G[2], 6, nP, 6, nP, 6, nD, S.tab, S.scr[0], S.scr[1], lane);
    addTable(0, -1, 432, false);
    // a mixed component: SS into tab[0, 216), then AA from the same first stage (scr[0])
    // into tab[216, 270), and the zero that pairs without an AA term read
    auto mixed = [&](double const * g) {
      contract3N(g, 6, nP, 6, nS, 6, nS, S.tab, S.scr[0], S.scr[1], lane);
      stageN(S.scr[0], 18, 3, nA, S.scr[1], lane);
      stageN(S.scr[1], 18, 3, nA, S.tab + 216, lane);
      if (lane == 0)
        S.tab[270] = 0.;
      __syncwarp();
    };
    mixed(S.G[3]); // [pz][sx][sy], [pz][ax][ay]
    addTable(1, 2, 648, false);
    mixed(S.G[4]); // [py][sx][sz], [py][ax][az]
    addTable(3, 4, 648 + (216 + kAA), false);
    mixed(S.G[5]); // [px][sy][sz], [px][ay][az]
    addTable(5, 6, 648 + 2 * (216 + kAA), false);
  }

  // ---- the scatter of the entries i <= j
  uint16_t const * rk = a.rank + e * (int64_t)(N * N);
  bool const anyBc = cons && bcOps;
#pragma unroll
  for (int k = 0; k < kPairsPerLane; ++k)
  {
    int const p = lane + 32 * k;
    if (p >= NP)
      break;
    uint16_t const pr = gPairsF[p];
    int const i = pr >> 8, j = pr & 0xff;
    int32_t const pij = S.rp[i] + rk[i * N + j], pji = S.rp[j] + rk[j * N + i];
    bool const ci = (cons >> i) & 1u, cj = (cons >> j) & 1u;
#pragma unroll
    for (int m = 0; m < 2; ++m)
    {
      LhsDev const & op = a.op[m];
      if (!op.on)
        continue;
      double val;
      if (op.stiff)
      {
        val = foldK ? kv[k] : (m ? ks1 : ks0) * kv[k];
        if (op.mass)
          val = foldM ? val + mv[k] : fma(m ? ms1 : ms0, mv[k], val);
      }
      else
        val = foldM ? mv[k] : (m ? ms1 : ms0) * mv[k];
      if (anyBc && op.bc && (ci || cj))
      {
        condenseF(op.vals + pij, a.bcDiag, a.b, S.dof[i], S.dof[j], S.bv[i], S.bv[j], ci, cj, i == j, val);
        continue;
      }
      atomicAdd(op.vals + pij, val);
      if (i != j)
        atomicAdd(op.vals + pji, val);
    }
  }
}

// ------------------------------------------------------------ the fixed-point kernel
// A block of four warps computes four elements in 64-bit fixed point (pxg_q2x.h); a thread
// works for element tid & 3 throughout:
//  0. coordinates, differences and Walsh-Hadamard transform by groups of eight lanes (one
//     coordinate of one element), units, shifts, and the sine series of the load;
//  1. one quadrature point per thread: columns, cofactors, |det|, products, then G and the
//     weighted determinant, and the load value;
//  2. the P axis that every table contracts first: 63 lines per element;
//  3. the two remaining axes of a table for one class of the first, nine values in, 36 out,
//     in registers: first S_x, S_y, S_z and the mass (while a warp sums the load to the
//     nodes), then the symmetric and antisymmetric tables of the mixed components; after
//     each of the two rounds every thread adds its pairs' terms into registers;
//  4. the scatter: a warp adds the 27 x 27 entries of one element row by row, so that lanes
//     read consecutive ranks and neighbouring columns share sectors.
// The FP64 form issues 509 FP64 instructions per element and warp, at 64 cycles each on
// this part; this one has none but the conversions of the results (26 per element).
namespace q2f
{
constexpr int E = 4;        // elements per block
constexpr int NT = 32 * E;  // threads per block
using q1x::Sp;

struct Shared
{
  int64_t H[E][3][8]; // H100, H010, H001, tH110, tH101, tH011, ttH111 at F = 60
  union
  {
    int64_t row[kRows][E];
    struct
    {
      int64_t s1[7][54][E];  // after the first axis
      int64_t G[7][NQ][E];   // xx yy zz xy xz yz, w |det| (before the tables)
    };
    struct
    {
      double kd[E][NP + 1], md[E][NP + 1]; // entries
    };
  };
  int64_t rq[NQ][E]; // load values (rqd: in FP64)
  int64_t coef[3][16][E];
  int64_t sm[6][E];
  double org[3][E];
  uint32_t cmax[E][9];
  int32_t dmax[3][E];
  int32_t se[6][E], ee[3][E];
  float bound[3][E];
  int32_t et[3][E];
  uint32_t lo[E], hi[E], ps[E], cons[E], ok[E];
  int32_t el[E];
  uint32_t dof[E][N];
  int32_t rp[E][N];
};
static_assert(sizeof(Smem) * E <= sizeof(Shared), "the refused elements' buffers fit the block's");

// x times s - 1, s in {0, 1, 2}
__device__ __forceinline__ int64_t times(int64_t x, int s) { return x * (int64_t)(s - 1); }

// contraction of a plane v[qs][ql] (first axis done) over its two axes
template <int KIND> // 0: P, D   1: P, P   2: S, S
__device__ __forceinline__ void plane(int64_t const (*in)[E], int64_t (*out)[E], int el)
{
  int64_t m[3][6]; // [ql][cs]
#pragma unroll
  for (int l = 0; l < 3; ++l)
  {
    if constexpr (KIND == 2)
      q2x::lineS(in[l][el], in[3 + l][el], in[6 + l][el], m[l]);
    else
      q2x::lineP(in[l][el], in[3 + l][el], in[6 + l][el], m[l]);
  }
#pragma unroll
  for (int c = 0; c < 6; ++c)
  {
    int64_t o[6];
    if constexpr (KIND == 0)
      q2x::lineD(m[0][c], m[1][c], m[2][c], o);
    else if constexpr (KIND == 1)
      q2x::lineP(m[0][c], m[1][c], m[2][c], o);
    else
      q2x::lineS(m[0][c], m[1][c], m[2][c], o);
#pragma unroll
    for (int k = 0; k < 6; ++k)
      out[c * 6 + k][el] = o[k];
  }
}
// the antisymmetric table of a component, and its negative 54 rows on
__device__ __forceinline__ void planeA(int64_t const (*in)[E], int64_t (*out)[E], int el)
{
  int64_t m[3][3];
#pragma unroll
  for (int l = 0; l < 3; ++l)
    q2x::lineA(in[l][el], in[3 + l][el], in[6 + l][el], m[l]);
#pragma unroll
  for (int c = 0; c < 3; ++c)
  {
    int64_t o[3];
    q2x::lineA(m[0][c], m[1][c], m[2][c], o);
#pragma unroll
    for (int k = 0; k < 3; ++k)
      out[c * 3 + k][el] = o[k], out[54 + c * 3 + k][el] = -o[k];
  }
}
// l_a of three doubles
__device__ __forceinline__ void lineLd(double v0, double v1, double v2, double (&o)[3])
{
  constexpr double t = 0.774596669241483;
  double const a = 0.5 * t * t * (v0 + v2), b = 0.5 * t * (v2 - v0);
  o[0] = a - b, o[1] = a + b, o[2] = fma(1. - t * t, v0 + v2, v1);
}

// the load's value at a point that is not a series or a constant: another function, a DOF
// field, a large element
__device__ __noinline__ double pointValue(AsmArgs const & a, Shared const & sh, int el, int q, double x, double y,
                                          double z)
{
  if (a.rkind == 1)
    return evalFn(a.fn, 1.0, x, y, z);
  int const qx = q / 9, qy = (q / 3) % 3, qz = q % 3;
  double s = 0.;
  for (int n = 0; n < N; ++n)
  {
    int const L = gLatOfNode[n];
    s = fma(gCoef[3 * (L / 9) + qx] * gCoef[3 * ((L / 3) % 3) + qy] * gCoef[3 * (L % 3) + qz],
            a.field[sh.dof[el][n]], s);
  }
  return s;
}

// entry (i, j) of element el for any operators and with the Dirichlet condensation
// (builder.hpp:76-124)
__device__ __noinline__ void scatterGeneral(AsmArgs const & a, Shared const & sh, int el, int64_t e, int i, int j,
                                            int p, int32_t pij)
{
  uint32_t const cons = sh.cons[el];
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
    double val = op.stiff ? kf * sh.kd[el][p] : mf * sh.md[el][p];
    if (op.stiff && op.mass)
      val = fma(mf, sh.md[el][p], val);
    if (!(op.bc && (ci || cj)))
      atomicAdd(op.vals + pij, val);
    else if (i == j)
      atomicAdd(op.vals + pij, a.bcDiag);
    else if (!ci && a.b)
    {
      double const z = val * a.bcVal[sh.dof[el][j]];
      if (z != 0.)
        atomicAdd(a.b + sh.dof[el][i], -z);
    }
  }
}
} // namespace q2f

__global__ void __launch_bounds__(q2f::NT, 5) kAssembleQ2Fx(AsmArgs const __grid_constant__ a)
{
  using namespace q2f;
  __shared__ Shared sh;
  int const tid = threadIdx.x, w = tid >> 5, l = tid & 31, el = tid & 3, x = tid >> 2;
  int64_t const i0 = blockIdx.x * (int64_t)E;
  auto element = [&](int k) { return elemOf(a, i0 + k < a.nelem ? i0 + k : a.nelem - 1); };
  int64_t const e = element(el);
  bool const needK = a.fold.needK, needM = a.fold.needM;
  // loads: sin sin sin by its series, a constant, and anything else point by point in FP64
  bool const analytic = a.rkind == 1 && a.fn != PXG_FN_CONST, sine = a.rkind == 1 && a.fn == PXG_FN_SIN3;
  double const kfac = a.fold.coef ? a.kE[e] : 1.0;

  // ---- 0. inputs
  // the ranks the warp's scatter will read
  if (l < (N * N * 2 + 255) / 128)
    asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<char const *>(a.rank + element(w) * (N * N)) +
                                                  min(128 * l, N * N * 2 - 2)));
  if (tid < E)
    sh.lo[tid] = 0xffffffffu, sh.hi[tid] = 0, sh.ps[tid] = 0, sh.cons[tid] = 0;
  // group of eight lanes g = 3 element + coordinate, lane v = lattice vertex
  int const g = tid >> 3, v = tid & 7, ge = g / 3, gr = g - 3 * ge;
  double d = 0.;
  if (tid < 8 * 3 * E)
  {
    // lattice order of the nodes: 0 1 3 2 4 5 7 6
    int const node = v ^ ((v >> 1) & 1);
    double const X = a.xyz[3 * (int64_t)a.conn[element(ge) * 8 + node] + gr];
    d = X - __shfl_sync(0xffffffffu, X, l & 24);
    int32_t m = q1x::hi32(q1x::doubleBits(d)) & 0x7fffffff;
    double o = X;
#pragma unroll
    for (int t = 1; t < 8; t *= 2)
    {
      m = max(m, __shfl_xor_sync(0xffffffffu, m, t));
      if (analytic)
        o += __shfl_xor_sync(0xffffffffu, o, t);
    }
    if (v == 0)
      sh.dmax[gr][ge] = m, sh.org[gr][ge] = 0.125 * o; // origin = vertex average (geo.hpp:721-728)
  }
  else
  {
    for (int k = tid - 8 * 3 * E; k < E * N; k += NT - 8 * 3 * E)
    {
      int const ke = k / N, n = k - ke * N;
      uint32_t const dof = a.emap[element(ke) * N + n];
      sh.dof[ke][n] = dof;
      sh.rp[ke][n] = a.rowPtr[dof];
    }
  }
  __syncthreads();
  int sc[3];
  bool ok = q1x::coordScales(sh.dmax[0][el], sh.dmax[1][el], sh.dmax[2][el], sc);
  int const scMin = min(sc[0], min(sc[1], sc[2]));
  if (tid < 8 * 3 * E)
  {
    int gs[3];
    q1x::coordScales(sh.dmax[0][ge], sh.dmax[1][ge], sh.dmax[2][ge], gs);
    int const sr = gr == 0 ? gs[0] : (gr == 1 ? gs[1] : gs[2]);
    int64_t h = q1x::roundToInt(q1x::scaleExp(d, 57 - sr));
#pragma unroll
    for (int t = 1; t < 8; t *= 2)
    {
      int64_t const o = __shfl_xor_sync(0xffffffffu, h, t);
      h = (v & t) ? h - o : h + o;
    }
    // lane v holds H_v (a set bit: difference), eight times the mean: F = 60.  times t per
    // axis beyond the first
    if (v == 3 || v == 5 || v == 6)
      h = 2 * q1x::mulc(q2x::kTh, h);
    if (v == 7)
      h = 2 * q1x::mulc(q2x::kT2h, h);
    if (v)
      sh.H[ge][gr][v] = h;
    // bounds of the columns: sums of their terms
    uint32_t const z = (uint32_t)abs(q1x::hi32(h)) + 1u;
    uint32_t const z1 = __shfl_sync(0xffffffffu, z, (l & 24) + 1), z2 = __shfl_sync(0xffffffffu, z, (l & 24) + 2),
                   z3 = __shfl_sync(0xffffffffu, z, (l & 24) + 3), z4 = __shfl_sync(0xffffffffu, z, (l & 24) + 4),
                   z5 = __shfl_sync(0xffffffffu, z, (l & 24) + 5), z6 = __shfl_sync(0xffffffffu, z, (l & 24) + 6),
                   z7 = __shfl_sync(0xffffffffu, z, (l & 24) + 7);
    if (v == 0)
    {
      uint32_t const c[3] = {z1 + z3 + z5 + z7, z2 + z3 + z6 + z7, z4 + z5 + z6 + z7};
      sh.cmax[ge][gr] = c[0], sh.cmax[ge][3 + gr] = c[1], sh.cmax[ge][6 + gr] = c[2];
      q1x::Bound const b = q1x::offsetBound(c, sr, q2x::kBoundRatio);
      // the offsets hold at F = 61 below 4
      sh.bound[gr][ge] = c[0] + c[1] + c[2] < (1u << 30) ? b.f : 1e30f;
      sh.et[gr][ge] = b.e;
      if (sine)
      {
        double t[2];
        sinCosPiTab(sh.org[gr][ge], t[0], t[1]);
#pragma unroll
        for (int i = 0; i < 2; ++i)
        {
          int64_t mt;
          int xt;
          q1x::sineParts(t[i], mt, xt);
          sh.sm[2 * gr + i][ge] = mt, sh.se[2 * gr + i][ge] = xt;
          if (i == 0)
            sh.ee[gr][ge] = q1x::seriesExponent<true>(xt, sr);
        }
      }
    }
  }
  else if (a.bcMask)
  {
    for (int k = tid - 8 * 3 * E; k < E * N; k += NT - 8 * 3 * E)
    {
      int const ke = k / N, n = k - ke * N;
      if (a.bcMask[sh.dof[ke][n]])
        atomicOr(&sh.cons[ke], 1u << n);
    }
  }
  __syncthreads();

  // ---- 1. scales, and one point per thread
  q1x::Shifts s;
  {
    uint32_t cm[9];
#pragma unroll
    for (int k = 0; k < 9; ++k)
      cm[k] = sh.cmax[el][k];
    ok = q1x::columnShifts(cm, s) && ok;
  }
  bool series = false;
  int deg = 0;
  if (sine)
  {
    float const bm = fmaxf(sh.bound[0][el], fmaxf(sh.bound[1][el], sh.bound[2][el]));
    series = ok && max(sc[0], max(sc[1], sc[2])) <= q1x::kLoadMaxScale && bm <= q1x::kLoadMaxT;
    // one degree for the block (every warp sees its four elements)
    deg = q1x::seriesDegree(__uint_as_float(__reduce_max_sync(0xffffffffu, series ? __float_as_uint(bm) : 0u)));
    for (int k = x; k < 3 * (deg + 1); k += 32)
    {
      int const r = k / (deg + 1), i = k - r * (deg + 1);
      sh.coef[r][i][el] = q1x::seriesCoef(q2x::kSeries[i], sh.ee[r][el], r == 0 ? sc[0] : (r == 1 ? sc[1] : sc[2]), i,
                                          sh.sm[2 * r + (i & 1)][el], sh.se[2 * r + (i & 1)][el]);
    }
  }
  int const q = x < NQ ? x : 0, qx = q / 9, qy = (q / 3) % 3, qz = q % 3;
  int64_t G[6], det, u[3];
  {
    Sp c1[3], c2[3], c3[3];
#pragma unroll
    for (int r = 0; r < 3; ++r)
    {
      int64_t const * const H = sh.H[el][r];
      int64_t const yz = times(times(H[7], qz), qy), xz = times(times(H[7], qz), qx), xy = times(times(H[7], qy), qx);
      int64_t const t1 = H[1] + times(H[3], qy) + times(H[5], qz) + yz;
      int64_t const t2 = H[2] + times(H[3], qx) + times(H[6], qz) + xz;
      int64_t const t3 = H[4] + times(H[5], qx) + times(H[6], qy) + xy;
      u[r] = 2 * (times(t1, qx) + times(t2, qy) + times(t3, qz)); // J xi / t at F = 61
      c1[r] = q1x::splitOdd(q1x::shl(t1, s.n[0]));
      c2[r] = q1x::splitOdd(q1x::shl(t2, s.n[1]));
      c3[r] = q1x::splitOdd(q1x::shl(t3, s.n[2]));
    }
    int const wt[3] = {sc[0] - scMin, sc[1] - scMin, sc[2] - scMin};
    det = q1x::pointProducts(c1, c2, c3, __any_sync(0xffffffffu, (wt[0] | wt[1] | wt[2]) != 0) != 0, wt, G);
    uint32_t lo = (uint32_t)q1x::hi32(det), hi = lo, ps = q1x::productSize(G, s);
#pragma unroll
    for (int t = 4; t < 32; t *= 2)
    {
      lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, t));
      hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, t));
      ps = max(ps, __shfl_xor_sync(0xffffffffu, ps, t));
    }
    if (l < E)
      atomicMin(&sh.lo[l], lo), atomicMax(&sh.hi[l], hi), atomicMax(&sh.ps[l], ps);
  }
  __syncthreads();
  int64_t km, mm;
  int ke, me, nd, k;
  ok = q1x::detShifts(sh.lo[el], sh.hi[el], nd, k) && ok;
  // the coefficient of a single stiffness (mass) operator is folded into its values
  // (their range keeps the products below 2^1023)
  ok = q1x::coefParts(a.fold.coefK ? a.fold.sK * kfac : a.fold.sK, km, ke) && ok;
  ok = q1x::coefParts(a.fold.coefM ? a.fold.sM * kfac : a.fold.sM, mm, me) && ok;
  int const sg = q1x::productShift(sh.ps[el]);
  int const eD = q1x::detExponent(sc, s, nd);
  q1x::limitFactor(mm, me, 60 - eD);
  int const eK = q1x::tensorExponent(sc, scMin, s, k, sg) + ke - 57, eM = eD + me - 60;
  if (x < NQ)
  {
    Sp const wq = q1x::split(gWx[q]);
    if (needK)
    {
      q1x::pointInverse(det, k, sg, q1x::split(q1x::shl(q1x::mul(q1x::split(km), wq), 2)), s, G);
#pragma unroll
      for (int c = 0; c < 6; ++c)
        sh.G[c][q][el] = G[c] >> 1; // F = 57: the entries reach 25 times the largest value
    }
    int64_t const dw = q1x::mul(q1x::split(q1x::shl(q1x::shl(det, nd), 2)), wq); // F = 60
    if (needM)
      sh.G[6][q][el] = q1x::mul(q1x::split(q1x::shl(dw, 2)), q1x::split(mm));
    if (series)
    {
      Sp const u0 = q1x::split(u[0]), u1 = q1x::split(u[1]), u2 = q1x::split(u[2]);
      int64_t f0 = sh.coef[0][deg][el], f1 = sh.coef[1][deg][el], f2 = sh.coef[2][deg][el];
      for (int i = deg - 1; i >= 0; --i)
      {
        f0 = q1x::mulAdd(q1x::split(f0), u0, sh.coef[0][i][el]);
        f1 = q1x::mulAdd(q1x::split(f1), u1, sh.coef[1][i][el]);
        f2 = q1x::mulAdd(q1x::split(f2), u2, sh.coef[2][i][el]);
      }
      int const n0 = q1x::seriesShift(sh.ee[0][el], sh.se[0][el], sh.et[0][el]),
                n1 = q1x::seriesShift(sh.ee[1][el], sh.se[2][el], sh.et[1][el]),
                n2 = q1x::seriesShift(sh.ee[2][el], sh.se[4][el], sh.et[2][el]);
      sh.rq[q][el] = q1x::pointLoad(q1x::shl(f0, n0), q1x::shl(f1, n1), q1x::shl(f2, n2), dw);
      if (q == 0)
        sh.el[el] = sh.ee[0][el] + sh.ee[1][el] + sh.ee[2][el] - (n0 + n1 + n2);
    }
    else if (a.rkind == 1 && !analytic)
      sh.rq[q][el] = dw >> 1;
    else if (a.rkind && ok)
    {
      double p[3] = {0., 0., 0.};
      if (a.rkind == 1)
#pragma unroll
        for (int r = 0; r < 3; ++r)
          p[r] = fma(0.774596669241483, q1x::toDouble(u[r], sc[r] - 61), sh.org[r][el]);
      sh.rq[q][el] =
          __double_as_longlong(a.rc * (q1x::toDoubleFlush(dw, eD - 60) * pointValue(a, sh, el, q, p[0], p[1], p[2])));
    }
  }
  if (tid < E)
    sh.ok[tid] = (ok ? 1u : 0u) | (i0 + tid < a.nelem ? 2u : 0u);
  __syncthreads();

  // ---- 2. the first axis (stride f; s, l the other two): P
  // S_x: y, z, x   S_y: x, z, y   S_z, mass: x, y, z   xy: z, x, y   xz: y, x, z   yz: x, y, z
  for (int k2 = x; k2 < 63; k2 += 32)
  {
    int const T = k2 / 9, r = k2 - 9 * T, q1 = r / 3, q2 = r - 3 * q1;
    if (T == 3 ? !needM : !needK)
      continue;
    int const f = (T == 0 || T == 5) ? 3 : (T == 4 ? 1 : 9), st = T <= 1 ? 1 : ((T == 4 || T == 5) ? 9 : 3),
              lt = T == 0 ? 9 : ((T == 1 || T == 4) ? 3 : 1);
    int64_t const(*in)[E] = sh.G[T < 3 ? T : (T == 3 ? 6 : T - 1)] + q1 * st + q2 * lt;
    int64_t o[6];
    q2x::lineP(in[0][el], in[f][el], in[2 * f][el], o);
#pragma unroll
    for (int c = 0; c < 6; ++c)
      sh.s1[T][c * 9 + r][el] = o[c];
  }
  __syncthreads();
  pdlWait(); // the writes start below

  // ---- 3. the tables S_x, S_y, S_z and mass; the load on the last warp
  if (x < 24)
  {
    int const T = x / 6, c = x - 6 * T;
    if (T < 3)
    {
      if (needK)
        plane<0>(sh.s1[T] + c * 9, sh.row + rowOf(0, x, 0, 0), el);
    }
    else if (needM)
      plane<1>(sh.s1[3] + c * 9, sh.row + rowOf(0, x, 0, 0), el);
  }
  else
  {
    // one line per lane pass: nine lines of four elements, three axes in place; the value
    // index is qx 9 + qy 3 + qz
    bool const mine = sh.ok[el] == 3u, fixedLoad = series || (a.rkind == 1 && !analytic);
    int64_t(*rq)[E] = sh.rq;
    if (a.rkind)
    {
#pragma unroll 1
      for (int ax = 0; ax < 3; ++ax)
      {
        int const f = ax == 0 ? 9 : (ax == 1 ? 3 : 1), g1 = ax == 0 ? 3 : 9, g2 = ax == 2 ? 3 : 1;
        for (int n = x - 24; n < 9; n += 8)
        {
          int const o0 = (n / 3) * g1 + (n % 3) * g2;
          int64_t const v0 = rq[o0][el], v1 = rq[o0 + f][el], v2 = rq[o0 + 2 * f][el];
          if (fixedLoad)
          {
            int64_t o[3];
            q2x::lineL(v0, v1, v2, o);
            rq[o0][el] = o[0], rq[o0 + f][el] = o[1], rq[o0 + 2 * f][el] = o[2];
          }
          else
          {
            double o[3];
            lineLd(__longlong_as_double(v0), __longlong_as_double(v1), __longlong_as_double(v2), o);
            rq[o0][el] = __double_as_longlong(o[0]), rq[o0 + f][el] = __double_as_longlong(o[1]),
            rq[o0 + 2 * f][el] = __double_as_longlong(o[2]);
          }
        }
        __syncwarp();
      }
    }
    if (mine && a.b && (a.rkind || a.fold.bc))
    {
      uint32_t const cons = sh.cons[el];
      int const ex = sine ? eD + sh.el[el] - 59 : eD - 59;
      for (int L = x - 24; L < N; L += 8)
      {
        int const n = gNodeOfLat[L];
        bool const c = (cons >> n) & 1u;
        uint32_t const dof = sh.dof[el][n];
        if (a.rkind && !(a.rbc && c))
          atomicAdd(a.b + dof,
                    fixedLoad ? a.rc * q1x::toDoubleFlush(rq[L][el], ex) : __longlong_as_double(rq[L][el]));
        if (c)
        {
          // buildLhs' Dirichlet values, once per operator with BCs (builder.hpp:119)
          double const h = a.bcVal[dof];
#pragma unroll
          for (int m = 0; m < 2; ++m)
            if (a.op[m].on && a.op[m].bc && h != 0.)
              atomicAdd(a.b + dof, h);
        }
      }
    }
  }
  __syncthreads();
  int64_t kv[kPairsPerLane], mv[kPairsPerLane];
#pragma unroll
  for (int t = 0; t < kPairsPerLane; ++t)
  {
    int const p = x + 32 * t;
    kv[t] = 0, mv[t] = 0;
    if (p < NP)
    {
      ushort4 const r = gPairA[p];
      if (needK)
        kv[t] = sh.row[r.x][el] + sh.row[r.y][el] + sh.row[r.z][el];
      if (needM)
        mv[t] = sh.row[r.w][el];
    }
  }
  __syncthreads();
  // the mixed components
  if (needK)
  {
    if (x < 18)
      plane<2>(sh.s1[4 + x / 6] + (x % 6) * 9, sh.row + rowOf(0, x, 0, 0), el);
    if (x >= 14)
    {
      int const z = x - 14;
      planeA(sh.s1[4 + z / 6] + (z % 6) * 9, sh.row + rowAA(z / 6) + (z % 6) * 9, el);
    }
    if (x == 31)
      sh.row[kZero][el] = 0;
    __syncthreads();
#pragma unroll
    for (int t = 0; t < kPairsPerLane; ++t)
    {
      int const p = x + 32 * t;
      if (p < NP)
      {
        uint4 const r = gPairB[p];
        kv[t] += 2 * (sh.row[r.x & 0xffffu][el] + sh.row[r.x >> 16][el] + sh.row[r.y & 0xffffu][el] +
                      sh.row[r.y >> 16][el] + sh.row[r.z & 0xffffu][el] + sh.row[r.z >> 16][el]);
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int t = 0; t < kPairsPerLane; ++t)
  {
    int const p = x + 32 * t;
    if (p < NP)
    {
      if (needK)
        sh.kd[el][p] = q1x::toDouble(kv[t], eK);
      if (needM)
        sh.md[el][p] = q1x::toDouble(mv[t], eM);
    }
  }
  __syncthreads();

  // ---- 4. scatter: warp w adds element w
  int64_t const ew = element(w);
  uint32_t const okw = sh.ok[w];
  if (okw == 3u && (needK || needM))
  {
    uint16_t const * const rk = a.rank + ew * (N * N);
    uint32_t const cons = a.fold.bc ? sh.cons[w] : 0u;
    if (a.fold.simple && !cons)
    {
#pragma unroll 12
      for (int f = l; f < N * N; f += 32)
      {
        uint32_t const ip = gEntry[f];
        int const p = ip >> 8;
        int32_t const pij = sh.rp[w][ip & 0xffu] + rk[f];
        if (a.fold.same)
          atomicAdd(a.fold.K + pij, sh.kd[w][p] + sh.md[w][p]);
        else
        {
          if (needK)
            atomicAdd(a.fold.K + pij, sh.kd[w][p]);
          if (needM)
            atomicAdd(a.fold.M + pij, sh.md[w][p]);
        }
      }
    }
    else if (a.fold.simple)
    {
      // with the Dirichlet condensation (builder.hpp:76-124): the diagonal of a
      // constrained DOF, the lift -K_ij h_j of a free row
      bool const one = needK && needM && !a.fold.same; // a second operator
#pragma unroll 4
      for (int f = l; f < N * N; f += 32)
      {
        uint32_t const ip = gEntry[f];
        int const i = ip & 0xffu, j = f - i * N, p = ip >> 8;
        int32_t const pij = sh.rp[w][i] + rk[f];
        bool const ci = (cons >> i) & 1u, c = ci || ((cons >> j) & 1u);
        // first operator: K, or K + M in one, or M alone; second: M
        double v0 = needK ? sh.kd[w][p] : sh.md[w][p], v1 = one ? sh.md[w][p] : 0.;
        if (a.fold.same)
          v0 += sh.md[w][p];
        double * const d0 = needK ? a.fold.K : a.fold.M;
        bool const c0 = c && (needK ? a.fold.bcK : a.fold.bcM), c1 = one && c && a.fold.bcM;
        if (!ci && (c0 || c1) && i != j && a.b)
        {
          double const z = ((c0 ? v0 : 0.) + (c1 ? v1 : 0.)) * a.bcVal[sh.dof[w][j]];
          if (z != 0.)
            atomicAdd(a.b + sh.dof[w][i], -z);
        }
        v0 = c0 ? a.bcDiag : v0, v1 = c1 ? a.bcDiag : v1;
        if (!c0 || i == j)
          atomicAdd(d0 + pij, v0);
        if (one && (!c1 || i == j))
          atomicAdd(a.fold.M + pij, v1);
      }
    }
    else
    {
#pragma unroll 1
      for (int f = l; f < N * N; f += 32)
      {
        uint32_t const ip = gEntry[f];
        int const i = ip & 0xffu;
        scatterGeneral(a, sh, w, ew, i, f - i * N, ip >> 8, sh.rp[w][i] + rk[f]);
      }
    }
  }
  // refused elements, each by its warp in FP64
  if (__syncthreads_or(okw == 2u))
    if (okw == 2u)
      elementQ2F64(a, ew, reinterpret_cast<Smem *>(&sh)[w]);
}

// The 1D tables, the lattice maps and the pair list, from the reference's rule and
// basis (the engine's host restatement of src/qr.cpp and src/reffe.cpp).
pxg_status initQ2F64Tables(pxg_ctx * c)
{
  using namespace q2f;
  std::vector<double> xi, w;
  hostRule(Q2HEX, xi, w);
  if ((int)w.size() != NQ)
    return fail(c, PXG_ERR_UNSUPPORTED, "Q2 rule: %d points", (int)w.size());
  // the three 1D points, ascending
  double t[3] = {1e300, 0., -1e300};
  for (int q = 0; q < NQ; ++q)
  {
    t[0] = xi[3 * q] < t[0] ? xi[3 * q] : t[0];
    t[2] = xi[3 * q] > t[2] ? xi[3 * q] : t[2];
  }
  auto idx = [&](double v) { return v == t[0] ? 0 : (v == t[2] ? 2 : 1); };
  t[1] = 0.;
  double wl[NQ];
  uint8_t ruleOfLat[NQ];
  for (int q = 0; q < NQ; ++q)
  {
    int const L = idx(xi[3 * q]) * 9 + idx(xi[3 * q + 1]) * 3 + idx(xi[3 * q + 2]);
    wl[L] = w[q];
    ruleOfLat[L] = (uint8_t)q;
  }
  // 1D functions of src/reffe.cpp:374-383 (index 0: node -1, 1: node +1, 2: node 0)
  auto f = [](int a, double x) { return a == 0 ? 0.5 * x * (x - 1.) : (a == 1 ? 0.5 * x * (x + 1.) : 1. - x * x); };
  auto df = [](int a, double x) { return a == 0 ? x - 0.5 : (a == 1 ? x + 0.5 : -2. * x); };
  int const cls[6][2] = {{0, 0}, {1, 1}, {2, 2}, {0, 1}, {0, 2}, {1, 2}};
  std::vector<double> coef(72);
  for (int a = 0; a < 3; ++a)
    for (int k = 0; k < 3; ++k)
      coef[3 * a + k] = f(a, t[k]);
  for (int cc = 0; cc < 6; ++cc)
    for (int k = 0; k < 3; ++k)
    {
      coef[9 + 3 * cc + k] = f(cls[cc][0], t[k]) * f(cls[cc][1], t[k]);
      coef[27 + 3 * cc + k] = df(cls[cc][0], t[k]) * df(cls[cc][1], t[k]);
    }
  int const anti[3][2] = {{0, 1}, {0, 2}, {1, 2}};
  for (int cc = 0; cc < 6; ++cc)
    for (int k = 0; k < 3; ++k)
    {
      int const a = cls[cc][0], b = cls[cc][1];
      coef[45 + 3 * cc + k] = 0.5 * (df(a, t[k]) * f(b, t[k]) + df(b, t[k]) * f(a, t[k]));
    }
  for (int cc = 0; cc < 3; ++cc)
    for (int k = 0; k < 3; ++k)
    {
      int const a = anti[cc][0], b = anti[cc][1];
      coef[63 + 3 * cc + k] = 0.5 * (df(a, t[k]) * f(b, t[k]) - df(b, t[k]) * f(a, t[k]));
    }
  // node n -> the 1D functions of its three factors: the lattice point where phi_n = 1
  uint8_t latOfNode[N], nodeOfLat[N];
  double const node1d[3] = {-1., 1., 0.};
  for (int L = 0; L < N; ++L)
  {
    double const p[3] = {node1d[L / 9], node1d[(L / 3) % 3], node1d[L % 3]};
    double phi[N], dphi[3 * N];
    hostShape(Q2HEX, p, phi, dphi);
    int found = -1;
    for (int n = 0; n < N; ++n)
      if (phi[n] > 0.5)
        found = n;
    if (found < 0)
      return fail(c, PXG_ERR_UNSUPPORTED, "Q2 node lattice");
    latOfNode[found] = (uint8_t)L;
    nodeOfLat[L] = (uint8_t)found;
  }
  std::vector<uint16_t> pairs;
  for (int i = 0; i < N; ++i)
    for (int j = i; j < N; ++j)
      pairs.push_back((uint16_t)(i << 8 | j));
  // the P, D, S, A classes divided by their first coefficient (the value at t_0, nonzero
  // for every class), and the deferred scale of each stiffness table value: the
  // product of its three classes' first coefficients, in the tables' layouts
  std::vector<double> coefN(coef);
  auto first = [&](int base, int cc) { return coef[base + 3 * cc]; };
  for (int k = 9; k < 72; k += 3)
    if (coef[k] == 0.)
      return fail(c, PXG_ERR_UNSUPPORTED, "Q2 tables: a class vanishes at the first Gauss point");
  for (int base : {9, 27, 45})
    for (int cc = 0; cc < 6; ++cc)
      for (int k = 0; k < 3; ++k)
        coefN[base + 3 * cc + k] = coef[base + 3 * cc + k] / first(base, cc);
  for (int cc = 0; cc < 3; ++cc)
    for (int k = 0; k < 3; ++k)
      coefN[63 + 3 * cc + k] = coef[63 + 3 * cc + k] / first(63, cc);
  std::vector<double> scale(kScales, 0.);
  auto sP = [&](int cc) { return first(9, cc); };
  auto sD = [&](int cc) { return first(27, cc); };
  auto sS = [&](int cc) { return first(45, cc); };
  auto sA = [&](int cc) { return first(63, cc); };
  for (int x = 0; x < 6; ++x)
    for (int y = 0; y < 6; ++y)
      for (int z = 0; z < 6; ++z)
      {
        int const k = x * 36 + y * 6 + z;
        scale[k] = sD(x) * sP(y) * sP(z);
        scale[216 + k] = sP(x) * sD(y) * sP(z);
        scale[432 + k] = sP(x) * sP(y) * sD(z);
      }
  // mixed component m: 2 x SS, and -2 x orientation x AA (index 64 + a: the negative
  // orientation; 54: no AA term, scale 0)
  for (int m = 0; m < 3; ++m)
  {
    int const base = 648 + m * (216 + kAA);
    for (int p = 0; p < 6; ++p)
    {
      for (int s1 = 0; s1 < 6; ++s1)
        for (int s2 = 0; s2 < 6; ++s2)
          scale[base + p * 36 + s1 * 6 + s2] = 2. * sP(p) * sS(s1) * sS(s2);
      for (int a1 = 0; a1 < 3; ++a1)
        for (int a2 = 0; a2 < 3; ++a2)
        {
          double const v = 2. * sP(p) * sA(a1) * sA(a2);
          scale[base + 216 + p * 9 + a1 * 3 + a2] = -v;
          scale[base + 216 + 64 + p * 9 + a1 * 3 + a2] = v;
        }
    }
  }
  PXG_CUDA(c, cudaMemcpyToSymbol(gCoef, coef.data(), 72 * 8));
  PXG_CUDA(c, cudaMemcpyToSymbol(gCoefN, coefN.data(), 72 * 8));
  PXG_CUDA(c, cudaMemcpyToSymbol(gScale, scale.data(), scale.size() * 8));
  PXG_CUDA(c, cudaMemcpyToSymbol(gT, t, 24));
  PXG_CUDA(c, cudaMemcpyToSymbol(gWl, wl, NQ * 8));
  PXG_CUDA(c, cudaMemcpyToSymbol(gRuleOfLat, ruleOfLat, NQ));
  PXG_CUDA(c, cudaMemcpyToSymbol(gLatOfNode, latOfNode, N));
  PXG_CUDA(c, cudaMemcpyToSymbol(gNodeOfLat, nodeOfLat, N));
  PXG_CUDA(c, cudaMemcpyToSymbol(gPairsF, pairs.data(), pairs.size() * 2));
  // each pair's index into the tables: S (and mass) [px][py][pz]; for the mixed
  // components xy, xz, yz the SS tables [pz][sx][sy], [py][sx][sz], [px][sy][sz] (the
  // symmetric classes of the two derivative axes) and the AA tables [pz][ax][ay], ... with
  // the antisymmetric class a + b - 1 of {a, b}, plus 64 when the orientation
  // sign(j_1 - i_1) sign(j_2 - i_2) is negative, and 54 when either axis pair is
  // diagonal (no AA term)
  std::vector<uint16_t> pidx(pairs.size() * 8, 0);
  auto aaIdx = [](int lead, int i1, int j1, int i2, int j2) -> uint16_t {
    if (i1 == j1 || i2 == j2)
      return 54;
    int const v = lead * 9 + (i1 + j1 - 1) * 3 + (i2 + j2 - 1);
    return (uint16_t)(((i1 < j1) == (i2 < j2)) ? v : 64 + v);
  };
  for (size_t q = 0; q < pairs.size(); ++q)
  {
    int const i = pairs[q] >> 8, j = pairs[q] & 0xff;
    int const Li = latOfNode[i], Lj = latOfNode[j];
    int const ix = Li / 9, iy = (Li / 3) % 3, iz = Li % 3, jx = Lj / 9, jy = (Lj / 3) % 3, jz = Lj % 3;
    int const px = symCls(ix, jx), py = symCls(iy, jy), pz = symCls(iz, jz);
    uint16_t * const o = &pidx[8 * q];
    o[0] = (uint16_t)(px * 36 + py * 6 + pz);
    o[1] = (uint16_t)(pz * 36 + px * 6 + py);
    o[2] = aaIdx(pz, ix, jx, iy, jy);
    o[3] = (uint16_t)(py * 36 + px * 6 + pz);
    o[4] = aaIdx(py, ix, jx, iz, jz);
    o[5] = (uint16_t)(px * 36 + py * 6 + pz);
    o[6] = aaIdx(px, iy, jy, iz, jz);
  }
  PXG_CUDA(c, cudaMemcpyToSymbol(gPairIdx, pidx.data(), pidx.size() * 2));
  std::vector<ushort4> pa(pairs.size());
  std::vector<uint4> pb(pairs.size());
  std::vector<uint32_t> entry(N * N);
  for (size_t q = 0; q < pairs.size(); ++q)
  {
    int const i = pairs[q] >> 8, j = pairs[q] & 0xff;
    int const Li = latOfNode[i], Lj = latOfNode[j];
    int const I[3] = {Li / 9, (Li / 3) % 3, Li % 3}, J[3] = {Lj / 9, (Lj / 3) % 3, Lj % 3};
    int const x = symCls(I[0], J[0]), y = symCls(I[1], J[1]), z = symCls(I[2], J[2]);
    pa[q] = make_ushort4((unsigned short)rowOf(0, y, z, x), (unsigned short)rowOf(1, x, z, y),
                         (unsigned short)rowOf(2, x, y, z), (unsigned short)rowOf(3, x, y, z));
    // the term is 2 SS - 2 s s' AA, s the sign of j - i on an axis
    auto anti = [&](int m, int lead, int u, int v) {
      if (I[u] == J[u] || I[v] == J[v])
        return kZero;
      bool const minus = (I[u] < J[u]) == (I[v] < J[v]);
      return rowAA(m) + (minus ? 54 : 0) + lead * 9 + (I[u] + J[u] - 1) * 3 + (I[v] + J[v] - 1);
    };
    auto two = [](int lo, int hi) { return (unsigned)lo | (unsigned)hi << 16; };
    pb[q] = make_uint4(two(rowOf(0, z, x, y), anti(0, z, 0, 1)), two(rowOf(1, y, x, z), anti(1, y, 0, 2)),
                       two(rowOf(2, x, y, z), anti(2, x, 1, 2)), 0u);
    entry[i * N + j] = (uint32_t)i | (uint32_t)q << 8;
    entry[j * N + i] = (uint32_t)j | (uint32_t)q << 8;
  }
  PXG_CUDA(c, cudaMemcpyToSymbol(gPairA, pa.data(), pa.size() * sizeof(ushort4)));
  PXG_CUDA(c, cudaMemcpyToSymbol(gPairB, pb.data(), pb.size() * sizeof(uint4)));
  PXG_CUDA(c, cudaMemcpyToSymbol(gEntry, entry.data(), entry.size() * 4));
  int64_t wx[NQ];
  for (int q = 0; q < NQ; ++q)
    wx[q] = (int64_t)(wl[q] * 4611686018427387904.0); // exact
  PXG_CUDA(c, cudaMemcpyToSymbol(gWx, wx, sizeof(wx)));
  return PXG_OK;
}

void launchAssembleQ2F64(AsmArgs const & args, cudaStream_t s)
{
  if (args.nelem <= 0)
    return;
  AsmArgs a = args;
  foldOps(a);
  launchElemKernel(kAssembleQ2Fx, (unsigned)((a.nelem + q2f::E - 1) / q2f::E), q2f::NT, 0, s, a);
}

} // namespace pxg
