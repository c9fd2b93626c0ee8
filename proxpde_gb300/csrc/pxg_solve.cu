// Device Jacobi-preconditioned CG and the adjoint gradient of the diffusion loss
//   K(k) u = b,   J(u) = 1/2 (u - u_t)^T M (u - u_t),   dJ/d log k_e = -(C u)_e^T K_e (C lambda)_e
// with K lambda = M (u - u_t), K_e = k_e K0_e the element stiffness and C zeroing the
// DOFs constrained by the essential BCs (the derivative of the condensed matrix
// C K C + D is C K0_e C).  proxpde itself solves with UmfPackLU
// (include/sparse_matrix.hpp:44).
//
// The solver is pxg_cg.h's, all rows as one group of blocks, one block per SM.
#include <cub/block/block_reduce.cuh>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "pxg_cg.h"
#include "pxg_internal.h"

namespace pxg
{
namespace
{

constexpr int kTpb = 256;
constexpr int kMaxPartBlocks = 1024;
// what the solver reports
enum : int
{
  S_RR = 0,
  S_BB,
  S_ITER,
  S_COUNT
};

inline int partBlocks(int64_t n)
{
  int64_t b = (n + kTpb - 1) / kTpb;
  return (int)(b < kMaxPartBlocks ? b : kMaxPartBlocks);
}

template <int NV>
__device__ __forceinline__ void blockSum(double (&v)[NV], double * out)
{
  using BR = cub::BlockReduce<double, kTpb>;
  __shared__ typename BR::TempStorage ts;
#pragma unroll
  for (int k = 0; k < NV; ++k)
  {
    double const s = BR(ts).Sum(v[k]);
    if (threadIdx.x == 0)
      out[k] = s;
    __syncthreads();
  }
}

__global__ void __launch_bounds__(kCgT, 1) kCgSolve(CgArgs const __grid_constant__ g, double * scal)
{
  extern __shared__ __align__(16) unsigned char dyn[];
  __shared__ CgShared sh;
  CgTile * const tiles = reinterpret_cast<CgTile *>(dyn);
  double * const vec = reinterpret_cast<double *>(dyn + kCgWarps * sizeof(CgTile));
  int64_t const r0 = cgRowStart(g, blockIdx.x), r1 = cgRowStart(g, blockIdx.x + 1);
  int const nr = (int)(r1 - r0);
  int const mean = nr > 0 ? (int)((g.rp[r1] - g.rp[r0]) / nr) + 1 : 1;
  cgLanes(nr, mean, [&](auto lanes) {
    CgCount count;
    CgResult res;
    if (cgRun<decltype(lanes)::value>(g, sh, tiles, vec, r0, nr, count, res) && blockIdx.x == 0 && threadIdx.x == 0)
    {
      scal[S_RR] = res.rr;
      scal[S_BB] = res.bb;
      scal[S_ITER] = res.it;
    }
  });
}

// y = A x and the dot x^T y (deterministic), for the loss
__global__ void __launch_bounds__(kTpb) kSpmvPlainDot(int32_t const * __restrict__ rp, int32_t const * __restrict__ ci,
                                                      double const * __restrict__ a, double const * __restrict__ x,
                                                      int64_t n, double * __restrict__ y, double * __restrict__ part)
{
  double acc[1] = {0.};
  constexpr int RPW = 32 / kLpr;
  int64_t const warps = (int64_t)gridDim.x * (blockDim.x / 32);
  int64_t const w = (int64_t)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
  int const lane = threadIdx.x & 31;
  for (int64_t r0 = w * RPW; r0 < n; r0 += warps * RPW)
  {
    int64_t const row = r0 + lane / kLpr;
    bool const valid = row < n;
    double const t = rowDot<>(rp, ci, a, x, row, valid);
    if (valid && (lane & (kLpr - 1)) == 0)
    {
      y[row] = t;
      acc[0] += x[row] * t;
    }
  }
  blockSum<1>(acc, part + blockIdx.x);
}

__global__ void kSub(double const * __restrict__ a, double const * __restrict__ b, int64_t n, double * __restrict__ c)
{
  int64_t const i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n)
    c[i] = a[i] - b[i];
}

__global__ void kScale(double * __restrict__ v, int64_t n, double s)
{
  int64_t const i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n)
    v[i] *= s;
}

} // namespace

// ------------------------------------------------------------------ CG driver
pxg_status cgSolve(pxg_ctx * c, int32_t const * rp, int32_t const * ci, double const * a, int64_t n,
                   double const * b, double * x, double rtol, int maxIter, int * itersOut, double * relOut,
                   cudaStream_t user)
{
  CgWork & w = c->cg;
  if (w.n < n)
  {
    PXG_CUDA(c, w.r.alloc(n));
    PXG_CUDA(c, w.z.alloc(n));
    PXG_CUDA(c, w.p.alloc(n));
    PXG_CUDA(c, w.dinv.alloc(n));
    PXG_CUDA(c, w.part.alloc(6 * c->sms));
    PXG_CUDA(c, w.scal.alloc(S_COUNT + 1)); // and the barrier's two counters
    w.n = n;
  }
  if (!w.stream)
    PXG_CUDA(c, cudaStreamCreateWithFlags(&w.stream, cudaStreamNonBlocking));
  if (!w.evIn)
  {
    PXG_CUDA(c, cudaEventCreateWithFlags(&w.evIn, cudaEventDisableTiming));
    PXG_CUDA(c, cudaEventCreateWithFlags(&w.evOut, cudaEventDisableTiming));
  }
  cudaStream_t const s = w.stream;
  PXG_CUDA(c, cudaEventRecord(w.evIn, user));
  PXG_CUDA(c, cudaStreamWaitEvent(s, w.evIn, 0));
  // one block per SM, at least 192 rows (six warps) each: fewer blocks exchange faster, more have
  // less work.  An iteration with 128, 192, 256, 384 rows, us: Q1 12^3 10.6, 10.4, 10.9, 12.2, 24^3
  // 12.6, 12.0, 12.1, 13.3, 30^3 13.1, 13.1, 14.2, 13.9; P1 24^3 x 6 11.6, 10.9, 11.2, 12.1.  The longer
  // rows of Q2 (64 entries) are faster with 128: 12^3 16.7, 18.6, 23.8, 26.1
  int64_t const grid = std::min<int64_t>(c->sms, (n + 191) / 192);
  cudaFuncAttributes fa;
  PXG_CUDA(c, cudaFuncGetAttributes(&fa, kCgSolve));
  int optin = 0;
  PXG_CUDA(c, cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, c->device));
  int const most = optin - (int)fa.sharedSizeBytes, tiles = kCgWarps * (int)sizeof(CgTile);
  PXG_CUDA(c, cudaFuncSetAttribute(kCgSolve, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
  // the vectors' shares in shared memory where all four fit beside the tiles (with room for
  // uneven shares); elsewhere that memory is better used as L1
  int64_t const rows = (n + grid - 1) / grid + (n + grid - 1) / grid / 4 + 64;
  int64_t const vec = rows * 4 * (int64_t)sizeof(double);
  int const cap = tiles + vec <= most ? (int)rows : 0, smem = tiles + (cap ? (int)vec : 0);
  int const aligned = ((uintptr_t)a | (uintptr_t)ci) % 16 == 0;
  unsigned * const counters = reinterpret_cast<unsigned *>(w.scal.p + S_COUNT);
  double * scal = w.scal.p;
  CgArgs g{rp, ci, a, b, x, w.p.p, w.r.p, w.z.p, w.dinv.p, reinterpret_cast<ulonglong2 *>(w.part.p), counters,
           counters + 1, 0, n, 0u, (unsigned)grid, barrierShortfall(), rtol * rtol, maxIter, cap, aligned, nullptr, 0};
  void * args[] = {&g, &scal};
  PXG_CUDA(c, cudaMemsetAsync(w.part.p, 0, 6 * grid * sizeof(double), s)); // no sum has the tag 0
  PXG_CUDA(c, cudaMemsetAsync(w.scal.p, 0, (S_COUNT + 1) * sizeof(double), s));
  PXG_CUDA(c, cudaLaunchCooperativeKernel((void const *)kCgSolve, dim3((unsigned)grid), dim3(kCgT), args, smem, s));
  double h[S_COUNT + 1];
  PXG_CUDA(c, cudaMemcpyAsync(h, w.scal.p, sizeof(h), cudaMemcpyDeviceToHost, s));
  PXG_CUDA(c, cudaStreamSynchronize(s));
  unsigned bar[2];
  std::memcpy(bar, &h[S_COUNT], sizeof(bar));
  if (bar[1])
    return fail(c, PXG_ERR_TIMEOUT, "CG: a grid barrier wait ran out");
  PXG_CUDA(c, cudaEventRecord(w.evOut, s));
  PXG_CUDA(c, cudaStreamWaitEvent(user, w.evOut, 0));
  double const rel = h[S_BB] > 0. ? std::sqrt(h[S_RR] / h[S_BB]) : 0.;
  if (itersOut)
    *itersOut = (int)h[S_ITER];
  if (relOut)
    *relOut = rel;
  if (!(rel <= rtol))
    return fail(c, PXG_ERR_NOT_CONVERGED, "CG stopped after %d iterations at relative residual %.3e (tol %.1e)",
                (int)h[S_ITER], rel, rtol);
  return PXG_OK;
}

} // namespace pxg

using namespace pxg;

extern "C"
{

pxg_status pxg_cg(pxg_ctx * c, int32_t const * row_ptr, int32_t const * col_idx, double const * vals, int64_t n,
                  double const * b, double * x, double rtol, int max_iter, int * iters, double * rel_res,
                  void * stream)
{
  if (!c || !row_ptr || !col_idx || !vals || !b || !x || n <= 0 || !(rtol > 0.) || max_iter <= 0)
    return c ? fail(c, PXG_ERR_INVALID_ARG, "pxg_cg: bad argument") : PXG_ERR_INVALID_ARG;
  pxg_status st = ensureDevice(c);
  if (st != PXG_OK)
    return st;
  return cgSolve(c, row_ptr, col_idx, vals, n, b, x, rtol, max_iter, iters, rel_res, (cudaStream_t)stream);
}

pxg_status pxg_adjoint_grad(pxg_ctx * c, double const * u, double const * lambda, double * g, void * stream)
{
  if (!c || !u || !lambda || !g)
    return PXG_ERR_INVALID_ARG;
  if (!c->emap.p || !c->hasCoef)
    return fail(c, PXG_ERR_INVALID_ARG, "adjoint gradient needs the DOF map and the coefficient");
  pxg_status st = ensureDevice(c);
  if (st != PXG_OK)
    return st;
  return launchAdjointGrad(c, u, lambda, g, (cudaStream_t)stream);
}

pxg_status pxg_adjoint_forward(pxg_ctx * c, pxg_rhs_op const * rhs, double const * u_target, double rtol,
                               int max_iter, double * u_out, double * loss, int * iters, void * stream)
{
  if (!c || !rhs || !u_target || !loss)
    return PXG_ERR_INVALID_ARG;
  if (!c->rowPtr.p || !c->hasCoef)
    return fail(c, PXG_ERR_INVALID_ARG, "forward needs the pattern and the coefficient");
  pxg_status st = ensureDevice(c);
  if (st != PXG_OK)
    return st;
  cudaStream_t const s = (cudaStream_t)stream;
  AdjState & A = c->adj;
  int64_t const n = c->ndof, nnz = c->nnz;
  if (A.n != n || A.nnz != nnz)
  {
    PXG_CUDA(c, A.K.alloc(nnz));
    PXG_CUDA(c, A.M.alloc(nnz));
    PXG_CUDA(c, A.b.alloc(n));
    PXG_CUDA(c, A.u.alloc(n));
    PXG_CUDA(c, A.w.alloc(n));
    PXG_CUDA(c, A.Mw.alloc(n));
    PXG_CUDA(c, A.lam.alloc(n));
    PXG_CUDA(c, A.part.alloc(kMaxPartBlocks));
    A.n = n;
    A.nnz = nnz;
  }
  A.valid = false;
  // K(k) with BCs, M without, b = rhs with BCs (and the BC lift of K)
  pxg_lhs_op const opK{2, 1.0, 0, 0.0, 1};
  pxg_lhs_op const opM{0, 0.0, 1, 1.0, 0};
  pxg_rhs_op r = *rhs;
  r.apply_bc = 1;
  if ((st = pxg_assemble(c, &opK, A.K.p, &opM, A.M.p, &r, A.b.p, 0u, stream)) != PXG_OK)
    return st;
  if ((st = cgSolve(c, c->rowPtr.p, c->colIdx.p, A.K.p, n, A.b.p, A.u.p, rtol, max_iter, iters, nullptr, s)) !=
      PXG_OK)
    return st;
  unsigned const blocks = (unsigned)((n + kTpb - 1) / kTpb);
  kSub<<<blocks, kTpb, 0, s>>>(A.u.p, u_target, n, A.w.p);
  int const nb = partBlocks(n);
  kSpmvPlainDot<<<nb, kTpb, 0, s>>>(c->rowPtr.p, c->colIdx.p, A.M.p, A.w.p, n, A.Mw.p, A.part.p);
  PXG_CUDA(c, cudaGetLastError());
  std::vector<double> hp(nb);
  PXG_CUDA(c, cudaMemcpyAsync(hp.data(), A.part.p, nb * sizeof(double), cudaMemcpyDeviceToHost, s));
  PXG_CUDA(c, cudaStreamSynchronize(s));
  double J = 0.;
  for (double v : hp)
    J += v;
  *loss = 0.5 * J;
  if (u_out)
    PXG_CUDA(c, cudaMemcpyAsync(u_out, A.u.p, n * sizeof(double), cudaMemcpyDeviceToDevice, s));
  A.rtol = rtol;
  A.maxIter = max_iter;
  A.valid = true;
  return PXG_OK;
}

pxg_status pxg_adjoint_backward(pxg_ctx * c, double dloss, double * grad, double * lambda_out, int * iters,
                                void * stream)
{
  if (!c || !grad)
    return PXG_ERR_INVALID_ARG;
  AdjState & A = c->adj;
  if (!A.valid)
    return fail(c, PXG_ERR_INVALID_ARG, "pxg_adjoint_backward needs a preceding pxg_adjoint_forward");
  pxg_status st = ensureDevice(c);
  if (st != PXG_OK)
    return st;
  cudaStream_t const s = (cudaStream_t)stream;
  // K lambda = M (u - u_t)  (K symmetric)
  if ((st = cgSolve(c, c->rowPtr.p, c->colIdx.p, A.K.p, A.n, A.Mw.p, A.lam.p, A.rtol, A.maxIter, iters, nullptr,
                    s)) != PXG_OK)
    return st;
  if ((st = launchAdjointGrad(c, A.u.p, A.lam.p, grad, s)) != PXG_OK)
    return st;
  if (dloss != 1.0)
    kScale<<<(unsigned)((c->nelem + kTpb - 1) / kTpb), kTpb, 0, s>>>(grad, c->nelem, dloss);
  if (lambda_out)
    PXG_CUDA(c, cudaMemcpyAsync(lambda_out, A.lam.p, A.n * sizeof(double), cudaMemcpyDeviceToDevice, s));
  PXG_CUDA(c, cudaGetLastError());
  return PXG_OK;
}

} // extern "C"
