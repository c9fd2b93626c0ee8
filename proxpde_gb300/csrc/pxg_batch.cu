// Batched adjoint gradients: many independent problems assembled, solved and
// differentiated together.
//
// A batch is the disjoint union of the problems of one element type, given to a
// context as one mesh whose elements are grouped by problem.  proxpde's first-touch
// numbering (include/dof.hpp:111-329) over such a union gives every problem a
// contiguous DOF range, and the union's pattern is block diagonal, so assembly and
// the gradient kernel need nothing new: one launch covers every problem.
//
// kBatchSolve is one persistent cooperative kernel, a block per SM, whose blocks are dealt
// to the problems in groups: for every problem a group runs Jacobi-CG (pxg_cg.h) on
// K u = b, forms J_p = 1/2 (u - u_t)^T M (u - u_t) and M (u - u_t), and runs the adjoint
// CG K lambda = M (u - u_t).  Only a group's blocks wait for one another, each problem
// stops at its own tolerance, and the groups are sized and fed so that they end about
// together (planBatch).  Waits are bounded: when
// one exceeds its limit the kernel sets an error flag and every block returns
// (PXG_ERR_TIMEOUT on the host).
// Before, all blocks went through all problems' rows with three grid barriers per
// iteration: 70 us each, whatever the batch's size (12 + 12 cubes of 8 .. 28: 16.7 ms,
// now 7.9 ms; 64 + 64 cubes of 8 .. 40: 108 ms, now 77 ms; 128 + 128 of 8 .. 48: 333 ms,
// now 286 ms, and 424 ms with a group for every problem that one block is too slow for).
// pxg_batch_adjoint captures the assembly, the persistent solve and the gradient
// kernels in one CUDA graph and replays it.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cmath>
#include <cstring>
#include <functional>
#include <queue>
#include <vector>

#include "pxg_cg.h"
#include "pxg_internal.h"

namespace pxg
{
namespace
{

struct SysDev
{
  int32_t const * rp;
  int32_t const * ci;
  double const * K;
  double const * M;
  double const * b;
  double const * ut;
  double * u;
  double * lam;
  double * r;
  double * z;
  double * p;
  double * dinv;
  double * w;
  double * Mw;
};

struct Problem
{
  int64_t row0, rows;
  int sys;
  int out; // place of its results
};

// a block's group (first block and size) and its problems: list entries beg .. end, taken one by
// one where queue < 0, or by the next free group of those that share the queue
struct Group
{
  int first, blocks;
  int beg, end;
  int queue;
};

struct BatchResult
{
  double J;
  int itF, itA; // iterations; the limit for a solve that did not converge
};

struct BatchDev
{
  SysDev sys[2];
  Group const * group; // [blocks], and the list entries that single warps solve
  Problem const * prob;
  BatchResult * res;
  ulonglong2 * part; // [3 * blocks]
  unsigned * bar;    // [blocks]
  unsigned * err;
  int * next;     // [0] entries of the shared queue taken; [1 + block] the entry its group takes;
                  // [1 + blocks] the warps' entries taken
  unsigned extra; // arrivals expected beyond a group (0; > 0 only to test the timeout path)
  double tol2;
  int maxIter;
  int cap;
  // optional timeline (PXG_BATCH_TRACE) of the first problem of block 0's group, a half per solve
  unsigned long long * trace;
  int traceCap;
};

// u, J, M (u - u_t) and lambda of one problem; false once a wait ran out
template <int LPR>
__device__ __forceinline__ bool batchProblem(BatchDev const & d, SysDev const & s, BatchResult & out, CgArgs & g,
                                             CgShared & sh, CgTile * tiles, double * vec, int64_t r0, int nr,
                                             CgCount & count)
{
  BatchResult res{0., 0, 0};
#pragma unroll 1
  for (int dir = 0; dir < 2; ++dir)
  {
    g.a = s.K;
    g.p = s.p;
    g.b = dir ? s.Mw : s.b;
    g.x = dir ? s.lam : s.u;
    CgResult c;
    if (!cgRun<LPR>(g, sh, tiles, vec, r0, nr, count, c))
      return false;
    int const it = c.bb == 0. || c.rr <= d.tol2 * c.bb ? c.it : d.maxIter;
    (dir ? res.itA : res.itF) = it;
    if (dir == 0)
    {
      for (int v = threadIdx.x; v < nr; v += kCgT)
        s.w[r0 + v] = s.u[r0 + v] - s.ut[r0 + v];
      if (!cgBarrier(g, sh, ++count.epoch))
        return false;
      g.a = s.M;
      g.p = s.w;
      CgRows<LPR> rows(tiles, r0, nr);
      rows.start(g);
      double const wMw[1] = {rows.product(g, s.Mw + r0)};
      if (!cgSum<1>(g, sh, ++count.tag, wMw, 1.))
        return false;
      res.J = 0.5 * sh.out[0];
      if (g.trace)
        g.trace += d.traceCap / 2;
    }
  }
  if (g.rank() == 0 && threadIdx.x == 0)
    out = res;
  return true;
}

// Small problems, where there are many: a warp each, its vectors in the place of its tile.  A block
// takes some 24 us for a problem of eight rows, most of it barriers and the latency of a few rows
// (a call on 20,000 cubes of one element: 3.2 ms, 1.35 here; 4,000 of one or two a side 0.89 and 0.40).
constexpr int kWarpRows = 64;
struct WarpVec
{
  double x[kWarpRows], r[kWarpRows], z[kWarpRows], p[kWarpRows], q[kWarpRows], di[kWarpRows];
};
static_assert(sizeof(WarpVec) <= sizeof(CgTile), "a warp's vectors in its tile");

__device__ __forceinline__ double warpAll(double v)
{
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
// q = A v on the problem's rows (a row per lane); returns v.q
__device__ __forceinline__ double warpProduct(SysDev const & s, Problem const & pr, double const * a,
                                              double const * v, double * q)
{
  double dot = 0.;
  for (int i = threadIdx.x & 31; i < (int)pr.rows; i += 32)
  {
    double t = 0.;
    for (int32_t k = s.rp[pr.row0 + i], e = s.rp[pr.row0 + i + 1]; k < e; ++k)
      t = fma(a[k], v[s.ci[k] - (int)pr.row0], t);
    q[i] = t;
    dot += v[i] * t;
  }
  __syncwarp();
  return warpAll(dot);
}
// the CG of cgRun on v.r = b; the iterations as batchProblem counts them
__device__ __forceinline__ int warpCg(BatchDev const & d, SysDev const & s, Problem const & pr, WarpVec & v)
{
  int const lane = threadIdx.x & 31, n = (int)pr.rows;
  double rz = 0., rr = 0.;
  for (int i = lane; i < n; i += 32)
  {
    double const b = v.r[i], z = v.di[i] * b;
    v.x[i] = 0.;
    v.p[i] = z;
    rz += b * z;
    rr += b * b;
  }
  rz = warpAll(rz);
  rr = warpAll(rr);
  __syncwarp();
  double const bb = rr;
  if (bb == 0.)
    return 0;
  for (int it = 1;; ++it)
  {
    double const al = rz / warpProduct(s, pr, s.K, v.p, v.q);
    double rz1 = 0.;
    rr = 0.;
    for (int i = lane; i < n; i += 32)
    {
      v.x[i] += al * v.p[i];
      double const r = v.r[i] - al * v.q[i], z = v.di[i] * r;
      v.r[i] = r;
      v.z[i] = z;
      rz1 += r * z;
      rr += r * r;
    }
    rz1 = warpAll(rz1);
    rr = warpAll(rr);
    if (rr <= d.tol2 * bb)
      return it;
    if (it >= d.maxIter || !(rr == rr))
      return d.maxIter;
    double const be = rz1 / rz;
    rz = rz1;
    for (int i = lane; i < n; i += 32)
      v.p[i] = v.z[i] + be * v.p[i];
    __syncwarp();
  }
}
__device__ __noinline__ void warpProblem(BatchDev const & d, Problem const & pr, WarpVec & v)
{
  SysDev const & s = d.sys[pr.sys];
  int const lane = threadIdx.x & 31, n = (int)pr.rows;
  BatchResult res{0., 0, 0};
  for (int i = lane; i < n; i += 32)
  {
    double di = 0.;
    for (int32_t k = s.rp[pr.row0 + i]; k < s.rp[pr.row0 + i + 1]; ++k)
      if (s.ci[k] == (int32_t)(pr.row0 + i))
        di = s.K[k];
    v.di[i] = di != 0. ? 1.0 / di : 1.0;
    v.r[i] = s.b[pr.row0 + i];
  }
  __syncwarp();
  res.itF = warpCg(d, s, pr, v);
  for (int i = lane; i < n; i += 32)
  {
    s.u[pr.row0 + i] = v.x[i];
    v.p[i] = v.x[i] - s.ut[pr.row0 + i];
  }
  __syncwarp();
  res.J = 0.5 * warpProduct(s, pr, s.M, v.p, v.r); // the right hand side of the adjoint
  res.itA = warpCg(d, s, pr, v);
  for (int i = lane; i < n; i += 32)
    s.lam[pr.row0 + i] = v.x[i];
  if (lane == 0)
    d.res[pr.out] = res;
  __syncwarp();
}

__global__ void __launch_bounds__(kCgT, 1) kBatchSolve(BatchDev const __grid_constant__ d)
{
  extern __shared__ __align__(16) unsigned char dyn[];
  __shared__ CgShared sh;
  CgTile * const tiles = reinterpret_cast<CgTile *>(dyn);
  double * const vec = reinterpret_cast<double *>(dyn + kCgWarps * sizeof(CgTile));
  Group const grp = d.group[blockIdx.x];
  CgCount count;
  // the entry that the group takes next; the other blocks learn it past the barrier, which also
  // keeps the next problem's sums from the words of this one's last
  auto take = [&](int i) {
    CgArgs g{};
    g.bar = d.bar + grp.first, g.err = d.err, g.block0 = grp.first, g.blocks = grp.blocks, g.extra = d.extra;
    if (grp.queue >= 0 && g.rank() == 0 && threadIdx.x == 0)
      __stcg(d.next + 1 + grp.first, grp.beg + atomicAdd(d.next, 1));
    if (!cgBarrier(g, sh, ++count.epoch))
      return grp.end;
    return grp.queue >= 0 ? __ldcg(d.next + 1 + grp.first) : i;
  };
  for (int i = take(grp.beg); i < grp.end; i = take(i + 1))
  {
    Problem const pr = d.prob[i];
    SysDev const & s = d.sys[pr.sys];
    bool const traced = d.trace && grp.first == 0 && i == 0;
    CgArgs g{s.rp, s.ci, s.K, s.b, s.u, s.p, s.r, s.z, s.dinv, d.part + 3 * grp.first, d.bar + grp.first, d.err,
             pr.row0, pr.rows, (unsigned)grp.first, (unsigned)grp.blocks, d.extra, d.tol2, d.maxIter, d.cap, 1,
             traced ? d.trace : nullptr, d.traceCap / 2};
    int64_t const r0 = cgRowStart(g, g.rank()), r1 = cgRowStart(g, g.rank() + 1);
    int const nr = (int)(r1 - r0);
    int const mean = nr > 0 ? (int)((s.rp[r1] - s.rp[r0]) / nr) + 1 : 1;
    bool ok = false;
    cgLanes(nr, mean, [&](auto lanes) {
      ok = batchProblem<decltype(lanes)::value>(d, s, d.res[pr.out], g, sh, tiles, vec, r0, nr, count);
    });
    if (!ok)
      return;
  }
  Group const small = d.group[gridDim.x];
  __syncthreads(); // the tiles are free
  for (;;)
  {
    int i = 0;
    if ((threadIdx.x & 31) == 0)
      i = small.beg < small.end ? small.beg + atomicAdd(d.next + 1 + gridDim.x, 1) : small.end;
    i = __shfl_sync(0xffffffffu, i, 0);
    if (i >= small.end)
      return;
    warpProblem(d, d.prob[i], *reinterpret_cast<WarpVec *>(tiles + threadIdx.x / 32));
  }
}

// Deals `blocks` blocks to the problems so that all end together, by the time an iteration takes: a
// block's FP64 operations (0.33 ns per entry of its rows, eight more per row) and the exchanges (4
// us in one block, 8 us in a few, 12 us in all), and iterations in proportion to the cube root of
// the rows.  Two kinds of plan, the shorter one is taken:
//  - few problems: the least end time for which the blocks suffice (bisection); a problem that
//    one block cannot solve in that time gets a group of its own, the others go, longest first,
//    to single blocks as these become free;
//  - many problems: groups of one size, which take the problems, longest first, as they become
//    free (groups of whole blocks per problem waste up to half of the last block each).
// Returns the largest share of rows.
int64_t planGroups(std::vector<Problem> & prob, std::vector<double> const & entries, int blocks,
                   std::vector<Group> & group)
{
  size_t const n = prob.size();
  if (n == 0)
  {
    for (int k = 0; k < blocks; ++k)
      group.push_back(Group{k, 1, 0, 0, -1});
    return 1;
  }
  std::vector<double> its(n), work(n);
  double lo = 0., hi = 0.;
  auto exchange = [](int b) { return b == 1 ? 4. : 7.5 + 0.6 * std::log2((double)b); };
  for (size_t p = 0; p < n; ++p)
  {
    its[p] = std::cbrt((double)prob[p].rows);
    work[p] = 0.33e-3 * (entries[p] + 8. * (double)prob[p].rows);
    hi += its[p] * (work[p] + 4.);
  }
  // blocks of problem p for the end time t (one: it may share); a share has at least 128 rows (a single
  // solve's 192 is within 5 % of it)
  auto need = [&](size_t p, double t) {
    if (its[p] * (work[p] + 4.) <= t)
      return 1;
    double const left = t / its[p] - 11.;
    double const most = (double)std::min<int64_t>(blocks, (prob[p].rows + 127) / 128);
    return left > 0. && work[p] / left <= most ? std::max(2, (int)std::ceil(work[p] / left)) : blocks + 1;
  };
  for (int k = 0; k < 40; ++k)
  {
    double const t = 0.5 * (lo + hi);
    double single = 0.;
    int64_t many = 0;
    for (size_t p = 0; p < n; ++p)
    {
      int const b = need(p, t);
      if (b == 1)
        single += its[p] * (work[p] + 4.);
      else
        many += b;
    }
    (many + (int64_t)std::ceil(single / t) <= blocks ? hi : lo) = t;
  }
  std::vector<size_t> order(n);
  for (size_t p = 0; p < n; ++p)
    order[p] = p;
  std::sort(order.begin(), order.end(), [&](size_t a, size_t b) { return its[a] * work[a] > its[b] * work[b]; });
  // groups of one size: the end time of a greedy deal, longest first
  int size = 0;
  for (int b = 1; b <= blocks / 2; b = b < 4 ? b + 1 : b + b / 4)
  {
    std::priority_queue<double, std::vector<double>, std::greater<double>> busy;
    for (int g = 0; g < blocks / b; ++g)
      busy.push(0.);
    double end = 0.;
    for (size_t p : order)
    {
      double const t = busy.top() + its[p] * (work[p] / b + exchange(b));
      busy.pop();
      busy.push(t);
      end = std::max(end, t);
    }
    if (end < hi)
    {
      hi = end;
      size = b;
    }
  }
  group.assign(blocks, Group{0, 1, 0, 0, -1});
  std::vector<Problem> list;
  int64_t share = 0;
  int used = 0;
  if (size == 0)
    for (size_t p : order)
    {
      int const b = need(p, hi);
      if (b == 1)
        continue;
      for (int k = 0; k < b; ++k)
        group[used + k] = Group{used, b, (int)list.size(), (int)list.size() + 1, -1};
      list.push_back(prob[p]);
      used += b;
      share = std::max(share, (prob[p].rows + b - 1) / b);
    }
  int const b = std::max(size, 1), beg = (int)list.size();
  for (size_t p : order)
    if (size > 0 || need(p, hi) == 1)
    {
      list.push_back(prob[p]);
      share = std::max(share, (prob[p].rows + b - 1) / b);
    }
  for (; used + b <= blocks; used += b)
    for (int k = 0; k < b; ++k)
      group[used + k] = Group{used, b, beg, (int)list.size(), 0};
  for (; used < blocks; ++used)
    group[used] = Group{used, 1, 0, 0, -1};
  prob = list;
  return share;
}

// The whole plan: groups for the larger problems, and a last entry of `group` for those that single
// warps take: the problems of up to kWarpRows rows, where these are more than two per block (fewer
// are done sooner by a block each).
int64_t planBatch(std::vector<Problem> & prob, std::vector<double> const & entries, int blocks,
                  std::vector<Group> & group)
{
  std::vector<Problem> large, small;
  std::vector<double> e;
  for (size_t p = 0; p < prob.size(); ++p)
    if (prob[p].rows <= kWarpRows)
      small.push_back(prob[p]);
  bool const warps = small.size() > 2 * (size_t)blocks;
  if (!warps)
    small.clear();
  for (size_t p = 0; p < prob.size(); ++p)
    if (!warps || prob[p].rows > kWarpRows)
    {
      large.push_back(prob[p]);
      e.push_back(entries[p]);
    }
  int64_t const share = planGroups(large, e, blocks, group);
  group.push_back(Group{0, 0, (int)large.size(), (int)(large.size() + small.size()), -1});
  prob = large;
  prob.insert(prob.end(), small.begin(), small.end());
  return share;
}

// DOF range of problem p: from the DOF of its first element's first slot (the first
// DOF it touches) to the next problem's
__global__ void kDofOff(uint32_t const * __restrict__ emap, int64_t const * __restrict__ elemOff, int nprob, int N,
                        int64_t ndof, int64_t * __restrict__ dofOff)
{
  int const p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p > nprob)
    return;
  dofOff[p] = (p == nprob) ? ndof : (int64_t)emap[elemOff[p] * N];
}

} // namespace
} // namespace pxg

using namespace pxg;

extern "C"
{

pxg_status pxg_batch_set(pxg_ctx * c, int64_t const * elem_offsets, int64_t nprob)
{
  if (!c || !elem_offsets || nprob <= 0)
    return PXG_ERR_INVALID_ARG;
  if (!c->rowPtr.p)
    return fail(c, PXG_ERR_INVALID_ARG, "build the pattern of the union mesh first");
  if (elem_offsets[0] != 0 || elem_offsets[nprob] != c->nelem)
    return fail(c, PXG_ERR_INVALID_ARG, "element offsets must run from 0 to nelem");
  for (int64_t p = 0; p < nprob; ++p)
    if (elem_offsets[p + 1] <= elem_offsets[p])
      return fail(c, PXG_ERR_INVALID_ARG, "problem %lld has no element", (long long)p);
  pxg_status st = ensureDevice(c);
  if (st != PXG_OK)
    return st;
  BatchState & B = c->batch;
  int64_t const n = c->ndof, nnz = c->nnz;
  B.ready = false;
  ++B.set;
  B.nprob = nprob;
  PXG_CUDA(c, B.elemOff.alloc(nprob + 1));
  PXG_CUDA(c, B.dofOff.alloc(nprob + 1));
  PXG_CUDA(c, cudaMemcpy(B.elemOff.p, elem_offsets, (nprob + 1) * 8, cudaMemcpyHostToDevice));
  kDofOff<<<(unsigned)((nprob + 1 + 255) / 256), 256>>>(c->emap.p, B.elemOff.p, (int)nprob, c->N, n, B.dofOff.p);
  PXG_CUDA(c, cudaGetLastError());
  // the DOF ranges must be contiguous and increasing (elements grouped by problem, no
  // node shared between problems)
  std::vector<int64_t> h(nprob + 1);
  PXG_CUDA(c, cudaMemcpy(h.data(), B.dofOff.p, (nprob + 1) * 8, cudaMemcpyDeviceToHost));
  for (int64_t p = 0; p < nprob; ++p)
    if (h[p + 1] <= h[p])
      return fail(c, PXG_ERR_INVALID_ARG, "problems share DOFs or are not grouped (problem %lld)", (long long)p);
  B.dofOffHost = h;
  for (DevBuf<double> * v : {&B.K, &B.M})
    PXG_CUDA(c, v->alloc(nnz));
  for (DevBuf<double> * v : {&B.b, &B.u, &B.lam, &B.r, &B.z, &B.p, &B.dinv, &B.w, &B.Mw})
    PXG_CUDA(c, v->alloc(n));
  B.ready = true;
  return PXG_OK;
}

pxg_status pxg_batch_adjoint(pxg_ctx * const * ctxs, int nctx, pxg_rhs_op const * rhs,
                             double const * const * u_targets, double rtol, int max_iter, double * losses,
                             double * const * grads, int * iters, int use_graph, void * stream)
{
  if (!ctxs || nctx < 1 || nctx > 2 || !rhs || !u_targets || !losses || !grads || !(rtol > 0.) || max_iter <= 0)
    return PXG_ERR_INVALID_ARG;
  pxg_ctx * c0 = ctxs[0];
  for (int i = 0; i < nctx; ++i)
  {
    if (!ctxs[i] || !ctxs[i]->batch.ready || !ctxs[i]->hasCoef || !u_targets[i] || !grads[i])
      return ctxs[i] ? fail(ctxs[i], PXG_ERR_INVALID_ARG, "batch %d: pxg_batch_set, the coefficient, the target "
                                                            "and the gradient output are required", i)
                     : PXG_ERR_INVALID_ARG;
    if (ctxs[i]->device != c0->device)
      return fail(c0, PXG_ERR_INVALID_ARG, "batches must live on one GPU");
  }
  pxg_status st = ensureDevice(c0);
  if (st != PXG_OK)
    return st;
  BatchShared & S = c0->bshared;
  int nprob = 0;
  for (int i = 0; i < nctx; ++i)
    nprob += (int)ctxs[i]->batch.nprob;
  int dev = c0->device, sms = 0, perSm = 0, optin = 0;
  PXG_CUDA(c0, cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  PXG_CUDA(c0, cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  cudaFuncAttributes fa;
  PXG_CUDA(c0, cudaFuncGetAttributes(&fa, kBatchSolve));
  int const most = optin - (int)fa.sharedSizeBytes, tiles = kCgWarps * (int)sizeof(CgTile), blocks = sms;
  PXG_CUDA(c0, cudaFuncSetAttribute(kBatchSolve, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
  std::vector<Problem> prob;
  std::vector<double> entries;
  for (int i = 0; i < nctx; ++i)
  {
    std::vector<int64_t> const & off = ctxs[i]->batch.dofOffHost;
    double const mean = (double)ctxs[i]->nnz / (double)ctxs[i]->ndof;
    for (int64_t q = 0; q < ctxs[i]->batch.nprob; ++q)
    {
      prob.push_back(Problem{off[q], off[q + 1] - off[q], i, (int)prob.size()});
      entries.push_back(mean * (double)(off[q + 1] - off[q]));
    }
  }
  // the plan depends on the problems' rows and entries alone, and the last call's, which is on the
  // device, is kept for calls with the same ones (with 4,000 problems it and its copies took 0.97 ms)
  auto same = [](auto const & v, std::vector<unsigned char> const & bytes) {
    return bytes.size() == v.size() * sizeof(v[0]) && std::memcmp(v.data(), bytes.data(), bytes.size()) == 0;
  };
  auto keep = [](auto const & v, std::vector<unsigned char> & bytes) {
    auto const * p = reinterpret_cast<unsigned char const *>(v.data());
    bytes.assign(p, p + v.size() * sizeof(v[0]));
  };
  if (!same(prob, S.planProb) || !same(entries, S.planEntries))
  {
    S.planProb.clear(); // until the new one is on the device
    std::vector<Problem> order = prob;
    std::vector<Group> group;
    int64_t const share = planBatch(order, entries, blocks, group);
    if (S.nprob < nprob)
    {
      if (S.exec) // the graph holds the old buffers
        cudaGraphExecDestroy(S.exec);
      S.exec = nullptr;
      S.nprob = 0;
      PXG_CUDA(c0, S.res.alloc(nprob * sizeof(BatchResult)));
      PXG_CUDA(c0, S.prob.alloc(nprob * sizeof(Problem)));
      PXG_CUDA(c0, S.group.alloc((blocks + 1) * sizeof(Group)));
      PXG_CUDA(c0, S.part.alloc(6 * blocks));
      PXG_CUDA(c0, S.bar.alloc(2 * blocks + 3)); // and the error flag, the queues
      S.nprob = nprob;
    }
    PXG_CUDA(c0, cudaMemcpy(S.prob.p, order.data(), order.size() * sizeof(Problem), cudaMemcpyHostToDevice));
    PXG_CUDA(c0, cudaMemcpy(S.group.p, group.data(), group.size() * sizeof(Group), cudaMemcpyHostToDevice));
    S.planShare = share;
    S.planBlocks0 = group[0].blocks;
    keep(entries, S.planEntries);
    keep(prob, S.planProb);
  }
  int64_t const share = S.planShare;
  // the vectors' shares in shared memory where the largest share's fit beside the tiles (with room
  // for uneven shares); elsewhere that memory is better used as L1
  int64_t const shareRows = share + share / 4 + 64, vecBytes = shareRows * 4 * (int64_t)sizeof(double);
  int const cap = tiles + vecBytes <= most ? (int)shareRows : 0, smem = tiles + (cap ? (int)vecBytes : 0);
  PXG_CUDA(c0, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, kBatchSolve, kCgT, smem));
  if (perSm < 1)
    return fail(c0, PXG_ERR_CUDA, "persistent solver does not fit on an SM");
  BatchDev d{};
  for (int i = 0; i < nctx; ++i)
  {
    pxg_ctx * c = ctxs[i];
    BatchState & B = c->batch;
    d.sys[i] = SysDev{c->rowPtr.p, c->colIdx.p, B.K.p, B.M.p, B.b.p, u_targets[i], B.u.p, B.lam.p,
                      B.r.p, B.z.p, B.p.p, B.dinv.p, B.w.p, B.Mw.p};
  }
  d.group = reinterpret_cast<Group const *>(S.group.p);
  d.prob = reinterpret_cast<Problem const *>(S.prob.p);
  d.res = reinterpret_cast<BatchResult *>(S.res.p);
  d.part = reinterpret_cast<ulonglong2 *>(S.part.p);
  d.bar = S.bar.p;
  d.err = S.bar.p + blocks;
  d.next = reinterpret_cast<int *>(S.bar.p) + blocks + 1;
  d.tol2 = rtol * rtol;
  d.maxIter = max_iter;
  d.cap = cap;
  // optional timeline of the persistent solver (not with graph replay: the buffer is
  // read back after the launch)
  char const * traceFile = getenv("PXG_BATCH_TRACE");
  DevBuf<unsigned long long> trace;
  if (traceFile && traceFile[0])
  {
    d.traceCap = 2 * (3 * std::min(max_iter, 4096) + 1);
    PXG_CUDA(c0, trace.alloc(d.traceCap));
    PXG_CUDA(c0, cudaMemset(trace.p, 0, d.traceCap * 8));
    d.trace = trace.p;
    use_graph = 0;
  }
  d.extra = barrierShortfall();

  cudaStream_t const s = (cudaStream_t)stream;
  auto record = [&](cudaStream_t rs) -> pxg_status {
    pxg_lhs_op const opK{2, 1.0, 0, 0.0, 1};
    pxg_lhs_op const opM{0, 0.0, 1, 1.0, 0};
    pxg_rhs_op r = *rhs;
    r.apply_bc = 1;
    for (int i = 0; i < nctx; ++i)
    {
      pxg_status e = pxg_assemble(ctxs[i], &opK, ctxs[i]->batch.K.p, &opM, ctxs[i]->batch.M.p, &r,
                                  ctxs[i]->batch.b.p, 0u, rs);
      if (e != PXG_OK)
        return e;
    }
    PXG_CUDA(c0, cudaMemsetAsync(S.part.p, 0, 6 * blocks * sizeof(double), rs)); // no sum has the tag 0
    PXG_CUDA(c0, cudaMemsetAsync(S.bar.p, 0, (2 * blocks + 3) * sizeof(unsigned), rs));
    void * args[] = {&d};
    PXG_CUDA(c0, cudaLaunchCooperativeKernel((void const *)kBatchSolve, dim3(blocks), dim3(kCgT), args, smem, rs));
    for (int i = 0; i < nctx; ++i)
    {
      pxg_status e = launchAdjointGrad(ctxs[i], ctxs[i]->batch.u.p, ctxs[i]->batch.lam.p, grads[i], rs);
      if (e != PXG_OK)
        return e;
    }
    return PXG_OK;
  };

  if (use_graph)
  {
    // the graph is rebuilt when the arguments change; replayed otherwise
    GraphKey key{};
    key.nctx = nctx;
    for (int i = 0; i < nctx; ++i)
    {
      key.ctx[i] = ctxs[i];
      key.ut[i] = u_targets[i];
      key.grad[i] = grads[i];
      key.scatter[i] = ctxs[i]->scatter;
      key.threads[i] = ctxs[i]->threads;
      key.arith[i] = ctxs[i]->arith;
      pxg_ctx const * c = ctxs[i];
      key.set[i] = c->batch.set;
      void const * const buf[] = {c->xyz.p, c->conn.p, c->emap.p, c->rowPtr.p, c->colIdx.p,
                                  c->rank.p, c->kE.p, c->bcMask.p, c->bcVal.p, c->colour.perm.p};
      static_assert(sizeof(buf) == sizeof(key.buf[0]), "one key entry per buffer");
      std::memcpy(key.buf[i], buf, sizeof(buf));
      key.nbc[i] = c->nbc;
      key.bcDiag[i] = c->bcDiag;
    }
    key.rhs = *rhs;
    key.rtol = rtol;
    key.maxIter = max_iter;
    key.smem = smem;
    if (!S.exec || !(S.key == key))
    {
      if (S.exec)
        cudaGraphExecDestroy(S.exec);
      S.exec = nullptr;
      cudaStream_t cs = nullptr;
      PXG_CUDA(c0, cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
      PXG_CUDA(c0, cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal));
      pxg_status e = record(cs);
      cudaGraph_t graph = nullptr;
      cudaError_t ce = cudaStreamEndCapture(cs, &graph);
      cudaStreamDestroy(cs);
      if (e != PXG_OK)
      {
        if (graph)
          cudaGraphDestroy(graph);
        return e;
      }
      if (ce == cudaSuccess)
        ce = cudaGraphInstantiate(&S.exec, graph, 0);
      if (graph)
        cudaGraphDestroy(graph);
      if (ce != cudaSuccess)
        return cudaFail(c0, ce, "batch graph capture");
      S.key = key;
    }
    PXG_CUDA(c0, cudaGraphLaunch(S.exec, s));
  }
  else
  {
    if ((st = record(s)) != PXG_OK)
      return st;
  }
  // per-problem results
  std::vector<BatchResult> res(nprob);
  unsigned err = 0;
  PXG_CUDA(c0, cudaMemcpyAsync(res.data(), S.res.p, res.size() * sizeof(BatchResult), cudaMemcpyDeviceToHost, s));
  PXG_CUDA(c0, cudaMemcpyAsync(&err, d.err, sizeof(err), cudaMemcpyDeviceToHost, s));
  PXG_CUDA(c0, cudaStreamSynchronize(s));
  if (err)
    return fail(c0, PXG_ERR_TIMEOUT, "persistent batch solver: a barrier wait ran out");
  if (d.trace)
  {
    // text: one line per CG iteration, "solve iteration ns_product ns_update ns_p blocks"
    std::vector<unsigned long long> t(d.traceCap);
    PXG_CUDA(c0, cudaMemcpy(t.data(), d.trace, t.size() * 8, cudaMemcpyDeviceToHost));
    if (FILE * f = fopen(traceFile, "a"))
    {
      int const half = d.traceCap / 2;
      for (int sv = 0; sv < 2; ++sv)
        for (int it = 0; 3 * it + 3 < half && t[sv * half + 3 * it + 3]; ++it)
        {
          unsigned long long const * r = &t[sv * half + 3 * it];
          fprintf(f, "%d %d %llu %llu %llu %d\n", sv, it, r[1] - r[0], r[2] - r[1], r[3] - r[2], S.planBlocks0);
        }
      fclose(f);
    }
  }
  int worst = 0;
  bool conv = true;
  for (int p = 0; p < nprob; ++p)
  {
    losses[p] = res[p].J;
    worst = std::max(worst, std::max(res[p].itF, res[p].itA));
    if (res[p].itF >= max_iter || res[p].itA >= max_iter)
      conv = false;
  }
  if (iters)
    *iters = worst;
  if (!conv)
    return fail(c0, PXG_ERR_NOT_CONVERGED, "a batched CG reached %d iterations", max_iter);
  return PXG_OK;
}

} // extern "C"
