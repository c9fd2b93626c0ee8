// Device Jacobi-preconditioned CG and the adjoint gradient of the diffusion loss
//   K(k) u = b,   J(u) = 1/2 (u - u_t)^T M (u - u_t),   dJ/d log k_e = -(C u)_e^T K_e (C lambda)_e
// with K lambda = M (u - u_t), K_e = k_e K0_e the element stiffness and C zeroing the
// DOFs constrained by the essential BCs (the derivative of the condensed matrix
// C K C + D is C K0_e C).  proxpde itself solves with UmfPackLU
// (include/sparse_matrix.hpp:44); the CG here is plain and not an optimisation
// target.
//
// CG design: one persistent cooperative kernel runs a whole solve, one block per SM.  A
// block owns a contiguous range of rows (equal shares of the work).  Its warps copy tiles
// of rows of the matrix into shared memory, ahead of their use; where the block's r, z, x
// and 1 / diagonal fit beside the tiles they stay there, and a share of one tile per warp
// (n up to 78,000 at 27 entries a row) is copied once per solve.  The dot products are
// reduced in a fixed order (per-block sums, which every block adds up), so a solve is
// reproducible; all blocks hold the same scalars and take the same branches.
// GB300's FP64 rate (1/64 of FP32) makes the product as FP64-bound as it is HBM-bound:
// an entry is one FMA, every unused slot and every shuffle addition costs one too, so a
// lane has a whole row where there are enough rows.
// 884,736 Q1 hexahedra (912,673 rows): 113 us an iteration as three kernels replayed from a
// captured graph (product 64-71), now 79 us (product 57, of which 42.5 is the FP64 pipe's
// and 42 the matrix's time in memory; the updates 11, the three exchanges the rest); at
// 32^3 elements 17 us, now 13 us, bound by the exchanges.
#include <cub/block/block_reduce.cuh>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "pxg_internal.h"

namespace pxg
{
namespace
{

constexpr int kTpb = 256;
constexpr int kMaxPartBlocks = 1024;
constexpr int kCgT = 512;               // threads of the solver's blocks (one per SM)
constexpr int kCgWarps = kCgT / 32;
constexpr int kCgEntries = 896;         // entries of a warp's tile in shared memory (32 rows of 27)
constexpr unsigned kCgPolls = 1u << 23; // polls of a barrier before giving up (some seconds)

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

struct CgArgs
{
  int32_t const * rp;
  int32_t const * ci;
  double const * a;
  double const * b;
  double * x;
  double * p;
  double * r, * z, * dinv; // for rows beyond a block's shared memory
  ulonglong2 * part;       // the blocks' sums: [grid] p.q, [grid][2] r.z and r.r
  double * scal;           // [S_COUNT]
  unsigned * bar;          // [0] arrivals, [1] a wait ran out
  int64_t n;
  double tol2;
  int maxIter;
  int cap;  // rows whose r, z, x and 1 / diagonal have room in shared memory
  int copy; // 1: the values and columns start at 16-byte boundaries
};

struct CgTile
{
  double a[kCgEntries];
  int32_t c[kCgEntries];
};

struct CgShared
{
  double red[2][kCgT];
  double warp[2][4];
  double out[3];
  int ok;
};

// Whether a wait ends after this many polls: its limit is reached, or another's was.  Uniform
// over the calling lanes up to one check.
__device__ __forceinline__ bool cgGiveUp(CgArgs const & g, unsigned polls)
{
  bool const up = __any_sync(__activemask(), polls >= kCgPolls || *(unsigned volatile *)(g.bar + 1) != 0u);
  if (up)
    atomicExch(g.bar + 1, 1u);
  return up;
}

// Thread 0's part of grid barrier number `epoch` (1, 2, ...): arrive and wait, within a limit;
// false once any wait ran out.  The block barriers before and after it and its acquire make the
// other blocks' plain stores visible to every thread.
__device__ __forceinline__ bool cgArriveWait(CgArgs const & g, unsigned epoch)
{
  __threadfence();
  atomicAdd(g.bar, 1u);
  unsigned const target = epoch * gridDim.x;
  bool ok = true;
  for (unsigned polls = 0;;)
  {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(g.bar) : "memory");
    if ((int)(v - target) >= 0)
      break;
    if ((++polls & 1023u) == 0 && cgGiveUp(g, polls))
    {
      ok = false;
      break;
    }
  }
  __threadfence();
  return ok;
}

__device__ __forceinline__ bool cgBarrier(CgArgs const & g, CgShared & sh, unsigned epoch)
{
  __syncthreads();
  if (threadIdx.x == 0)
    sh.ok = cgArriveWait(g, epoch);
  __syncthreads();
  return sh.ok != 0;
}

// Sums over the warp of s[0] (in lane 0) and, for two values, of s[1] (in lane 16): the first
// stage gives each half warp one of them.
template <int NV>
__device__ __forceinline__ double cgWarpSum(double const (&s)[NV])
{
  bool const upper = NV == 2 && (threadIdx.x & 16);
  double t = (upper ? s[NV - 1] : s[0]) + __shfl_xor_sync(0xffffffffu, NV == 1 || upper ? s[0] : s[NV - 1], 16);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1)
    t += __shfl_xor_sync(0xffffffffu, t, o);
  return t;
}

// A block's sums go to the others as 16-byte words of a value and the number of the sum it
// belongs to, stored and loaded whole, so that a word is its own flag.
__device__ __forceinline__ void putTagged(ulonglong2 * to, double v, unsigned tag)
{
  asm volatile("{ .reg .b128 w; mov.b128 w, {%1, %2}; st.relaxed.gpu.global.b128 [%0], w; }" ::"l"(to),
               "l"(__double_as_longlong(v)), "l"((long long)tag)
               : "memory");
}
__device__ __forceinline__ bool getTagged(ulonglong2 const * from, unsigned tag, double & v)
{
  long long lo, hi;
  asm volatile("{ .reg .b128 w; ld.relaxed.gpu.global.b128 w, [%2]; mov.b128 {%0, %1}, w; }"
               : "=l"(lo), "=l"(hi)
               : "l"(from)
               : "memory");
  v = __longlong_as_double(lo);
  return hi == (long long)tag;
}

// Sums of NV values over all threads of the grid in sh.out[0 .. NV), and their quotient
// with `rz` in sh.out[NV] (rz / sum for one value, sum / rz for two), with a bounded wait for
// the other blocks' (no barrier: it makes none of their stores visible).  An FP64 addition
// holds the pipe for 64 cycles, so as few as possible are in a row: four warps add the block's
// 512 values, four per lane, then warp 0 the four sums and, once they are there, the blocks'.
// A counter that all blocks wait for and then loads of their sums took 4.3 us or more, this takes
// 2.9 us (32^3 elements, 152 blocks).  A sum's words are written again two sums of the same kind
// later at the earliest after a barrier that all readers have passed.
template <int NV>
__device__ __forceinline__ bool cgSum(CgArgs const & g, CgShared & sh, unsigned tag, double const (&v)[NV], double rz)
{
  static_assert(kCgT == 4 * 128, "the first stage adds four values per lane");
  int const t = threadIdx.x, lane = t & 31, half = NV == 2 ? lane >> 4 : 0;
  bool const holds = lane == 0 || (NV == 2 && lane == 16);
  ulonglong2 * const part = g.part + (NV == 1 ? 0 : gridDim.x);
  double s[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k)
    sh.red[k][t] = v[k];
  __syncthreads();
  if (t < 128)
  {
#pragma unroll
    for (int k = 0; k < NV; ++k)
    {
      double const * const w = sh.red[k] + t;
      s[k] = (w[0] + w[128]) + (w[256] + w[384]);
    }
    double const x = cgWarpSum<NV>(s);
    if (holds)
      sh.warp[half][t / 32] = x;
  }
  __syncthreads();
  if (t < 32)
  {
    double x = sh.warp[half][lane & 3];
    x += __shfl_xor_sync(0xffffffffu, x, 2);
    x += __shfl_xor_sync(0xffffffffu, x, 1);
    if (holds)
      putTagged(part + NV * blockIdx.x + half, x, tag);
#pragma unroll
    for (int k = 0; k < NV; ++k)
      s[k] = 0.;
    bool ok = true;
    for (unsigned b0 = 0; b0 < gridDim.x; b0 += 160)
    {
      double w[5][NV];
      for (unsigned polls = 0;;)
      {
        bool here = true;
#pragma unroll
        for (int i = 0; i < 5; ++i)
#pragma unroll
          for (int k = 0; k < NV; ++k)
          {
            unsigned const b = b0 + 32 * i + lane;
            w[i][k] = 0.;
            if (b < gridDim.x)
              here = getTagged(part + NV * b + k, tag, w[i][k]) && here;
          }
        if (__all_sync(0xffffffffu, here))
          break;
        if ((++polls & 1023u) == 0 && cgGiveUp(g, polls))
        {
          ok = false;
          break;
        }
      }
#pragma unroll
      for (int k = 0; k < NV; ++k)
        s[k] += ((w[0][k] + w[1][k]) + (w[2][k] + w[3][k])) + w[4][k];
    }
    x = cgWarpSum<NV>(s);
    if (holds)
    {
      sh.out[half] = x;
      if (half == 0)
        sh.out[NV] = NV == 1 ? rz / x : x / rz;
    }
    if (lane == 0)
      sh.ok = ok;
  }
  __syncthreads();
  return sh.ok != 0;
}

// First row of block k's share: the first multiple of 32 rows whose rows before it carry
// k / grid of the work.  A lane's row costs its tile's longest row, so most of a row's weight
// is the matrix's mean row; by entries alone the blocks with many short rows were last.
// Every thread of the block probes; three rounds cover 1e8 multiples.
__device__ __forceinline__ int64_t cgRowStart(CgArgs const & g, unsigned k)
{
  int64_t const tiles = (g.n + 31) / 32;
  if (k >= gridDim.x)
    return g.n;
  double const want = (double)(4 * (int64_t)g.rp[g.n]) * (double)k / (double)gridDim.x;
  double const mean = (double)g.rp[g.n] / (double)g.n; // a row's weight beside its entries'
  int64_t lo = 0, hi = tiles;
  while (hi > lo)
  {
    int64_t const step = (hi - lo + kCgT - 1) / kCgT, t = lo + threadIdx.x * step;
    int64_t const r = min(32 * t, g.n);
    int const below = __syncthreads_count(t < hi && (double)g.rp[r] + 3. * mean * (double)r < want);
    if (below == 0)
      hi = lo;
    else
    {
      int64_t const last = lo + (below - 1) * step;
      hi = min(hi, last + step);
      lo = last + 1;
    }
  }
  return min(32 * lo, g.n);
}

__device__ __forceinline__ void copy16(void * to, void const * from, int bytes, uint64_t policy)
{
  asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2, %3;" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(to)),
               "l"(from), "r"(bytes), "l"(policy)
               : "memory");
}

// The product's rows: a warp takes tiles of 32 / LPR consecutive rows, LPR lanes a row, whose
// values and columns it copies into shared memory with whole-line accesses (lanes reading their
// rows from memory touch a line each, 1,000 L1 cycles per 32 rows of 27 entries: 81 us at 96^3).
// One buffer a warp is enough, as the FP64 pipe has three other warps meanwhile, once the tile
// after has been asked into L2 (72 us without, 60 us with).  After a warp's last tile its first
// is copied again, so that the copy runs during the updates; a warp with a single tile copies it
// once per solve.  U gathers are in flight at a time: 9, 14 and 27 measured alike.
template <int LPR>
struct CgRows
{
  static constexpr int R = 32 / LPR, U = LPR == 1 ? 9 : LPR == 2 ? 14 : 8;
  CgTile & tile;
  int64_t r0;
  int nr, lane, beg, end, first; // the lane's row in the copied tile; entry that the buffer starts with
  bool staged;
  uint64_t policy;

  // row pointers of the tile at row v0 (rows past the block's last are empty)
  __device__ __forceinline__ void range(CgArgs const & g, int v0, int & b, int & e) const
  {
    int const v = v0 + lane / LPR;
    b = g.rp[r0 + min(v, nr)];
    e = g.rp[r0 + min(v + 1, nr)];
  }
  __device__ __forceinline__ void copy(CgArgs const & g)
  {
    first = __shfl_sync(0xffffffffu, beg, 0) & ~3;
    int const n = __shfl_sync(0xffffffffu, end, 31) - first;
    staged = g.copy && n <= kCgEntries;
    if (staged)
    {
      for (int k = 2 * lane; k < n; k += 64)
        copy16(tile.a + k, g.a + first + k, min(16, 8 * (n - k)), policy);
      for (int k = 4 * lane; k < n; k += 128)
        copy16(tile.c + k, g.ci + first + k, min(16, 4 * (n - k)), policy);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  // the tile at row v0 into L2
  __device__ __forceinline__ void prefetch(CgArgs const & g, int v0) const
  {
    if (lane != 0 || !g.copy)
      return;
    int64_t const b = (g.rp[r0 + v0] + 3) & ~3, e = g.rp[r0 + min(v0 + R, nr)] & ~3;
    if (e <= b)
      return;
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(g.a + b), "r"((uint32_t)(8 * (e - b))) : "memory");
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(g.ci + b), "r"((uint32_t)(4 * (e - b))) : "memory");
  }
  __device__ __forceinline__ void start(CgArgs const & g)
  {
    int const v0 = (threadIdx.x / 32) * R;
    range(g, min(v0, nr), beg, end);
    copy(g);
  }
  // q = A p; returns the thread's share of p.q
  __device__ __forceinline__ double product(CgArgs const & g, double * q)
  {
    double pq = 0.;
    int const w0 = (threadIdx.x / 32) * R;
    for (int v0 = w0; v0 < nr; v0 += kCgWarps * R)
    {
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncwarp();
      int const next = v0 + kCgWarps * R < nr ? v0 + kCgWarps * R : w0;
      int nb, ne;
      range(g, next, nb, ne);
      int const v = v0 + lane / LPR;
      double t = 0.;
      if (staged)
      {
        int const n = end - first;
        int const most = (int)__reduce_max_sync(0xffffffffu, (unsigned)(end - beg)); // the longest row
        for (int j = 0; j < most; j += U * LPR)
        {
          int const k = beg - first + j + lane % LPR;
          double pv[U];
#pragma unroll
          for (int u = 0; u < U; ++u)
            pv[u] = k + u * LPR < n ? g.p[tile.c[k + u * LPR]] : 0.;
#pragma unroll
          for (int u = 0; u < U; ++u)
          {
            if (j + u * LPR >= most)
              break;
            if (k + u * LPR < n)
              t = fma(tile.a[k + u * LPR], pv[u], t);
          }
        }
#pragma unroll
        for (int o = LPR / 2; o > 0; o >>= 1)
          t += __shfl_xor_sync(0xffffffffu, t, o);
      }
      else
        t = rowDot<false, LPR, 8>(g.rp, g.ci, g.a, g.p, r0 + v, v < nr);
      if (v < nr && lane % LPR == 0)
      {
        q[v] = t;
        pq += g.p[r0 + v] * t;
      }
      __syncwarp();
      if (next != v0)
      {
        beg = nb;
        end = ne;
        copy(g);
        prefetch(g, next + kCgWarps * R < nr ? next + kCgWarps * R : w0);
      }
    }
    return pq;
  }
};

template <int LPR>
__device__ __forceinline__ void cgRun(CgArgs const & g, CgShared & sh, CgTile * tiles, double * vec, int64_t r0, int nr)
{
  int const t = threadIdx.x;
  bool const fit = nr <= g.cap;
  double * const r = fit ? vec : g.r + r0;
  double * const z = fit ? vec + nr : g.z + r0;
  double * const x = fit ? vec + 2 * nr : g.x + r0;
  double * const di = fit ? vec + 3 * nr : g.dinv + r0;
  double * const p = g.p + r0;
  uint64_t policy;
  asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
  CgRows<LPR> rows{tiles[t / 32], r0, nr, t & 31, 0, 0, 0, false, policy};
  rows.start(g);
  unsigned epoch = 0, tag = 0;
  double s2[2] = {0., 0.};
  // x = 0, r = b, z = p = D^-1 b; four lanes look for a row's diagonal (the last of its
  // entries there, 1 where there is none)
  for (int v0 = 0; v0 < nr; v0 += kCgT / 4)
  {
    int const v = v0 + t / 4;
    int at = -1;
    if (v < nr)
      for (int32_t k = g.rp[r0 + v] + (t & 3); k < g.rp[r0 + v + 1]; k += 4)
        if (g.ci[k] == (int32_t)(r0 + v))
          at = k;
    at = max(at, __shfl_xor_sync(0xffffffffu, at, 1));
    at = max(at, __shfl_xor_sync(0xffffffffu, at, 2));
    if (v < nr && (t & 3) == 0)
    {
      double const d = at >= 0 ? g.a[at] : 0., b = g.b[r0 + v], dv = d != 0. ? 1.0 / d : 1.0, zv = dv * b;
      di[v] = dv;
      x[v] = 0.;
      r[v] = b;
      p[v] = zv;
      s2[0] += b * zv;
      s2[1] += b * b;
    }
  }
  if (!cgSum<2>(g, sh, ++tag, s2, 1.))
    return;
  double rz = sh.out[0], rr = sh.out[1];
  if (!cgBarrier(g, sh, ++epoch)) // p is there
    return;
  double const bb = rr;
  int it = 0;
  while (bb != 0.)
  {
    double const pq[1] = {rows.product(g, z)};
    if (!cgSum<1>(g, sh, ++tag, pq, rz))
      return;
    // x += alpha p, r -= alpha q, z = D^-1 r
    double const al = sh.out[1];
    constexpr int U = 2; // rows per thread whose loads are issued before any store
    s2[0] = s2[1] = 0.;
    for (int v0 = t; v0 < nr; v0 += U * kCgT)
    {
      double xv[U], pv[U], rv[U], qv[U], dv[U];
#pragma unroll
      for (int u = 0; u < U; ++u)
      {
        int const v = min(v0 + u * kCgT, nr - 1);
        xv[u] = x[v], pv[u] = p[v], rv[u] = r[v], qv[u] = z[v], dv[u] = di[v];
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
      {
        int const v = v0 + u * kCgT;
        if (v >= nr)
          break;
        x[v] = xv[u] + al * pv[u];
        double const ri = rv[u] - al * qv[u], zi = dv[u] * ri;
        r[v] = ri;
        z[v] = zi;
        s2[0] += ri * zi;
        s2[1] += ri * ri;
      }
    }
    if (!cgSum<2>(g, sh, ++tag, s2, rz))
      return;
    rz = sh.out[0], rr = sh.out[1];
    ++it;
    if (rr <= g.tol2 * bb || it >= g.maxIter || !(rr == rr))
      break;
    // p = z + beta p
    double const be = sh.out[2];
    for (int v0 = t; v0 < nr; v0 += U * kCgT)
    {
      double zv[U], pv[U];
#pragma unroll
      for (int u = 0; u < U; ++u)
      {
        int const v = min(v0 + u * kCgT, nr - 1);
        zv[u] = z[v], pv[u] = p[v];
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (v0 + u * kCgT < nr)
          p[v0 + u * kCgT] = zv[u] + be * pv[u];
    }
    if (!cgBarrier(g, sh, ++epoch))
      return;
  }
  if (x != g.x + r0)
    for (int v = t; v < nr; v += kCgT)
      g.x[r0 + v] = x[v];
  if (blockIdx.x == 0 && t == 0)
  {
    g.scal[S_RR] = rr;
    g.scal[S_BB] = bb;
    g.scal[S_ITER] = it;
  }
}

__global__ void __launch_bounds__(kCgT, 1) kCgSolve(CgArgs const __grid_constant__ g)
{
  extern __shared__ __align__(16) unsigned char dyn[];
  __shared__ CgShared sh;
  CgTile * const tiles = reinterpret_cast<CgTile *>(dyn);
  double * const vec = reinterpret_cast<double *>(dyn + kCgWarps * sizeof(CgTile));
  int64_t const r0 = cgRowStart(g, blockIdx.x), r1 = cgRowStart(g, blockIdx.x + 1);
  int const nr = (int)(r1 - r0);
  // lanes per row: more where the block has fewer than 32 rows for each warp, and so that a
  // tile's entries fit its buffer
  int const mean = nr > 0 ? (int)((g.rp[r1] - g.rp[r0]) / nr) + 1 : 1;
  int const need = (32 * mean - 1) / kCgEntries + 1;
  if (need <= 1 && 2 * nr > kCgT)
    cgRun<1>(g, sh, tiles, vec, r0, nr);
  else if (need <= 2 && 4 * nr > kCgT)
    cgRun<2>(g, sh, tiles, vec, r0, nr);
  else if (need <= 4 && 8 * nr > kCgT)
    cgRun<4>(g, sh, tiles, vec, r0, nr);
  else
    cgRun<8>(g, sh, tiles, vec, r0, nr);
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
    double const t = rowDot<false>(rp, ci, a, x, row, valid);
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
  // one block per SM, at least 128 rows (four warps) each
  int64_t const grid = std::min<int64_t>(c->sms, (n + 127) / 128);
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
  CgArgs g{rp, ci, a, b, x, w.p.p, w.r.p, w.z.p, w.dinv.p, reinterpret_cast<ulonglong2 *>(w.part.p),
           w.scal.p, reinterpret_cast<unsigned *>(w.scal.p + S_COUNT), n, rtol * rtol, maxIter, cap, aligned};
  void * args[] = {&g};
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
