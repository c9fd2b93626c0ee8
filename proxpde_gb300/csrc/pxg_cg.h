// Jacobi-preconditioned CG inside a persistent kernel: a group of blocks, one per SM, solves one
// system.  Used by the single solves (pxg_solve.cu) and the batches (pxg_batch.cu).
//
// A block owns a contiguous range of rows (equal shares of the work).  Its warps copy tiles
// of rows of the matrix into shared memory, ahead of their use; where the block's r, z, x
// and 1 / diagonal fit beside the tiles they stay there, and a share of one tile per warp
// (n up to 78,000 at 27 entries a row) is copied once per solve.  The dot products are
// reduced in a fixed order (per-block sums, which every block adds up), so a solve is
// reproducible; all blocks hold the same scalars and take the same branches.
// GB300's FP64 rate (1/64 of FP32) makes the product as FP64-bound as it is HBM-bound:
// an entry is one FMA, every unused slot and every shuffle addition costs one too, so a
// lane has a whole row where there are enough rows.
// 884,736 Q1 hexahedra (912,673 rows): 113 us an iteration as three kernels replayed from a
// captured graph (product 64-71), now 82 us (product 57, of which 42.5 is the FP64 pipe's
// and 42 the matrix's time in memory; the updates 11, the three exchanges the rest); at
// 32^3 elements 17 us, now 13 us, bound by the exchanges.
#pragma once

#include <cstdint>
#include <cstdlib>
#include <type_traits>

#include "pxg_internal.h"

namespace pxg
{
namespace
{
constexpr int kCgT = 512;               // threads of the solver's blocks (one per SM)
constexpr int kCgWarps = kCgT / 32;
constexpr int kCgEntries = 896;         // entries of a warp's tile in shared memory (32 rows of 27)
// Polls of a wait before giving up (about half a minute): a block may have to wait for SMs that
// another stream's kernel holds.  With arrivals missing on purpose (tests): some seconds.
constexpr unsigned kCgPolls = 1u << 25, kCgPollsTest = 1u << 21;

// PXG_TEST_BARRIER_SHORTFALL=1 makes every barrier wait for one block more than the group has, so
// that the bounded waits run out (tests of the timeout path)
inline unsigned barrierShortfall()
{
  char const * t = std::getenv("PXG_TEST_BARRIER_SHORTFALL");
  return t && t[0] == '1' ? 1u : 0u;
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
  unsigned * bar;          // arrivals
  unsigned * err;          // a wait ran out
  int64_t first, n;        // the system's rows: first .. first + n of all arrays
  unsigned block0, blocks; // the group of blocks that solves it: the first one and how many
  unsigned extra;          // arrivals waited for beyond the group's (0; > 0 to test the limit)
  double tol2;
  int maxIter;
  int cap;  // rows whose r, z, x and 1 / diagonal have room in shared memory
  int copy; // 1: the values and columns start at 16-byte boundaries
  // optional timeline of the group's first block: the global timer after the start and after each
  // iteration's product, update and barrier; nullptr when off
  unsigned long long * trace;
  int traceCap;

  __device__ __forceinline__ unsigned rank() const { return blockIdx.x - block0; }
};

// a block's running counts of its group's barriers and sums
struct CgCount
{
  unsigned epoch = 0, tag = 0;
};

__device__ __forceinline__ void cgMark(CgArgs const & g, int k)
{
  if (g.trace && g.rank() == 0 && threadIdx.x == 0 && k < g.traceCap)
  {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    g.trace[k] = t;
  }
}

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
  unsigned const most = g.extra ? kCgPollsTest : kCgPolls;
  bool const up = __any_sync(__activemask(), polls >= most || *(unsigned volatile *)g.err != 0u);
  if (up)
    atomicExch(g.err, 1u);
  return up;
}

// Thread 0's part of group barrier number `epoch` (1, 2, ...): arrive and wait, within a limit;
// false once any wait ran out.  The block barriers before and after it and its acquire make the
// other blocks' plain stores visible to every thread.
__device__ __forceinline__ bool cgArriveWait(CgArgs const & g, unsigned epoch)
{
  __threadfence();
  atomicAdd(g.bar, 1u);
  unsigned const target = epoch * g.blocks + g.extra;
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
  if (g.blocks + g.extra == 1)
    return true;
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

// Sums of NV values over all threads of the group in sh.out[0 .. NV), and their quotient
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
  ulonglong2 * const part = g.part + (NV == 1 ? 0 : g.blocks);
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
    if (holds && g.blocks > 1)
      putTagged(part + NV * g.rank() + half, x, tag);
#pragma unroll
    for (int k = 0; k < NV; ++k)
      s[k] = 0.;
    bool ok = true;
    for (unsigned b0 = 0; b0 < g.blocks && g.blocks > 1; b0 += 160)
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
            if (b < g.blocks)
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
    if (g.blocks > 1)
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
  int32_t const * const rp = g.rp + g.first;
  if (k >= g.blocks)
    return g.first + g.n;
  double const entries = (double)(rp[g.n] - rp[0]), mean = entries / (double)g.n; // a row's weight beside its entries'
  double const want = 4. * entries * (double)k / (double)g.blocks;
  int64_t lo = 0, hi = tiles;
  while (hi > lo)
  {
    int64_t const step = (hi - lo + kCgT - 1) / kCgT, t = lo + threadIdx.x * step;
    int64_t const r = min(32 * t, g.n);
    int const below = __syncthreads_count(t < hi && (double)(rp[r] - rp[0]) + 3. * mean * (double)r < want);
    if (below == 0)
      hi = lo;
    else
    {
      int64_t const last = lo + (below - 1) * step;
      hi = min(hi, last + step);
      lo = last + 1;
    }
  }
  return g.first + min(32 * lo, g.n);
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
  int nr, lane, beg = 0, end = 0, first = 0; // the lane's row in the copied tile; entry that the buffer starts with
  bool staged = false;
  uint64_t policy;

  __device__ __forceinline__ CgRows(CgTile * tiles, int64_t row0, int rows)
      : tile(tiles[threadIdx.x / 32]), r0(row0), nr(rows), lane(threadIdx.x & 31)
  {
    asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
  }
  __device__ __forceinline__ ~CgRows() { asm volatile("cp.async.wait_all;" ::: "memory"); }

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
        t = rowDot<LPR, 8>(g.rp, g.ci, g.a, g.p, r0 + v, v < nr);
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

// how a solve ended
struct CgResult
{
  double rr, bb; // r.r and b.b
  int it;
};

// Jacobi-preconditioned CG on the group's system, the calling block's rows r0 .. r0 + nr; `vec`
// holds their r, z, x and 1 / diagonal where nr <= g.cap.  False once a wait ran out.
template <int LPR>
__device__ __forceinline__ bool cgRun(CgArgs const & g, CgShared & sh, CgTile * tiles, double * vec, int64_t r0, int nr,
                                      CgCount & count, CgResult & res)
{
  int const t = threadIdx.x;
  bool const fit = nr <= g.cap;
  double * const r = fit ? vec : g.r + r0;
  double * const z = fit ? vec + nr : g.z + r0;
  double * const x = fit ? vec + 2 * nr : g.x + r0;
  double * const di = fit ? vec + 3 * nr : g.dinv + r0;
  double * const p = g.p + r0;
  CgRows<LPR> rows(tiles, r0, nr);
  rows.start(g);
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
  if (!cgSum<2>(g, sh, ++count.tag, s2, 1.))
    return false;
  double rz = sh.out[0], rr = sh.out[1];
  if (!cgBarrier(g, sh, ++count.epoch)) // p is there
    return false;
  double const bb = rr;
  int it = 0;
  cgMark(g, 0);
  while (bb != 0.)
  {
    double const pq[1] = {rows.product(g, z)};
    if (!cgSum<1>(g, sh, ++count.tag, pq, rz))
      return false;
    cgMark(g, 3 * it + 1);
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
    if (!cgSum<2>(g, sh, ++count.tag, s2, rz))
      return false;
    cgMark(g, 3 * it + 2);
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
    if (!cgBarrier(g, sh, ++count.epoch))
      return false;
    cgMark(g, 3 * it);
  }
  if (x != g.x + r0)
    for (int v = t; v < nr; v += kCgT)
      g.x[r0 + v] = x[v];
  res = {rr, bb, it};
  return true;
}

// f(integral_constant LPR): lanes per row for `nr` rows of `mean` entries, more where the block
// has fewer than 32 rows for each warp, and so that a tile's entries fit its buffer
template <class F>
__device__ __forceinline__ void cgLanes(int nr, int mean, F && f)
{
  int const need = (32 * mean - 1) / kCgEntries + 1;
  if (need <= 1 && 2 * nr > kCgT)
    f(std::integral_constant<int, 1>{});
  else if (need <= 2 && 4 * nr > kCgT)
    f(std::integral_constant<int, 2>{});
  else if (need <= 4 && 8 * nr > kCgT)
    f(std::integral_constant<int, 4>{});
  else
    f(std::integral_constant<int, 8>{});
}
} // namespace
} // namespace pxg
