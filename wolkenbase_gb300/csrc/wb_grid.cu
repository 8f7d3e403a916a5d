/* Column grid over the point store, the spatial index of the tile gather and
 * of classify.
 *
 * The reference answers every neighbourhood query by descending the octree
 * (Octree::findBlocks, octree.cpp:234-251).  Both queries of this path are
 * vertical: a cylinder (any z) and a downward hyperboloid whose horizontal
 * reach grows with depth.  A 2-D grid of square columns answers them with
 * plain ring walks: cells are visited outward from the query axis, so the
 * directions a classify query collects spread around the point early and the
 * surround test can stop after a few rings.
 *
 * Cells hold store positions sorted by height (so a query can stop reading a
 * column once its points are above the hyperboloid), a copy of the points'
 * integer X/Y/Z in grid order for coalesced reads, and per-cell integer
 * bounds for pruning.  A point that
 * lies outside the octree root cube is flagged: the reference's queries treat
 * such points through their leaf's cube, and the kernels do the same for them.
 */
#include <cuda_runtime.h>
#include <cstdint>
#include <cmath>
#include <cstring>
#include "wb_internal.h"
#include "wb_device.cuh"
#include "wb_warpsort.cuh"

namespace
{
struct GridArgs
{
  uint64_t nd;
  double off[3], scale[3], unit;
  double x0, y0, cell;
  int nx, ny;
  double rootLo[3], rootHi[3];
  /* integer thresholds (thr = 1: the decode increases with the record integer
     on every axis): xb[0..nx], yb[0..ny], then the root cube's faces
     {x, y, z lo, x, y, z hi} */
  const long long *bounds;
  int thr;
  float colPerUnit[2];
};

/* Smallest record integer X in [-2^31, 2^31) with pred(X), for a predicate
 * that is false then true as X grows; 2^31 when it never holds. */
template <typename P>
__device__ long long firstTrue(double guess, P pred)
{
  long long lo = -2147483648LL, hi = 2147483648LL;   // pred(lo) false, pred(hi) taken as true
  // a bracket of eight integers around the guess, if it holds the answer (the
  // whole search is a chain of 33 FP64 divisions: 44 us whatever the cloud, now 13)
  const long long near = (long long)fmin(fmax(guess, -2147483640.0), 2147483640.0);
  if (near - 4 > lo && near + 4 < hi && !pred(near - 4) && pred(near + 4))
  {
    lo = near - 4;
    hi = near + 4;
  }
  else if (pred(lo))
    return lo;
  while (hi - lo > 1)
  {
    const long long mid = lo + (hi - lo) / 2;
    if (pred(mid))
      hi = mid;
    else
      lo = mid;
  }
  return hi;
}

/* The record-integer thresholds of the column boundaries and the root cube's
 * faces, one thread each, found with the same FP64 arithmetic the per-point
 * tests use: with a decode that increases with X, floor((dec(X) - x0) / cell)
 * >= i exactly when X >= xb[i], and dec(X) < lo exactly when X < xlo. */
__global__ void gridBoundsKernel(GridArgs g, long long *__restrict__ bounds)
{
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int nb = (g.nx + 1) + (g.ny + 1);
  auto guess = [&](int ax, double v) { return (v / g.unit - g.off[ax]) / g.scale[ax]; };
  if (t <= g.nx)
    bounds[t] = firstTrue(guess(0, g.x0 + t * g.cell), [&](long long X) {
      return floor((wb_decode((int32_t)X, g.off[0], g.scale[0], g.unit) - g.x0) / g.cell) >= (double)t;
    });
  else if (t < nb)
  {
    const int i = t - (g.nx + 1);
    bounds[t] = firstTrue(guess(1, g.y0 + i * g.cell), [&](long long X) {
      return floor((wb_decode((int32_t)X, g.off[1], g.scale[1], g.unit) - g.y0) / g.cell) >= (double)i;
    });
  }
  else if (t < nb + 6)
  {
    const int ax = (t - nb) % 3;
    const double lim = (t - nb) < 3 ? g.rootLo[ax] : g.rootHi[ax];
    bounds[t] = firstTrue(guess(ax, lim), [&](long long X) { return wb_decode((int32_t)X, g.off[ax], g.scale[ax], g.unit) >= lim; });
  }
}

/* Column of record integer X on an axis with thresholds b[0..n]: X lies in
 * [b[0], b[n]); a guess from the mean column width, then the thresholds. */
__device__ __forceinline__ int columnOf(const long long *__restrict__ b, int n, long long X, float perUnit)
{
  int k = (int)((float)(uint32_t)(X - b[0]) * perUnit);   // (a 64-bit conversion is an FP64 instruction)
  k = min(max(k, 0), n - 1);
  while (k > 0 && X < b[k])
    k--;
  while (k < n - 1 && X >= b[k + 1])
    k++;
  return k;
}

__global__ void cellKernel(GridArgs g, const int32_t *__restrict__ sx, const int32_t *__restrict__ sy,
                           const int32_t *__restrict__ sz, uint32_t *__restrict__ count, uint32_t *__restrict__ rank,
                           uint8_t *__restrict__ stray, unsigned long long *__restrict__ nStray,
                           int *__restrict__ ext, const double *__restrict__ xyzd, int2 *__restrict__ colOf)
{
  // record-integer extent of the points ({min x, y, z}, {max x, y, z})
  int mn[3] = {INT32_MAX, INT32_MAX, INT32_MAX}, mx[3] = {INT32_MIN, INT32_MIN, INT32_MIN};
  // whole warps step together, for the counts' runs
  const int lane = threadIdx.x & 31;
  const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
  int next[3] = {0, 0, 0};   // the next point, read while this one is placed
  auto read = [&](uint64_t j) {
    if (j < g.nd)
    {
      next[0] = __ldg(sx + j);
      next[1] = __ldg(sy + j);
      next[2] = __ldg(sz + j);
    }
  };
  read((uint64_t)blockIdx.x * blockDim.x + threadIdx.x);
  for (uint64_t j0 = (uint64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31u); j0 < g.nd; j0 += step)
  {
    const uint64_t j = j0 + lane;
    const int q[3] = {next[0], next[1], next[2]};
    read(j + step);
    uint32_t cell = 0xffffffffu;
    if (j < g.nd)
    {
      for (int a = 0; a < 3; a++)
      {
        mn[a] = min(mn[a], q[a]);
        mx[a] = max(mx[a], q[a]);
      }
      // the point's column as the classify set-up needs it (unclamped, within
      // +-1e9), and clamped into the grid for the sort key; from the integer
      // thresholds where they apply, else in FP64
      int ci, cj;
      bool beside, s;   // beside or above the root cube; outside it at all
      if (g.thr)
      {
        const long long *xb = g.bounds, *yb = g.bounds + g.nx + 1, *face = g.bounds + g.nx + g.ny + 2;
        const long long X = q[0], Y = q[1], Z = q[2];
        if (X >= xb[0] && X < xb[g.nx])
          ci = columnOf(xb, g.nx, X, g.colPerUnit[0]);
        else
          ci = (int)fmax(fmin(floor((xyzd[j] - g.x0) / g.cell), 1e9), -1e9);
        if (Y >= yb[0] && Y < yb[g.ny])
          cj = columnOf(yb, g.ny, Y, g.colPerUnit[1]);
        else
          cj = (int)fmax(fmin(floor((xyzd[g.nd + j] - g.y0) / g.cell), 1e9), -1e9);
        beside = X < face[0] || Y < face[1] || X >= face[3] || Y >= face[4] || Z >= face[5];
        s = beside || Z < face[2];
      }
      else
      {
        const double x = xyzd[j], y = xyzd[g.nd + j], z = xyzd[2 * g.nd + j];
        ci = (int)fmax(fmin(floor((x - g.x0) / g.cell), 1e9), -1e9);
        cj = (int)fmax(fmin(floor((y - g.y0) / g.cell), 1e9), -1e9);
        beside = x < g.rootLo[0] || y < g.rootLo[1] || x >= g.rootHi[0] || y >= g.rootHi[1] || z >= g.rootHi[2];
        s = beside || z < g.rootLo[2];
      }
      colOf[j] = make_int2(ci, cj);
      const int cx = min(max(ci, 0), g.nx - 1), cy = min(max(cj, 0), g.ny - 1);
      cell = (uint32_t)cy * (uint32_t)g.nx + cx;
      stray[j] = (uint8_t)((s ? 1 : 0) | (beside ? 2 : 0));
      if (s)
        atomicAdd(nStray, beside ? (1ull << 32) + 1 : 1ull);   // those beside or above in the upper half
    }
    // the point's place among its column's points: the store order is local,
    // so neighbouring lanes share columns and each run of them takes its
    // places with one atomic
    const uint32_t left = __shfl_up_sync(0xffffffffu, cell, 1);
    const unsigned heads = __ballot_sync(0xffffffffu, lane == 0 || cell != left);
    const int head = 31 - __clz(heads & ((2u << lane) - 1));
    const unsigned after = lane == 31 ? 0u : heads >> (lane + 1);
    const int len = (after ? lane + __ffs(after) : 32) - head;
    uint32_t base = 0;
    if (lane == head && j < g.nd)
      base = atomicAdd(&count[cell], (uint32_t)len);
    base = __shfl_sync(0xffffffffu, base, head);
    if (j < g.nd)
      rank[j] = base + (uint32_t)(lane - head);
  }
  for (int a = 0; a < 3; a++)
    for (int o = 16; o; o >>= 1)
    {
      mn[a] = min(mn[a], __shfl_xor_sync(0xffffffffu, mn[a], o));
      mx[a] = max(mx[a], __shfl_xor_sync(0xffffffffu, mx[a], o));
    }
  if ((threadIdx.x & 31) == 0)
    for (int a = 0; a < 3; a++)
    {
      atomicMin(&ext[a], mn[a]);
      atomicMax(&ext[3 + a], mx[a]);
    }
}

__device__ __forceinline__ uint32_t cellOf(int2 col, int nx, int ny)
{
  return (uint32_t)min(max(col.y, 0), ny - 1) * (uint32_t)nx + (uint32_t)min(max(col.x, 0), nx - 1);
}

/* Order of a column's points: by height, then store position. */
__device__ __forceinline__ uint64_t heightKey(int32_t z, uint64_t j)
{
  return ((uint64_t)(uint32_t)(z ^ (int32_t)0x80000000) << 32) | (uint32_t)j;
}

/* Puts every point's (height, store position) at its place in its column. */
__global__ void cellScatterKernel(uint64_t nd, int nx, int ny, const int2 *__restrict__ colOf,
                                  const uint32_t *__restrict__ rank, const uint32_t *__restrict__ start,
                                  const int32_t *__restrict__ sz, uint64_t *__restrict__ slots, const int *__restrict__ err)
{
  if (*err)
    return;   // start was not written
  for (uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; j < nd; j += (uint64_t)gridDim.x * blockDim.x)
    slots[start[cellOf(colOf[j], nx, ny)] + rank[j]] = heightKey(sz[j], j);
}

/* The same as sort keys, for the radix sort: the column above. */
__global__ void cellKeyKernel(uint64_t nd, int nx, int ny, const int2 *__restrict__ colOf, const int32_t *__restrict__ sz,
                              uint64_t *__restrict__ key)
{
  for (uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; j < nd; j += (uint64_t)gridDim.x * blockDim.x)
    key[j] = ((uint64_t)cellOf(colOf[j], nx, ny) << 32) | (uint32_t)(sz[j] ^ (int32_t)0x80000000);
}

/* Gathers a column's points, in the order of `at(i)` (store positions), as
 * int4 {X, Y, Z, position} and forms the column's record. */
template <typename At>
__device__ __forceinline__ void fillColumn(uint64_t c, uint32_t b, uint32_t e, int lane, int lanes, At at,
                                           const int32_t *__restrict__ sx, const int32_t *__restrict__ sy,
                                           const int32_t *__restrict__ sz, const uint8_t *__restrict__ stray,
                                           int4 *__restrict__ gpt, int32_t mn[3], int32_t mx[3], bool &beside)
{
  for (uint32_t i = b + lane; i < e; i += lanes)
  {
    const uint32_t j = at(i);
    const int32_t q[3] = {sx[j], sy[j], sz[j]};
    const uint8_t st = stray[j];
    gpt[i] = make_int4(q[0], q[1], q[2], (int)(j | ((st & 1) ? 0x80000000u : 0u)));
    beside |= (st & 2) != 0;
    for (int a = 0; a < 3; a++)
    {
      mn[a] = min(mn[a], q[a]);
      mx[a] = max(mx[a], q[a]);
    }
  }
}

/* Warp-wide part of a column's record; lane 0 writes it. */
__device__ __forceinline__ void writeColumn(uint64_t c, uint32_t b, uint32_t e, int lane, int32_t mn[3], int32_t mx[3],
                                            bool beside, int4 *__restrict__ rec)
{
  for (int a = 0; a < 3; a++)
  {
    mn[a] = __reduce_min_sync(0xffffffffu, mn[a]);
    mx[a] = __reduce_max_sync(0xffffffffu, mx[a]);
  }
  // a column holding a point beside or above the root cube is read in full: a
  // shape can hold that point's block without holding the point
  const bool any = __any_sync(0xffffffffu, beside);
  if (lane == 0)
  {
    rec[2 * c] = make_int4(mn[0], mn[1], mx[0], mx[1]);
    rec[2 * c + 1] = make_int4(mn[2], (int)b, (int)e, any ? 1 : 0);
  }
}

/* Sorts and fills the columns, one warp each: up to 256 points in registers, up
 * to kColumnMax in shared memory (8M points: 155 us; 196 with those from 65 points
 * on in shared memory); larger columns are listed for bigColumnKernel.  Replaces the radix sort of all points by (column, height)
 * where columns are of ordinary size: five passes over 12-byte pairs. */
constexpr int kColumnWarps = 4, kColumnMax = 512, kBigColumnMax = 4096;
__global__ void __launch_bounds__(32 * kColumnWarps) columnKernel(uint64_t ncell, const uint32_t *__restrict__ start,
                                                                  const uint64_t *__restrict__ slots,
                                                                  const int32_t *__restrict__ sx,
                                                                  const int32_t *__restrict__ sy,
                                                                  const int32_t *__restrict__ sz,
                                                                  const uint8_t *__restrict__ stray,
                                                                  int4 *__restrict__ gpt, int4 *__restrict__ rec,
                                                                  uint32_t *__restrict__ big, uint32_t *__restrict__ nBig,
                                                                  const int *__restrict__ err)
{
  __shared__ uint64_t buf[kColumnWarps][kColumnMax];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint64_t c = (uint64_t)blockIdx.x * kColumnWarps + w;
  if (c >= ncell || *err)   // err: start was not written, nothing is listed for bigColumnKernel
    return;
  const uint32_t b = start[c], e = start[c + 1], n = e - b;
  int32_t mn[3] = {INT32_MAX, INT32_MAX, INT32_MAX}, mx[3] = {INT32_MIN, INT32_MIN, INT32_MIN};
  bool beside = false;
  uint64_t *k = buf[w];
  if (n > kColumnMax)
  {
    if (lane == 0)
      big[atomicAdd(nBig, 1u)] = (uint32_t)c;
    return;
  }
  if (n <= 64)
    wb_warp_sort_to<2>(slots + b, k, n, lane);
  else if (n <= 128)
    wb_warp_sort_to<4>(slots + b, k, n, lane);
  else if (n <= 256)
    wb_warp_sort_to<8>(slots + b, k, n, lane);
  else
  {
    int P = 512;
    while (P < (int)n)
      P <<= 1;
    for (int q = lane; q < P; q += 32)
      k[q] = q < (int)n ? slots[b + q] : ~0ull;
    __syncwarp();
    for (int size = 2; size <= P; size <<= 1)
      for (int j = size >> 1; j > 0; j >>= 1)
      {
        for (int t = lane; t < P / 2; t += 32)
        {
          const int i = 2 * t - (t & (j - 1)), u = i + j;
          const uint64_t x = k[i], y = k[u];
          if ((x > y) == ((i & size) == 0))
          {
            k[i] = y;
            k[u] = x;
          }
        }
        __syncwarp();
      }
  }
  fillColumn(c, b, e, lane, 32, [&](uint32_t i) { return (uint32_t)k[i - b]; }, sx, sy, sz, stray, gpt, mn, mx, beside);
  writeColumn(c, b, e, lane, mn, mx, beside, rec);
}

/* The listed columns, one block each, up to kBigColumnMax points in shared
 * memory; a larger one raises *unsorted and the caller sorts by radix passes. */
__global__ void __launch_bounds__(512) bigColumnKernel(const uint32_t *__restrict__ big, const uint32_t *__restrict__ nBig,
                                                       const uint32_t *__restrict__ start,
                                                       const uint64_t *__restrict__ slots, const int32_t *__restrict__ sx,
                                                       const int32_t *__restrict__ sy, const int32_t *__restrict__ sz,
                                                       const uint8_t *__restrict__ stray, int4 *__restrict__ gpt,
                                                       int4 *__restrict__ rec, uint32_t *__restrict__ unsorted)
{
  __shared__ uint64_t k[kBigColumnMax];
  __shared__ int32_t ext[6];
  __shared__ int flag;
  const uint32_t nb = *nBig;
  for (uint32_t r = blockIdx.x; r < nb; r += gridDim.x)
  {
    const uint32_t c = big[r], b = start[c], e = start[c + 1], n = e - b;
    __syncthreads();
    if (n > kBigColumnMax)
    {
      if (threadIdx.x == 0)
        *unsorted = 1;
      continue;
    }
    int P = 1024;
    while (P < (int)n)
      P <<= 1;
    for (int q = threadIdx.x; q < P; q += 512)
      k[q] = q < (int)n ? slots[b + q] : ~0ull;
    if (threadIdx.x < 6)
      ext[threadIdx.x] = threadIdx.x < 3 ? INT32_MAX : INT32_MIN;
    if (threadIdx.x == 0)
      flag = 0;
    __syncthreads();
    for (int size = 2; size <= P; size <<= 1)
      for (int j = size >> 1; j > 0; j >>= 1)
      {
        for (int t = threadIdx.x; t < P / 2; t += 512)
        {
          const int i = 2 * t - (t & (j - 1)), u = i + j;
          const uint64_t x = k[i], y = k[u];
          if ((x > y) == ((i & size) == 0))
          {
            k[i] = y;
            k[u] = x;
          }
        }
        __syncthreads();
      }
    int32_t mn[3] = {INT32_MAX, INT32_MAX, INT32_MAX}, mx[3] = {INT32_MIN, INT32_MIN, INT32_MIN};
    bool beside = false;
    fillColumn(c, b, e, (int)threadIdx.x, 512, [&](uint32_t i) { return (uint32_t)k[i - b]; }, sx, sy, sz, stray, gpt, mn, mx,
               beside);
    for (int a = 0; a < 3; a++)
    {
      atomicMin(&ext[a], mn[a]);
      atomicMax(&ext[3 + a], mx[a]);
    }
    if (beside)
      flag = 1;
    __syncthreads();
    if (threadIdx.x == 0)
    {
      rec[2 * (uint64_t)c] = make_int4(ext[0], ext[1], ext[3], ext[4]);
      rec[2 * (uint64_t)c + 1] = make_int4(ext[2], (int)b, (int)e, flag);
    }
  }
}

/* Fills columns whose points are already in order (pos), one warp each. */
__global__ void cellFillKernel(uint64_t ncell, const uint32_t *__restrict__ start, const uint32_t *__restrict__ pos,
                               const int32_t *__restrict__ sx, const int32_t *__restrict__ sy,
                               const int32_t *__restrict__ sz, const uint8_t *__restrict__ stray,
                               int4 *__restrict__ gpt, int4 *__restrict__ rec, const int *__restrict__ err)
{
  const uint64_t c = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (c >= ncell || *err)   // err: pos was not written
    return;
  const uint32_t b = start[c], e = start[c + 1];
  int32_t mn[3] = {INT32_MAX, INT32_MAX, INT32_MAX}, mx[3] = {INT32_MIN, INT32_MIN, INT32_MIN};
  bool beside = false;
  fillColumn(c, b, e, lane, 32, [&](uint32_t i) { return pos[i]; }, sx, sy, sz, stray, gpt, mn, mx, beside);
  writeColumn(c, b, e, lane, mn, mx, beside, rec);
}

/* Column groups (the work items of the margin pass): a column of n points is
 * ceil(n / 32) groups of consecutive points. */
__global__ void groupCountKernel(uint64_t ncell, const int4 *__restrict__ rec, uint32_t *__restrict__ cnt)
{
  for (uint64_t c = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; c < ncell; c += (uint64_t)gridDim.x * blockDim.x)
  {
    int4 r1 = rec[2 * c + 1];
    cnt[c] = ((uint32_t)(r1.z - r1.y) + 31) / 32;
  }
}

__global__ void groupFillKernel(uint64_t ncell, const int4 *__restrict__ rec, const uint32_t *__restrict__ first,
                                uint2 *__restrict__ groups, const int *__restrict__ err)
{
  if (*err)
    return;   // first was not written
  for (uint64_t c = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; c < ncell; c += (uint64_t)gridDim.x * blockDim.x)
  {
    int4 r1 = rec[2 * c + 1];
    uint32_t g = first[c];
    for (uint32_t t = (uint32_t)r1.y; t < (uint32_t)r1.z; t += 32)
      groups[g++] = make_uint2((uint32_t)c, t);
  }
}

/* Position of cell (x, y) of an 8 x 8 block along a Hilbert curve. */
__device__ __forceinline__ int hilbert8(int x, int y)
{
  int d = 0;
#pragma unroll
  for (int s = 4; s; s >>= 1)
  {
    const int rx = (x & s) != 0, ry = (y & s) != 0;
    d += s * s * ((3 * rx) ^ ry);
    if (!ry)
    {
      if (rx)
      {
        x = 7 - x;
        y = 7 - y;
      }
      const int t = x;
      x = y;
      y = t;
    }
  }
  return d;
}

/* The point groups of classify: the points of each super-cell in an order
 * whose runs of 32 are compact (and whose runs of 8 are still more so), and the
 * runs.  Points near their column's lowest (mostly ground) follow a Hilbert
 * curve over an 8 x 8 division of the super-cell; points more than a column's
 * width above it (roofs, walls, trees) come after them by height, so that they
 * do not stretch the ground groups.  One block per super-cell, a warp
 * per row of its columns: a histogram of the points' buckets, its prefix, and a
 * scatter; the blocks take their places in the two lists from one counter
 * (points in the low 36 bits, groups above).  A super-cell's groups are
 * consecutive: its record gets the first one and their number.  8M points take
 * 0.088 ms, 10,000 points 15 us (0.13 ms and 37 us with a warp per super-cell
 * that met its columns one after another).
 *
 * The order in which classify takes the groups, after the records: those of
 * points high above their column from the front, the others from the back
 * (taken[1] counts both, the high ones in its lower half).  A group under
 * trees reads up to 20 times the groups an average one does, and the last
 * groups to start hold a few warps while the rest of the GPU idles.  With the
 * high ones first the fast pass takes 1.41 ms instead of 1.61 for 1M points and
 * 6.16 instead of 6.63 for 5M; for 50M it is the same. */
constexpr int kOrderThreads = 32 * WB_SUPER, kOrderBuckets = 96;
__global__ void __launch_bounds__(kOrderThreads) groupOrderKernel(int nx, int ny, int snx, int sny, float colUnits,
                                                                     const int4 *__restrict__ rec,
                                                                     int4 *__restrict__ srec,
                                                                     const int4 *__restrict__ gpt,
                                                                     int2 *__restrict__ bxy, int2 *__restrict__ bzw,
                                                                     int4 *__restrict__ groups, uint64_t maxGroups,
                                                                     unsigned long long *__restrict__ taken)
{
  __shared__ uint32_t hist[WB_SUPER][kOrderBuckets];
  __shared__ uint32_t lowS, totalS;
  __shared__ unsigned long long atS, turnS;
  const int lane = threadIdx.x & 31, r = threadIdx.x >> 5;
  uint32_t *h = hist[r];
  const uint64_t s = blockIdx.x;
  const int si = (int)(s % snx), sj = (int)(s / snx);
  const int4 box = srec[2 * s];
  if (box.x == INT32_MAX)
    return;
  for (int b = lane; b < kOrderBuckets; b += 32)
    h[b] = 0;
  __syncwarp();
  const int i0 = si * WB_SUPER, ni = min(WB_SUPER, nx - i0);
  const float fx = 8.f / ((float)((int64_t)box.z - box.x) + 1.f), fy = 8.f / ((float)((int64_t)box.w - box.y) + 1.f);
  const float perCol = 1.f / colUnits;
  // the super-cell's columns, one per lane
  constexpr int S = WB_SUPER;
  static_assert(S * S <= 32, "a lane per column");
  int4 mine = make_int4(0, 0, 0, 0);
  if (lane < S * S && lane % S < ni && sj * S + lane / S < ny)
    mine = rec[2 * ((uint64_t)(sj * S + lane / S) * nx + i0 + lane % S) + 1];
  const unsigned full = __ballot_sync(0xffffffffu, mine.y != mine.z);
  // the points of warp r's row of columns, which are consecutive: f(point, bucket)
  const unsigned row = (full >> (r * S)) & ((1u << S) - 1);
  const uint32_t b0 = (uint32_t)__shfl_sync(0xffffffffu, mine.y, row ? r * S + __ffs(row) - 1 : 0),
                 e0 = (uint32_t)__shfl_sync(0xffffffffu, mine.z, row ? r * S + 31 - __clz(row) : 0);
  // where each column's points begin, and its lowest point
  uint32_t from[S];
  int zlow[S];
#pragma unroll
  for (int q = 0; q < S; q++)
  {
    from[q] = (uint32_t)__shfl_sync(0xffffffffu, mine.y, r * S + q);
    zlow[q] = __shfl_sync(0xffffffffu, mine.x, r * S + q);
    if (!((row >> q) & 1))
      from[q] = 0xffffffffu;
  }
  auto forPoints = [&](auto f) {
    if (!row)
      return;
    int4 next = make_int4(0, 0, 0, 0);
    if (b0 + lane < e0)
      next = gpt[b0 + lane];
    for (uint32_t t = b0 + lane; t < e0; t += 32)
    {
      const int4 p = next;
      if (t + 32 < e0)
        next = gpt[t + 32];
      int zmin = zlow[0];
#pragma unroll
      for (int q = 1; q < S; q++)
        zmin = t >= from[q] ? zlow[q] : zmin;
      // (differences in 32 bits: a 64-bit conversion is an FP64 instruction)
      const float up = (float)((uint32_t)p.z - (uint32_t)zmin) * perCol;   // column widths above the column's lowest point
      int b;
      if (up > 1.f)
        b = 64 + (int)fminf(up - 1.f, 31.f);
      else
        b = hilbert8(min(7, (int)((float)((uint32_t)p.x - (uint32_t)box.x) * fx)),
                     min(7, (int)((float)((uint32_t)p.y - (uint32_t)box.y) * fy)));
      f(p, b);
    }
  };
  forPoints([&](const int4 &, int b) { atomicAdd(&h[b], 1u); });
  __syncthreads();
  if (threadIdx.x < 32)
  {
    // exclusive prefix over the buckets, three per lane; points of the first 64
    uint32_t sum = 0, low = 0;
    for (int q = 0; q < 3; q++)
      for (int k = 0; k < S; k++)
      {
        const uint32_t v = hist[k][lane * 3 + q];
        sum += v;
        if (lane * 3 + q < 64)
          low += v;
      }
    uint32_t inc = sum;
    for (int o = 1; o < 32; o <<= 1)
    {
      const uint32_t v = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o)
        inc += v;
    }
    uint32_t run = inc - sum;
    for (int q = 0; q < 3; q++)
      for (int k = 0; k < S; k++)   // within a bucket row by row
      {
        const uint32_t v = hist[k][lane * 3 + q];
        hist[k][lane * 3 + q] = run;
        run += v;
      }
    low = __reduce_add_sync(0xffffffffu, low);
    if (lane == 31)
    {
      const uint32_t gLow = (low + 31) / 32, gAll = gLow + (inc - low + 31) / 32;
      lowS = low;
      totalS = inc;
      atS = atomicAdd(taken, ((unsigned long long)gAll << 36) | inc);
      turnS = atomicAdd(taken + 1, ((unsigned long long)gLow << 32) | (gAll - gLow));
    }
  }
  __syncthreads();
  const uint32_t low = lowS, total = totalS, gLow = (low + 31) / 32, gAll = gLow + (total - low + 31) / 32;
  const unsigned long long at = atS, turn = turnS;
  uint32_t *order = (uint32_t *)(groups + 2 * maxGroups);
  const uint32_t base = (uint32_t)(at & ((1ull << 36) - 1)), g0 = (uint32_t)(at >> 36);
  // first point, points and super-cell of each group; groupBoxKernel adds the bounds
  for (uint32_t k = threadIdx.x; k < gAll; k += kOrderThreads)
  {
    order[k < gLow ? maxGroups - 1 - ((turn >> 32) + k) : (uint32_t)turn + (k - gLow)] = g0 + k;
    groups[2 * (uint64_t)(g0 + k) + 1] =
        k < gLow ? make_int4(0, (int)(base + 32 * k), (int)min(32u, low - 32 * k), 0)
                 : make_int4(0, (int)(base + low + 32 * (k - gLow)), (int)min(32u, total - low - 32 * (k - gLow)), 0);
  }
  if (threadIdx.x == 0)
  {
    srec[2 * s + 1].y = (int)g0;
    srec[2 * s + 1].z = (int)gAll;
  }
  forPoints([&](const int4 &p, int b) {
    const uint32_t at = base + atomicAdd(&h[b], 1u);
    bxy[at] = make_int2(p.x, p.y);
    bzw[at] = make_int2(p.z, p.w);
  });
}

/* What the blocks of points outside the root cube are found from. */
struct StrayArgs
{
  const uint32_t *leafId;
  const uint64_t *leafKey;
  const uint8_t *leafLev;
  const uint8_t *stray;
  double unitOff[3], perStep[3], rootLo[3], rootSide;   /* off * unit, 1 / (scale * unit) */
  int imin[3], imax[3];   /* the cloud's record integers */
};

/* The box of the blocks of outside points in record integers, and the lowest of
 * their cubes' tops and bottoms: a shape that takes such a point by its block,
 * without holding the point, reaches the box at that top; one that takes it at
 * all reaches it at that bottom. */
struct StrayBox
{
  int x0, y0, x1, y1, top, bottom;
  __device__ void clear()
  {
    x0 = y0 = top = bottom = INT32_MAX;
    x1 = y1 = INT32_MIN;
  }
  __device__ void add(const StrayBox &b)
  {
    x0 = min(x0, b.x0);
    y0 = min(y0, b.y0);
    x1 = max(x1, b.x1);
    y1 = max(y1, b.y1);
    top = min(top, b.top);
    bottom = min(bottom, b.bottom);
  }
  __device__ void warpAdd()
  {
    x0 = __reduce_min_sync(0xffffffffu, x0);
    y0 = __reduce_min_sync(0xffffffffu, y0);
    x1 = __reduce_max_sync(0xffffffffu, x1);
    y1 = __reduce_max_sync(0xffffffffu, y1);
    top = __reduce_min_sync(0xffffffffu, top);
    bottom = __reduce_min_sync(0xffffffffu, bottom);
  }
  __device__ void store(int4 *r) const
  {
    r[0] = make_int4(x0, y0, x1, y1);
    r[1] = make_int4(top, bottom, 0, 0);
  }
  __device__ void load(const int4 *r)
  {
    x0 = r[0].x;
    y0 = r[0].y;
    x1 = r[0].z;
    y1 = r[0].w;
    top = r[1].x;
    bottom = r[1].y;
  }
};

/* The block of stored point j, a record unit wider on every side and within the
 * cloud's extent (which holds every query's own point, so that nothing is nearer
 * to one than before), its heights at most 2^29 units below it. */
__device__ __noinline__ StrayBox strayBlock(const StrayArgs &a, uint32_t j)
{
  const uint32_t l = a.leafId[j];
  double c[3], side;
  wb_leaf_cube(a.leafKey[l], a.leafLev[l], a.rootLo, a.rootSide, c[0], c[1], c[2], side);
  int lo[3], hi[3];
#pragma unroll
  for (int k = 0; k < 3; k++)
  {
    const double p = (c[k] - side / 2 - a.unitOff[k]) * a.perStep[k], q = (c[k] + side / 2 - a.unitOff[k]) * a.perStep[k];
    const double least = k < 2 ? (double)a.imin[k] : fmax((double)a.imin[k] - 536870912.0, -2147483648.0);
    lo[k] = (int)fmin(fmax(floor(fmin(p, q)) - 1, least), (double)a.imax[k]);
    hi[k] = (int)fmin(fmax(k < 2 ? ceil(fmax(p, q)) + 1 : floor(fmax(p, q)) - 1, least), (double)a.imax[k]);
  }
  StrayBox b;
  b.x0 = lo[0];
  b.y0 = lo[1];
  b.x1 = hi[0];
  b.y1 = hi[1];
  b.top = hi[2];
  b.bottom = lo[2];
  return b;
}

/* The records of the columns that hold points beside or above the root cube, of all
 * their points outside it; one warp each (run only for clouds with such
 * points).  Bound by the FP64 pipe: with straySuperKernel 0.08 ms for 52,000 such
 * points of 1.56M (0.16 with divisions by the step). */
__global__ void strayColumnKernel(uint64_t ncell, StrayArgs a, const int4 *__restrict__ rec, const int4 *__restrict__ gpt,
                                  int4 *__restrict__ out)
{
  const int lane = threadIdx.x & 31;
  const uint64_t warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t c = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; c < ncell; c += warps)
  {
    const int4 r1 = rec[2 * c + 1];
    if (!r1.w)
      continue;
    StrayBox b;
    b.clear();
    uint32_t l0 = 0xffffffffu, l1 = 0;   // the least and the greatest of their leaves
    for (uint32_t i = (uint32_t)r1.y + lane; i < (uint32_t)r1.z; i += 32)
    {
      const int w = gpt[i].w;
      if (w < 0)
      {
        const uint32_t j = (uint32_t)w & 0x7fffffffu;
        b.add(strayBlock(a, j));
        l0 = min(l0, a.leafId[j]);
        l1 = max(l1, a.leafId[j]);
      }
    }
    __syncwarp();
    b.warpAdd();
    l0 = __reduce_min_sync(0xffffffffu, l0);
    l1 = __reduce_max_sync(0xffffffffu, l1);
    if (lane == 0)
    {
      b.store(out + 2 * c);
      out[2 * c + 1].z = l0 == l1;   // one block: its bounds also tell for certain
    }
  }
}

/* The same per super-cell. */
__global__ void straySuperKernel(int nx, int ny, int snx, int sny, const int4 *__restrict__ rec,
                                 const int4 *__restrict__ srec, const int4 *__restrict__ col, int4 *__restrict__ out)
{
  const uint64_t ns = (uint64_t)snx * sny;
  for (uint64_t s = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; s < ns; s += (uint64_t)gridDim.x * blockDim.x)
  {
    if (!srec[2 * s + 1].w)
      continue;
    StrayBox b;
    b.clear();
    for (int q = 0; q < WB_SUPER * WB_SUPER; q++)
    {
      const int i = (int)(s % snx) * WB_SUPER + q % WB_SUPER, j = (int)(s / snx) * WB_SUPER + q / WB_SUPER;
      const uint64_t c = (uint64_t)j * nx + i;
      if (i < nx && j < ny && rec[2 * c + 1].w)
      {
        StrayBox o;
        o.load(col + 2 * c);
        b.add(o);
      }
    }
    b.store(out + 2 * s);
  }
}

/* The groups' records: two int4 per group, {x0, y0, x1, y1} and {zmin, first,
 * points, flags} (flags: holds a point beside or above the root cube, which
 * the queries can take with its block without the hyperboloid holding the point
 * itself: strayGrp then has the blocks' box); one warp per group. */
__global__ void groupBoxKernel(StrayArgs a, const unsigned long long *__restrict__ taken, const int2 *__restrict__ bxy,
                               const int2 *__restrict__ bzw, int4 *__restrict__ groups, int4 *__restrict__ strayGrp)
{
  const int lane = threadIdx.x & 31;
  const uint64_t n = *taken >> 36, warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t k = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; k < n; k += warps)
  {
    const int4 r1 = groups[2 * k + 1];
    const bool ok = lane < r1.z;
    int2 p = make_int2(0, 0), q = make_int2(0, 0);
    if (ok)
    {
      p = bxy[(uint32_t)r1.y + lane];
      q = bzw[(uint32_t)r1.y + lane];
    }
    const int x0 = __reduce_min_sync(0xffffffffu, ok ? p.x : INT32_MAX), x1 = __reduce_max_sync(0xffffffffu, ok ? p.x : INT32_MIN);
    const int y0 = __reduce_min_sync(0xffffffffu, ok ? p.y : INT32_MAX), y1 = __reduce_max_sync(0xffffffffu, ok ? p.y : INT32_MIN);
    const int z0 = __reduce_min_sync(0xffffffffu, ok ? q.x : INT32_MAX);
    const bool mine = ok && q.y < 0;   // outside the root cube
    const bool stray = __any_sync(0xffffffffu, mine && (a.stray[(uint32_t)q.y & 0x7fffffffu] & 2));
    if (stray)
    {
      StrayBox b;
      b.clear();
      if (mine)
        b = strayBlock(a, (uint32_t)q.y & 0x7fffffffu);
      __syncwarp();
      b.warpAdd();
      if (lane == 0)
        b.store(strayGrp + 2 * k);
    }
    if (lane == 0)
    {
      groups[2 * k] = make_int4(x0, y0, x1, y1);
      groups[2 * k + 1] = make_int4(z0, r1.y, r1.z, stray ? 1 : 0);
    }
  }
}

/* Records of each block of WB_SUPER x WB_SUPER columns (the column record
 * layout; begin/end unused; flags: some column's flags). */
__global__ void superKernel(int nx, int ny, int snx, int sny, const int4 *__restrict__ rec, int4 *__restrict__ srec)
{
  uint64_t ns = (uint64_t)snx * sny;
  for (uint64_t s = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; s < ns; s += (uint64_t)gridDim.x * blockDim.x)
  {
    int si = (int)(s % snx), sj = (int)(s / snx);
    int32_t mn[3] = {INT32_MAX, INT32_MAX, INT32_MAX}, mx[2] = {INT32_MIN, INT32_MIN};
    int flags = 0;
    for (int dj = 0; dj < WB_SUPER; dj++)
      for (int di = 0; di < WB_SUPER; di++)
      {
        int i = si * WB_SUPER + di, j = sj * WB_SUPER + dj;
        if (i >= nx || j >= ny)
          continue;
        uint64_t c = (uint64_t)j * nx + i;
        int4 r0 = rec[2 * c], r1 = rec[2 * c + 1];
        if (r1.y == r1.z)
          continue;
        mn[0] = min(mn[0], r0.x);
        mn[1] = min(mn[1], r0.y);
        mx[0] = max(mx[0], r0.z);
        mx[1] = max(mx[1], r0.w);
        mn[2] = min(mn[2], r1.x);
        flags |= r1.w;
      }
    srec[2 * s] = make_int4(mn[0], mn[1], mx[0], mx[1]);
    srec[2 * s + 1] = make_int4(mn[2], 0, 0, flags);   // y, z: groupOrderKernel
  }
}
}  // namespace

static GridArgs gridArgs(const wb_ctx *c)
{
  GridArgs a{};
  const WbGeom &g = c->g;
  a.nd = c->nd;
  for (int k = 0; k < 3; k++)
  {
    a.off[k] = g.off[k];
    a.scale[k] = g.scale[k];
    a.rootLo[k] = g.root_lo[k];
    a.rootHi[k] = g.root_lo[k] + g.root_side;
  }
  a.unit = g.unit;
  return a;
}

static StrayArgs strayArgs(const wb_ctx *c)
{
  StrayArgs a{};
  const WbGeom &g = c->g;
  a.leafId = (const uint32_t *)c->leafId.p;
  a.leafKey = (const uint64_t *)c->leafKey.p;
  a.leafLev = (const uint8_t *)c->leafLevel.p;
  a.stray = (const uint8_t *)c->stray.p;
  for (int k = 0; k < 3; k++)
  {
    a.unitOff[k] = g.off[k] * g.unit;
    a.perStep[k] = 1.0 / (g.scale[k] * g.unit);
    a.rootLo[k] = g.root_lo[k];
    a.imin[k] = c->grid.imin[k];
    a.imax[k] = c->grid.imax[k];
  }
  a.rootSide = g.root_side;
  return a;
}

int wb_grid_impl(wb_ctx *c, double x0, double y0, double x1, double y1)
{
  uint64_t nd = c->nd;
  WbGeom &g = c->g;
  double w = fmax(x1 - x0, 1e-9), h = fmax(y1 - y0, 1e-9);
  // about grid_points points per occupied column, at most 2^24 columns
  double cell = sqrt(w * h * c->grid_points / (double)(nd ? nd : 1));
  double minCell = sqrt(w * h / (double)(1u << 24));
  if (cell < minCell)
    cell = minCell;
  int nx = (int)ceil(w / cell) + 1, ny = (int)ceil(h / cell) + 1;
  c->grid.x0 = x0;
  c->grid.y0 = y0;
  c->grid.cell = cell;
  c->grid.nx = nx;
  c->grid.ny = ny;
  uint64_t ncell = (uint64_t)nx * ny;
  c->grid.ncell = ncell;
  int rc;
  if ((rc = wb_ensure(c, c->gKey0, nd * 8 + 64)) || (rc = wb_ensure(c, c->gKey1, nd * 8 + 64)) ||
      (rc = wb_ensure(c, c->gVal0, nd * 4 + 64)) || (rc = wb_ensure(c, c->gVal1, nd * 4 + 64)) ||
      (rc = wb_ensure(c, c->stray, nd + 64)) || (rc = wb_ensure(c, c->cellStart, (ncell + 1) * 8 + 64)) ||
      (rc = wb_ensure(c, c->gpt, nd * 16 + 64)) || (rc = wb_ensure(c, c->cellRec, ncell * 32 + 64)) ||
      (rc = wb_ensure(c, c->colOf, nd * 8 + 64)))
    return rc;
  GridArgs a = gridArgs(c);
  a.x0 = x0;
  a.y0 = y0;
  a.cell = cell;
  a.nx = nx;
  a.ny = ny;
  // integer thresholds where every axis decodes increasingly
  a.thr = 0;
  a.bounds = nullptr;
  if (g.scale[0] * g.unit > 0 && g.scale[1] * g.unit > 0 && g.scale[2] * g.unit > 0)
  {
    const int nb = (nx + 1) + (ny + 1) + 6;
    if ((rc = wb_ensure(c, c->gridBounds, (size_t)nb * 8 + 64)))
      return rc;
    a.thr = 1;
    a.bounds = (const long long *)c->gridBounds.p;
    a.colPerUnit[0] = (float)(g.scale[0] * g.unit / cell);
    a.colPerUnit[1] = (float)(g.scale[1] * g.unit / cell);
    { gridBoundsKernel<<<(unsigned)((nb + 127) / 128), 128, 0, c->stream>>>(a, (long long *)c->gridBounds.p); ++c->launches; }
  }
  unsigned long long *dStray = (unsigned long long *)((char *)c->small.p + 256);
  int *dExt = (int *)((char *)c->small.p + 512);
  static const int kExtInit[6] = {INT32_MAX, INT32_MAX, INT32_MAX, INT32_MIN, INT32_MIN, INT32_MIN};
  WB_CUDA(c, cudaMemsetAsync(dStray, 0, 8, c->stream));
  WB_CUDA(c, cudaMemcpyAsync(dExt, kExtInit, 24, cudaMemcpyDefault, c->stream));
  unsigned blocks = (unsigned)std::min<uint64_t>((nd + 255) / 256 + 1, (uint64_t)c->sm_count * 16);
  // a counting sort by column (counts, their prefix, the points' places), then
  // each column by height
  uint32_t *start = (uint32_t *)c->cellStart.p, *count = start + ncell + 1, *rank = (uint32_t *)c->gVal0.p;
  uint32_t *dBig = (uint32_t *)((char *)c->small.p + 640);   // big columns, and whether one was too big
  uint64_t *slots = (uint64_t *)c->gKey0.p;
  const int32_t *sx = (const int32_t *)c->sx.p, *sy = (const int32_t *)c->sy.p, *sz = (const int32_t *)c->sz.p;
  const uint8_t *stray = (const uint8_t *)c->stray.p;
  const int2 *colOf = (const int2 *)c->colOf.p;
  int4 *gpt = (int4 *)c->gpt.p, *cellRec = (int4 *)c->cellRec.p;
  const int *err = wb_lookback_err(c);
  WB_CUDA(c, cudaMemsetAsync(count, 0, (ncell + 1) * 4, c->stream));
  WB_CUDA(c, cudaMemsetAsync(dBig, 0, 8, c->stream));
  { cellKernel<<<blocks, 256, 0, c->stream>>>(a, sx, sy, sz, count, rank, (uint8_t *)c->stray.p, dStray, dExt,
                                              (const double *)c->xyzd.p, (int2 *)c->colOf.p); ++c->launches; }
  if ((rc = wb_exclusive_scan_u32(c, count, start, ncell + 1, nullptr)))
    return rc;
  { cellScatterKernel<<<blocks, 256, 0, c->stream>>>(nd, nx, ny, colOf, rank, start, sz, slots, err); ++c->launches; }
  { columnKernel<<<(unsigned)((ncell + kColumnWarps - 1) / kColumnWarps), 32 * kColumnWarps, 0, c->stream>>>(
        ncell, start, slots, sx, sy, sz, stray, gpt, cellRec, count, dBig, err); ++c->launches; }
  { bigColumnKernel<<<(unsigned)c->sm_count, 512, 0, c->stream>>>(count, dBig, start, slots, sx, sy, sz, stray, gpt, cellRec,
                                                                  dBig + 1); ++c->launches; }
  WB_CUDA(c, cudaGetLastError());
  unsigned char back[WB_SMALL_LOOKBACK + 4];   // the scratch block's words, in one copy
  WB_CUDA(c, cudaMemcpyAsync(back, c->small.p, sizeof back, cudaMemcpyDefault, c->stream));
  WB_CUDA(c, cudaStreamSynchronize(c->stream));
  unsigned long long ns;
  int ext[6], gaveUp;
  uint32_t bigs[2];
  memcpy(&ns, back + 256, 8);
  memcpy(ext, back + 512, 24);
  memcpy(bigs, back + 640, 8);
  memcpy(&gaveUp, back + WB_SMALL_LOOKBACK, 4);
  if (gaveUp)
    return wb_lookback_failed(c, "column grid");
  if (bigs[1])
  {
    // a column of more than kBigColumnMax points (an outlier far from the rest
    // stretches the grid): all points by radix passes
    uint64_t *key = (uint64_t *)c->gKey0.p;
    uint32_t *val = (uint32_t *)c->gVal0.p;
    int bits = 1;
    while ((1ull << bits) < ncell)
      bits++;
    { cellKeyKernel<<<blocks, 256, 0, c->stream>>>(nd, nx, ny, colOf, sz, key); ++c->launches; }
    if ((rc = wb_radix_sort_pairs(c, key, val, (uint64_t *)c->gKey1.p, (uint32_t *)c->gVal1.p, nd, 0, 32 + bits, ~0ull, true)))
      return rc;
    { cellFillKernel<<<(unsigned)((ncell * 32 + 255) / 256), 256, 0, c->stream>>>(ncell, start, val, sx, sy, sz, stray, gpt,
                                                                                 cellRec, err); ++c->launches; }
    WB_CUDA(c, cudaMemcpyAsync(&gaveUp, err, 4, cudaMemcpyDefault, c->stream));
    WB_CUDA(c, cudaStreamSynchronize(c->stream));
    if (gaveUp)
      return wb_lookback_failed(c, "column grid");
  }
  int snx = (nx + WB_SUPER - 1) / WB_SUPER, sny = (ny + WB_SUPER - 1) / WB_SUPER;
  c->grid.snx = snx;
  c->grid.sny = sny;
  uint64_t nsup = (uint64_t)snx * sny;
  if ((rc = wb_ensure(c, c->superRec, nsup * 32 + 64)))
    return rc;
  { superKernel<<<(unsigned)std::min<uint64_t>((nsup + 255) / 256, (uint64_t)c->sm_count * 16), 256, 0, c->stream>>>(
        nx, ny, snx, sny, (const int4 *)c->cellRec.p, (int4 *)c->superRec.p); ++c->launches; }
  WB_CUDA(c, cudaGetLastError());
  c->grid.grouped = c->grid.colGrouped = false;
  c->grid.nColGroups = 0;
  c->grid.nStray = (uint32_t)ns;
  c->grid.nBeside = ns >> 32;
  for (int k = 0; k < 3; k++)
  {
    c->grid.imin[k] = ext[k];
    c->grid.imax[k] = ext[3 + k];
  }
  if (c->grid.nBeside)
  {
    if ((rc = wb_ensure(c, c->strayCol, ncell * 32 + 64)) || (rc = wb_ensure(c, c->straySuper, nsup * 32 + 64)))
      return rc;
    { strayColumnKernel<<<(unsigned)std::min<uint64_t>((ncell * 32 + 255) / 256, (uint64_t)c->sm_count * 32), 256, 0, c->stream>>>(
          ncell, strayArgs(c), cellRec, gpt, (int4 *)c->strayCol.p); ++c->launches; }
    { straySuperKernel<<<(unsigned)std::min<uint64_t>((nsup + 255) / 256, (uint64_t)c->sm_count * 16), 256, 0, c->stream>>>(
          nx, ny, snx, sny, cellRec, (const int4 *)c->superRec.p, (const int4 *)c->strayCol.p, (int4 *)c->straySuper.p); ++c->launches; }
    WB_CUDA(c, cudaGetLastError());
  }
  return 0;
}

/* The column groups of the margin pass (groups of consecutive points of a
 * column), formed once per grid when a classify first wants margins;
 * synchronises then. */
int wb_column_groups(wb_ctx *c, const uint2 **groups, uint64_t *count)
{
  const uint64_t ncell = c->grid.ncell, nd = c->nd;
  uint32_t *gTot = (uint32_t *)((char *)c->small.p + 640);
  int rc;
  *groups = (const uint2 *)c->colGroups.p;
  *count = c->grid.nColGroups;
  if (c->grid.colGrouped || !nd)
    return 0;
  if ((rc = wb_ensure(c, c->groupCnt, (ncell + 1) * 8 + 64)))
    return rc;
  uint32_t *gcnt = (uint32_t *)c->groupCnt.p, *gfirst = gcnt + ncell + 1;
  const unsigned blocks = (unsigned)std::min<uint64_t>((ncell + 255) / 256, (uint64_t)c->sm_count * 16);
  { groupCountKernel<<<blocks, 256, 0, c->stream>>>(ncell, (const int4 *)c->cellRec.p, gcnt); ++c->launches; }
  if ((rc = wb_exclusive_scan_u32(c, gcnt, gfirst, ncell, gTot)))
    return rc;
  // at most nd / 32 + ncell groups
  if ((rc = wb_ensure(c, c->colGroups, (nd / 32 + ncell + 1) * 8 + 64)))
    return rc;
  { groupFillKernel<<<blocks, 256, 0, c->stream>>>(ncell, (const int4 *)c->cellRec.p, gfirst, (uint2 *)c->colGroups.p,
                                                    wb_lookback_err(c)); ++c->launches; }
  WB_CUDA(c, cudaGetLastError());
  uint32_t ngroups = 0;
  int gaveUp = 0;
  WB_CUDA(c, cudaMemcpyAsync(&ngroups, gTot, 4, cudaMemcpyDefault, c->stream));
  WB_CUDA(c, cudaMemcpyAsync(&gaveUp, wb_lookback_err(c), 4, cudaMemcpyDefault, c->stream));
  WB_CUDA(c, cudaStreamSynchronize(c->stream));
  if (gaveUp)
    return wb_lookback_failed(c, "wb_classify");
  *groups = (const uint2 *)c->colGroups.p;
  *count = c->grid.nColGroups = ngroups;
  c->grid.colGrouped = true;
  return 0;
}

/* The point groups of the fast pass, formed once per grid when a classify
 * first wants them (an octree or a scan alone does not).  Their number stays on
 * the device: *taken, groups above the low 36 bits. */
int wb_point_groups(wb_ctx *c, const unsigned long long **taken, uint64_t *maxGroups)
{
  unsigned long long *gTot = (unsigned long long *)((char *)c->small.p + 704);
  const uint64_t nd = c->nd, nsup = (uint64_t)c->grid.snx * c->grid.sny;
  // at most 32 points each, two partly filled ones per super-cell
  const uint64_t most = nd / 32 + 2 * std::min<uint64_t>(nsup, nd) + 1;
  *taken = gTot;
  *maxGroups = most;
  if (c->grid.grouped)
    return 0;
  int rc;
  if ((rc = wb_ensure(c, c->groups, most * 36 + 64)) || (c->grid.nBeside && (rc = wb_ensure(c, c->strayGrp, most * 32 + 64))))
    return rc;
  WB_CUDA(c, cudaMemsetAsync(gTot, 0, 16, c->stream));
  if (nd)
  {
    const WbGeom &g = c->g;
    // the points in group order take the place of the grid sort's key buffers
    { groupOrderKernel<<<(unsigned)nsup, kOrderThreads, 0, c->stream>>>(
          c->grid.nx, c->grid.ny, c->grid.snx, c->grid.sny, (float)(c->grid.cell / fabs(g.scale[2] * g.unit)),
          (const int4 *)c->cellRec.p, (int4 *)c->superRec.p, (const int4 *)c->gpt.p, (int2 *)c->gKey0.p,
          (int2 *)c->gKey1.p, (int4 *)c->groups.p, most, gTot); ++c->launches; }
    { groupBoxKernel<<<(unsigned)std::min<uint64_t>((nd / 32 + 8) / 8, (uint64_t)c->sm_count * 16), 256, 0, c->stream>>>(
          strayArgs(c), gTot, (const int2 *)c->gKey0.p, (const int2 *)c->gKey1.p, (int4 *)c->groups.p,
          (int4 *)c->strayGrp.p); ++c->launches; }
    WB_CUDA(c, cudaGetLastError());
  }
  c->grid.grouped = true;
  return 0;
}
