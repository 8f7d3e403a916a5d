/* Octree build on the GPU: the replacement for OctStore::put / split.
 *
 * The reference inserts points one at a time and splits a block when a 538th
 * distinct point arrives (octree.cpp:620-662, 1295-1338).  Because a split
 * never merges and de-duplication is by exact xyz, the final tree depends only
 * on the set of distinct points: a node is internal iff its cube holds more
 * than 537 distinct points (the root is always internal), and every non-empty
 * octant of an internal node that is not itself internal is a leaf block.
 * The build therefore needs no insertion order:
 *
 *   K1  decode X,Y,Z like las.cpp:808 and compute a 63-bit Morton key whose
 *       every bit is one of the reference's x>=center decisions
 *   K2  stable radix sort of (key, input index)
 *   K3  mark duplicates (same doubles; the last one read survives, as
 *       OctBuffer::put overwrites) and compact
 *   K4  common-prefix level of keys 537 apart; the leaf level of a point is
 *       1 + the largest such level over the 538-point windows that contain it
 *       (a node holds >537 points iff one window fits inside it)
 *   K5  leaf starts, leaf table, per-leaf order by input index
 */
#include <cuda_runtime.h>
#include <cstdint>
#include <cstring>
#include <cmath>
#include "wb_internal.h"
#include "wb_device.cuh"
#include "wb_lookback.cuh"
#include "wb_warpsort.cuh"

namespace
{
constexpr int kWindow = WB_RECORDS + 1;   // 538 points: the first that forces a split

struct KeyArgs
{
  const uint8_t *rec;
  uint64_t n;
  uint32_t stride;
  double off[3], scale[3], unit;
  double lo[3], cell;
  /* Fixed-point form of the level-21 cell coordinate, per axis:
     t(X) = (C + (X - x0) * R) / 2^shift, with |X - x0| <= dmax.  A point
     whose fraction lies more than eps from an integer takes floor(t); for the
     rest the decoded coordinate is compared with that one boundary (eps is
     below half of 2^shift).  All of an axis with fixed = 0 take the general
     FP64 path. */
  int fixed[3], shift[3];
  long long x0[3], dmax[3], rfix[3], cfix[3], eps[3];
};

__device__ __forceinline__ void loadXYZ(const uint8_t *rec, uint32_t stride, uint64_t i, int32_t &x, int32_t &y,
                                        int32_t &z)
{
  const uint8_t *p = rec + i * (uint64_t)stride;
  if ((stride & 3) == 0)
  {
    const int32_t *q = (const int32_t *)p;
    x = q[0];
    y = q[1];
    z = q[2];
  }
  else
  {
    int32_t v[3];
    memcpy(v, p, 12);
    x = v[0];
    y = v[1];
    z = v[2];
  }
}

__global__ void keyKernel(KeyArgs a, uint64_t *__restrict__ keys)
{
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < a.n; i += (uint64_t)gridDim.x * blockDim.x)
  {
    int32_t q[3];
    loadXYZ(a.rec, a.stride, i, q[0], q[1], q[2]);
    uint32_t k[3];
#pragma unroll
    for (int ax = 0; ax < 3; ax++)
    {
      const long long d = (long long)q[ax] - a.x0[ax];
      const long long kMax = (1 << WB_LEVELS) - 1;
      if (a.fixed[ax] && d >= -a.dmax[ax] && d <= a.dmax[ax])
      {
        const long long tf = d * a.rfix[ax] + a.cfix[ax];
        long long k0 = tf >> a.shift[ax];
        const long long fr = tf - k0 * (1ll << a.shift[ax]);
        // within eps of cell boundary kb: the decoded coordinate decides (cell
        // sides are dyadic, so with decimal coordinates one point in 125 lies
        // on a boundary and most warps hold one: six FP64 instructions here,
        // where the general search took 40 and the FP64 pipe bounded the kernel)
        const bool below = fr <= a.eps[ax], above = fr >= (1ll << a.shift[ax]) - a.eps[ax];
        if (below || above)
        {
          const long long kb = k0 + above;
          k0 = wb_decode(q[ax], a.off[ax], a.scale[ax], a.unit) >= a.lo[ax] + wb_double((int)kb) * a.cell ? kb : kb - 1;
        }
        k[ax] = (uint32_t)(k0 < 0 ? 0 : (k0 > kMax ? kMax : k0));
      }
      else
        k[ax] = wb_cell_index(wb_decode(q[ax], a.off[ax], a.scale[ax], a.unit), a.lo[ax], a.cell);
    }
    keys[i] = wb_morton(k[0], k[1], k[2]);
  }
}

__device__ __forceinline__ bool sameDoubles(const KeyArgs &a, uint32_t i, uint32_t j)
{
  int32_t p[3], q[3];
  loadXYZ(a.rec, a.stride, i, p[0], p[1], p[2]);
  loadXYZ(a.rec, a.stride, j, q[0], q[1], q[2]);
#pragma unroll
  for (int ax = 0; ax < 3; ax++)
    if (wb_decode(p[ax], a.off[ax], a.scale[ax], a.unit) != wb_decode(q[ax], a.off[ax], a.scale[ax], a.unit))
      return false;
  return true;
}

/* The counters of a build, in the context's scratch block from
 * WB_SMALL_LOOKBACK on. */
struct BuildFlags
{
  int lookback;        /* a look-back gave up (kept by the primitives too)    */
  uint32_t dups;       /* records a later identical point replaced            */
  uint32_t longRuns;   /* runs of equal sorted bits too long for runKernel     */
  uint32_t unsorted;   /* one of them was too long for longRunKernel as well   */
  uint32_t leaves;
  int tooDeep, maxLevel;
};

/* Whether sorted record i survives: no later record of its key has the same xyz. */
__device__ __forceinline__ bool survives(const KeyArgs &a, const uint64_t *keys, const uint32_t *idx, uint64_t i)
{
  const uint64_t k = keys[i];
  for (uint64_t j = i + 1; j < a.n && keys[j] == k; j++)
    if (sameDoubles(a, idx[i], idx[j]))
      return false;
  return true;
}

__device__ __forceinline__ void countDups(uint32_t dups, BuildFlags *f)
{
  dups = __reduce_add_sync(0xffffffffu, dups);
  if ((threadIdx.x & 31) == 0 && dups)
    atomicAdd(&f->dups, dups);
}

/* The radix sort orders the keys' bits from `begin` up, enough of them to tell
 * almost all points apart; this finishes the order and marks the survivors.
 * One thread per run of equal sorted bits (its first record's): runs are one or
 * two points long, and the run is in input order for equal keys, so a stable
 * insertion sort of the rest of the key gives the full sort's order.  Longer
 * runs are listed for longRunKernel.
 * 145 us for 20M points (keys read, flags written); with it five radix passes do
 * where eight did (50M points: sort 4.4 -> 2.3 ms). */
constexpr int kRunMax = 32;
__global__ void runKernel(KeyArgs a, int begin, uint64_t *keys, uint32_t *idx, uint8_t *__restrict__ surv,
                          uint32_t *__restrict__ longRuns, BuildFlags *f)
{
  uint32_t dups = 0;
  if (!f->lookback)
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < a.n; i += (uint64_t)gridDim.x * blockDim.x)
    {
      const uint64_t p = keys[i] >> begin;
      if (i && (keys[i - 1] >> begin) == p)
        continue;
      int m = 1;
      while (m <= kRunMax && i + m < a.n && (keys[i + m] >> begin) == p)
        m++;
      if (m > kRunMax)
      {
        longRuns[atomicAdd(&f->longRuns, 1u)] = (uint32_t)i;
        continue;
      }
      for (int q = 1; q < m; q++)
      {
        const uint64_t k = keys[i + q];
        const uint32_t v = idx[i + q];
        int b = q;
        for (; b > 0 && keys[i + b - 1] > k; b--)
        {
          keys[i + b] = keys[i + b - 1];
          idx[i + b] = idx[i + b - 1];
        }
        if (b != q)
        {
          keys[i + b] = k;
          idx[i + b] = v;
        }
      }
      for (int q = 0; q < m; q++)
      {
        // later records of the run only: another run may be on the move
        bool s = true;
        const uint64_t k = keys[i + q];
        for (int u = q + 1; s && u < m && keys[i + u] == k; u++)
          s = !sameDoubles(a, idx[i + q], idx[i + u]);
        surv[i + q] = s;
        dups += !s;
      }
    }
  countDups(dups, f);
}

/* The listed runs, one block each: sorted by (key, input index) in shared
 * memory up to kLongRunMax points (lines and stacks of points); a longer one
 * raises `unsorted` and the caller sorts all bits. */
constexpr int kLongRunMax = 2048;
__global__ void __launch_bounds__(256) longRunKernel(KeyArgs a, int begin, uint64_t *keys, uint32_t *idx,
                                                     uint8_t *__restrict__ surv, const uint32_t *__restrict__ longRuns,
                                                     BuildFlags *f)
{
  __shared__ uint64_t k[kLongRunMax];
  __shared__ uint32_t v[kLongRunMax];
  __shared__ int len;
  uint32_t dups = 0;
  const uint32_t runs = f->longRuns;
  for (uint32_t r = blockIdx.x; r < runs; r += gridDim.x)
  {
    const uint64_t i = longRuns[r], p = keys[i] >> begin;
    __syncthreads();
    if (threadIdx.x == 0)
      len = kLongRunMax + 1;
    __syncthreads();
    for (int q = threadIdx.x; q <= kLongRunMax; q += 256)
      if (i + q >= a.n || (keys[i + q] >> begin) != p)
      {
        atomicMin(&len, q);
        break;
      }
    __syncthreads();
    const int m = len;
    if (m > kLongRunMax)
    {
      if (threadIdx.x == 0)
        f->unsorted = 1;
      continue;
    }
    int P = 64;
    while (P < m)
      P <<= 1;
    for (int q = threadIdx.x; q < P; q += 256)
    {
      k[q] = q < m ? keys[i + q] : ~0ull;
      v[q] = q < m ? idx[i + q] : ~0u;
    }
    __syncthreads();
    for (int size = 2; size <= P; size <<= 1)
      for (int j = size >> 1; j > 0; j >>= 1)
      {
        for (int q = threadIdx.x; q < P; q += 256)
        {
          const int u = q ^ j;
          if (u > q)
          {
            const bool up = (q & size) == 0;
            const uint64_t kx = k[q], ky = k[u];
            const uint32_t vx = v[q], vy = v[u];
            if ((kx > ky || (kx == ky && vx > vy)) == up)
            {
              k[q] = ky;
              k[u] = kx;
              v[q] = vy;
              v[u] = vx;
            }
          }
        }
        __syncthreads();
      }
    for (int q = threadIdx.x; q < m; q += 256)
    {
      keys[i + q] = k[q];
      idx[i + q] = v[q];
      bool s = true;
      for (int u = q + 1; s && u < m && k[u] == k[q]; u++)
        s = !sameDoubles(a, v[q], v[u]);
      surv[i + q] = s;
      dups += !s;
    }
  }
  countDups(dups, f);
}

/* The survivors of fully sorted keys. */
__global__ void survivorKernel(KeyArgs a, const uint64_t *__restrict__ keys, const uint32_t *__restrict__ idx,
                               uint8_t *__restrict__ surv, BuildFlags *f)
{
  uint32_t dups = 0;
  if (!f->lookback)
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < a.n; i += (uint64_t)gridDim.x * blockDim.x)
    {
      const bool s = survives(a, keys, idx, i);
      surv[i] = s;
      dups += !s;
    }
  countDups(dups, f);
}

/* The survivors' keys and indices, closed up. */
struct CompactScan
{
  const uint8_t *surv;
  const uint64_t *keys;
  const uint32_t *idx;
  uint64_t *dkey;
  uint32_t *didx;
  __device__ uint32_t value(uint64_t i, bool ok) const { return ok ? __ldg(surv + i) : 0; }
  __device__ void put(uint64_t i, uint32_t before, uint32_t v) const
  {
    if (v)
    {
      dkey[before] = __ldg(keys + i);   // (read past the stores of the items before)
      didx[before] = __ldg(idx + i);
    }
  }
};
template <int ITEMS>
__global__ void __launch_bounds__(256) compactKernel(uint64_t n, CompactScan f, unsigned *counter,
                                                     unsigned long long *status, int *err)
{
  lookbackScan<ITEMS>(n, f, counter, status, nullptr, err);
}

/* Prefix and suffix maxima, inside aligned segments of kWindow windows, of
 * the common levels of keys kWindow - 1 apart (van Herk / Gil-Werman): one warp
 * per segment, the levels of its windows in registers between the two. */
__global__ void segMaxKernel(const uint64_t *__restrict__ dkey, uint64_t nw, uint8_t *__restrict__ pre,
                             uint8_t *__restrict__ suf)
{
  constexpr int ROWS = (kWindow + 31) / 32;
  const uint64_t seg = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const uint64_t b = seg * kWindow;
  if (b >= nw)
    return;
  const uint64_t e = b + kWindow < nw ? b + kWindow : nw;
  int v[ROWS];
#pragma unroll
  for (int r = 0; r < ROWS; r++)
  {
    const uint64_t s = b + 32 * r + lane;
    v[r] = s < e ? wb_common_levels(dkey[s], dkey[s + kWindow - 1]) : 0;
  }
  int run = 0;
#pragma unroll
  for (int r = 0; r < ROWS; r++)
  {
    const uint64_t s = b + 32 * r + lane;
    int x = v[r];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
      const int t = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o)
        x = max(x, t);
    }
    x = max(x, run);
    if (s < e)
      pre[s] = (uint8_t)x;
    run = __shfl_sync(0xffffffffu, x, 31);
  }
  run = 0;
#pragma unroll
  for (int r = ROWS - 1; r >= 0; r--)
  {
    const uint64_t s = b + 32 * r + lane;
    int x = v[r];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
      const int t = __shfl_down_sync(0xffffffffu, x, o);
      if (lane + o < 32)
        x = max(x, t);
    }
    x = max(x, run);
    if (s < e)
      suf[s] = (uint8_t)x;
    run = __shfl_sync(0xffffffffu, x, 0);
  }
}

__device__ __forceinline__ uint64_t prefixAt(uint64_t key, int level)
{
  return level <= 0 ? 0 : key >> (63 - 3 * level);
}

/* The leaves: point i's leaf level is 1 + the largest common level over the
 * windows [s, s + 537] that contain it; a leaf starts where the level or the
 * key's prefix at that level changes.  One pass forms the leaf of every point
 * and the leaf table (up to cap entries: the caller makes room and runs it
 * again when there are more). */
struct LeafScan
{
  uint64_t nw, cap;
  const uint64_t *dkey;
  const uint8_t *pre, *suf;
  uint32_t *leafId, *first;
  uint8_t *leafLev;
  uint64_t *leafKey;
  BuildFlags *f;
  __device__ int level(uint64_t i) const
  {
    int d = 0;
    if (nw > 0)
    {
      const uint32_t at = (uint32_t)i, last = (uint32_t)nw - 1;
      const uint32_t a = at >= (uint32_t)(kWindow - 1) ? at - (kWindow - 1) : 0;
      const uint32_t b = min(at, last);
      if (a <= b)
      {
        const uint32_t sa = a / kWindow, sb = b / kWindow;
        if (sa != sb)
          d = max((int)__ldg(suf + a), (int)__ldg(pre + b));
        else if (a == sa * kWindow)
          d = __ldg(pre + b);
        else
          d = __ldg(suf + a);
      }
    }
    if (d >= WB_LEVELS)
    {
      f->tooDeep = 1;
      d = WB_LEVELS - 1;
    }
    return d + 1;
  }
  /* Of a warp's 32 consecutive points, together: each has its neighbour's level
   * and key from the lane before. */
  __device__ uint32_t value(uint64_t i, bool ok) const
  {
    const int l = ok ? level(i) : 0;
    const uint64_t key = ok ? __ldg(dkey + i) : 0;
    int lb = __shfl_up_sync(0xffffffffu, l, 1);
    uint64_t kb = __shfl_up_sync(0xffffffffu, key, 1);
    if ((threadIdx.x & 31) == 0 && ok && i)
    {
      lb = level(i - 1);
      kb = __ldg(dkey + i - 1);
    }
    return ok && (i == 0 || lb != l || prefixAt(kb, l) != prefixAt(key, l));
  }
  __device__ void put(uint64_t i, uint32_t before, uint32_t v) const
  {
    const uint32_t l = before + v - 1;
    leafId[i] = l;
    if (v && l < cap)
    {
      const int lv = level(i);
      first[l] = (uint32_t)i;
      leafLev[l] = (uint8_t)lv;
      const uint64_t mask = (lv >= WB_LEVELS) ? ~0ULL : ~((1ULL << (63 - 3 * lv)) - 1);
      leafKey[l] = dkey[i] & mask;
      if (lv > f->maxLevel)
        atomicMax(&f->maxLevel, lv);
    }
  }
};
template <int ITEMS>
__global__ void __launch_bounds__(256) leafKernel(uint64_t nd, LeafScan f, unsigned *counter, unsigned long long *status,
                                                  int *err)
{
  lookbackScan<ITEMS>(nd, f, counter, status, &f.f->leaves, err);
}

/* One warp per leaf: its input indices (<= 537) sorted in registers, X/Y/Z
 * gathered into store order, and each stored record's store slot.  50M points
 * in random order take 3.2 ms, bound by DRAM (53% of its rate: 135 bytes read and
 * 68 written a point, most for the record and the store slot, each alone in its
 * sector); 8M take 0.30 ms, 1M 0.047 (0.072 with a block per leaf and the sort in
 * shared memory, 11,300 warp instructions a leaf at 80% of the issue slots). */
constexpr int kLeafWarps = 4, kLeafRows = 4;
__global__ void __launch_bounds__(32 * kLeafWarps, 10) leafSortKernel(KeyArgs a, const uint32_t *__restrict__ first,
                                                               uint32_t *__restrict__ count,
                                                               const uint32_t *__restrict__ didx,
                                                               uint32_t *__restrict__ sidx, int32_t *__restrict__ sx,
                                                               int32_t *__restrict__ sy, int32_t *__restrict__ sz,
                                                               uint32_t *__restrict__ storeOf,
                                                               uint64_t L,
                                                               double *__restrict__ xyzd, uint64_t nd)
{
  __shared__ __align__(16) uint32_t buf[kLeafWarps][544];
  const int lane = threadIdx.x & 31;
  const uint64_t l = (uint64_t)blockIdx.x * kLeafWarps + (threadIdx.x >> 5);
  if (l >= L)
    return;
  uint32_t *v = buf[threadIdx.x >> 5];
  const uint32_t f = first[l], cnt = (uint32_t)((l + 1 < L ? first[l + 1] : nd) - f);
  if (lane == 0)
    count[l] = cnt;
  for (uint32_t t = lane; t < cnt; t += 32)
    v[t] = didx[f + t];
  __syncwarp();
  wb_warp_sort_1024(v, cnt, lane);
  // kLeafRows rows' records at once: they lie anywhere in the input
  for (uint32_t t0 = lane; t0 < cnt; t0 += 32 * kLeafRows)
  {
    uint32_t id[kLeafRows];
    int32_t q[kLeafRows][3];
#pragma unroll
    for (int r = 0; r < kLeafRows; r++)
      if (t0 + 32 * r < cnt)
      {
        id[r] = v[t0 + 32 * r];
        loadXYZ(a.rec, a.stride, id[r], q[r][0], q[r][1], q[r][2]);
      }
#pragma unroll
    for (int r = 0; r < kLeafRows; r++)
      if (t0 + 32 * r < cnt)
      {
        const uint32_t at = f + t0 + 32 * r;
        sidx[at] = id[r];
        sx[at] = q[r][0];
        sy[at] = q[r][1];
        sz[at] = q[r][2];
#pragma unroll
        for (int ax = 0; ax < 3; ax++)
          xyzd[(uint64_t)ax * nd + at] = wb_decode(q[r][ax], a.off[ax], a.scale[ax], a.unit);
        storeOf[id[r]] = at;
      }
  }
}

/* Records overwritten by a later duplicate point at the survivor's slot. */
__global__ void dupMapKernel(KeyArgs a, const uint64_t *__restrict__ keys, const uint32_t *__restrict__ idx,
                             const uint8_t *__restrict__ surv, uint32_t *__restrict__ storeOf)
{
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < a.n; i += (uint64_t)gridDim.x * blockDim.x)
    if (!surv[i])
    {
      uint64_t k = keys[i];
      uint64_t last = i;
      for (uint64_t j = i + 1; j < a.n && keys[j] == k; j++)
        if (sameDoubles(a, idx[i], idx[j]))
          last = j;
      storeOf[idx[i]] = storeOf[idx[last]];
    }
}

__global__ void pointLeafKernel(uint64_t n, const uint32_t *__restrict__ storeOf, const uint32_t *__restrict__ leafId,
                                uint32_t *__restrict__ pointLeaf)
{
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
    pointLeaf[i] = leafId[storeOf[i]];
}

}  // namespace

static unsigned gridFor(wb_ctx *c, uint64_t n, int threads = 256)
{
  uint64_t b = (n + threads - 1) / threads;
  uint64_t cap = (uint64_t)c->sm_count * 16;
  if (b > cap)
    b = cap;
  if (b < 1)
    b = 1;
  return (unsigned)b;
}

/* Sets up the fixed-point cell coordinate of axis k (see KeyArgs).  t is
 * the coordinate in cell units, (decode(X) - lo) / cell, linear in X up to
 * the rounding of decode; the error allowed for (eps) covers the rounding of
 * R and C to 2^-shift, the decode's two roundings and the double arithmetic
 * here, with a factor of 16 to spare. */
static void keyFixedPoint(const WbGeom &g, double mn, double mx, int k, KeyArgs &a)
{
  a.fixed[k] = 0;
  a.shift[k] = 0;
  a.x0[k] = a.dmax[k] = a.rfix[k] = a.cfix[k] = a.eps[k] = 0;
  const double u = g.scale[k] * g.unit;
  if (!(u > 0) || !(g.unit > 0) || !(g.cell > 0))
    return;
  const double R = u / g.cell;   // the cell is a power of two: exact
  double xlo = (fmin(mn, mx) / g.unit - g.off[k]) / g.scale[k], xhi = (fmax(mn, mx) / g.unit - g.off[k]) / g.scale[k];
  if (!(fabs(xlo) < 2e9) || !(fabs(xhi) < 2e9))
    return;
  const long long X0 = llround((xlo + xhi) / 2);
  const long long dmax = (long long)ceil(fmax(fabs(xlo - X0), fabs(xhi - X0))) + 4;
  const double x0d = (g.off[k] + g.scale[k] * (double)X0) * g.unit;
  const double C = (x0d - g.root_lo[k]) / g.cell;
  const double B = fabs(C) + (double)dmax * R + 4;
  int shift = 62 - (int)ceil(log2(B));
  if (shift > 40)
    shift = 40;
  if (shift < 24)
    return;
  const double one = ldexp(1.0, shift);
  // decode error: two roundings of |x| (<= |x0d| + dmax*u) and the subtraction of lo
  const double mag = fabs(x0d) + (double)dmax * u + fabs(g.root_lo[k]);
  const double errCells = (double)dmax / one + 1.0 / one + 8 * ldexp(mag, -52) / g.cell + ldexp(B, -50);
  // eps below half a cell, so that a point can be in doubt about one boundary
  // only, the one keyKernel compares it with: a cloud whose coordinates round
  // to more than that (a root cube of centimetres at 1e9) is searched in FP64
  if (!(16 * errCells < 0.5 - 32 / one))
    return;
  a.fixed[k] = 1;
  a.shift[k] = shift;
  a.x0[k] = X0;
  a.dmax[k] = dmax;
  a.rfix[k] = llround(R * one);
  a.cfix[k] = llround(C * one);
  a.eps[k] = (long long)ceil(16 * errCells * one) + 16;
}

/* The point -> leaf map of every record (leaf of its store slot), formed when
 * a caller asks for it: the pipeline itself reads store slots only. */
int wb_point_leaf_map(wb_ctx *c)
{
  const uint64_t n = c->n;
  int rc;
  if (!n)
    return 0;
  if ((rc = wb_ensure(c, c->pointLeaf, n * 4 + 64)))
    return rc;
  { pointLeafKernel<<<gridFor(c, n), 256, 0, c->stream>>>(n, (const uint32_t *)c->storeOf.p,
                                                          (const uint32_t *)c->leafId.p, (uint32_t *)c->pointLeaf.p); ++c->launches; }
  WB_CUDA(c, cudaGetLastError());
  return 0;
}

int wb_build_impl(wb_ctx *c, const wb_cloud *cl)
{
  if (!cl || !cl->records || cl->stride < 12)
    return wb_fail(c, WB_EINVAL, "wb_octree_build: records must be non-null with stride >= 12");
  if (cl->n > 0xfffffff0ull)
    return wb_fail(c, WB_EINVAL, "wb_octree_build: at most 2^32-16 points per cloud");
  uint64_t n = cl->n;
  // with paging, a cloud whose working set (about 340 B per point plus the
  // records) is above the HBM budget keeps its scratch buffers in host memory
  c->spill_cold = c->host_budget && c->budget &&
                  n * (340ull + (cl->device_resident ? 0 : cl->stride)) > c->budget;
  WbGeom &g = c->g;
  for (int a = 0; a < 3; a++)
  {
    g.off[a] = cl->offset[a];
    g.scale[a] = cl->scale[a];
  }
  g.unit = cl->unit;
  double mn[3], mx[3];
  for (int a = 0; a < 3; a++)
  {
    mn[a] = cl->minc[a] * cl->unit;
    mx[a] = cl->maxc[a] * cl->unit;
  }
  wb_size_fit(mn, mx, g.root_c, &g.root_side);
  if (!(g.root_side > 0))
    return wb_fail(c, WB_EINVAL, "wb_octree_build: header min/max enclose no volume");
  for (int a = 0; a < 3; a++)
    g.root_lo[a] = g.root_c[a] - g.root_side / 2;
  g.cell = ldexp(g.root_side, -WB_LEVELS);
  wb_tile_cube(mn, mx, g.tile_c, &g.tile_side);
  c->n = n;
  c->stage = 0;

  KeyArgs a;
  a.n = n;
  a.stride = cl->stride;
  for (int k = 0; k < 3; k++)
  {
    a.off[k] = g.off[k];
    a.scale[k] = g.scale[k];
    a.lo[k] = g.root_lo[k];
  }
  a.unit = g.unit;
  a.cell = g.cell;
  for (int k = 0; k < 3; k++)
    keyFixedPoint(g, mn[k], mx[k], k, a);

  int rc;
  if (cl->device_resident && n && !wb_device_accessible(cl->records))
    return wb_fail(c, WB_EINVAL, "wb_octree_build: device_resident records must be device memory");
  if (cl->device_resident)
    a.rec = (const uint8_t *)cl->records;
  else
  {
    if ((rc = wb_ensure(c, c->rec, n * (uint64_t)cl->stride)))
      return rc;
    if ((rc = wb_copy_in(c, c->rec.p, cl->records, n * (uint64_t)cl->stride)))
      return rc;
    a.rec = (const uint8_t *)c->rec.p;
  }
  wb_mark(c, "upload");
  if (n == 0)
  {
    c->nd = c->n_leaves = 0;
    c->grid = GridInfo{};   // no columns or groups of an earlier cloud
    c->stage = 1;
    return 0;
  }
  if ((rc = wb_ensure(c, c->key0, n * 8)) || (rc = wb_ensure(c, c->key1, n * 8)) ||
      (rc = wb_ensure(c, c->idx0, n * 4)) || (rc = wb_ensure(c, c->idx1, n * 4)) ||
      (rc = wb_ensure(c, c->tmp8, n)) || (rc = wb_ensure(c, c->storeOf, n * 4)) || (rc = wb_small(c)))
    return rc;
  BuildFlags *flags = (BuildFlags *)((char *)c->small.p + WB_SMALL_LOOKBACK), fl;
  auto readFlags = [&]() -> int {
    WB_CUDA(c, cudaMemcpyAsync(&fl, flags, sizeof fl, cudaMemcpyDefault, c->stream));
    WB_CUDA(c, cudaStreamSynchronize(c->stream));
    return fl.lookback ? wb_lookback_failed(c, "wb_octree_build") : 0;
  };
  WB_CUDA(c, cudaMemsetAsync(&flags->dups, 0, sizeof(BuildFlags) - 4, c->stream));
  uint64_t *keys = (uint64_t *)c->key0.p, *kAlt = (uint64_t *)c->key1.p;
  uint32_t *idx = (uint32_t *)c->idx0.p, *iAlt = (uint32_t *)c->idx1.p;
  uint8_t *surv = (uint8_t *)c->tmp8.p;
  { keyKernel<<<gridFor(c, n), 256, 0, c->stream>>>(a, keys); ++c->launches; }
  WB_CUDA(c, cudaGetLastError());
  wb_mark(c, "decode_key");
  auto swapIfMoved = [&]() {
    kAlt = (keys == (uint64_t *)c->key0.p) ? (uint64_t *)c->key1.p : (uint64_t *)c->key0.p;
    iAlt = (idx == (uint32_t *)c->idx0.p) ? (uint32_t *)c->idx1.p : (uint32_t *)c->idx0.p;
  };
  // The points lie on surfaces, so about log4(n) levels (three key bits each)
  // and one more tell nearly all apart; the nearest whole number of passes.
  const int passes = std::min(8, std::max(2, (int)((3 * (std::log2((double)n) / 2 + 1) + 4) / 8)));
  const int begin = std::max(0, 63 - 8 * passes);
  if ((rc = wb_radix_sort_pairs(c, keys, idx, kAlt, iAlt, n, begin, 63, ~0ull, true)))
    return rc;
  swapIfMoved();
  wb_mark(c, "sort");
  // (the list of long runs takes the free half of the index buffers)
  { runKernel<<<gridFor(c, n), 256, 0, c->stream>>>(a, begin, keys, idx, surv, iAlt, flags); ++c->launches; }
  { longRunKernel<<<(unsigned)c->sm_count, 256, 0, c->stream>>>(a, begin, keys, idx, surv, iAlt, flags); ++c->launches; }
  WB_CUDA(c, cudaGetLastError());
  if ((rc = readFlags()))
    return rc;
  if (fl.unsorted)
  {
    // the runs' partial order is stable, so sorting all bits gives the full order
    WB_CUDA(c, cudaMemsetAsync(&flags->dups, 0, 4, c->stream));
    if ((rc = wb_radix_sort_pairs(c, keys, idx, kAlt, iAlt, n, 0, 63)))
      return rc;
    swapIfMoved();
    { survivorKernel<<<gridFor(c, n), 256, 0, c->stream>>>(a, keys, idx, surv, flags); ++c->launches; }
    if ((rc = readFlags()))
      return rc;
  }
  const uint64_t nd = n - fl.dups;
  c->nd = nd;
  uint64_t *dkey = keys;
  uint32_t *didx = idx;
  unsigned *counter;
  unsigned long long *status;
  // Scans of less than a tile per SM use tiles of a quarter: a thread's items
  // come one after another (10,000 points: leafKernel 29 us with 16 a thread, 9.6 with 4)
  const bool few = n <= (uint64_t)c->sm_count * kScanTile;
  const uint64_t scanTile = few ? kScanTile / 4 : kScanTile;
  if (nd != n)
  {
    dkey = kAlt;
    didx = iAlt;
    const uint64_t tiles = (n + scanTile - 1) / scanTile;
    if ((rc = wb_lookback_words(c, tiles, &counter, &status)))
      return rc;
    { (few ? compactKernel<4> : compactKernel<kScanItems>)<<<(unsigned)tiles, 256, 0, c->stream>>>(n, CompactScan{surv, keys, idx, dkey, didx}, counter, status,
                                                            &flags->lookback); ++c->launches; }
  }
  wb_mark(c, "dedup");

  const uint64_t nw = nd >= (uint64_t)kWindow ? nd - kWindow + 1 : 0;
  if ((rc = wb_ensure(c, c->pre, nw + 64)) || (rc = wb_ensure(c, c->suf, nw + 64)) ||
      (rc = wb_ensure(c, c->leafId, nd * 4 + 64)))
    return rc;
  uint8_t *pre = (uint8_t *)c->pre.p, *suf = (uint8_t *)c->suf.p;
  if (nw)
  {
    const uint64_t segs = (nw + kWindow - 1) / kWindow;
    { segMaxKernel<<<(unsigned)((segs * 32 + 255) / 256), 256, 0, c->stream>>>(dkey, nw, pre, suf); ++c->launches; }
  }
  // room for the leaves a surface usually has (200 to 300 points each); more
  // are counted, then made room for
  uint64_t L = std::min<uint64_t>(nd, nd / 64 + 4096);
  for (int tries = 0;; tries++)
  {
    if ((rc = wb_ensure(c, c->leafFirst, L * 4 + 64)) || (rc = wb_ensure(c, c->leafCount, L * 4 + 64)) ||
        (rc = wb_ensure(c, c->leafLevel, L + 64)) || (rc = wb_ensure(c, c->leafKey, L * 8 + 64)))
      return rc;
    const uint64_t tiles = (nd + scanTile - 1) / scanTile;
    if ((rc = wb_lookback_words(c, tiles, &counter, &status)))
      return rc;
    { (few ? leafKernel<4> : leafKernel<kScanItems>)<<<(unsigned)tiles, 256, 0, c->stream>>>(
          nd, LeafScan{nw, L, dkey, pre, suf, (uint32_t *)c->leafId.p, (uint32_t *)c->leafFirst.p,
                       (uint8_t *)c->leafLevel.p, (uint64_t *)c->leafKey.p, flags}, counter, status,
          &flags->lookback); ++c->launches; }
    WB_CUDA(c, cudaGetLastError());
    if ((rc = readFlags()))
      return rc;
    if (fl.tooDeep)
      return wb_fail(c, WB_EDEPTH, "wb_octree_build: more than 537 distinct points in a cell 21 levels below the root");
    const bool fits = fl.leaves <= L;
    L = fl.leaves;
    if (fits || tries)
      break;
  }
  c->n_leaves = L;
  c->max_depth = (uint32_t)fl.maxLevel;
  if ((rc = wb_ensure(c, c->sidx, nd * 4 + 64)) || (rc = wb_ensure(c, c->sx, nd * 4 + 64)) ||
      (rc = wb_ensure(c, c->sy, nd * 4 + 64)) || (rc = wb_ensure(c, c->sz, nd * 4 + 64)) ||
      (rc = wb_ensure(c, c->xyzd, nd * 24 + 64)))
    return rc;
  wb_mark(c, "leaves");
  uint32_t *storeOf = (uint32_t *)c->storeOf.p;
  { leafSortKernel<<<(unsigned)((L + kLeafWarps - 1) / kLeafWarps), 32 * kLeafWarps, 0, c->stream>>>(a, (const uint32_t *)c->leafFirst.p,
                                                               (uint32_t *)c->leafCount.p, didx, (uint32_t *)c->sidx.p,
                                                               (int32_t *)c->sx.p, (int32_t *)c->sy.p, (int32_t *)c->sz.p,
                                                               storeOf, L, (double *)c->xyzd.p, nd); ++c->launches; }
  // records a later identical point overwrote take their survivor's slot
  if (nd != n)
    { dupMapKernel<<<gridFor(c, n), 256, 0, c->stream>>>(a, keys, idx, surv, storeOf); ++c->launches; }
  WB_CUDA(c, cudaGetLastError());
  wb_mark(c, "leaf_order");
  c->grid_bounds[0] = mn[0];
  c->grid_bounds[1] = mn[1];
  c->grid_bounds[2] = mx[0];
  c->grid_bounds[3] = mx[1];
  if ((rc = wb_grid_impl(c, mn[0], mn[1], mx[0], mx[1])))
    return rc;
  wb_mark(c, "grid");
  c->stage = 1;
  return 0;
}
