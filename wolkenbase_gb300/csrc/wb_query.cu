/* Shape queries over the device-resident octree: Octree::findBlocks
 * (octree.cpp:234-251) and OctStore::pointsIn (octree.cpp:1214-1242) for the
 * two shapes the classification path asks about, a Cylinder (shape.cpp:
 * 214-238) and a downward Hyperboloid (shape.cpp:119-159).
 *
 * findBlocks descends from the root into every octant whose cube the shape
 * intersects (Shape::intersect: the shape holds the cube's closest point,
 * shape.cpp:63-66).  For these convex shapes a cube that meets the shape has
 * every ancestor meeting it too, so the blocks found are exactly the leaves
 * whose own cube meets the shape, in depth-first order -- the leaf table's
 * order.  pointsIn then takes a whole block when all eight corners of its
 * cube are inside (Shape::in(Cube), shape.cpp:50-61) and otherwise every
 * point the shape holds, in store order; sorted=true orders the result by
 * height (the reference's std::sort by z leaves ties in no particular order;
 * here ties keep the unsorted order).
 *
 * One thread per leaf lists the leaves that meet the shape, in order, in one
 * pass (a look-back scan).  A query that meets few leaves (up to kFewLeaves: a
 * neighbourhood) is answered by one block, which tests the leaves' points, places
 * them, sorts them when asked and writes them to pinned host memory, so the
 * call is two kernels and one wait.  Larger ones count, scan, fill and
 * radix-sort over the listed leaves.  Points are tested in FP32 relative to the
 * shape, exactly in FP64 within 1e-5 of its surface: FP64 issues at 1/64 rate.
 * A sorted hyperboloid query of 2M points: 388 us before (a warp per leaf, FP64
 * throughout, eight allocations and waits), of which 80% was allocation,
 * launches and waits.
 */
#include <cuda_runtime.h>
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <string>
#include <vector>
#include "wb_internal.h"
#include "wb_device.cuh"
#include "wb_lookback.cuh"

namespace
{
struct QShape
{
  int kind;
  double cx, cy, cz;   /* cylinder: centre (z unused); hyperboloid: centre v + (0, 0, por) */
  double r;            /* cylinder radius */
  double por2, slope;  /* hyperboloid */
};

struct QArgs
{
  QShape s;
  uint64_t L;
  const uint64_t *leafKey;
  const uint8_t *leafLev;
  const uint32_t *first, *count;
  const double *xyzd;   /* decoded x, y, z planes of nd doubles */
  uint64_t nd;
  const uint32_t *sidx;
  double rootLo[3], rootSide;
};

__device__ __forceinline__ bool shapeIn(const QShape &s, double x, double y, double z)
{
  if (s.kind == WB_SHAPE_CYLINDER)
    return wb_hypot(s.cx - x, s.cy - y) <= s.r;
  return wb_hyp_in(s.cx, s.cy, s.cz, s.por2, s.slope, x, y, z);
}

/* Shape::intersect (shape.cpp:63-66) with closestPoint of the Cylinder
 * (shape.cpp:220-238: the cube's centre height) or the Hyperboloid
 * (shape.cpp:137-159: the cube's bottom for a downward one, top otherwise). */
__device__ __forceinline__ bool shapeMeets(const QShape &s, double cx, double cy, double cz, double side)
{
  const double x = wb_clamp_toward(s.cx, cx, side), y = wb_clamp_toward(s.cy, cy, side);
  double z = cz;
  if (s.kind == WB_SHAPE_HYPERBOLOID)
  {
    if (s.slope > 0)
      z -= side / 2;
    if (s.slope < 0)
      z += side / 2;
  }
  return shapeIn(s, x, y, z);
}

/* Shape::in(Cube): all eight corners inside. */
__device__ __forceinline__ bool shapeHolds(const QShape &s, double cx, double cy, double cz, double side)
{
  const double h = side / 2;
  bool all = true;
  for (int n = 0; n < 8 && all; n++)
    all = shapeIn(s, (n & 1) ? cx + h : cx - h, (n & 2) ? cy + h : cy - h, (n & 4) ? cz + h : cz - h);
  return all;
}

/* The shape against leaf l's cube; cubes far from it are told by their centre
 * alone, with half a side to spare. */
__device__ __forceinline__ bool leafMeets(const QArgs &a, uint64_t l)
{
  double cx, cy, cz, side;
  wb_leaf_cube(a.leafKey[l], a.leafLev[l], a.rootLo, a.rootSide, cx, cy, cz, side);
  const double ax = fabs(a.s.cx - cx) - side, ay = fabs(a.s.cy - cy) - side;
  if (a.s.kind == WB_SHAPE_CYLINDER)
  {
    if (ax > a.s.r || ay > a.s.r)
      return false;
  }
  else if (a.s.slope > 0)
  {
    const double zd = a.s.cz - (cz - side / 2);
    if (!(zd > 0) || ax * a.s.slope > zd || ay * a.s.slope > zd)
      return false;
  }
  return shapeMeets(a.s, cx, cy, cz, side);
}

/* The listed leaves, in depth-first order. */
struct MeetScan
{
  QArgs a;
  uint32_t *list;
  __device__ uint32_t value(uint64_t l, bool ok) const { return ok && leafMeets(a, l); }
  __device__ void put(uint64_t l, uint32_t before, uint32_t v) const
  {
    if (v)
      list[before] = (uint32_t)l;
  }
};
__global__ void __launch_bounds__(256) meetKernel(MeetScan f, unsigned *counter, unsigned long long *status,
                                                  uint32_t *total, int *err)
{
  lookbackScan<1>(f.a.L, f, counter, status, total, err);
}

/* shapeIn of stored point j. */
__device__ __forceinline__ bool pointIn(const QArgs &a, uint64_t j)
{
  const double x = a.xyzd[j], y = a.xyzd[a.nd + j], z = a.xyzd[2 * a.nd + j];
  const float dx = (float)(a.s.cx - x), dy = (float)(a.s.cy - y), d2 = dx * dx + dy * dy;
  if (a.s.kind == WB_SHAPE_CYLINDER)
  {
    const float r = (float)a.s.r, r2 = r * r;
    if (r2 > 1e-30f && r2 < 1e30f)
    {
      if (d2 < r2 * (1 - 1e-5f))
        return true;
      if (d2 > r2 * (1 + 1e-5f))
        return false;
    }
  }
  else if (a.s.slope > 0)
  {
    const float zd = (float)(a.s.cz - z), s = (float)a.s.slope, w = zd * zd, r2 = s * s * d2, p = (float)a.s.por2;
    const float f = w - r2 - p, tol = 1e-5f * (w + r2 + p);
    if (tol > 1e-30f && tol < 1e30f)
    {
      if (zd < 0 || f < -tol)
        return false;
      if (f > tol)
        return true;
    }
  }
  return shapeIn(a.s, x, y, z);
}

/* Order-preserving key of a height. */
__device__ __forceinline__ uint64_t heightBits(double z)
{
  if (z == 0)
    z = 0;   // -0 and +0 compare equal
  uint64_t u;
  memcpy(&u, &z, 8);
  return (u >> 63) ? ~u : (u | 0x8000000000000000ull);
}

/* A warp tests leaf l's points, 32 a row (at most 17 rows): lane r keeps row
 * r's hits; returns how many. */
constexpr int kLeafRows = (WB_RECORDS + 31) / 32;
__device__ __forceinline__ uint32_t leafRows(const QArgs &a, uint32_t l, unsigned &hits)
{
  const int lane = threadIdx.x & 31;
  double cx, cy, cz, side;
  wb_leaf_cube(a.leafKey[l], a.leafLev[l], a.rootLo, a.rootSide, cx, cy, cz, side);
  const bool whole = shapeHolds(a.s, cx, cy, cz, side);
  const uint32_t f = a.first[l], n = a.count[l];
  uint32_t taken = 0;
  hits = 0;
  for (int r = 0; 32u * r < n; r++)
  {
    const uint32_t t = 32u * r + lane;
    const bool in = t < n && (whole || pointIn(a, f + t));
    const unsigned b = __ballot_sync(0xffffffffu, in);
    if (lane == r)
      hits = b;
    taken += __popc(b);
  }
  return taken;
}

/* What the one-block answer leaves in pinned host memory. */
constexpr int kFewLeaves = 128, kFewPoints = 8192, kFewSorted = 2048;
struct QueryAnswer
{
  uint32_t leaves, points;
  uint32_t complete;   /* rec holds the answer */
  uint32_t failed;     /* the listing's look-back gave up */
  uint32_t rec[kFewPoints];
};

/* One block answers a query of at most kFewLeaves leaves.  want: capacity of
 * the caller (0: the count only). */
__global__ void __launch_bounds__(1024) fewLeavesKernel(QArgs a, const uint32_t *__restrict__ list,
                                                        const uint32_t *__restrict__ nList, uint64_t want, int sorted,
                                                        const int *__restrict__ err, QueryAnswer *ans)
{
  __shared__ uint32_t cnt[kFewLeaves + 1];
  __shared__ uint64_t key[kFewSorted];
  __shared__ uint32_t ord[kFewSorted], rec[kFewSorted];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint32_t n = *nList;
  const bool failed = *err != 0;
  if (threadIdx.x == 0)
    ans->failed = failed;
  if (failed || n > kFewLeaves)
  {
    if (threadIdx.x == 0)
    {
      ans->leaves = n;
      ans->complete = 0;
    }
    return;
  }
  constexpr int ROUNDS = kFewLeaves / 32;
  unsigned hits[ROUNDS];
#pragma unroll
  for (int q = 0; q < ROUNDS; q++)
  {
    const uint32_t i = q * 32 + w;
    hits[q] = 0;
    uint32_t taken = 0;
    if (i < n)
      taken = leafRows(a, list[i], hits[q]);
    if (lane == 0)
      cnt[i] = taken;
  }
  __syncthreads();
  if (w == 0)
  {
    // exclusive prefix of the leaves' counts
    uint32_t run = 0;
    for (int q = 0; q < ROUNDS; q++)
    {
      const uint32_t v = cnt[q * 32 + lane];
      uint32_t inc = v;
      for (int o = 1; o < 32; o <<= 1)
      {
        const uint32_t u = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o)
          inc += u;
      }
      cnt[q * 32 + lane] = run + inc - v;
      run += __shfl_sync(0xffffffffu, inc, 31);
    }
    if (lane == 0)
      cnt[kFewLeaves] = run;
  }
  __syncthreads();
  const uint32_t total = cnt[kFewLeaves];
  const bool sort = sorted && total > 1, fits = total <= want && total <= (sort ? kFewSorted : kFewPoints);
  if (threadIdx.x == 0)
  {
    ans->leaves = n;
    ans->points = total;
    ans->complete = fits || total > want;
  }
  if (!fits)
    return;
#pragma unroll
  for (int q = 0; q < ROUNDS; q++)
  {
    const uint32_t i = q * 32 + w;
    if (i >= n)
      continue;
    const uint32_t f = a.first[list[i]];
    uint32_t at = cnt[i];
    for (int r = 0; r < kLeafRows; r++)
    {
      const unsigned b = __shfl_sync(0xffffffffu, hits[q], r);
      if ((b >> lane) & 1)
      {
        const uint32_t j = f + 32 * r + lane, p = at + __popc(b & ((1u << lane) - 1));
        if (sort)
        {
          key[p] = heightBits(a.xyzd[2 * a.nd + j]);
          ord[p] = p;
          rec[p] = a.sidx[j];
        }
        else
          ans->rec[p] = a.sidx[j];
      }
      at += __popc(b);
    }
  }
  if (!sort)
    return;
  int P = 64;
  while (P < (int)total)
    P <<= 1;
  for (int q = threadIdx.x + (int)total; q < P; q += 1024)
  {
    key[q] = ~0ull;
    ord[q] = ~0u;
  }
  __syncthreads();
  // by height, ties in the order found
  for (int size = 2; size <= P; size <<= 1)
    for (int j = size >> 1; j > 0; j >>= 1)
    {
      for (int t = threadIdx.x; t < P / 2; t += 1024)
      {
        const int i = 2 * t - (t & (j - 1)), u = i + j;
        const uint64_t x = key[i], y = key[u];
        const uint32_t ox = ord[i], oy = ord[u];
        if ((x > y || (x == y && ox > oy)) == ((i & size) == 0))
        {
          key[i] = y;
          key[u] = x;
          ord[i] = oy;
          ord[u] = ox;
        }
      }
      __syncthreads();
    }
  for (uint32_t t = threadIdx.x; t < total; t += 1024)
    ans->rec[t] = rec[ord[t]];
}

/* FILL false: cnt[i] = points of listed leaf i that pointsIn returns; true:
 * their record indices (and, with keys, heights: record integers where sz gives
 * them) written from off[i] on. */
template <bool FILL>
__global__ void listedKernel(QArgs a, const uint32_t *__restrict__ list, uint32_t n, uint32_t *__restrict__ cnt,
                             const uint32_t *__restrict__ off, uint32_t *__restrict__ out, uint64_t *__restrict__ keys,
                             const int32_t *__restrict__ sz)
{
  const int lane = threadIdx.x & 31;
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += warps)
  {
    unsigned hits;
    const uint32_t taken = leafRows(a, list[i], hits);
    if (!FILL)
    {
      if (lane == 0)
        cnt[i] = taken;
      continue;
    }
    const uint32_t f = a.first[list[i]];
    uint32_t at = off[i];
    for (int r = 0; r < kLeafRows; r++)
    {
      const unsigned b = __shfl_sync(0xffffffffu, hits, r);
      if ((b >> lane) & 1)
      {
        const uint32_t j = f + 32 * r + lane, p = at + __popc(b & ((1u << lane) - 1));
        out[p] = a.sidx[j];
        if (keys)
          keys[p] = sz ? (uint64_t)((uint32_t)sz[j] ^ 0x80000000u) : heightBits(a.xyzd[2 * a.nd + j]);
      }
      at += __popc(b);
    }
  }
}

int shapeArgs(wb_ctx *c, const wb_shape *sh, QArgs &a, const char *who)
{
  if (!sh)
    return wb_fail(c, WB_EINVAL, std::string(who) + ": shape is NULL");
  memset(&a, 0, sizeof a);
  a.s.kind = sh->kind;
  if (sh->kind == WB_SHAPE_CYLINDER)
  {
    if (!(sh->r >= 0))
      return wb_fail(c, WB_EINVAL, std::string(who) + ": cylinder radius must be >= 0");
    a.s.cx = sh->v[0];
    a.s.cy = sh->v[1];
    a.s.r = sh->r;
  }
  else if (sh->kind == WB_SHAPE_HYPERBOLOID)
  {
    // Hyperboloid(v, r, s): por = r*s^2, centre = v + (0, 0, por) (shape.cpp:119-125)
    const double por = sh->r * (sh->s * sh->s);
    a.s.por2 = por * por;
    a.s.slope = sh->s;
    a.s.cx = sh->v[0] + 0;
    a.s.cy = sh->v[1] + 0;
    a.s.cz = sh->v[2] + por;
  }
  else
    return wb_fail(c, WB_EINVAL, std::string(who) + ": unknown shape kind");
  if (c->stage < 1)
    return wb_fail(c, WB_ESTATE, std::string(who) + ": no octree built");
  a.L = c->n_leaves;
  a.leafKey = (const uint64_t *)c->leafKey.p;
  a.leafLev = (const uint8_t *)c->leafLevel.p;
  a.first = (const uint32_t *)c->leafFirst.p;
  a.count = (const uint32_t *)c->leafCount.p;
  a.xyzd = (const double *)c->xyzd.p;
  a.nd = c->nd;
  a.sidx = (const uint32_t *)c->sidx.p;
  for (int k = 0; k < 3; k++)
    a.rootLo[k] = c->g.root_lo[k];
  a.rootSide = c->g.root_side;
  return 0;
}

/* Lists the leaves that meet the shape: *list on the device, their number at
 * *nList; behind the list, room for two more words a leaf and one. */
int listLeaves(wb_ctx *c, const QArgs &a, uint32_t **list, uint32_t **nList)
{
  const uint64_t tiles = (a.L + 255) / 256;   // a leaf a thread: FP64 cube tests, spread over the SMs
  unsigned *counter;
  unsigned long long *status;
  int rc = wb_lookback_words(c, tiles, &counter, &status);
  if (rc || (rc = wb_ensure(c, c->queryBuf, a.L * 12 + 128)))
    return rc;
  *nList = (uint32_t *)c->queryBuf.p;
  *list = *nList + 16;
  { meetKernel<<<(unsigned)tiles, 256, 0, c->stream>>>(MeetScan{a, *list}, counter, status, *nList, wb_lookback_err(c)); ++c->launches; }
  WB_CUDA(c, cudaGetLastError());
  return 0;
}
}  // namespace

extern "C" int wb_find_blocks(wb_ctx *c, const wb_shape *sh, int64_t *leaves, uint64_t capacity, uint64_t *count)
{
  if (!c || (capacity && !leaves))
    return WB_EINVAL;
  WbDeviceGuard deviceGuard(c->device);
  QArgs a;
  int rc = shapeArgs(c, sh, a, "wb_find_blocks");
  if (rc)
    return rc;
  if (count)
    *count = 0;
  const uint64_t L = a.L;
  if (L == 0)
    return 0;
  uint32_t *list, *nList, total = 0;
  int err = 0;
  if ((rc = listLeaves(c, a, &list, &nList)))
    return rc;
  WB_CUDA(c, cudaMemcpyAsync(&total, nList, 4, cudaMemcpyDefault, c->stream));
  WB_CUDA(c, cudaMemcpyAsync(&err, wb_lookback_err(c), 4, cudaMemcpyDefault, c->stream));
  WB_CUDA(c, cudaStreamSynchronize(c->stream));
  if (err)
    return wb_lookback_failed(c, "wb_find_blocks");
  if (count)
    *count = total;
  if (total > capacity)
    return wb_fail(c, WB_EINVAL, "wb_find_blocks: " + std::to_string(total) + " blocks, capacity " +
                                     std::to_string(capacity));
  if (!total)
    return 0;
  std::vector<uint32_t> l(total);
  WB_CUDA(c, cudaMemcpyAsync(l.data(), list, (size_t)total * 4, cudaMemcpyDefault, c->stream));
  WB_CUDA(c, cudaStreamSynchronize(c->stream));
  if (wb_device_accessible(leaves))
  {
    const std::vector<int64_t> wide(l.begin(), l.end());
    WB_CUDA(c, cudaMemcpyAsync(leaves, wide.data(), (size_t)total * 8, cudaMemcpyDefault, c->stream));
    WB_CUDA(c, cudaStreamSynchronize(c->stream));
  }
  else
    std::copy(l.begin(), l.end(), leaves);
  return 0;
}

extern "C" int wb_points_in(wb_ctx *c, const wb_shape *sh, int sorted, uint32_t *records, uint64_t capacity,
                            uint64_t *count)
{
  if (!c || (capacity && !records))
    return WB_EINVAL;
  WbDeviceGuard deviceGuard(c->device);
  QArgs a;
  int rc = shapeArgs(c, sh, a, "wb_points_in");
  if (rc)
    return rc;
  if (count)
    *count = 0;
  const uint64_t L = a.L;
  if (L == 0)
    return 0;
  uint32_t *list, *nList;
  if ((rc = listLeaves(c, a, &list, &nList)) || (rc = wb_host_stage(c, sizeof(QueryAnswer))))
    return rc;
  QueryAnswer *ans = (QueryAnswer *)c->hostStage;
  { fewLeavesKernel<<<1, 1024, 0, c->stream>>>(a, list, nList, capacity, sorted, wb_lookback_err(c), ans); ++c->launches; }
  WB_CUDA(c, cudaGetLastError());
  WB_CUDA(c, cudaStreamSynchronize(c->stream));
  if (ans->failed)
    return wb_lookback_failed(c, "wb_points_in");
  auto tooMany = [&](uint64_t total) {
    return wb_fail(c, WB_EINVAL, "wb_points_in: " + std::to_string(total) + " points, capacity " +
                                     std::to_string(capacity));
  };
  if (ans->complete)
  {
    const uint32_t total = ans->points;
    if (count)
      *count = total;
    if (total > capacity)
      return tooMany(total);
    if (total && wb_device_accessible(records))
    {
      WB_CUDA(c, cudaMemcpyAsync(records, ans->rec, (size_t)total * 4, cudaMemcpyDefault, c->stream));
      WB_CUDA(c, cudaStreamSynchronize(c->stream));
    }
    else if (total)
      memcpy(records, ans->rec, (size_t)total * 4);
    return 0;
  }
  // many leaves or points: counts, their prefix, the points, a radix sort
  const uint32_t n = ans->leaves;
  const unsigned grid = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(((uint64_t)n * 32 + 255) / 256, (uint64_t)c->sm_count * 32));
  uint32_t *cnt = list + L, *ex = cnt + L, *dTot = ex + L;
  { listedKernel<false><<<grid, 256, 0, c->stream>>>(a, list, n, cnt, nullptr, nullptr, nullptr, nullptr); ++c->launches; }
  if ((rc = wb_exclusive_scan_u32(c, cnt, ex, n, dTot)))
    return rc;
  uint32_t total = 0;
  int err = 0;
  auto failed = [&]() -> int {
    WB_CUDA(c, cudaMemcpyAsync(&err, wb_lookback_err(c), 4, cudaMemcpyDefault, c->stream));
    WB_CUDA(c, cudaStreamSynchronize(c->stream));
    return err ? wb_lookback_failed(c, "wb_points_in") : 0;
  };
  WB_CUDA(c, cudaMemcpyAsync(&total, dTot, 4, cudaMemcpyDefault, c->stream));
  if ((rc = failed()))
    return rc;
  if (count)
    *count = total;
  if (total > capacity)
    return tooMany(total);
  if (total == 0)
    return 0;
  // the build's sort buffers serve again (an allocation costs as much as a pass)
  const bool sort = sorted && total > 1;
  if ((rc = wb_ensure(c, c->idx0, (uint64_t)total * 4)) || (rc = wb_ensure(c, c->idx1, (uint64_t)total * 4)) ||
      (sort && ((rc = wb_ensure(c, c->key0, (uint64_t)total * 8)) || (rc = wb_ensure(c, c->key1, (uint64_t)total * 8)))))
    return rc;
  uint32_t *vals = (uint32_t *)c->idx0.p;
  uint64_t *keys = (uint64_t *)c->key0.p;
  // where the decode increases with the record integer in steps FP64 resolves,
  // that integer orders as the height does, in as many bits as the cloud's vary
  const double step = c->g.scale[2] * c->g.unit;
  const double mag = std::max(std::fabs((c->g.off[2] + c->g.scale[2] * c->grid.imin[2]) * c->g.unit),
                              std::fabs((c->g.off[2] + c->g.scale[2] * c->grid.imax[2]) * c->g.unit)) +
                     std::fabs(c->g.off[2] * c->g.unit) + step;
  const bool ints = step > 0 && step >= 4 * std::ldexp(mag, -52);
  int bits = 64;
  if (ints)
    for (bits = 0; bits < 32 && (((uint32_t)c->grid.imin[2] ^ (uint32_t)c->grid.imax[2]) >> bits);)
      bits++;
  { listedKernel<true><<<grid, 256, 0, c->stream>>>(a, list, n, nullptr, ex, vals, sort ? keys : nullptr,
                                                   ints ? (const int32_t *)c->sz.p : nullptr); ++c->launches; }
  if (sort && bits &&
      (rc = wb_radix_sort_pairs(c, keys, vals, (uint64_t *)c->key1.p, (uint32_t *)c->idx1.p, total, 0, bits)))
    return rc;
  WB_CUDA(c, cudaGetLastError());
  WB_CUDA(c, cudaMemcpyAsync(records, vals, (size_t)total * 4, cudaMemcpyDefault, c->stream));
  return failed();
}
