/* Device-wide primitives written for this library: exclusive scan of u32 and
 * a stable LSD radix sort of (u64 key, u32 value) pairs, both in one pass over
 * the data per step (wb_lookback.cuh).
 *
 * Radix sort: 8-bit digits.  One kernel counts all passes' digits in one read
 * of the keys; then each pass is one kernel: a block takes the next tile, ranks
 * its keys with warp __match_any_sync groups (stable: a warp walks its keys in
 * order, 32 at a time), publishes the tile's digit counts, puts the tile in
 * digit order in shared memory, looks back for its digits' places (one thread a
 * digit) and writes each digit's run with consecutive threads.  A pass over 20M
 * pairs takes 150-200 us (2.4-3.2 TB/s; issue 43-58%, ranking and look-back);
 * counting, scanning and scattering in three to five kernels took 220.
 */
#include <cuda_runtime.h>
#include <cstdint>
#include "wb_internal.h"
#include "wb_lookback.cuh"

namespace
{
struct PlainScan
{
  const uint32_t *in;
  uint32_t *out;
  __device__ uint32_t value(uint64_t i, bool ok) const { return ok ? in[i] : 0; }
  __device__ void put(uint64_t i, uint32_t before, uint32_t) const { out[i] = before; }
};

__global__ void __launch_bounds__(256) scanKernel(uint64_t n, PlainScan f, unsigned *counter, unsigned long long *status,
                                                  uint32_t *total, int *err)
{
  lookbackScan<kScanItems>(n, f, counter, status, total, err);
}

/* ---------------- radix sort ---------------- */
constexpr int kSortThreads = 256;
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kSortPasses = 8;

/* Digit counts of every pass (digits `begin + 8 p` of the keys). */
__global__ void __launch_bounds__(kSortThreads) radixCounts(const uint64_t *__restrict__ keys, uint64_t n, int begin,
                                                           int passes, uint32_t *__restrict__ hist)
{
  __shared__ uint32_t h[kSortPasses * 256];
  for (int i = threadIdx.x; i < passes * 256; i += kSortThreads)
    h[i] = 0;
  __syncthreads();
  for (uint64_t i = (uint64_t)blockIdx.x * kSortThreads + threadIdx.x; i < n; i += (uint64_t)gridDim.x * kSortThreads)
  {
    const uint64_t k = keys[i] >> begin;
    for (int p = 0; p < passes; p++)
      atomicAdd(&h[p * 256 + ((k >> (8 * p)) & 255)], 1u);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < passes * 256; i += kSortThreads)
    if (h[i])
      atomicAdd(&hist[i], h[i]);
}

/* One stable pass of an 8-bit digit; vals NULL: a key's value is its index.
 * Full tiles (all but the last) run without bounds checks.  The values are read
 * after the keys are out, so that only the ranks are in registers during the
 * look-back. */
template <int ITEMS, typename Word>
__global__ void __launch_bounds__(kSortThreads, ITEMS == 16 ? 3 : 4)
    radixPass(const uint64_t *__restrict__ keys, const uint32_t *__restrict__ vals, uint64_t n, int shift,
              const uint32_t *__restrict__ hist, unsigned *counter, Word *status, unsigned tag,
              uint64_t *__restrict__ keysOut, uint32_t *__restrict__ valsOut, int *err)
{
  constexpr int TILE = ITEMS * kSortThreads;
  __shared__ uint32_t wcount[kSortWarps][256];
  __shared__ uint32_t localStart[256], globalStart[256];
  __shared__ uint64_t skeys[TILE];   // then the values
  __shared__ uint32_t warpSums[kSortWarps];
  __shared__ unsigned tileS;
  __shared__ int failed;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, d0 = threadIdx.x;
  if (threadIdx.x == 0)
  {
    tileS = atomicAdd(counter, 1u);
    failed = 0;
  }
#pragma unroll
  for (int i = 0; i < kSortWarps; i++)
    wcount[i][threadIdx.x] = 0;
  __syncthreads();
  const unsigned tile = tileS;
  const uint64_t tbase = (uint64_t)tile * TILE;
  const uint32_t tileN = (uint32_t)(n - tbase < (uint64_t)TILE ? n - tbase : (uint64_t)TILE);
  const bool full = tileN == TILE;
  const uint32_t at0 = (uint32_t)warp * (ITEMS * 32) + lane;   // the thread's first item
  const uint64_t *kin = keys + tbase + at0;
  uint64_t key[ITEMS];
  uint32_t at[ITEMS];
  const unsigned lt = (1u << lane) - 1;
  uint32_t *wc = wcount[warp];
  if (full)
  {
#pragma unroll
    for (int s = 0; s < ITEMS; s++)
      key[s] = kin[32 * s];
#pragma unroll
    for (int s = 0; s < ITEMS; s++)
    {
      const uint32_t d = (uint32_t)(key[s] >> shift) & 255;
      const unsigned peers = __match_any_sync(0xffffffffu, d);   // a vote per bit took half as many instructions again
      const uint32_t pre = wc[d];
      at[s] = pre + __popc(peers & lt);
      __syncwarp();
      if ((peers & lt) == 0)
        wc[d] = pre + __popc(peers);
      __syncwarp();
    }
  }
  else
  {
#pragma unroll
    for (int s = 0; s < ITEMS; s++)
    {
      const bool ok = at0 + 32 * s < tileN;
      key[s] = ok ? kin[32 * s] : 0;
      const uint32_t d = ok ? (uint32_t)(key[s] >> shift) & 255 : 256u;
      const unsigned peers = __match_any_sync(0xffffffffu, d);
      const uint32_t pre = ok ? wc[d & 255] : 0;
      at[s] = pre + __popc(peers & lt);
      __syncwarp();
      if (ok && (peers & lt) == 0)
        wc[d & 255] = pre + __popc(peers);
      __syncwarp();
    }
  }
  __syncthreads();
  // per digit (one thread each): exclusive prefix over the warps and the tile's count
  uint32_t cnt = 0;
#pragma unroll
  for (int w = 0; w < kSortWarps; w++)
  {
    const uint32_t c = wcount[w][d0];
    wcount[w][d0] = cnt;
    cnt += c;
  }
  lookbackPut(status + (uint64_t)tile * 256 + d0, DigitWord<Word>::make(tag, tile == 0, cnt));
  uint32_t total;
  const uint32_t start = blockExclusive256(cnt, warpSums, total), bin = blockExclusive256(hist[d0], warpSums, total);
#pragma unroll
  for (int w = 0; w < kSortWarps; w++)
    wcount[w][d0] += start;
  localStart[d0] = start;
  __syncthreads();
#pragma unroll
  for (int s = 0; s < ITEMS; s++)
    if (full || at0 + 32 * s < tileN)
    {
      at[s] += wc[(uint32_t)(key[s] >> shift) & 255];
      skeys[at[s]] = key[s];
    }
  Word before = 0;
  if (tile && !lookbackColumn<Word, sizeof(Word) == 4 ? 32 : 16>(status + d0, 256, tag, (int64_t)tile, before, err))
    failed = 1;
  else if (tile)
    lookbackPut(status + (uint64_t)tile * 256 + d0, DigitWord<Word>::make(tag, true, before + cnt));
  globalStart[d0] = bin + (uint32_t)before - start;
  __syncthreads();
  if (failed)
    return;
  uint32_t pos[ITEMS];
#pragma unroll
  for (int s = 0; s < ITEMS; s++)
  {
    const uint32_t t = threadIdx.x + s * kSortThreads;
    if (full || t < tileN)
    {
      const uint64_t k = skeys[t];
      pos[s] = globalStart[(uint32_t)(k >> shift) & 255] + t;
      if (pos[s] < n)
        keysOut[pos[s]] = k;
    }
  }
  uint32_t val[ITEMS];
  const uint32_t *vin = vals + tbase + at0;
#pragma unroll
  for (int s = 0; s < ITEMS; s++)
    val[s] = vals ? (full || at0 + 32 * s < tileN ? vin[32 * s] : 0u) : (uint32_t)tbase + at0 + 32 * s;
  __syncthreads();
  uint32_t *svals = (uint32_t *)skeys;
#pragma unroll
  for (int s = 0; s < ITEMS; s++)
    if (full || at0 + 32 * s < tileN)
      svals[at[s]] = val[s];
  __syncthreads();
#pragma unroll
  for (int s = 0; s < ITEMS; s++)
  {
    const uint32_t t = threadIdx.x + s * kSortThreads;
    if ((full || t < tileN) && pos[s] < n)
      valsOut[pos[s]] = svals[t];
  }
}

__global__ void pullKernel(const uint4 *__restrict__ src, uint4 *__restrict__ dst, uint64_t n16)
{
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n16; i += (uint64_t)gridDim.x * blockDim.x)
    dst[i] = src[i];
}
}  // namespace

/* Copy of a caller's host buffer into device memory, in stream order.  Pinned
 * host memory is read in place by a kernel over the CPU link (GB300: NVLink-C2C,
 * the same rate as the copy engine); anything else goes through
 * cudaMemcpyAsync. */
int wb_copy_in(wb_ctx *c, void *dst, const void *src, size_t bytes)
{
  cudaPointerAttributes at;
  const void *view = nullptr;
  if (cudaPointerGetAttributes(&at, src) == cudaSuccess)
  {
    if (at.type == cudaMemoryTypeHost && at.devicePointer)
      view = at.devicePointer;
  }
  else
    cudaGetLastError();
  if (view && bytes >= (1u << 20) && (uintptr_t)view % 16 == 0 && (uintptr_t)dst % 16 == 0)
  {
    const uint64_t n16 = bytes / 16;
    const unsigned grid = (unsigned)c->sm_count * 8;
    { pullKernel<<<grid, 256, 0, c->stream>>>((const uint4 *)view, (uint4 *)dst, n16); ++c->launches; }
    WB_CUDA(c, cudaGetLastError());
    if (bytes > n16 * 16)
      WB_CUDA(c, cudaMemcpyAsync((uint8_t *)dst + n16 * 16, (const uint8_t *)src + n16 * 16, bytes - n16 * 16,
                                 cudaMemcpyDefault, c->stream));
    return 0;
  }
  WB_CUDA(c, cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDefault, c->stream));
  return 0;
}

/* Whether kernels can dereference p: device or managed memory, or host memory
 * mapped for the device.  A pageable host pointer passed where the API wants
 * a device pointer is refused with WB_EINVAL instead of reaching a kernel. */
bool wb_device_accessible(const void *p)
{
  if (!p)
    return false;
  cudaPointerAttributes at;
  if (cudaPointerGetAttributes(&at, p) != cudaSuccess)
  {
    cudaGetLastError();
    return false;
  }
  return at.type == cudaMemoryTypeDevice || at.type == cudaMemoryTypeManaged ||
         (at.type == cudaMemoryTypeHost && at.devicePointer == p);
}

int wb_small(wb_ctx *c)
{
  if (c->small.p)
    return 0;
  int rc = wb_ensure(c, c->small, 4096);
  if (rc)
    return rc;
  WB_CUDA(c, cudaMemsetAsync(c->small.p, 0, 4096, c->stream));
  return 0;
}

int wb_host_stage(wb_ctx *c, size_t bytes)
{
  if (c->hostStageCap >= bytes)
    return 0;
  WB_CUDA(c, cudaStreamSynchronize(c->stream));
  if (c->hostStage)
    cudaFreeHost(c->hostStage);
  c->hostStage = nullptr;
  c->hostStageCap = 0;
  WB_CUDA(c, cudaHostAlloc(&c->hostStage, bytes, cudaHostAllocDefault));
  c->hostStageCap = bytes;
  return 0;
}

int *wb_lookback_err(wb_ctx *c)
{
  return (int *)((char *)c->small.p + WB_SMALL_LOOKBACK);
}

/* The answer of a call whose look-back gave up; the next call starts afresh. */
int wb_lookback_failed(wb_ctx *c, const char *who)
{
  cudaMemsetAsync(wb_lookback_err(c), 0, 4, c->stream);
  return wb_fail(c, WB_ETIMEDOUT, std::string(who) + ": a look-back wait gave up");
}

/* Counter and status words of a look-back sequence of `words` words, cleared. */
int wb_lookback_words(wb_ctx *c, uint64_t words, unsigned **counter, unsigned long long **status)
{
  int rc = wb_small(c);
  if (rc || (rc = wb_ensure(c, c->scanTmp, words * 8 + 64)))
    return rc;
  WB_CUDA(c, cudaMemsetAsync(c->scanTmp.p, 0, words * 8 + 64, c->stream));
  *counter = (unsigned *)c->scanTmp.p;
  *status = (unsigned long long *)((char *)c->scanTmp.p + 64);
  return 0;
}

int wb_exclusive_scan_u32(wb_ctx *c, const uint32_t *in, uint32_t *out, uint64_t n, uint32_t *total_dev)
{
  if (n == 0)
    return 0;
  const uint64_t tiles = (n + kScanTile - 1) / kScanTile;
  unsigned *counter;
  unsigned long long *status;
  int rc = wb_lookback_words(c, tiles, &counter, &status);
  if (rc)
    return rc;
  { scanKernel<<<(unsigned)tiles, 256, 0, c->stream>>>(n, PlainScan{in, out}, counter, status, total_dev,
                                                       wb_lookback_err(c)); ++c->launches; }
  WB_CUDA(c, cudaGetLastError());
  return 0;
}

int wb_radix_sort_pairs(wb_ctx *c, uint64_t *&keys, uint32_t *&vals, uint64_t *keysAlt, uint32_t *valsAlt,
                        uint64_t n, int beginBit, int endBit, uint64_t varying, bool iota)
{
  if (n <= 1 && !iota)
    return 0;
  const int passes = (endBit - beginBit + 7) / 8;
  // keys a tile: enough tiles to fill the GPU, else large ones (fewer look-backs)
  const int items = n >= (1ull << 21) ? 16 : (n >= (1ull << 19) ? 8 : 4);
  const uint64_t tiles = (n + (uint64_t)items * kSortThreads - 1) / ((uint64_t)items * kSortThreads);
  const size_t head = kSortPasses * 256 * 4 + 64;   // digit counts, tile counters
  const bool small = n < (1ull << 26);
  const size_t words = tiles * 256 * (small ? 4 : 8);
  int rc = wb_small(c);
  if (rc || (rc = wb_ensure(c, c->scanTmp, head + words + 64)))
    return rc;
  uint32_t *hist = (uint32_t *)c->scanTmp.p;
  unsigned *counter = (unsigned *)(hist + kSortPasses * 256);
  void *status = (char *)c->scanTmp.p + head;
  WB_CUDA(c, cudaMemsetAsync(c->scanTmp.p, 0, head + words, c->stream));
  { radixCounts<<<(unsigned)std::min<uint64_t>((n + 2047) / 2048, (uint64_t)c->sm_count * 4), kSortThreads, 0,
                  c->stream>>>(keys, n, beginBit, passes, hist); ++c->launches; }
  int *err = wb_lookback_err(c);
  const uint32_t *in = iota ? nullptr : vals;
  for (int p = 0; p < passes; p++)
  {
    const int shift = beginBit + 8 * p;
    if (!((varying >> shift) & 255) && in)
      continue;   // digit the same for all keys: the pass would be the identity
    auto launch = [&](auto pass, auto *words) {
      pass<<<(unsigned)tiles, kSortThreads, 0, c->stream>>>(keys, in, n, shift, hist + p * 256, counter + p, words,
                                                            (unsigned)p + 1, keysAlt, valsAlt, err);
      ++c->launches;
    };
    if (small)
      launch(items == 16 ? radixPass<16, uint32_t> : (items == 8 ? radixPass<8, uint32_t> : radixPass<4, uint32_t>),
             (uint32_t *)status);
    else
      launch(radixPass<16, unsigned long long>, (unsigned long long *)status);
    std::swap(keys, keysAlt);
    std::swap(vals, valsAlt);
    in = vals;
  }
  WB_CUDA(c, cudaGetLastError());
  return 0;
}
