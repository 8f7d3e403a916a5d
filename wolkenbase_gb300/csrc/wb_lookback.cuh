/* Decoupled look-back: a block learns the sum over all blocks before it while
 * they run, so a prefix takes one pass over the data.
 *
 * Blocks take their tile numbers from a counter, so the tiles before a running
 * one are running or finished, and each publishes its own sum before it waits
 * for anyone.  A wait is bounded all the same: after kLookbackSpins polls, or
 * when another block gave up, the block sets *err and gives up: its caller
 * returns without writing.  What it would have written then holds whatever was
 * there before, so every kernel that takes an address from it returns when *err
 * is set, and the host reads *err with the stage's own read-back, clears it and
 * answers WB_ETIMEDOUT.
 *
 * A status word holds a tag (which pass of a kernel sequence it belongs to, 0
 * never), whether the value is the tile's own sum or includes everything
 * before it, and the value: words of an earlier pass read as not there yet, so
 * the words are cleared once per sequence. */
#ifndef WB_LOOKBACK_CUH
#define WB_LOOKBACK_CUH
#include <cstdint>
#include <cuda_runtime.h>

#ifndef WB_LOOKBACK_SPINS
#define WB_LOOKBACK_SPINS (1 << 20)   /* about a second */
#endif
constexpr int kLookbackSpins = WB_LOOKBACK_SPINS;
constexpr int kLookbackValueBits = 48;   /* tag 15 bits, inclusive 1 bit, value 48 bits */

__device__ __forceinline__ unsigned long long lookbackWord(unsigned tag, bool inclusive, unsigned long long v)
{
  return ((unsigned long long)tag << (kLookbackValueBits + 1)) | ((unsigned long long)inclusive << kLookbackValueBits) | v;
}

__device__ __forceinline__ void lookbackPut(unsigned long long *p, unsigned long long v)
{
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

__device__ __forceinline__ unsigned long long lookbackGet(const unsigned long long *p)
{
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

/* Whether poll number `spins` of a wait is its last: the limit, or another
 * block's error, looked at every 64 polls so that later blocks need not wait. */
__device__ __forceinline__ bool lookbackGivesUp(int spins, const int *err)
{
  return spins > kLookbackSpins || (spins % 64 == 0 && *(const volatile int *)err);
}

/* Status words of the radix passes, one per digit and tile: 32 bits while the
 * counts fit 26 of them (tag 5 bits, inclusive 1 bit), else 64. */
template <typename Word>
struct DigitWord
{
  static constexpr int kBits = sizeof(Word) == 4 ? 26 : 48;
  static __device__ __forceinline__ Word make(unsigned tag, bool inclusive, Word v)
  {
    return ((Word)tag << (kBits + 1)) | ((Word)inclusive << kBits) | v;
  }
  static __device__ __forceinline__ unsigned tag(Word w) { return (unsigned)(w >> (kBits + 1)); }
  static __device__ __forceinline__ bool inclusive(Word w) { return (w >> kBits) & 1; }
  static __device__ __forceinline__ Word value(Word w) { return w & (((Word)1 << kBits) - 1); }
};
__device__ __forceinline__ void lookbackPut(uint32_t *p, uint32_t v)
{
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t lookbackGet(const uint32_t *p)
{
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

/* One thread's look back along its own column of status words (tile t's word
 * at status[t * stride]): the sum over the tiles before `tile`.  False when it
 * gave up.  WINDOW tiles at a time with their loads in flight together: all
 * tiles that wait for the same frontier learn it in one round trip, so the
 * frontier moves WINDOW tiles per round trip (at 8, 112 cycles a tile: 0.66 of
 * the 0.75 ms that a pass over 50M pairs took). */
template <typename Word, int WINDOW>
__device__ __forceinline__ bool lookbackColumn(const Word *status, uint64_t stride, unsigned tag, int64_t tile,
                                               Word &sum, int *err)
{
  typedef DigitWord<Word> D;
  sum = 0;
  int64_t t = tile - 1;
  int spins = 0;
  while (t >= 0)
  {
    Word w[WINDOW];
#pragma unroll
    for (int q = 0; q < WINDOW; q++)
      w[q] = t - q >= 0 ? lookbackGet(status + (uint64_t)(t - q) * stride) : 0;
    bool ready = true, end = false;
    int step = 0;
#pragma unroll
    for (int q = 0; q < WINDOW; q++)
    {
      const bool there = t - q >= 0 && D::tag(w[q]) == tag;
      ready = ready && there;
      if (ready && !end)
      {
        sum += D::value(w[q]);
        step = q + 1;
        end = D::inclusive(w[q]);
      }
    }
    if (end)
      return true;
    t -= step;
    if (t >= 0 && step < WINDOW && lookbackGivesUp(++spins, err))
    {
      *err = 1;
      return false;
    }
  }
  return true;
}

/* A warp's look back along one word per tile: 32 tiles at a time.  Every lane
 * gets the sum. */
__device__ __forceinline__ bool lookbackWarp(const unsigned long long *status, unsigned tag, int64_t tile,
                                             unsigned long long &sum, int *err)
{
  constexpr unsigned long long kValue = (1ull << kLookbackValueBits) - 1;
  const int lane = threadIdx.x & 31;
  sum = 0;
  int64_t t = tile - 1;
  int spins = 0;
  while (t >= 0)
  {
    unsigned long long w = 0;
    bool there = true, incl = false;
    if (t - lane >= 0)
    {
      w = lookbackGet(status + (t - lane));
      there = (unsigned)(w >> (kLookbackValueBits + 1)) == tag;
      incl = there && ((w >> kLookbackValueBits) & 1);
    }
    const unsigned ok = __ballot_sync(0xffffffffu, there), in = __ballot_sync(0xffffffffu, incl);
    // the tiles up to the first one that is not there yet, or that includes the rest
    int n = __ffs(~ok) - 1;
    if (n < 0)
      n = 32;
    const int first = __ffs(in) - 1;
    const bool end = first >= 0 && first < n;
    if (end)
      n = first + 1;
    unsigned long long v = lane < n && t - lane >= 0 ? w & kValue : 0;
    for (int o = 16; o; o >>= 1)
      v += __shfl_xor_sync(0xffffffffu, v, o);
    sum += v;
    if (end)
      return true;
    t -= n;
    if (n < 32 && __any_sync(0xffffffffu, lookbackGivesUp(++spins, err)))
    {
      if (lane == 0)
        *err = 1;
      return false;
    }
  }
  return true;
}

/* Exclusive prefix over a block of 256 threads of one value each, and the
 * block's total; warpSums is 8 words of shared memory. */
__device__ __forceinline__ uint32_t blockExclusive256(uint32_t v, uint32_t *warpSums, uint32_t &total)
{
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint32_t inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1)
  {
    const uint32_t u = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o)
      inc += u;
  }
  if (lane == 31)
    warpSums[w] = inc;
  __syncthreads();
  uint32_t before = 0;
  total = 0;
#pragma unroll
  for (int q = 0; q < 8; q++)
  {
    const uint32_t s = warpSums[q];
    before += q < w ? s : 0;
    total += s;
  }
  __syncthreads();
  return before + inc - v;
}

/* One-pass scan of 256-thread tiles of ITEMS items a thread: value(i, i < n) is
 * item i's value (0 past the end), asked of a warp's 32 consecutive items
 * together; put(i, before, value) receives the sum before it.  The last tile
 * writes the total.  counter and status (one word per tile) are zero on
 * entry. */
constexpr int kScanItems = 16, kScanTile = 256 * kScanItems;
template <int ITEMS, typename F>
__device__ __forceinline__ void lookbackScan(uint64_t n, F &f, unsigned *counter, unsigned long long *status,
                                             uint32_t *total, int *err)
{
  __shared__ uint32_t warpSums[8];
  __shared__ unsigned tileS;
  __shared__ unsigned long long beforeS;
  __shared__ int failed;
  if (threadIdx.x == 0)
  {
    tileS = atomicAdd(counter, 1u);
    failed = 0;
  }
  __syncthreads();
  const unsigned tile = tileS;
  const uint64_t base = (uint64_t)tile * (256 * ITEMS);
  // a warp's items lie together, a lane's 32 apart
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint64_t wbase = base + (uint64_t)w * (32 * ITEMS);
  uint32_t v[ITEMS], ex[ITEMS], run = 0;
#pragma unroll
  for (int k = 0; k < ITEMS; k++)
  {
    const uint64_t i = wbase + 32 * k + lane;
    v[k] = f.value(i, i < n);
  }
#pragma unroll
  for (int k = 0; k < ITEMS; k++)
  {
    uint32_t inc = v[k];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
      const uint32_t u = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o)
        inc += u;
    }
    ex[k] = run + inc - v[k];
    run += __shfl_sync(0xffffffffu, inc, 31);
  }
  if (lane == 0)
    warpSums[w] = run;
  __syncthreads();
  uint32_t before = 0, sum = 0;
#pragma unroll
  for (int q = 0; q < 8; q++)
  {
    const uint32_t s = warpSums[q];
    before += q < w ? s : 0;
    sum += s;
  }
  if (w == 0)
  {
    unsigned long long b = 0;
    if (lane == 0)
      lookbackPut(status + tile, lookbackWord(1, tile == 0, sum));
    const bool ok = lookbackWarp(status, 1, tile, b, err);
    if (lane == 0)
    {
      if (ok && tile)
        lookbackPut(status + tile, lookbackWord(1, true, b + sum));
      beforeS = b;
      failed = !ok;
      if (ok && base + 256 * ITEMS >= n && total)
        *total = (uint32_t)(b + sum);
    }
  }
  __syncthreads();
  if (failed)
    return;
  const uint32_t off = (uint32_t)beforeS + before;
#pragma unroll
  for (int k = 0; k < ITEMS; k++)
  {
    const uint64_t i = wbase + 32 * k + lane;
    if (i < n)
      f.put(i, off + ex[k], v[k]);
  }
}

#endif
