/* A bitonic sort of 32 * E unsigned integers (32 or 64 bits) by one warp, in registers.
 *
 * Lane l holds the elements l * E to l * E + E - 1.  The network's first step
 * of each phase compares element i with its mirror image i ^ (k - 1), so every
 * comparator puts the smaller value at the lower index and no direction has to
 * be looked up; partners within a lane cost a minimum and a maximum, partners
 * in two lanes a shuffle and one of the two.  A stage of the same network over
 * shared memory costs two loads, up to two stores and their addresses per
 * comparator: with it the sorts issued five times as many instructions.
 */
#ifndef WB_WARPSORT_CUH
#define WB_WARPSORT_CUH
#include <cstdint>
#include <cuda_runtime.h>

template <int E, class T>
__device__ __forceinline__ void wb_warp_sort(T (&v)[E], int lane)
{
  constexpr unsigned kAll = 0xffffffffu;
#pragma unroll
  for (int k = 2; k <= 32 * E; k <<= 1)
  {
    if (k <= E)
    {
#pragma unroll
      for (int e = 0; e < E; e++)
        if ((e ^ (k - 1)) > e)
        {
          const T x = v[e], y = v[e ^ (k - 1)];
          v[e] = min(x, y);
          v[e ^ (k - 1)] = max(x, y);
        }
    }
    else
    {
      const bool lower = (lane & (k / E / 2)) == 0;
#pragma unroll
      for (int e = 0; e < (E + 1) / 2; e++)
      {
        const T x = __shfl_xor_sync(kAll, v[E - 1 - e], k / E - 1);
        if (E > 1)
        {
          const T y = __shfl_xor_sync(kAll, v[e], k / E - 1);
          v[E - 1 - e] = lower ? min(v[E - 1 - e], y) : max(v[E - 1 - e], y);
        }
        v[e] = lower ? min(v[e], x) : max(v[e], x);
      }
    }
#pragma unroll
    for (int j = k / 4; j > 0; j >>= 1)
    {
      if (j >= E)
      {
        const bool lower = (lane & (j / E)) == 0;
#pragma unroll
        for (int e = 0; e < E; e++)
        {
          const T x = __shfl_xor_sync(kAll, v[e], j / E);
          v[e] = lower ? min(v[e], x) : max(v[e], x);
        }
      }
      else
      {
#pragma unroll
        for (int e = 0; e < E; e++)
          if ((e ^ j) > e)
          {
            const T x = v[e], y = v[e ^ j];
            v[e] = min(x, y);
            v[e ^ j] = max(x, y);
          }
      }
    }
  }
}

/* Sorts n <= 32 * E values through registers, from src to dst (the same array or
 * another, 16-byte aligned); up to three entries after them are written too. */
template <int E, class T>
__device__ __forceinline__ void wb_warp_sort_to(const T *src, T *dst, uint32_t n, int lane)
{
  T v[E];
#pragma unroll
  for (int e = 0; e < E; e++)
    v[e] = e * 32 + lane < (int)n ? src[e * 32 + lane] : ~(T)0;
  __syncwarp();
  wb_warp_sort<E>(v, lane);
  if constexpr (sizeof(T) == 4 && E % 4 == 0)
  {
#pragma unroll
    for (int e = 0; e < E; e += 4)
      if (lane * E + e < (int)n)
        ((uint4 *)dst)[(lane * E + e) / 4] = make_uint4(v[e], v[e + 1], v[e + 2], v[e + 3]);
  }
  else
  {
#pragma unroll
    for (int e = 0; e < E; e++)
      if (lane * E + e < (int)n)
        dst[lane * E + e] = v[e];
  }
  __syncwarp();
}

/* The same for any n up to 1024. */
__device__ __forceinline__ void wb_warp_sort_1024(uint32_t *b, uint32_t n, int lane)
{
  if (n <= 32)
    wb_warp_sort_to<1>(b, b, n, lane);
  else if (n <= 64)
    wb_warp_sort_to<2>(b, b, n, lane);
  else if (n <= 128)
    wb_warp_sort_to<4>(b, b, n, lane);
  else if (n <= 256)
    wb_warp_sort_to<8>(b, b, n, lane);
  else if (n <= 512)
    wb_warp_sort_to<16>(b, b, n, lane);
  else
    wb_warp_sort_to<32>(b, b, n, lane);
}
#endif
