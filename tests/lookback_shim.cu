/* Reaches into the library for test_gpu_lookback.py: waits that run out, in
 * kernels of its own with a short limit, and the contexts' error word. */
#include <cstdint>
#include <cuda_runtime.h>
#include "wb_internal.h"
#include "wb_lookback.cuh"

struct CopyScan
{
  uint32_t *out;
  __device__ uint32_t value(uint64_t, bool ok) const { return ok ? 1u : 0u; }
  __device__ void put(uint64_t i, uint32_t before, uint32_t) const { out[i] = before; }
};

__global__ void __launch_bounds__(256) scanOnce(uint64_t n, CopyScan f, unsigned *counter, unsigned long long *status,
                                                uint32_t *total, int *err)
{
  lookbackScan<1>(n, f, counter, status, total, err);
}

__global__ void columnOnce(const uint32_t *status, int64_t tile, int *err, int *gaveUp)
{
  uint32_t sum;
  if (!lookbackColumn<uint32_t, 4>(status + threadIdx.x, 32, 1, tile, sum, err))
    atomicAdd(gaveUp, 1);
}

/* Scans n items by blocks that take their tiles from `first` on, so that tile 0
 * is never published when it is above zero: out (n words, 7 before), the total
 * (7 before) and the error word. */
extern "C" int shim_scan(uint32_t n, unsigned first, uint32_t *out, uint32_t *total, int *err)
{
  const unsigned tiles = (n + 255) / 256;
  uint32_t *d = nullptr;
  if (first > tiles || cudaMalloc(&d, n * 4 + 64 + (tiles + 1) * 8 + 64))
    return -1;
  unsigned long long *status = (unsigned long long *)(d + ((n + 1) / 2 * 2));
  unsigned *counter = (unsigned *)(status + tiles);   // counter, total, error word
  unsigned init[3] = {first, 7, 0};
  cudaMemset(status, 0, tiles * 8);
  cudaMemcpy(counter, init, sizeof init, cudaMemcpyHostToDevice);
  for (uint32_t i = 0; i < n; i++)
    out[i] = 7;
  cudaMemcpy(d, out, n * 4, cudaMemcpyHostToDevice);
  if (tiles > first)
    scanOnce<<<tiles - first, 256>>>(n, CopyScan{d}, counter, status, counter + 1, (int *)(counter + 2));
  cudaMemcpy(out, d, n * 4, cudaMemcpyDeviceToHost);
  cudaMemcpy(init, counter, sizeof init, cudaMemcpyDeviceToHost);
  *total = init[1];
  *err = (int)init[2];
  const cudaError_t e = cudaGetLastError();
  cudaFree(d);
  return (int)e;
}

/* 32 threads look back from tile 3 over words of which `there` tiles are
 * published: how many gave up, and the error word. */
extern "C" int shim_column(int there, int *gaveUp, int *err)
{
  uint32_t host[4 * 32] = {0};
  for (int t = 0; t < there && t < 3; t++)
    for (int d = 0; d < 32; d++)
      host[t * 32 + d] = (1u << 27) | ((t == 0) << 26) | 5u;   // tag 1, inclusive at tile 0, value 5
  uint32_t *p = nullptr;
  if (cudaMalloc(&p, sizeof host))
    return -1;
  cudaMemcpy(p, host, sizeof host, cudaMemcpyHostToDevice);
  columnOnce<<<1, 32>>>(p, 3, (int *)(p + 96), (int *)(p + 97));
  cudaMemcpy(host, p, sizeof host, cudaMemcpyDeviceToHost);
  *err = (int)host[96];
  *gaveUp = (int)host[97];
  const cudaError_t e = cudaGetLastError();
  cudaFree(p);
  return (int)e;
}

extern "C" int shim_set(wb_ctx *c, int v)
{
  cudaDeviceSynchronize();
  if (wb_small(c) || cudaDeviceSynchronize())
    return -1;
  return (int)cudaMemcpy(wb_lookback_err(c), &v, 4, cudaMemcpyHostToDevice);
}

extern "C" int shim_get(wb_ctx *c, int *v)
{
  cudaDeviceSynchronize();
  return (int)cudaMemcpy(v, wb_lookback_err(c), 4, cudaMemcpyDeviceToHost);
}

extern "C" int shim_grid(wb_ctx *c)
{
  const double *b = c->grid_bounds;
  return wb_grid_impl(c, b[0], b[1], b[2], b[3]);
}
