// Linked with fcb200.cu's object, answers the CUDA runtime calls of prepare_kernel:
// preparing a kernel again (a second plan) must at no time show another bound than the
// one that calls on other threads go by.
#include "fcb_internal.h"

#include <cstdio>

static const fcb::KernelInfo *g_k = nullptr;
static long long g_seen = -1;

extern "C" {
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *n, const void *, int, size_t) { *n = 4; return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned) { *n = 4; return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveClusters(int *n, const void *, const cudaLaunchConfig_t *)
{
  g_seen = g_k->few->resident_tiles;  // what a call on another thread would read now
  *n = 16;
  return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
}

int main()
{
  fcb::KernelInfo few, k;
  few.cluster = 8;
  k.cluster = 4;
  k.few = &few;
  g_k = &k;
  if (fcb::prepare_kernel(&k)) return 2;
  const long long first = few.resident_tiles;
  if (fcb::prepare_kernel(&k)) return 2;
  std::printf("bound %lld, while prepared again %lld\n", first, g_seen);
  return first == 16 && g_seen == first ? 0 : 1;
}
