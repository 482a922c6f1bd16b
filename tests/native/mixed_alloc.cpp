// Linked with fcb_mixed.cu's object: making a mixed-radix plan with every one of its
// allocations failing in turn reports an error; no exception leaves it (it is called from
// C functions).  The first argument is the length.
#include "fcb200.h"
#include "fcb_internal.h"

#include <cstdio>
#include <cstdlib>
#include <new>

static int g_left = -1;  // allocations until one fails; negative: none does

static void *get(std::size_t n) { return g_left >= 0 && g_left-- == 0 ? nullptr : std::malloc(n); }
void *operator new(std::size_t n)
{
  if (void *p = get(n)) return p;
  throw std::bad_alloc();
}
void *operator new[](std::size_t n) { return operator new(n); }
void *operator new(std::size_t n, const std::nothrow_t &) noexcept { return get(n); }
void *operator new[](std::size_t n, const std::nothrow_t &) noexcept { return get(n); }
void operator delete(void *p) noexcept { std::free(p); }
void operator delete[](void *p) noexcept { std::free(p); }
void operator delete(void *p, std::size_t) noexcept { std::free(p); }
void operator delete[](void *p, std::size_t) noexcept { std::free(p); }

extern "C" {
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaFree(void *) { return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaErrorNotSupported; }
}

namespace fcb {
int set_error(int code, const char *, ...) { return code; }
int cuda_error(cudaError_t, const char *) { return FCB_ERR_CUDA; }
const void *mixed_rows_fn(bool) { return nullptr; }
const void *mixed_conv_fn(bool) { return nullptr; }
const void *mixed_cols_fn(bool) { return nullptr; }
}

int main(int argc, char **argv)
{
  const long long n = argc > 1 ? std::atoll(argv[1]) : 1144;
  for (int fail = 0; fail < 64; ++fail)
  {
    g_left = fail;
    fcb::MixedPlan *p = nullptr;
    int rc = 0;
    try
    {
      rc = fcb::mixed_create(n, &p, nullptr);
    }
    catch (...)
    {
      std::printf("allocation %d: an exception\n", fail);
      return 1;
    }
    const bool all = g_left >= 0;  // none was left to fail: stopped by the runtime call above
    g_left = -1;
    if (rc != (all ? FCB_ERR_CUDA : FCB_ERR_NOMEM) || p) return 2;
    if (all) return 0;
  }
  return 3;
}
