// Mixed-radix plans: factors, tables, CTA shapes and launches (kernel and
// algorithm: fcb_mixed.cuh).
#include "fcb200.h"
#include "fcb_internal.h"
#include "fcb_mixed.cuh"

#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <memory>
#include <new>

namespace fcb {

namespace {

// Twiddles W_L^{n' q} of all stages but the last, FP64 rounded to float.
__global__ void mixed_tw_kernel(float4 *tw, MrStage s)
{
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (long long)(s.R / 2) * s.S) return;
  const long long q = 2 * (i / s.S) + 1, np = i % s.S;
  double s0, c0, s1, c1;
  sincospi(-2.0 * (double)((q * np) % s.L) / (double)s.L, &s0, &c0);
  sincospi(-2.0 * (double)(((q + 1) * np) % s.L) / (double)s.L, &s1, &c1);
  tw[s.tw + i] = make_float4((float)c0, (float)s0, (float)c1, (float)s1);
}

// rep[r][q * nb + b] = spec[r][kprev(b) + nb q] * scale
__global__ void mixed_rep_kernel(const float2 *spec, long long spec_rs, float2 *rep, long long rows, int n, int nb,
                                 const unsigned short *rev, float scale)
{
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= rows * n) return;
  const long long r = i / n;
  const int e = (int)(i % n), q = e / nb, j = e % nb;
  const float2 v = spec[r * spec_rs + e];  // output j + nb q, which block rev[j] holds
  rep[r * n + q * nb + rev[j]] = make_float2(v.x * scale, v.y * scale);
}

// Arithmetic of one DFT of R samples in registers, in operations per sample.
float dft_cost(int R)
{
  static const float c[17] = {0, 0, 2, 5.3f, 4, 7.2f, 7.3f, 10, 6.5f, 9.8f, 9.2f, 17, 9.3f, 20, 12, 12.5f, 9.2f};
  return c[R];
}
// A pass through shared memory with its twiddles, on the same scale (a pass moves 16 bytes of shared memory and 8 of
// twiddles per sample, about the issue slots of 16 operations).
constexpr float kPassCost = 16.f;

struct Radices
{
  int r[kMrStages];
  int count = 0;
};

// Radices of n with the least cost, in descending order of their share of two: the last stage reads R adjacent samples
// per thread, which is free of bank conflicts only for odd R.
bool factor(int n, Radices &best)
{
  Radices cur;
  float best_cost = 1e30f;
  auto rec = [&](auto &&self, int left, int from, float cost) -> void {
    if (cost >= best_cost) return;
    if (left == 1)
    {
      best_cost = cost;
      best = cur;
      return;
    }
    if (cur.count == kMrStages) return;
    for (int R = from; R >= 2; --R)
      if (left % R == 0)
      {
        cur.r[cur.count++] = R;
        self(self, left / R, R, cost + dft_cost(R) + kPassCost);
        --cur.count;
      }
  };
  rec(rec, n, 16, 0.f);
  // insertion, equal shares in the order found
  for (int i = 1; i < best.count; ++i)
    for (int j = i; j > 0 && (best.r[j] & -best.r[j]) > (best.r[j - 1] & -best.r[j - 1]); --j)
      std::swap(best.r[j], best.r[j - 1]);
  return best.count > 0;
}

struct MrConfig { int C, threads; };

}  // namespace

struct MixedPlan
{
  int n = 0, ns = 0;
  MrStage st[kMrStages] = {};
  int sms = 148;
  float4 *tw = nullptr;
  unsigned short *rev = nullptr;
  // the last call's CTA shape: transforms << 24 | C << 12 | threads (rows, columns); a
  // different count computes it again (about 1 us)
  std::atomic<unsigned long long> last[2] = {};
};

namespace {

// CTA shape for `count` transforms.  Rows: of all C and thread counts the one with the least modelled time: a step is
// one butterfly per thread, an SM issues about 256 threads' worth of a step at once and needs about 512 resident to hide
// latency, and CTAs that do not fit at once queue.
MrConfig configure_rows(const MixedPlan &p, long long count, int sms)
{
  MrConfig best = {1, 256};
  float best_time = 1e30f;
  for (int C : {1, 2, 3, 4, 6, 8, 12, 16, 24, 32, 48, 64})
  {
    const long long smem = 8LL * C * p.n;
    if (C > 1 && (smem > 64 * 1024 || C >= 2 * count)) break;
    const int tmax = smem > kMrSmem / 2 ? 512 : 256;
    for (int T = 64; T <= tmax; T += tmax / 8)
    {
      float steps = 0;
      for (int k = 0; k < p.ns; ++k) steps += (float)((C * p.st[k].nb + T - 1) / T) * p.st[k].R;
      const int ctas = (int)std::max<long long>(1, std::min<long long>(std::min(32, 768 / T), kMrSmem / (smem + 1024)));
      const long long grid = (count + C - 1) / C, per_sm = (grid + sms - 1) / sms;
      const float waves = (float)((per_sm + ctas - 1) / ctas);
      const float time = steps * waves * std::max(2.f, (float)std::min<long long>(ctas, per_sm) * T / 256.f);
      if (time < best_time)
      {
        best_time = time;
        best = {C, T};
      }
    }
  }
  return best;
}

// Columns: C adjacent ones per CTA, so that accesses cover 8 C bytes side by side.  Up to 4 (a 32-byte sector) only as
// many as bring the call down to one CTA an SM (100 columns of 7000: C = 1 15.3 us, 2 17.6, 4 24.6; 256 of 4096: 20.4,
// 12.4, -), from there as many as leave every SM a CTA and room for two.
MrConfig configure_cols(const MixedPlan &p, long long count, long long groups, int sms)
{
  auto grid = [&](int C) { return (count + C - 1) / C * groups; };
  int C = 1;
  while (C < 32 && C < count)
  {
    const long long smem = 16LL * C * p.n;
    if (smem > kMrSmem || (C < 4 ? grid(C) <= sms : smem > kMrSmem / 2 || grid(2 * C) < sms)) break;
    C *= 2;
  }
  // enough threads for one butterfly each, at most 256 where several CTAs share an SM
  int most = 0;
  for (int k = 0; k < p.ns; ++k) most = std::max(most, p.st[k].nb * C);
  const int cap = 8LL * C * p.n > kMrSmem / 2 || (count + C - 1) / C * groups <= sms ? 512 : 256;
  return {C, std::max(64, std::min(cap, (most + 31) / 32 * 32))};
}

const void *mixed_fn(int kind, bool col, bool big)
{
  return col ? mixed_cols_fn(big) : kind == kMrConv ? mixed_conv_fn(big) : mixed_rows_fn(big);
}

int mixed_launch(MixedPlan *p, int kind, bool col, MrArgs &a, cudaStream_t st, long long groups = 1)
{
  if (a.count <= 0) return FCB_OK;
  MrConfig c;
  const unsigned long long seen = p->last[col].load(std::memory_order_relaxed);
  if (groups == 1 && (long long)(seen >> 24) == a.count)
    c = {(int)(seen >> 12 & 0xfff), (int)(seen & 0xfff)};
  else
  {
    c = col ? configure_cols(*p, a.count, groups, p->sms) : configure_rows(*p, a.count, p->sms);
    if (a.count < 1LL << 40 && groups == 1)
      p->last[col].store((unsigned long long)a.count << 24 | (unsigned)c.C << 12 | (unsigned)c.threads,
                         std::memory_order_relaxed);
  }
  a.n = p->n;
  a.ns = p->ns;
  a.C = c.C;
  a.logC = 0;
  while ((1 << a.logC) < c.C) ++a.logC;
  for (int k = 0; k < p->ns; ++k) a.st[k] = p->st[k];
  a.tw = p->tw;
  a.rev = p->rev;
  const long long grid = (a.count + c.C - 1) / c.C;
  if (grid > 0x7fffffffLL || groups > 65535) return set_error(FCB_ERR_INVALID, "too many rows in one call");
  const size_t smem = p->ns > 1 ? sizeof(float2) * (size_t)c.C * p->n : 0;
  const void *fn = mixed_fn(kind, col, c.threads > 256);
  void *params[] = {&a};
  return launch_kernel(fn, dim3((unsigned)grid, (unsigned)groups), c.threads, 1, smem, params, st,
                       "mixed-radix kernel launch");
}

}  // namespace

bool mixed_columns(long long n) { return n <= kMrMaxCol && mixed_length(n); }

bool mixed_length(long long n)
{
  if (n < 2 || n > kMrMaxN) return false;
  for (int f : {2, 3, 5, 7, 11, 13})
    while (n % f == 0) n /= f;
  return n == 1;
}

// The last stage of a row takes its blocks in output order: those of adjacent threads lie n / (first radix) samples
// apart, and where that is a multiple of 16 (128 bytes) as many of a half-warp's threads as the radix read the same bank.
bool mixed_conflicts(long long n)
{
  Radices radix;
  return mixed_length(n) && factor((int)n, radix) && radix.r[0] >= 14 && n / radix.r[0] % 16 == 0;
}

void mixed_free(MixedPlan *p)
{
  if (!p) return;
  cudaFree(p->tw);
  cudaFree(p->rev);
  delete p;
}

int mixed_create(long long n, MixedPlan **out, cudaStream_t st)
{
  *out = nullptr;
  Radices radix;
  if (!mixed_length(n) || !factor((int)n, radix))
    return set_error(FCB_ERR_UNSUPPORTED, "length %lld has no mixed-radix plan", n);
  MixedPlan *p = new (std::nothrow) MixedPlan;
  if (!p) return set_error(FCB_ERR_NOMEM, "mixed-radix plan");
  p->n = (int)n;
  p->ns = radix.count;
  auto magic = [](int d) { return d == 1 ? 0u : (unsigned)(((1ULL << 32) + d - 1) / d); };
  int L = (int)n, tw = 0;
  for (int k = 0; k < p->ns; ++k)
  {
    MrStage &s = p->st[k];
    s.R = radix.r[k];
    s.L = L;
    s.S = L / s.R;
    s.nb = (int)n / s.R;
    s.mS = magic(s.S);
    s.mNB = magic(s.nb);
    s.tw = tw;
    tw += k + 1 < p->ns ? (s.R / 2) * s.S : 0;
    L = s.S;
  }
  // block b of the last stage has the digits q1 .. q(ns-1), the first one the most significant;
  // its first output is q1 + R1 (q2 + R2 (q3 + ...))
  const int nb = p->st[p->ns - 1].nb;
  const std::unique_ptr<unsigned short[]> rev(new (std::nothrow) unsigned short[nb]);
  if (!rev)
  {
    mixed_free(p);
    return set_error(FCB_ERR_NOMEM, "mixed-radix tables");
  }
  for (int b = 0; b < nb; ++b)
  {
    int rest = b, j = 0;
    for (int k = p->ns - 2; k >= 0; --k)
    {
      j = rest % p->st[k].R + p->st[k].R * j;
      rest /= p->st[k].R;
    }
    rev[j] = (unsigned short)b;
  }
  int dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&p->sms, cudaDevAttrMultiProcessorCount, dev);
  cudaError_t e = cudaSuccess;
  for (const void *fn : {mixed_rows_fn(false), mixed_rows_fn(true), mixed_conv_fn(false), mixed_conv_fn(true),
                         mixed_cols_fn(false), mixed_cols_fn(true)})
    if (e == cudaSuccess) e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kMrSmem);
  if (e != cudaSuccess)
  {
    mixed_free(p);
    return cuda_error(e, "cudaFuncSetAttribute(smem)");
  }
  e = cudaMalloc(&p->rev, sizeof(unsigned short) * (size_t)nb);
  if (e == cudaSuccess) e = cudaMalloc(&p->tw, sizeof(float4) * (size_t)std::max(tw, 1));
  if (e != cudaSuccess)
  {
    mixed_free(p);
    return set_error(FCB_ERR_NOMEM, "mixed-radix tables: %s", cudaGetErrorString(e));
  }
  // from pageable memory: the host buffer has been read when the call returns
  e = cudaMemcpyAsync(p->rev, rev.get(), sizeof(unsigned short) * (size_t)nb, cudaMemcpyHostToDevice, st);
  for (int k = 0; e == cudaSuccess && k + 1 < p->ns; ++k)
  {
    const long long m = (long long)(p->st[k].R / 2) * p->st[k].S;
    mixed_tw_kernel<<<(unsigned)((m + 255) / 256), 256, 0, st>>>(p->tw, p->st[k]);
    e = cudaGetLastError();
  }
  if (e != cudaSuccess)
  {
    mixed_free(p);
    return cuda_error(e, "mixed-radix tables");
  }
  *out = p;
  return FCB_OK;
}

void mixed_info(const MixedPlan *p, long long rows, int *rows_per_cta, int *smem, int *threads)
{
  const MrConfig c = configure_rows(*p, std::max<long long>(rows, 1), p->sms);
  if (rows_per_cta) *rows_per_cta = c.C;
  if (smem) *smem = p->ns > 1 ? 8 * c.C * p->n : 0;
  if (threads) *threads = c.threads;
}

int mixed_replica(const MixedPlan *p, const float2 *spec, long long spec_rs, long long rows, float scale, float2 *rep,
                  cudaStream_t st)
{
  const long long total = rows * p->n;
  mixed_rep_kernel<<<(unsigned)((total + 255) / 256), 256, 0, st>>>(spec, spec_rs, rep, rows, p->n,
                                                                   p->st[p->ns - 1].nb, p->rev, scale);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? FCB_OK : cuda_error(e, "replica table build");
}

int mixed_transform(MixedPlan *p, bool columns, const float2 *in, long long in_ld, float2 *out, long long out_ld,
                    long long count, bool inverse, float scale, cudaStream_t st)
{
  MrArgs a = {};
  a.in = in;
  a.out = out;
  a.in_bs = columns ? 1 : in_ld;
  a.in_es = columns ? in_ld : 1;
  a.out_bs = columns ? 1 : out_ld;
  a.out_es = columns ? out_ld : 1;
  a.count = count;
  a.inverse = inverse;
  a.scale = scale;
  return mixed_launch(p, kMrTransform, columns, a, st);
}

int mixed_column_groups(MixedPlan *p, const float2 *in, long long in_ld, long long in_gs, float2 *out,
                        long long out_ld, long long out_gs, long long cols, long long groups, bool inverse,
                        float scale, cudaStream_t st)
{
  MrArgs a = {};
  a.in = in;
  a.out = out;
  a.in_bs = a.out_bs = 1;
  a.in_es = in_ld;
  a.out_es = out_ld;
  a.in_gs = in_gs;
  a.out_gs = out_gs;
  a.count = cols;
  a.inverse = inverse;
  a.scale = scale;
  return mixed_launch(p, kMrTransform, true, a, st, groups);
}

int mixed_conv(MixedPlan *p, const float2 *in, long long in_rs, float2 *out, long long out_rs, long long rows,
               const float2 *rep, long long rep_rs, cudaStream_t st)
{
  MrArgs a = {};
  a.in = in;
  a.out = out;
  a.in_bs = in_rs;
  a.out_bs = out_rs;
  a.in_es = a.out_es = 1;
  a.count = rows;
  a.rep = rep;
  a.rep_bs = rep_rs;
  return mixed_launch(p, kMrConv, false, a, st);
}

}  // namespace fcb
