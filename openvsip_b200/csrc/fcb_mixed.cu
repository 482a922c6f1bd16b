// Mixed-radix FFT of any length n whose prime factors are 2, 3, 5, 7, 11 and
// 13, along rows or columns, and the fused fast convolution on such lengths.
//
// Reference behaviour replaced: the FFTW backend plans any length directly
// (src/ovxx/fftw/fftw.cpp:39-116) and takes either axis of an Fftm
// (fftw.cpp:904-977); its tests use 18, 68, 252 and 768, the SAR application
// 480, 756, 1072 and 1144.
//
// Algorithm: decimation in frequency, in place in shared memory.  Stage s (of
// radix R, sub-length L, stride S = L / R) takes the R elements base + S r of
// each butterfly, transforms them in registers, multiplies output q by
// W_L^{n' q} (n' the butterfly's place in its block) and puts it back at
// base + S q.  The first stage reads the row from global memory and the last
// one (S = 1, no twiddles) writes the result there, so ns stages make ns - 1
// passes through shared memory.  After the last stage, block b holds the
// outputs k = kprev(b) + (n / R) q, kprev the mixed-radix digit reversal, which
// a table gives.  The fast convolution multiplies by the replica in registers
// there and runs the transposed stages back (twiddle first, natural order out):
// 2 (ns - 1) passes and no reordering.  An inverse transform is the forward one
// on samples with real and imaginary parts exchanged on the way in and out.
//
// A thread holds one butterfly (at most 16 samples) at a time, so several CTAs
// share an SM and hide each other's latencies; a CTA takes as many rows as
// keep its threads busy in every stage (see configure_rows).  Columns: a CTA takes C
// adjacent ones, adjacent threads adjacent columns, so that global accesses
// cover C samples side by side and shared-memory accesses have no conflicts
// whatever the stride.
//
// Bound by latency and by the L1 / shared-memory path (16 bytes of exchange and
// 8 of twiddles per sample and pass) rather than by HBM.  Measured, 2^22 samples
// per call, against two Bluestein transforms in the row kernels: transform at
// 480 / 756 / 1000 / 1144 / 3000 samples 43.7 / 52.7 / 43.4 / 65.6 / 69.6 us ->
// 20.5 / 20.5 / 22.6 / 18.9 / 23.1 us (67 MB: 2.9 - 3.6 TB/s); fast convolution
// at 480 / 1144 / 3000: 88 / 134 / 131 us -> 28.7 / 30.7 / 38.7 us.  Columns,
// against transposing copies around the row kernels: 1144 columns of 756 24.4 ->
// 6.0 us, 1024 of 4096 61 -> 19 us, 4096 of 4096 219 -> 104 us.
#include "fcb200.h"
#include "fcb_internal.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <new>
#include <type_traits>
#include <vector>

namespace fcb {

namespace {

constexpr int kMrStages = 8;
constexpr int kMrSmem = 227 * 1024;  // shared memory of one CTA, and of an SM
constexpr int kMrMaxN = 28 * 1024;   // longest row that fits
// Longest column: two side by side fit.  Measured against transposing into rows and back:
// 8192 columns of 512 45 against 62 us; one column per CTA (16384 columns of 256, 8-byte
// accesses) 80 against 67 us.
constexpr int kMrMaxCol = kMrMaxN / 2;

struct MrStage
{
  int R, S, L;       // radix, stride, sub-length (L = R S)
  int nb;            // butterflies per transform, n / R
  unsigned mS, mNB;  // ceil(2^32 / S) and ceil(2^32 / nb): exact quotients of numbers below 2^16
  int tw;            // the stage's twiddles: tw + (q - 1) S + n', q = 1 .. R - 1
};

struct MrArgs
{
  const float2 *in;
  long long in_bs, in_es;  // element k of transform r: in[r * in_bs + k * in_es]
  float2 *out;
  long long out_bs, out_es;
  long long in_gs, out_gs;  // columns: distance of the matrices of a stack (blockIdx.y)
  long long count;         // transforms (of one matrix)
  int n, ns, C, logC;      // length, stages, transforms per CTA (columns: a power of two)
  MrStage st[kMrStages];
  const float2 *tw;
  const unsigned short *rev;  // block of the last stage whose first output is j, j < n / R
  const float2 *rep;       // convolution: multipliers in last-stage order [q * nb + b], with the 1/n
  long long rep_bs;
  float scale;             // transform: output scale
  int inverse;             // transform: exchange re and im on the way in and out
  // chirp convolution (Bluestein rows): in[k] * cin[r * cin_bs + k] for k < n_in and 0 beyond;
  // outputs k < n_out only, times cout[k] when set
  const float2 *cin;
  long long cin_bs;
  int n_in;
  const float2 *cout;
  int n_out;
};

enum MrKind { kMrTransform = 0, kMrConv = 1, kMrChirp = 2 };

// ---------------------------------------------------------------------------
// cos and sin of 2 pi k / R, evaluated by the compiler in double (Taylor series
// in the first octant) and rounded once.
constexpr double kTwoPi = 6.28318530717958647692528676655900577;
__host__ __device__ constexpr double taylor_sin(double x)
{
  double term = x, sum = x;
  for (int i = 1; i < 12; ++i)
  {
    term *= -x * x / ((2 * i) * (2 * i + 1));
    sum += term;
  }
  return sum;
}
__host__ __device__ constexpr double taylor_cos(double x)
{
  double term = 1, sum = 1;
  for (int i = 1; i < 12; ++i)
  {
    term *= -x * x / ((2 * i - 1) * (2 * i));
    sum += term;
  }
  return sum;
}
__host__ __device__ constexpr double cos_frac(int k, int R)
{
  k = ((k % R) + R) % R;
  if (2 * k > R) k = R - k;
  if (4 * k > R) return -cos_frac(R - 2 * k, 2 * R);
  return 8 * k <= R ? taylor_cos(kTwoPi * k / R) : taylor_sin(kTwoPi * (R - 4 * k) / (4.0 * R));
}
__host__ __device__ constexpr double sin_frac(int k, int R) { return cos_frac(4 * k - R, 4 * R); }

template <int N, class F, int... I>
__device__ __forceinline__ void static_for_impl(F &&f, std::integer_sequence<int, I...>)
{
  (f(std::integral_constant<int, I>{}), ...);
}
template <int N, class F>
__device__ __forceinline__ void static_for(F &&f)
{
  static_for_impl<N>(f, std::make_integer_sequence<int, N>{});
}

__device__ __forceinline__ float2 p_add(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 p_sub(float2 a, float2 b)
{
  unsigned long long d;
  const unsigned long long x = *reinterpret_cast<unsigned long long *>(&a);
  const unsigned long long y = *reinterpret_cast<unsigned long long *>(&b);
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(x), "l"(y));
  return *reinterpret_cast<float2 *>(&d);
}
__device__ __forceinline__ float2 p_fma(float s, float2 a, float2 c) { return __ffma2_rn(make_float2(s, s), a, c); }
__device__ __forceinline__ float2 mr_cmul(float2 a, float2 b)
{
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float2 swap_if(float2 a, bool s) { return s ? make_float2(a.y, a.x) : a; }

// x * exp(-2 pi i K / R)
template <int K, int R>
__device__ __forceinline__ float2 rot(float2 x)
{
  constexpr int k = ((K % R) + R) % R;
  if constexpr (k == 0) return x;
  else if constexpr (4 * k == R) return make_float2(x.y, -x.x);
  else if constexpr (2 * k == R) return make_float2(-x.x, -x.y);
  else if constexpr (4 * k == 3 * R) return make_float2(-x.y, x.x);
  else
  {
    constexpr float c = (float)cos_frac(k, R), s = (float)sin_frac(k, R);
    if constexpr (8 * k == R) return make_float2(c * (x.x + x.y), c * (x.y - x.x));
    else if constexpr (8 * k == 3 * R) return make_float2(s * (x.y - x.x), -s * (x.x + x.y));
    else return make_float2(fmaf(x.y, s, x.x * c), fmaf(x.x, -s, x.y * c));
  }
}

__host__ __device__ constexpr int gcd_(int a, int b) { return b ? gcd_(b, a % b) : a; }
__host__ __device__ constexpr int inv_mod(int a, int m)
{
  for (int i = 1; i < m; ++i)
    if (a * i % m == 1) return i;
  return 0;
}
// The radices that split as A x B (0: a prime, or 4)
__host__ __device__ constexpr int split(int R)
{
  return R == 6 ? 2 : R == 8 ? 2 : R == 9 ? 3 : R == 10 ? 2 : R == 12 ? 4 : R == 14 ? 2 : R == 15 ? 3 : R == 16 ? 4 : 0;
}

// Forward DFT of R values in registers, natural order in and out.
template <int R>
struct Dft
{
  __device__ __forceinline__ static void run(float2 *x)
  {
    if constexpr (R == 1) return;
    else if constexpr (R == 2)
    {
      const float2 a = x[0];
      x[0] = p_add(a, x[1]);
      x[1] = p_sub(a, x[1]);
    }
    else if constexpr (R == 4)
    {
      const float2 s0 = p_add(x[0], x[2]), d0 = p_sub(x[0], x[2]);
      const float2 s1 = p_add(x[1], x[3]), d1 = p_sub(x[1], x[3]);
      x[0] = p_add(s0, s1);
      x[2] = p_sub(s0, s1);
      x[1] = make_float2(d0.x + d1.y, d0.y - d1.x);
      x[3] = make_float2(d0.x - d1.y, d0.y + d1.x);
    }
    else if constexpr (split(R) != 0)
    {
      constexpr int A = split(R), B = R / A;
      constexpr bool PF = gcd_(A, B) == 1;  // coprime: no inner twiddles
      float2 y[B][A];
      static_for<B>([&](auto n2c) {
        constexpr int n2 = decltype(n2c)::value;
        static_for<A>([&](auto n1c) {
          constexpr int n1 = decltype(n1c)::value;
          y[n2][n1] = x[PF ? (B * n1 + A * n2) % R : n2 + B * n1];
        });
        Dft<A>::run(y[n2]);
      });
      static_for<A>([&](auto k1c) {
        constexpr int k1 = decltype(k1c)::value;
        float2 z[B];
        static_for<B>([&](auto n2c) {
          constexpr int n2 = decltype(n2c)::value;
          z[n2] = rot<PF ? 0 : n2 * k1, R>(y[n2][k1]);
        });
        Dft<B>::run(z);
        static_for<B>([&](auto k2c) {
          constexpr int k2 = decltype(k2c)::value;
          constexpr int k = PF ? (B * inv_mod(B % A, A) * k1 + A * inv_mod(A % B, B) * k2) % R : k1 + A * k2;
          x[k] = z[k2];
        });
      });
    }
    else
    {
      // odd prime: sums and differences of x[j], x[R - j]
      constexpr int H = (R - 1) / 2;
      float2 t[H], d[H];
      const float2 x0 = x[0];
      static_for<H>([&](auto jc) {
        constexpr int j = decltype(jc)::value;
        t[j] = p_add(x[j + 1], x[R - 1 - j]);
        d[j] = p_sub(x[j + 1], x[R - 1 - j]);
        x[0] = p_add(x[0], t[j]);
      });
      static_for<H>([&](auto kc) {
        constexpr int k = decltype(kc)::value + 1;
        float2 C = x0, S = make_float2(0.f, 0.f);
        static_for<H>([&](auto jc) {
          constexpr int j = decltype(jc)::value + 1;
          constexpr float c = (float)cos_frac(j * k, R), s = (float)sin_frac(j * k, R);
          C = p_fma(c, t[j - 1], C);
          if constexpr (j == 1) S = __fmul2_rn(make_float2(s, s), d[0]);
          else S = p_fma(s, d[j - 1], S);
        });
        x[k] = make_float2(C.x + S.y, C.y - S.x);      // C - i S
        x[R - k] = make_float2(C.x - S.y, C.y + S.x);
      });
    }
  }
};

// Calls f with the radix as a compile-time constant.
template <class F>
__device__ __forceinline__ void with_radix(int R, F &&f)
{
  switch (R)
  {
#define FCB_RADIX(r) \
  case r: f(std::integral_constant<int, r>{}); break;
    FCB_RADIX(2) FCB_RADIX(3) FCB_RADIX(4) FCB_RADIX(5) FCB_RADIX(6) FCB_RADIX(7) FCB_RADIX(8) FCB_RADIX(9)
    FCB_RADIX(10) FCB_RADIX(11) FCB_RADIX(12) FCB_RADIX(13) FCB_RADIX(14) FCB_RADIX(15) FCB_RADIX(16)
#undef FCB_RADIX
    default: break;
  }
}

// d >= 1, m = ceil(2^32 / d) (0 for d = 1), i < 2^16: i / d
__device__ __forceinline__ int quot(int i, int d, unsigned m) { return d == 1 ? i : (int)__umulhi((unsigned)i, m); }

template <int KIND, bool COL, int MAXT, int MINB>
__global__ void __launch_bounds__(MAXT, MINB) mixed_kernel(const __grid_constant__ MrArgs a)
{
  extern __shared__ float2 sm[];
  const int t = threadIdx.x, T = blockDim.x;
  const long long r0 = (long long)blockIdx.x * a.C;
  const int cnt = (int)min((long long)a.C, a.count - r0);  // transforms of this CTA
  const bool inv = KIND == kMrTransform && a.inverse;
  const int C = a.C, n = a.n, ns = a.ns;
  // distance of neighbouring elements of a transform in shared memory, and of transforms
  const int es = COL ? C : 1, cs = COL ? 1 : n;

  // item i of a stage: transform c of the CTA, butterfly b of the transform
  auto items = [&](const MrStage &s) { return COL ? s.nb << a.logC : cnt * s.nb; };
  auto item = [&](const MrStage &s, int i, int &c, int &b) {
    if (COL)
    {
      c = i & (C - 1);
      b = i >> a.logC;
    }
    else
    {
      c = quot(i, s.nb, s.mNB);
      b = i - c * s.nb;
    }
    return !COL || c < cnt;
  };
  auto base_of = [&](const MrStage &s, int b, int &np) {
    const int blk = quot(b, s.S, s.mS);
    np = b - blk * s.S;
    return blk * s.L + np;
  };
  auto load_global = [&](const MrStage &s, int c, int b, auto rc, float2 *x) {
    constexpr int R = decltype(rc)::value;
    const float2 *p = a.in + (COL ? blockIdx.y * a.in_gs : 0) + (r0 + c) * a.in_bs + b * a.in_es;
    const long long step = s.S * a.in_es;
    if constexpr (KIND == kMrChirp)
    {
      const float2 *m = a.cin + (r0 + c) * a.cin_bs + b;
#pragma unroll
      for (int r = 0; r < R; ++r)
        x[r] = b + s.S * r < a.n_in ? mr_cmul(__ldg(p + r * step), __ldg(m + s.S * r)) : make_float2(0.f, 0.f);
    }
    else
    {
#pragma unroll
      for (int r = 0; r < R; ++r) x[r] = swap_if(__ldg(p + r * step), inv);
    }
  };
  // natural-order outputs of the last inverse stage (re and im exchanged)
  auto store_conv = [&](const MrStage &s, int c, int b, auto rc, const float2 *x) {
    constexpr int R = decltype(rc)::value;
    float2 *p = a.out + (r0 + c) * a.out_bs + b;
#pragma unroll
    for (int r = 0; r < R; ++r)
    {
      const int k = b + s.S * r;
      const float2 v = make_float2(x[r].y, x[r].x);
      if constexpr (KIND == kMrChirp)
      {
        if (k < a.n_out) p[s.S * r] = a.cout ? mr_cmul(v, __ldg(a.cout + k)) : v;
      }
      else
        p[s.S * r] = v;
    }
  };
  auto times_replica = [&](const MrStage &s, int c, int b, auto rc, float2 *x) {
    constexpr int R = decltype(rc)::value;
    const float2 *w = a.rep + (r0 + c) * a.rep_bs + b;
#pragma unroll
    for (int q = 0; q < R; ++q)
    {
      const float2 v = mr_cmul(x[q], __ldg(w + q * s.nb));
      x[q] = make_float2(v.y, v.x);
    }
  };

  if (ns == 1)
  {
    // the whole transform in registers
    const MrStage &s = a.st[0];
    with_radix(s.R, [&](auto rc) {
      constexpr int R = decltype(rc)::value;
      for (int i = t; i < items(s); i += T)
      {
        int c, b;
        if (!item(s, i, c, b)) continue;
        float2 x[R];
        load_global(s, c, b, rc, x);
        Dft<R>::run(x);
        if constexpr (KIND == kMrTransform)
        {
          float2 *p = a.out + (COL ? blockIdx.y * a.out_gs : 0) + (r0 + c) * a.out_bs;
#pragma unroll
          for (int q = 0; q < R; ++q)
            p[q * a.out_es] = swap_if(make_float2(x[q].x * a.scale, x[q].y * a.scale), inv);
        }
        else
        {
          times_replica(s, c, b, rc, x);
          Dft<R>::run(x);
          store_conv(s, c, b, rc, x);
        }
      }
    });
    return;
  }

  {
    const MrStage &s = a.st[0];
    with_radix(s.R, [&](auto rc) {
      constexpr int R = decltype(rc)::value;
      for (int i = t; i < items(s); i += T)
      {
        int c, b;
        if (!item(s, i, c, b)) continue;
        float2 x[R];
        load_global(s, c, b, rc, x);
        Dft<R>::run(x);
        const float2 *w = a.tw + s.tw + b;
        float2 *y = sm + c * cs + b * es;
        y[0] = x[0];
#pragma unroll
        for (int q = 1; q < R; ++q) y[s.S * q * es] = mr_cmul(x[q], __ldg(w + (q - 1) * s.S));
      }
    });
    __syncthreads();
  }
#pragma unroll 1
  for (int k = 1; k < ns - 1; ++k)
  {
    const MrStage &s = a.st[k];
    with_radix(s.R, [&](auto rc) {
      constexpr int R = decltype(rc)::value;
      for (int i = t; i < items(s); i += T)
      {
        int c, b, np;
        if (!item(s, i, c, b)) continue;
        float2 *y = sm + c * cs + base_of(s, b, np) * es;
        float2 x[R];
#pragma unroll
        for (int r = 0; r < R; ++r) x[r] = y[s.S * r * es];
        Dft<R>::run(x);
        const float2 *w = a.tw + s.tw + np;
        y[0] = x[0];
#pragma unroll
        for (int q = 1; q < R; ++q) y[s.S * q * es] = mr_cmul(x[q], __ldg(w + (q - 1) * s.S));
      }
    });
    __syncthreads();
  }
  {
    const MrStage &s = a.st[ns - 1];
    with_radix(s.R, [&](auto rc) {
      constexpr int R = decltype(rc)::value;
      for (int i = t; i < items(s); i += T)
      {
        int c, b;
        if (!item(s, i, c, b)) continue;
        // a transform takes its blocks in output order, the convolution in place
        const int blk = KIND == kMrTransform ? a.rev[b] : b;
        float2 *y = sm + c * cs + blk * R * es;
        float2 x[R];
#pragma unroll
        for (int r = 0; r < R; ++r) x[r] = y[r * es];
        Dft<R>::run(x);
        if constexpr (KIND == kMrTransform)
        {
          float2 *p = a.out + (COL ? blockIdx.y * a.out_gs : 0) + (r0 + c) * a.out_bs + b * a.out_es;
          const long long step = s.nb * a.out_es;
#pragma unroll
          for (int q = 0; q < R; ++q)
            p[q * step] = swap_if(make_float2(x[q].x * a.scale, x[q].y * a.scale), inv);
        }
        else
        {
          times_replica(s, c, b, rc, x);
          Dft<R>::run(x);
#pragma unroll
          for (int r = 0; r < R; ++r) y[r * es] = x[r];
        }
      }
    });
  }
  if constexpr (KIND != kMrTransform)
  {
#pragma unroll 1
    for (int k = ns - 2; k >= 0; --k)
    {
      __syncthreads();
      const MrStage &s = a.st[k];
      with_radix(s.R, [&](auto rc) {
        constexpr int R = decltype(rc)::value;
        for (int i = t; i < items(s); i += T)
        {
          int c, b, np;
          if (!item(s, i, c, b)) continue;
          float2 *y = sm + c * cs + base_of(s, b, np) * es;
          const float2 *w = a.tw + s.tw + np;
          float2 x[R];
          x[0] = y[0];
#pragma unroll
          for (int q = 1; q < R; ++q) x[q] = mr_cmul(y[s.S * q * es], __ldg(w + (q - 1) * s.S));
          Dft<R>::run(x);
          if (k == 0)
            store_conv(s, c, b, rc, x);
          else
          {
#pragma unroll
            for (int r = 0; r < R; ++r) y[s.S * r * es] = x[r];
          }
        }
      });
    }
  }
}

// Twiddles W_L^{n' q} of all stages but the last, FP64 rounded to float.
__global__ void mixed_tw_kernel(float2 *tw, MrStage s)
{
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (long long)(s.R - 1) * s.S) return;
  const long long q = i / s.S + 1, np = i % s.S;
  double sn, cs;
  sincospi(-2.0 * (double)((q * np) % s.L) / (double)s.L, &sn, &cs);
  tw[s.tw + i] = make_float2((float)cs, (float)sn);
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

// Radices of n with the least cost, in ascending order of their share of two: the last stage reads R adjacent samples
// per thread, which is free of bank conflicts only for odd R.
bool factor(int n, int max_stages, std::vector<int> &best)
{
  std::vector<int> cur;
  float best_cost = 1e30f;
  auto rec = [&](auto &&self, int left, int from, float cost) -> void {
    if (cost >= best_cost) return;
    if (left == 1)
    {
      best_cost = cost;
      best = cur;
      return;
    }
    if ((int)cur.size() == max_stages) return;
    for (int R = from; R >= 2; --R)
      if (left % R == 0)
      {
        cur.push_back(R);
        self(self, left / R, R, cost + dft_cost(R) + kPassCost);
        cur.pop_back();
      }
  };
  rec(rec, n, 16, 0.f);
  if (best.empty()) return false;
  std::stable_sort(best.begin(), best.end(), [](int x, int y) { return (x & -x) > (y & -y); });
  return true;
}

struct MrConfig { int C, threads; };

}  // namespace

struct MixedPlan
{
  int n = 0, ns = 0;
  MrStage st[kMrStages] = {};
  int sms = 148;
  float2 *tw = nullptr;
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

// Columns: C adjacent ones per CTA, so that accesses cover 8 C bytes side by side.  At least 4 (a 32-byte sector)
// where they fit, more while two CTAs fit an SM and every SM has one.
MrConfig configure_cols(const MixedPlan &p, long long count, long long groups, int sms)
{
  int C = 1;
  while (C < 32 && C < count)
  {
    const long long smem = 16LL * C * p.n;
    if (smem > kMrSmem) break;
    if (C >= 4 && (smem > kMrSmem / 2 || (count + 2 * C - 1) / (2 * C) * groups < sms)) break;
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
  if (col) return big ? (const void *)&mixed_kernel<kMrTransform, true, 512, 1> : (const void *)&mixed_kernel<kMrTransform, true, 256, 3>;
  switch (kind)
  {
    case kMrTransform: return big ? (const void *)&mixed_kernel<kMrTransform, false, 512, 1> : (const void *)&mixed_kernel<kMrTransform, false, 256, 3>;
    case kMrConv: return big ? (const void *)&mixed_kernel<kMrConv, false, 512, 1> : (const void *)&mixed_kernel<kMrConv, false, 256, 3>;
    default: return big ? (const void *)&mixed_kernel<kMrChirp, false, 512, 1> : (const void *)&mixed_kernel<kMrChirp, false, 256, 3>;
  }
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
  const cudaError_t e = cudaLaunchKernel(fn, dim3((unsigned)grid, (unsigned)groups), dim3(c.threads), params, smem, st);
  return e == cudaSuccess ? FCB_OK : cuda_error(e, "mixed-radix kernel launch");
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
  std::vector<int> radix;
  if (!mixed_length(n) || !factor((int)n, kMrStages, radix))
    return set_error(FCB_ERR_UNSUPPORTED, "length %lld has no mixed-radix plan", n);
  MixedPlan *p = new (std::nothrow) MixedPlan;
  if (!p) return set_error(FCB_ERR_NOMEM, "mixed-radix plan");
  p->n = (int)n;
  p->ns = (int)radix.size();
  auto magic = [](int d) { return d == 1 ? 0u : (unsigned)(((1ULL << 32) + d - 1) / d); };
  int L = (int)n, tw = 0;
  for (int k = 0; k < p->ns; ++k)
  {
    MrStage &s = p->st[k];
    s.R = radix[k];
    s.L = L;
    s.S = L / s.R;
    s.nb = (int)n / s.R;
    s.mS = magic(s.S);
    s.mNB = magic(s.nb);
    s.tw = tw;
    tw += k + 1 < p->ns ? (s.R - 1) * s.S : 0;
    L = s.S;
  }
  // block b of the last stage has the digits q1 .. q(ns-1), the first one the most significant;
  // its first output is q1 + R1 (q2 + R2 (q3 + ...))
  const int nb = p->st[p->ns - 1].nb;
  std::vector<unsigned short> rev(nb);
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
  for (int i = 0; e == cudaSuccess && i < 8; ++i)
    e = cudaFuncSetAttribute(mixed_fn(i / 2, i / 2 == 3, i & 1), cudaFuncAttributeMaxDynamicSharedMemorySize, kMrSmem);
  if (e != cudaSuccess)
  {
    mixed_free(p);
    return cuda_error(e, "cudaFuncSetAttribute(smem)");
  }
  e = cudaMalloc(&p->rev, sizeof(unsigned short) * (size_t)nb);
  if (e == cudaSuccess) e = cudaMalloc(&p->tw, sizeof(float2) * (size_t)std::max(tw, 1));
  if (e != cudaSuccess)
  {
    mixed_free(p);
    return set_error(FCB_ERR_NOMEM, "mixed-radix tables: %s", cudaGetErrorString(e));
  }
  // from pageable memory: the host buffer has been read when the call returns
  e = cudaMemcpyAsync(p->rev, rev.data(), sizeof(unsigned short) * (size_t)nb, cudaMemcpyHostToDevice, st);
  for (int k = 0; e == cudaSuccess && k + 1 < p->ns; ++k)
  {
    const long long m = (long long)(p->st[k].R - 1) * p->st[k].S;
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

int mixed_chirp(MixedPlan *p, const float2 *in, long long in_rs, float2 *out, long long out_rs, long long rows,
                long long n, const float2 *cin, long long cin_rs, const float2 *cout, const float2 *rep, cudaStream_t st)
{
  MrArgs a = {};
  a.in = in;
  a.out = out;
  a.in_bs = in_rs;
  a.out_bs = out_rs;
  a.in_es = a.out_es = 1;
  a.count = rows;
  a.rep = rep;
  a.cin = cin;
  a.cin_bs = cin_rs;
  a.cout = cout;
  a.n_in = a.n_out = (int)n;
  return mixed_launch(p, kMrChirp, false, a, st);
}

}  // namespace fcb
