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
// 8 of twiddles per sample and pass) rather than by HBM: rows of 1144 use 45 % of
// the issue slots and 49 % of the shared-memory path with 18 warps an SM, most of
// their stalls on global loads.  Measured, 2^22 samples per call, against two Bluestein transforms in the row kernels: transform at
// 480 / 756 / 1000 / 1144 / 3000 samples 43.7 / 52.7 / 43.4 / 65.6 / 69.6 us ->
// 18.7 / 20.5 / 21 / 18 / 20.6 us (67 MB: 3.2 - 3.7 TB/s); fast convolution
// at 480 / 1144 / 3000: 88 / 134 / 131 us -> 27.2 / 29 / 35.2 us.  Columns,
// against transposing copies around the row kernels: 1144 columns of 756 24.4 ->
// 5.9 us, 1024 of 4096 61 -> 18.3 us, 4096 of 4096 219 -> 102 us.  80 registers, three
// CTAs of 256 threads an SM: two transforms a thread (packed arithmetic, 128
// registers) measured 0.6 to 1.1 of this speed, 64 registers (four CTAs) 0.73 to
// 1.13.
#pragma once

#include "fcb_engine.cuh"

#include <cuda_runtime.h>

#include <type_traits>
#include <utility>

namespace fcb {

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
  int tw;            // the stage's twiddles, in pairs q, q + 1: tw + (q / 2) S + n', q = 1, 3, ..
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
  const float4 *tw;
  const unsigned short *rev;  // block of the last stage whose first output is j, j < n / R
  const float2 *rep;       // convolution: multipliers in last-stage order [q * nb + b], with the 1/n
  long long rep_bs;
  float scale;             // transform: output scale
  int inverse;             // transform: exchange re and im on the way in and out
};

enum MrKind { kMrTransform = 0, kMrConv = 1 };

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
  begin_after_previous();
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
#pragma unroll
    for (int r = 0; r < R; ++r) x[r] = swap_if(p[r * step], inv);
  };
  // natural-order outputs of the last inverse stage (re and im exchanged)
  auto store_conv = [&](const MrStage &s, int c, int b, auto rc, const float2 *x) {
    constexpr int R = decltype(rc)::value;
    float2 *p = a.out + (r0 + c) * a.out_bs + b;
#pragma unroll
    for (int r = 0; r < R; ++r) p[s.S * r] = make_float2(x[r].y, x[r].x);
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

  // the twiddles w(q), q = 1 .. R - 1, of a butterfly, two per load (half the load
  // instructions: 1400 rows of 3000 samples 23.1 -> 20.6 us, fast convolution
  // 38.9 -> 35.2 us)
  auto twiddles = [&](const MrStage &s, int np, auto rc, float2 *w) {
    constexpr int R = decltype(rc)::value;
    const float4 *p = a.tw + s.tw + np;
#pragma unroll
    for (int q = 1; q < R; q += 2)
    {
      const float4 m = __ldg(p + (q / 2) * s.S);
      w[q] = make_float2(m.x, m.y);
      if (q + 1 < R) w[q + 1] = make_float2(m.z, m.w);
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
        float2 w[R];
        twiddles(s, b, rc, w);
        float2 *y = sm + c * cs + b * es;
        y[0] = x[0];
#pragma unroll
        for (int q = 1; q < R; ++q) y[s.S * q * es] = mr_cmul(x[q], w[q]);
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
        float2 w[R];
        twiddles(s, np, rc, w);
        y[0] = x[0];
#pragma unroll
        for (int q = 1; q < R; ++q) y[s.S * q * es] = mr_cmul(x[q], w[q]);
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
          float2 w[R], x[R];
          twiddles(s, np, rc, w);
          x[0] = y[0];
#pragma unroll
          for (int q = 1; q < R; ++q) x[q] = mr_cmul(y[s.S * q * es], w[q]);
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

// Kernels (fcb_mixed_rows.cu, fcb_mixed_conv.cu, fcb_mixed_cols.cu) for CTAs of up
// to 256 or (big) 512 threads.
const void *mixed_rows_fn(bool big);
const void *mixed_conv_fn(bool big);
const void *mixed_cols_fn(bool big);

}  // namespace fcb
