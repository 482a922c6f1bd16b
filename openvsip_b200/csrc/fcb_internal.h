// Internal declarations shared by the fcb200 translation units.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cstddef>

namespace fcb {

struct RowArgs;

// Runtime copy of the compile-time schedule (see Sched<> in fcb_engine.cuh).
struct SchedRT
{
  int logn, n, ns, r1, d, half;
  int ept, rb, lrb;    // samples per thread, later-stage radix and its log2
  long long tw2_size;  // float2 entries of the stage >= 2 twiddle tables
};
SchedRT sched_rt(int logn, int ept = 32);

// A number that every plan's creation stores (always the same one) and every call reads.
struct SharedCount
{
  std::atomic<long long> v{0};
  SharedCount() = default;
  SharedCount(const SharedCount &o) : v(o.v.load(std::memory_order_relaxed)) {}
  SharedCount &operator=(const SharedCount &o) { return *this = (long long)o; }
  SharedCount &operator=(long long n)
  {
    v.store(n, std::memory_order_relaxed);
    return *this;
  }
  operator long long() const { return v.load(std::memory_order_relaxed); }
};

struct KernelInfo
{
  const void *fn = nullptr;
  int threads = 256;     // threads per CTA
  int cluster = 1;       // CTAs per row (thread-block cluster size)
  int rows_per_cta = 1;  // rows per CTA when cluster == 1
  int smem = 0;          // dynamic shared memory per CTA, bytes
  long long tw_bytes = 0; // twiddle table size
  int ept = 32;          // samples per thread (the tables depend on it)
  bool overlapped = true;        // the launch overlaps the kernel before (begin_after_previous)
  mutable SharedCount resident_tiles;  // CTAs (or clusters) resident at once, set by prepare_kernel
  const KernelInfo *few = nullptr;     // the kernel for calls whose rows are all resident at once in it
};

constexpr int kMin512 = 12;  // 512-thread variants exist for rows of 4096 samples and more
constexpr int kMin128 = 8, kMax128 = 13;  // 128-thread variants: rows of 256 .. 8192 samples
constexpr int kWideLog = 14;     // the wide variant (256 threads x 64 samples): rows of 16384 samples,
constexpr int kWideMaxLog = 15;  // and 32768 on clusters of two CTAs
// Variant ids: [0] 256, [1] 512, [2] 128 threads with 32 samples each, [3] the
// wide one.  Its public tuning value is -256.
constexpr int kVariants = 4;

// Entries [logn][variant] of one mode (fcb_rows_*.cu)
void rows_table_fwd(KernelInfo (*tab)[kVariants]);
void rows_table_inv(KernelInfo (*tab)[kVariants]);
void rows_table_conv(KernelInfo (*tab)[kVariants]);
void rows_table_coefs(KernelInfo (*tab)[kVariants]);
void rows_table_r2c(KernelInfo (*tab)[kVariants]);
void rows_table_c2r(KernelInfo (*tab)[kVariants]);
const KernelInfo *kernel_info(int logn, int mode);
// Fused kernel with element-wise multipliers (kChirpconv, fcb_bluestein.cu)
// for work rows of 2^logn samples, in the same variant as `like` (whose
// tables it reads).
const KernelInfo *chirp_kernel(int logn, const KernelInfo *like);
// Real-row kernel (inverse: kC2R, else kR2C) of 2^logn complex samples, in the
// same variant as `like` (whose tables it reads); NULL where there is none (the
// split of rows that span a cluster: measured 125 us against 89 us for two passes
// over 256 rows of 65536, each bin pair reading two slots of other CTAs).
const KernelInfo *real_kernel(int logn, bool inverse, const KernelInfo *like);
// Fused kernel for a replica row per data row, in the same variant as `like`; NULL
// where there is none (rows that span a cluster).
const KernelInfo *coefs_kernel(int logn, const KernelInfo *like);
// Row pass of a 2-D transform that combines `radix` rows (fcb_rows_cross.cu):
// rows of 64 .. 8192 samples.
struct CrossKernel
{
  KernelInfo k;
  int radix = 1;
};
constexpr int kCrossMinLog = 6, kCrossMaxLog = 13;
const CrossKernel *cross_kernel(int logn, bool inverse);
int set_variant(int logn, int mode, int threads);
const KernelInfo *kernel_variant(int logn, int mode, int threads);
int get_variant(int logn, int mode);
int prepare_kernel(const KernelInfo *k);
// Launches a kernel in clusters of `cluster` CTAs; one that starts with
// begin_after_previous() (overlapped) so that its launch overlaps the end of the
// kernel before it in the stream.
int launch_kernel(const void *fn, dim3 grid, dim3 threads, int cluster, size_t smem, void **params, cudaStream_t st,
                  const char *what, bool overlapped = true);
int launch_rows(const KernelInfo *k, long long rows, const RowArgs &args, cudaStream_t st);

int build_twiddles(int logn, int ept, float4 **out, cudaStream_t st);
int build_replica_table(int logn, int ept, const float2 *spec_dev, long long spec_rs, long long rows,
                        float4 *rep_dev, cudaStream_t st);
int replica_spectrum_dev(const float2 *rep_dev, long long n, int matched, float2 *spec_dev,
                         cudaStream_t st);
int launch_vmmul(const float2 *v, const float2 *m, long long m_rs, float2 *out, long long out_rs,
                 long long rows, long long cols, cudaStream_t st);
// out[c][r] = in[r][c], rows x cols (strides in complex elements)
int launch_transpose(const float2 *in, long long in_rs, float2 *out, long long out_rs, long long rows,
                     long long cols, cudaStream_t st);
int launch_scale_rows(const float2 *in, long long in_rs, float2 *out, long long out_rs, long long rows,
                      const float4 *rep, long long rep_rs, float scale, cudaStream_t st);

// Bluestein chirp-z pieces (fcb_bluestein.cu) for rows of non-power-of-two
// length N, computed through power-of-two work rows of M >= 2N - 1 samples.
int bluestein_tables(long long N, long long M, int sign, float2 **chirp, float2 **spectrum, cudaStream_t st);
int scale_copy(const float2 *in, float2 *out, long long total, float s, cudaStream_t st);

// Mixed-radix plans (fcb_mixed.cu): lengths whose prime factors are at most 13,
// one row in shared memory.  Device tables only; a plan may be used from several
// streams and threads at once.
struct MixedPlan;
bool mixed_length(long long n);
bool mixed_columns(long long n);  // lengths whose columns mixed_transform takes
bool mixed_conflicts(long long n);  // adjacent blocks of a row's last stage share a bank
int mixed_create(long long n, MixedPlan **out, cudaStream_t st);
void mixed_free(MixedPlan *p);
void mixed_info(const MixedPlan *p, long long rows, int *rows_per_cta, int *smem, int *threads);
// replica table: rows spectra of n values, times scale (the 1/n belongs in it), into rows * n values
int mixed_replica(const MixedPlan *p, const float2 *spec, long long spec_rs, long long rows, float scale, float2 *rep,
                  cudaStream_t st);
// `count` rows (or, with columns, columns) of a matrix whose rows are in_ld / out_ld apart
int mixed_transform(MixedPlan *p, bool columns, const float2 *in, long long in_ld, float2 *out, long long out_ld,
                    long long count, bool inverse, float scale, cudaStream_t st);
// Columns of a stack of `groups` matrices, in_gs / out_gs elements apart, whose rows
// are in_ld / out_ld apart
int mixed_column_groups(MixedPlan *p, const float2 *in, long long in_ld, long long in_gs, float2 *out,
                        long long out_ld, long long out_gs, long long cols, long long groups, bool inverse,
                        float scale, cudaStream_t st);
int mixed_conv(MixedPlan *p, const float2 *in, long long in_rs, float2 *out, long long out_rs, long long rows,
               const float2 *rep, long long rep_rs, cudaStream_t st);
// Real-input row FFTs (fcb_real.cu).
int real_twiddles(long long n, long long count, float2 **out, cudaStream_t st);
int real_twiddle_pairs(long long n, float4 **out, cudaStream_t st);
int r2c_post(float2 *y, long long rs, long long m, long long rows, const float2 *w, float scale, cudaStream_t st);
int c2r_pre(const float2 *x, long long x_rs, float2 *z, long long z_rs, long long m, long long rows,
            const float2 *w, cudaStream_t st);
int real_expand(const float *x, long long x_rs, float2 *z, long long n, long long rows, cudaStream_t st);
int herm_expand(const float2 *x, long long x_rs, float2 *z, long long n, long long rows, cudaStream_t st);
int take_real(const float2 *z, long long n, float *out, long long out_rs, long long rows, cudaStream_t st);

// Host-side copies (fcb_hostcopy.cu): rows x row_bytes between host buffers
// with the given pitches, split over the copy threads; and whether a host
// range is pageable (not pinned or registered with CUDA).
void host_copy_rows(void *dst, size_t dst_pitch, const void *src, size_t src_pitch, size_t row_bytes, size_t rows);
bool host_pageable(const void *ptr, size_t bytes);

int set_error(int code, const char *fmt, ...);
const char *error_text();
int cuda_error(cudaError_t e, const char *what);

}  // namespace fcb
