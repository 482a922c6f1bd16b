// Kernel table entries of the row kernels (the variants of every length).  Each
// mode is instantiated in a translation unit of its own, so that they compile
// side by side.
#pragma once

#include "fcb_engine.cuh"
#include "fcb_internal.h"

#include <mutex>

namespace fcb {

template <int LOGN, int MODE, int T, int EPTW = 32, bool FEW = false>
KernelInfo rows_info()
{
  using S = Sched<LOGN, T, EPTW>;
  KernelInfo k;
  // the split of real rows and the replica-per-row form have no cluster form (entry left empty)
  if constexpr ((MODE != kR2C && MODE != kCoefs) || S::CS == 1) k.fn = (const void *)&rows_kernel<LOGN, MODE, T, EPTW, FEW>;
  k.ept = EPTW;
  k.overlapped = overlapped_rows(EPTW);
  k.threads = T;
  k.cluster = S::CS;
  k.rows_per_cta = S::ROWS;
  k.smem = S::SMEM;
  k.tw_bytes = S::tw_bytes();
  // The kernel for calls of few rows (same tables, same arithmetic), for the default variants of
  // 32 samples a thread: the FEW form of the same CTA up to 8192 samples; from 16384 up, where a
  // CTA of 512 threads fills an SM anyway, twice as many CTAs of 256 threads for a row.  The wide
  // variant, the default of the fused convolution at 16384 and the transforms at 32768, has none:
  // its tables and stages are others, and rows would come out differently.
  if constexpr (!FEW && EPTW == 32 && MODE != kCoefs)
  {
    constexpr bool same = (T == 128 && LOGN <= 12) || (T == 256 && (LOGN < kMin128 || LOGN == 13));
    constexpr bool split = T == 512 && LOGN >= 14 && MODE != kR2C;
    if constexpr (same || split)
    {
      static const KernelInfo few = rows_info<LOGN, MODE, split ? 256 : T, 32, true>();
      k.few = &few;
    }
  }
  return k;
}

template <int MODE, int LOGN = kMaxLogN>
void fill_rows_table(KernelInfo (*tab)[kVariants])
{
  if constexpr (LOGN >= 1)
  {
    tab[LOGN][0] = rows_info<LOGN, MODE, 256>();
    if constexpr (LOGN >= kMin512) tab[LOGN][1] = rows_info<LOGN, MODE, 512>();
    if constexpr (LOGN >= kMin128 && LOGN <= kMax128) tab[LOGN][2] = rows_info<LOGN, MODE, 128>();
    if constexpr (LOGN >= kWideLog && LOGN <= kWideMaxLog) tab[LOGN][3] = rows_info<LOGN, MODE, 256, 64>();
    fill_rows_table<MODE, LOGN - 1>(tab);
  }
}

}  // namespace fcb
