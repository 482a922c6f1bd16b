// Row kernels: the row pass of 2-D transforms with the columns' first stage
// (512-thread CTAs, the variant whose CTAs hold the most rows).
#include "fcb_rows.cuh"

namespace fcb {

template <int MODE, int LOGN>
static void fill(CrossKernel *tab)
{
  if constexpr (LOGN >= kCrossMinLog)
  {
    tab[LOGN].k = rows_info<LOGN, MODE, 512>();
    tab[LOGN].radix = cross_radix<Sched<LOGN, 512>>();
    fill<MODE, LOGN - 1>(tab);
  }
}

const CrossKernel *cross_kernel(int logn, bool inverse)
{
  static CrossKernel tab[2][kCrossMaxLog + 1];
  static std::once_flag once;
  std::call_once(once, [] {
    fill<kFwdCross, kCrossMaxLog>(tab[0]);
    fill<kInvCross, kCrossMaxLog>(tab[1]);
  });
  return logn >= kCrossMinLog && logn <= kCrossMaxLog ? &tab[inverse][logn] : nullptr;
}

}  // namespace fcb
