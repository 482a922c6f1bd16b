// Mixed-radix kernels: transforms of columns.
#include "fcb_mixed.cuh"

namespace fcb {

const void *mixed_cols_fn(bool big)
{
  return big ? (const void *)&mixed_kernel<kMrTransform, true, 512, 1> : (const void *)&mixed_kernel<kMrTransform, true, 256, 3>;
}

}  // namespace fcb
