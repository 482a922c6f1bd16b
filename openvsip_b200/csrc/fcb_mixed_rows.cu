// Mixed-radix kernels: transforms of rows.
#include "fcb_mixed.cuh"

namespace fcb {

const void *mixed_rows_fn(bool big)
{
  return big ? (const void *)&mixed_kernel<kMrTransform, false, 512, 1> : (const void *)&mixed_kernel<kMrTransform, false, 256, 3>;
}

}  // namespace fcb
