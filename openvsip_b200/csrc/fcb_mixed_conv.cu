// Mixed-radix kernels: fast convolution of rows.
#include "fcb_mixed.cuh"

namespace fcb {

const void *mixed_conv_fn(bool big)
{
  return big ? (const void *)&mixed_kernel<kMrConv, false, 512, 1> : (const void *)&mixed_kernel<kMrConv, false, 256, 3>;
}

}  // namespace fcb
