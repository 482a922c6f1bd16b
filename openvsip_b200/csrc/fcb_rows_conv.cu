// Row kernels: fused fast convolutions.
#include "fcb_rows.cuh"

namespace fcb {

void rows_table_conv(KernelInfo (*tab)[kVariants]) { fill_rows_table<kFastconv>(tab); }

}  // namespace fcb
