// Row kernels: inverse transforms.
#include "fcb_rows.cuh"

namespace fcb {

void rows_table_inv(KernelInfo (*tab)[kVariants]) { fill_rows_table<kInv>(tab); }

}  // namespace fcb
