// Row kernels: transforms of real rows.
#include "fcb_rows.cuh"

namespace fcb {

void rows_table_r2c(KernelInfo (*tab)[kVariants]) { fill_rows_table<kR2C>(tab); }

}  // namespace fcb
