// Row kernels: inverse transforms to real rows.
#include "fcb_rows.cuh"

namespace fcb {

void rows_table_c2r(KernelInfo (*tab)[kVariants]) { fill_rows_table<kC2R>(tab); }

}  // namespace fcb
