// Row kernels: fused fast convolutions with a replica row for every data row.
#include "fcb_rows.cuh"

namespace fcb {

void rows_table_coefs(KernelInfo (*tab)[kVariants]) { fill_rows_table<kCoefs>(tab); }

}  // namespace fcb
