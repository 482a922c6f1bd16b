// Row kernels: forward transforms.
#include "fcb_rows.cuh"

namespace fcb {

void rows_table_fwd(KernelInfo (*tab)[kVariants]) { fill_rows_table<kFwd>(tab); }

}  // namespace fcb
