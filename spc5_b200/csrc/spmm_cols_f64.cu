// spmm_cols_f64.cu -- FP64: the kernels of spmm_cols.cuh.
#include "spmm_cols.cuh"

namespace spc5cuda {
SPC5_COLS_KIND(f64, double, double, double, double, double)
}  // namespace spc5cuda
