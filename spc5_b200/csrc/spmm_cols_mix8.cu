// spmm_cols_mix8.cu -- 8-column layout, mixed: the kernels of spmm_cols.cuh.
#include "spmm_cols.cuh"

namespace spc5cuda {
SPC5_COLS_KIND(mix8, double, float, float, double, double)
}  // namespace spc5cuda
