// spmm_cols_f32.cu -- float layout, float: the kernels of spmm_cols.cuh.
#include "spmm_cols.cuh"

namespace spc5cuda {
SPC5_COLS_KIND(f32, float, float, float, float, float)
}  // namespace spc5cuda
