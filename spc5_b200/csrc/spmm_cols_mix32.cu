// spmm_cols_mix32.cu -- float layout, mixed: the kernels of spmm_cols.cuh.
#include "spmm_cols.cuh"

namespace spc5cuda {
SPC5_COLS_KIND(mix32, float, float, float, double, double)
}  // namespace spc5cuda
