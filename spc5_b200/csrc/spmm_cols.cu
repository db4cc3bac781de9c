// spmm_cols.cu -- the staged SpMM with a lane per column (spmm_cols.cuh): the kinds'
// launches (kernels.h says which kind is which).
#include "kernels.h"

namespace spc5cuda {

#define SPC5_COLS_DECLARE(NAME)                                                                                    \
    void launch_spmm_cols_##NAME(const BetaView&, int, const void*, long, long, void*, long, long, cudaStream_t);  \
    void launch_batch_cols_##NAME(int, int, const BatchMat*, const BatchJob*, int, cudaStream_t);
SPC5_COLS_DECLARE(f64)
SPC5_COLS_DECLARE(f32)
SPC5_COLS_DECLARE(mix32)
SPC5_COLS_DECLARE(mix8)

int spmm_cols_kc(int vs, int r, int k) {
    const int lanes = (vs == 16 && r == 8) ? 16 : 8;
    const int kmax = mm_kc_limit(vs, r, lanes);
    int kc = 1;
    while (kc * 2 <= k && kc * 2 <= kmax) kc *= 2;
    return kc;
}

void launch_spmm_cols(int kind, const BetaView& m, int kc, const void* x, long ldx, long xcs, void* y, long ldy,
                      long ycs, cudaStream_t s) {
    const auto launch = kind == 0   ? launch_spmm_cols_f64
                        : kind == 1 ? launch_spmm_cols_f32
                        : kind == 2 ? launch_spmm_cols_mix32
                                    : launch_spmm_cols_mix8;
    launch(m, kc, x, ldx, xcs, y, ldy, ycs, s);
}

void launch_batch_cols(int kind, int r, int kc, const BatchMat* mats, const BatchJob* jobs, int njobs,
                       cudaStream_t s) {
    if (njobs <= 0) return;
    const auto launch = kind == 0   ? launch_batch_cols_f64
                        : kind == 1 ? launch_batch_cols_f32
                        : kind == 2 ? launch_batch_cols_mix32
                                    : launch_batch_cols_mix8;
    launch(r, kc, mats, jobs, njobs, s);
}

}  // namespace spc5cuda
