// kernels.h -- host-side launchers of the sm_100a kernels (internal).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace spc5cuda {

// ---- scan ---------------------------------------------------------------
// out[0..n] = exclusive prefix sum of in[0..n), out[n] = total.  tmp must
// hold scan_tmp_ints(n) ints.  in and out may alias.
long scan_tmp_ints(long n);
void exclusive_scan_i32(const int* in, int* out, long n, int* tmp, cudaStream_t s);

// ---- CSR checks and conversion (convert.cu) -------------------------------
// Writes two zeros to d_out when the CSR is well formed (monotone rowptr
// starting at 0, columns in [0, ncols), strictly increasing inside a row);
// d_out[0]: 1 rowptr, 2 column range; d_out[1]: order or duplicate.  colidx is
// 16-byte aligned.
void launch_validate_csr(int nrows, int ncols, long nnz, const int* rowptr, const int* colidx,
                         int* d_out, cudaStream_t s);

// counts[br] = blocks of block-row br for rows-per-block r and VS columns.
void launch_blockrow_counts(int vs, int r, int nrows, const int* rowptr, const int* colidx,
                            int* counts, cudaStream_t s);

// Emits headers and reordered values of every block-row (brptr = exclusive
// scan of the counts).  value_bytes is 8 or 4.
void launch_emit(int vs, int r, int nrows, const int* rowptr, const int* colidx,
                 const void* vin, int value_bytes, const int* brptr, uint8_t* headers,
                 void* vout, cudaStream_t s);

// valptr[br] = rowptr[min(br*r, nrows)] for br in [0, nbr].
void launch_valptr_from_csr(int r, int nrows, const int* rowptr, int* valptr, cudaStream_t s);

// counts[br] = number of values of block-row br, from the header masks.
void launch_blockrow_value_counts(int mask_bytes, int r, int nbr, const int* brptr,
                                  const uint8_t* headers, int* counts, cudaStream_t s);

// ---- SpMV (spmv.cu) ------------------------------------------------------
struct BetaView {
    int r = 0;
    int nrows = 0;
    int nbr = 0;                    // ceil(nrows / r)
    const int* brptr = nullptr;     // nbr + 1 block offsets
    const uint8_t* headers = nullptr;
    const void* values = nullptr;
    const int* valptr = nullptr;    // nbr + 1 value offsets
    const int* gstart = nullptr;    // ngroups + 1 block-row starts of the group ranges
    int ngroups = 0;
    // thread-per-sub-row kernel (short block-rows): nwarps + 1 block-row
    // starts of the per-warp ranges; null selects the group kernel
    const int* wstart = nullptr;
    int nwarps = 0;
    int form = 0;  // of the row kernel: rows::WIDE, NARROW or DEEP (rows_blocks.cuh)
    float fill = 0.f;     // values per sub-row and block on average
    int chunk_rows = 32;  // sub-rows of an average chunk of the row kernel (rows::chunk_rows),
    int list_rows = 32;   // and of one of the value lists' (spmm_rows.cu: 4 KB of headers at least)
    // when set, the launch does its work only if *run_if == run_if_value (a
    // device word written by an earlier kernel on the same stream)
    const int* run_if = nullptr;
    int run_if_value = 0;
    bool follows = false;  // may become resident before the launch before it ends (run_if launches wait for it)
};

// Number of VS-lane groups the SpMV kernels launch on the current device
// for rows-per-block r: one wave of resident CTAs.
int spmv_groups(int vs, int r);

// gstart[0..ngroups] = block-row ranges holding ~nblocks/ngroups blocks each.
void launch_partition(int nbr, const int* brptr, int ngroups, int* gstart, cudaStream_t s);

void launch_spmv_f64(const BetaView& m, const double* x, double* y, cudaStream_t s);

// Thread-per-sub-row kernel (spmv_rows.cu): resident warps on this device,
// whether block-rows of at most max_blocks blocks / max_values values fit its
// staging buffers, and what a converted matrix asks of it (synchronises s).
// (vt: the handle's value type, SPC5CUDA_F64 / F32 / F32_V8.)
int rows_warps(int vt, int r, int form);
struct RowStats {
    bool fits;    // every block-row fits the row kernel's buffers
    int form;     // of the row kernel that suits the matrix
};
// (headers may be null: the form is not asked for.)
RowStats row_stats(int vt, int r, int nbr, const int* brptr, const int* valptr, const uint8_t* headers,
                   long nblocks, long nnz, cudaStream_t s);
// What the drop-in symbols find out about bare arrays, without a host round
// trip (core_prep.cu): byte offsets in a 256-byte aligned scratch block of
// valptr, gstart and wstart (as in BetaView) and of flag = 0 when some
// block-row does not fit the row kernel's buffers, else 1 for its wide, 2 for
// its narrow instantiation.
struct CoreScratch {
    size_t valptr, stats, before, gstart, wstart, flag, bytes;
};
CoreScratch core_scratch(int nbr, int ngroups, int nwarps);
void launch_core_prep(int value_type, int r, int nbr, const int* brptr, const uint8_t* headers, int ngroups, int nwarps,
                      const CoreScratch& c, unsigned char* mem, cudaStream_t s);
// The row SpMV of a kind (below).
void launch_rows_kind(int kind, const BetaView& m, const void* x, void* y, cudaStream_t s);
void launch_rows_f64(const BetaView& m, const double* x, double* y, cudaStream_t s);
void launch_rows_f32(const BetaView& m, const float* x, float* y, cudaStream_t s);
void launch_rows_mixed(const BetaView& m, const float* x, double* y, cudaStream_t s);
// Float values in the 8-column layout (F32_V8), float x, FP64 accumulation and y.
void launch_rows_mixed8(const BetaView& m, const float* x, double* y, cudaStream_t s);
void launch_spmv_f32(const BetaView& m, const float* x, float* y, cudaStream_t s);
void launch_spmv_mixed(const BetaView& m, const float* x, double* y, cudaStream_t s);
void launch_spmv_mixed8(const BetaView& m, const float* x, double* y, cudaStream_t s);

// ---- SpMM (spmm.cu): Y += A X.  Element (row i, right-hand side q) of X
// is x[i * ldx + q * xcs] (row-major: xcs = 1; column-major: ldx = 1,
// xcs = leading dimension), likewise Y with ldy, ycs.
void launch_spmm_f64(const BetaView& m, int k, const double* x, long ldx, long xcs, double* y,
                     long ldy, long ycs, cudaStream_t s);
void launch_spmm_f32(const BetaView& m, int k, const float* x, long ldx, long xcs, float* y,
                     long ldy, long ycs, cudaStream_t s);
void launch_spmm_mixed(const BetaView& m, int k, const float* x, long ldx, long xcs, double* y,
                       long ldy, long ycs, cudaStream_t s);
void launch_spmm_mixed8(const BetaView& m, int k, const float* x, long ldx, long xcs, double* y,
                        long ldy, long ycs, cudaStream_t s);

// ---- staged SpMM (spmm_rows.cu) over the per-warp ranges m.wstart /
// m.nwarps of a matrix whose block-rows fit the row kernels' buffers; same
// arguments and results as launch_spmm_*.
void launch_spmm_rows_f64(const BetaView& m, int k, const double* x, long ldx, long xcs, double* y,
                          long ldy, long ycs, cudaStream_t s);
void launch_spmm_rows_f32(const BetaView& m, int k, const float* x, long ldx, long xcs, float* y,
                          long ldy, long ycs, cudaStream_t s);
void launch_spmm_rows_mixed(const BetaView& m, int k, const float* x, long ldx, long xcs, double* y,
                            long ldy, long ycs, cudaStream_t s);
void launch_spmm_rows_mixed8(const BetaView& m, int k, const float* x, long ldx, long xcs, double* y,
                             long ldy, long ycs, cudaStream_t s);

// ---- batched SpMM (spmm.cu): many matrices, one launch per (r, kc) class
struct BatchMat {
    const int* brptr;
    const uint8_t* headers;
    const void* values;
    const int* valptr;
    const void* x;  // row-major ncols x k (ldx)
    long ldx;
    void* y;        // row-major nrows x k (ldy)
    long ldy;
    long xcs;       // stride between right-hand sides (1: row-major)
    long ycs;
    int nrows;
    int k;          // right-hand sides
};
struct BatchJob {
    int mat;      // index into the BatchMat array
    int r_begin;  // block-row range
    int r_end;
    int kofs;     // first right-hand side of this pass
};
// right-hand sides per pass for rows-per-block r and k right-hand sides
int batch_kc(int r, int k);
// kind 0 = f64, 1 = f32, 2 = mixed (f32 values and x, f64 y), 3 = mixed in the
// 8-column layout (F32_V8 matrices)
void launch_batch(int kind, int r, int kc, const BatchMat* mats, const BatchJob* jobs, int njobs,
                  int ctas, cudaStream_t s);
// Right-hand sides per pass of the staged SpMM with k left: 2, 4, 8 or 16 (the
// last pass may have fewer).
int spmm_rows_kc(int k);
// Whether a pass with k right-hand sides left runs with a lane per column
// (spmm_cols.cu) instead (fill, list_rows, chunk_rows: as in BetaView), and whether
// one contiguous right-hand side does instead of the row SpMV.
bool spmm_columns(int vs, int value_bytes, int r, float fill, int list_rows, int k);
bool spmv_columns(int vs, int r, float fill, int chunk_rows);
// Right-hand sides of such a pass (a power of two), and its launch for a kind.
int spmm_cols_kc(int vs, int r, int k);
void launch_spmm_cols(int kind, const BetaView& m, int kc, const void* x, long ldx, long xcs, void* y, long ldy,
                      long ycs, cudaStream_t s);
void launch_batch_cols(int kind, int r, int kc, const BatchMat* mats, const BatchJob* jobs, int njobs,
                       cudaStream_t s);
// Most right-hand sides of such a pass: r x (vs / lanes columns per lane) x kc
// accumulators stay at most 32, kc at most 16 (r <= 2) or 8.
constexpr int mm_kc_limit(int vs, int r, int lanes) {
    const int most = r <= 2 ? 16 : 8, kc = 32 / (r * (vs / lanes));
    return kc > most ? most : kc;
}
// The same for matrices whose block-rows fit the row kernels' buffers
// (spmm_rows.cu): one warp per job at a time; kc from spmm_rows_kc, or 1 for
// jobs of one right-hand side with contiguous x and y, which run the row SpMV's
// wide or narrow form.
void launch_batch_rows(int kind, int r, int kc, bool narrow, const BatchMat* mats, const BatchJob* jobs, int njobs,
                       cudaStream_t s);

}  // namespace spc5cuda
