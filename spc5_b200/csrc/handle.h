// handle.h -- host-side internals shared by the C ABI translation units:
// device buffers, status plumbing and the matrix handle (spc5cuda_mat).
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <memory>
#include <new>

#include "common.cuh"
#include "kernels.h"
#include "memory.h"
#include "rows_stage.cuh"

namespace spc5cuda {

inline bool aligned(const void* p, size_t a) { return (reinterpret_cast<uintptr_t>(p) % a) == 0; }

inline int format_to_r(int format) {
    switch (format) {
        case SPC5CUDA_FORMAT_1rVc_WT: return 1;
        case SPC5CUDA_FORMAT_2rVc: return 2;
        case SPC5CUDA_FORMAT_4rVc: return 4;
        case SPC5CUDA_FORMAT_8rVc: return 8;
        default: return 0;
    }
}

inline int r_to_format(int r) {
    switch (r) {
        case 1: return SPC5CUDA_FORMAT_1rVc_WT;
        case 2: return SPC5CUDA_FORMAT_2rVc;
        case 4: return SPC5CUDA_FORMAT_4rVc;
        case 8: return SPC5CUDA_FORMAT_8rVc;
        default: return SPC5CUDA_UNDEFINED_FORMAT;
    }
}

// F64 and F32_V8 use the 8-column layout (uint8 masks), F32 the 16-column one.
inline bool valid_value_type(int value_type) {
    return value_type == SPC5CUDA_F64 || value_type == SPC5CUDA_F32 || value_type == SPC5CUDA_F32_V8;
}
inline int vs_of(int value_type) { return value_type == SPC5CUDA_F32 ? 16 : 8; }
inline int mask_bytes_of(int value_type) { return value_type == SPC5CUDA_F32 ? 2 : 1; }
inline int value_bytes_of(int value_type) { return value_type == SPC5CUDA_F64 ? 8 : 4; }

template <class F>
inline spc5cuda_status guarded(F&& f) {
    try {
        f();
        return SPC5CUDA_OK;
    } catch (const Error& e) {
        return e.status;
    } catch (const std::bad_alloc&) {
        return SPC5CUDA_ERR_NOMEM;
    } catch (...) {
        return SPC5CUDA_ERR_INVALID;
    }
}

inline void require(bool cond, spc5cuda_status s, const char* what) {
    if (!cond) throw Error(s, what);
}


// The sorted plan of an irregular matrix (plan.cu): the rows sorted by size,
// the long rows stored as warp streams or chains, the short rows one per lane
// (stream.cuh); it holds the plan's only copy of the values.  Launches share
// no state (the chains' sums are scratch of the call), so calls on different
// streams overlap freely.
struct SortedPlan {
    static constexpr int CLASSES = 5;
    static constexpr int SHORT_VALUES = 16;
    Owned perm;   // nrows: matrix row of each sorted row
    Owned key;    // nrows: sort key of each sorted row (stream.cuh)
    Owned val;    // values: the long rows' in step order, then the short rows' in lane order
    Owned col;    // their x indices
    Owned mask;   // long rows: active-lane mask of every step
    Owned sstep;  // long slabs + 1: first step of each
    Owned sval;   // long slabs + 1: first value of each
    Owned chains; // short rows: mask of the non-empty chains
    int row_end[CLASSES] = {0};   // sorted rows up to the end of each class of long rows
    int slab_end[CLASSES] = {0};  // slabs up to the end of each class
    int short_rows[SHORT_VALUES + 1] = {0};  // rows of n values; they follow the long ones
    int short_slabs = 0;
    long long_values = 0;
    // the chain part: the first chain_rows sorted rows
    int chain_rows = 0;
    long nchains = 0;       // non-empty chains
    long chain_values = 0;  // their values
    Owned chain;            // all of it, in one buffer:
    void* cval = nullptr;         // entries: values,
    int* ccol = nullptr;          // x indices
    int* clen = nullptr;          // per chain: entries,
    int* cid = nullptr;           // id
    long* cfirst = nullptr;       // chain slabs + 1: first entry of each
    uint16_t* cmask = nullptr;    // per row: its non-empty chains
    long bytes() const {
        return long(perm.bytes + key.bytes + val.bytes + col.bytes + mask.bytes + sstep.bytes + sval.bytes +
                    chains.bytes + chain.bytes);
    }
    // kernel launches of one SpMV: the chains' and their rows', the long rows', the short rows'
    int launches() const {
        return (chain_rows > 0 ? 2 : 0) + (slab_end[CLASSES - 1] > 0 ? 1 : 0) + (short_slabs > 0 ? 1 : 0);
    }
};

// The sorted plan of a converted matrix (synchronises s).
void build_sorted_plan(spc5cuda_mat* m, cudaStream_t s);
// The reference-order values of a handle whose plan holds the only copy,
// written to a device buffer of m->value_bytes().
void rebuild_values(const spc5cuda_mat* m, void* values, cudaStream_t s);
// y += A x through the plan (x, y of the handle's types; mixed: F32 or
// F32_V8 handle, float x, double y).
void plan_spmv(const spc5cuda_mat* m, const void* x, void* y, bool mixed, cudaStream_t s);
// Y += A X through the plan (element (row i, rhs q) of X at
// x[i * ldx + q * xcs], likewise Y).
void plan_spmm(const spc5cuda_mat* m, int k, const void* x, long ldx, long xcs, void* y, long ldy, long ycs,
               bool mixed, cudaStream_t s);

}  // namespace spc5cuda

// The device-resident SPC5Mat<T> (src/spc5.hpp:44-62).
struct spc5cuda_mat {
    using Owned = spc5cuda::Owned;
    using BetaView = spc5cuda::BetaView;
    int value_type = SPC5CUDA_F64;
    int format = SPC5CUDA_UNDEFINED_FORMAT;
    int r = 0;
    int nrows = 0, ncols = 0;
    long nnz = 0;
    long nblocks = 0;
    Owned rowptr;   // CSR row pointer (nrows+1); dropped after conversion
    Owned colidx;   // CSR column indices; dropped after conversion
    Owned values;   // nnz values (CSR order, then beta order)
    Owned brptr;    // rowsSize after conversion: ceil(nrows/r)+1 block offsets
    Owned headers;  // blocksColumnIndexesWithMasks
    Owned valptr;   // ceil(nrows/r)+1 value offsets (not in the reference format)
    Owned gstart;   // ngroups+1 block-row starts of the per-group ranges
    int ngroups = 0;
    Owned wstart;   // nwarps+1 block-row starts of the thread-per-sub-row kernel's warps
    int nwarps = 0;
    int kernel = SPC5CUDA_KERNEL_AUTO;  // SpMV kernel choice (spc5cuda_mat_set_kernel)
    bool rows_ok = false;               // every block-row fits the row kernel's buffers
    int rows_form = 0;                  // its form that suits the matrix
    std::unique_ptr<spc5cuda::SortedPlan> plan;  // rows sorted by size (irregular matrices)
    // the plan holds the only copy of the values (set when the plan is built
    // and serves SpMV): the reference order is rebuilt on demand
    bool values_dropped = false;

    int nbr() const { return r ? spc5cuda::div_up(nrows, r) : 0; }
    BetaView view() const {
        BetaView v;
        v.r = r;
        v.nrows = nrows;
        v.nbr = nbr();
        v.brptr = brptr.as<int>();
        v.headers = headers.as<uint8_t>();
        v.values = values.p;
        v.valptr = valptr.as<int>();
        v.gstart = gstart.as<int>();
        v.ngroups = ngroups;
        v.fill = fill();
        v.chunk_rows = chunk_rows();
        v.list_rows = list_rows();
        if (use_rows()) {
            v.wstart = wstart.as<int>();
            v.nwarps = nwarps;
            v.form = rows_form;
        }
        return v;
    }
    // Values per sub-row and block, and sub-rows per chunk, on average.
    float fill() const { return nblocks > 0 ? float(double(nnz) / (double(r) * double(nblocks))) : 0.f; }
    int chunk_rows() const { return spc5cuda::rows::chunk_rows(value_type, r, nbr(), nblocks, nnz); }
    int list_rows() const { return spc5cuda::rows::chunk_rows(value_type, r, nbr(), nblocks, nnz, 4096); }
    // The view of the SpMM kernels: the per-warp ranges of the staged kernel
    // whenever every block-row fits its buffers, unless the group kernel was
    // requested.
    BetaView spmm_view() const {
        BetaView v = view();
        v.wstart = nullptr;
        v.nwarps = 0;
        if (rows_ok && nwarps > 0 && kernel != SPC5CUDA_KERNEL_GROUPS) {
            v.wstart = wstart.as<int>();
            v.nwarps = nwarps;
            v.form = rows_form;
        }
        return v;
    }
    // The thread-per-sub-row kernel runs when every block-row fits its
    // staging buffers, on request or by default (it is faster than the group
    // kernel on the B200 for every r).
    bool use_rows() const {
        if (!rows_ok || nwarps <= 0) return false;
        return kernel == SPC5CUDA_KERNEL_ROWS || kernel == SPC5CUDA_KERNEL_AUTO;
    }
    // The length-sorted plan runs on request, or by default when some
    // block-row is too large for the row kernel (irregular matrices).
    bool use_plan() const {
        if (!plan) return false;
        return kernel == SPC5CUDA_KERNEL_SORTED || (kernel == SPC5CUDA_KERNEL_AUTO && !rows_ok);
    }
    bool wants_plan() const {
        return kernel == SPC5CUDA_KERNEL_SORTED || (kernel == SPC5CUDA_KERNEL_AUTO && !rows_ok);
    }
    size_t header_bytes() const {
        return size_t(nblocks) * size_t(4 + r * spc5cuda::mask_bytes_of(value_type));
    }
    size_t value_bytes() const { return size_t(nnz) * size_t(spc5cuda::value_bytes_of(value_type)); }
    // Bring the reference-order values back into the handle (synchronises s);
    // a no-op unless the plan holds the only copy.
    void restore_values(cudaStream_t s) {
        if (!values_dropped) return;
        Owned v;
        v.alloc(std::max<size_t>(value_bytes(), 16));
        spc5cuda::rebuild_values(this, v.p, s);
        SPC5_CUDA(cudaStreamSynchronize(s));
        values = std::move(v);
        values_dropped = false;
    }
    long device_bytes() const {
        return long(rowptr.bytes + colidx.bytes + values.bytes + brptr.bytes + headers.bytes +
                    valptr.bytes + gstart.bytes + wstart.bytes) + (plan ? plan->bytes() : 0L);
    }
    // The same without a plan: the reference order alone.
    long beta_bytes() const {
        return device_bytes() - (plan ? plan->bytes() : 0L) +
               (values_dropped ? std::max(long(value_bytes()), 16L) : 0L);
    }
    // The per-group block-row ranges for the current device, and the per-warp
    // ranges of the thread-per-sub-row kernel when every block-row fits it.
    void build_partition(cudaStream_t s) {
        const int vs = spc5cuda::vs_of(value_type);
        ngroups = spc5cuda::spmv_groups(vs, r);
        gstart.alloc(sizeof(int) * size_t(ngroups + 1));
        spc5cuda::launch_partition(nbr(), brptr.as<int>(), ngroups, gstart.as<int>(), s);
        const spc5cuda::RowStats stats = spc5cuda::row_stats(value_type, r, nbr(), brptr.as<int>(), valptr.as<int>(),
                                                             headers.as<uint8_t>(), nblocks, nnz, s);
        rows_ok = stats.fits;
        rows_form = stats.form;
        if (rows_ok) {
            nwarps = spc5cuda::rows_warps(value_type, r, rows_form);
            wstart.alloc(sizeof(int) * size_t(nwarps + 1));
            spc5cuda::launch_partition(nbr(), brptr.as<int>(), nwarps, wstart.as<int>(), s);
        } else {
            nwarps = 0;
            wstart.release();
        }
        restore_values(s);  // the plan may hold the only copy
        plan.reset();
        if (wants_plan()) spc5cuda::build_sorted_plan(this, s);
    }
};


namespace spc5cuda {

// Block counts per block-row of a CSR handle for rows-per-block r, scanned
// into brptr_out (ceil(nrows/r)+1 ints); returns the total (synchronises s).
long count_blocks(const spc5cuda_mat* m, int r, int* brptr_out, cudaStream_t s);

// Value offsets of every block-row from the header masks.
void valptr_from_headers(int mask_bytes, int r, int nbr, const int* brptr, const uint8_t* headers,
                         int* valptr, cudaStream_t s);

}  // namespace spc5cuda
