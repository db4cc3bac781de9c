// spmv_rows.cu -- thread-per-sub-row beta(r,VS) SpMV, y += A x, for
// matrices whose block-rows are short (every block-row's headers and values
// fit one per-warp staging buffer: stencils, Poisson, banded and FEM-like
// matrices).
//
// Work split: warp w owns the contiguous block-rows [wstart[w], wstart[w+1])
// (balanced by blocks).  It walks them in chunks of at most 32 / r block-rows:
// the chunk's packed headers and values are copied into the warp's
// shared-memory buffer with coalesced 16-byte cp.async (rows_stage.cuh), then
// lane s of a block-row works on its sub-row s from shared memory, all VS
// columns, with VS accumulators in registers.
//
// Three forms.  The wide one tests every column of a block; the deep one is the wide
// one with twice the blocks per step, for long block-rows.  The narrow
// one is for matrices whose sub-row masks span at most NS columns (stencils:
// 3 of 8 or 16): a lane's masks keep to one window of NS columns from its
// block-row's first column on (at r = 8, VS = 8 modulo VS), so it tests NS
// columns per block; a step with a wider mask in some lane runs block by block
// over all columns.  The window starts at accumulator 0: the row's
// accumulators are rotated, which the reduce tree (it pairs accumulators VS/2,
// ..., 1 apart, and addition commutes) does not see.  The wide kernel spent 165
// warp instructions per step of 8 block-rows on the 27-point stencil and was
// bound by issue.  Measured on B200, wide before / narrow now: stencil 160^3
// r = 4 FP64 278 / 201 us, 127^3 r = 8 FP64 234 / 181 us, 140^3 r = 1 FP64 201 /
// 145 us, 140^3 r = 2 mixed 182 / 135 us, 101^3 r = 1 f32 93 / 46 us.
//
// Arithmetic (bit-identical to the reference kernels core_SPC5_{r}rVc_Spmv_*,
// src/spc5.hpp:2309-2715): accumulator c of sub-row s receives
// fma(value, x[col + c], acc[c]) for every block in order whose mask s has
// bit c, reading the values at the sub-row's compact offset in the block
// (the masks of the sub-rows below s, then popcount of the bits below c) --
// the expand-load of the vector kernel.  The row sum is the
// _mm512_reduce_add tree over the accumulators (distance VS/2, then VS/4,
// ..., 1) and y[row] += sum.  Clear bits skip the FMA, which leaves the
// accumulator unchanged for finite x (it starts at +0.0 and never becomes
// -0.0), so y is bit-identical for finite x.
#include <algorithm>
#include <climits>
#include <map>
#include <mutex>
#include <tuple>
#include <type_traits>

#include "common.cuh"
#include "handle.h"
#include "rows_blocks.cuh"

namespace spc5cuda {

namespace {

using namespace rows;
constexpr int ROWS_THREADS = rows::THREADS;
constexpr int ROWS_WARPS = rows::WARPS;
constexpr int ROWS_CTAS_PER_SM = 16;

// CTAs per SM asked of the compiler.  Wide: 6 (80 registers).  Narrow: 7 (72 registers: the 5-point Poisson
// 512^2 at r = 2 then takes two chunks per warp instead of three, 8.3 against
// 9.4 us on the device; 160^3 at r = 4 197 against 203 us), 6 at r = 8, whose
// window wraps (127^3: 7 was 7% slower).  5 where 16 double accumulators (the
// float layout in mixed precision) need the registers.
// Deep: 4 for double x (106 and 121 registers), 7 for float x.
template <class LT, int R, class X, class A>
constexpr int row_ctas(int form) {
    constexpr int VS = Layout<LT>::VS;
    if (form == DEEP) return sizeof(X) == 8 ? 4 : 7;
    if (VS * sizeof(A) > 64) return 5;
    return form == NARROW && R < 8 ? 7 : 6;
}

// Whether the deep form runs instead of the wide one: 8 columns, r >= 4, and long
// block-rows, of which a chunk holds few, so that steps that wait for one another
// count for more than warps in flight.  Measured on B200 (us, wide / deep, 60,000
// rows of 41 values in a band of 401): FP64 r = 4 28.5 / 25.8, r = 8 31.9 / 28.2; float
// values r = 8 50.8 / 40.2 (4 CTAs 52.9); 200,000 rows of 31 values in a band of 301,
// 24 sub-rows per chunk, float values r = 8 73.2 / 71.0.  With float values only where
// sub-rows have few values per block: 32^3 grid of 3 unknowns, three, r = 8 39 / 45.
bool deep(int vt, int r, int nbr, long nblocks, long nnz) {
    if (vt == SPC5CUDA_F32 || r < 4) return false;
    const int rows = chunk_rows(vt, r, nbr, nblocks, nnz);
    return vt == SPC5CUDA_F64 ? rows < 24 : rows <= 24 && 2 * nnz < 3L * r * nblocks;
}

template <class LT, int R, class V, class X, class A, class Y, int FORM>
__global__ void __launch_bounds__(ROWS_THREADS, row_ctas<LT, R, X, A>(FORM))
    k_rows(int nrows, const int* __restrict__ brptr, const uint8_t* __restrict__ headers,
           const V* __restrict__ values, const int* __restrict__ valptr, const int* __restrict__ wstart, int nwarps,
           const X* __restrict__ x, Y* __restrict__ y, const int* __restrict__ run_if, int run_if_value) {
    // a launch gated on a device word (see BetaView::run_if): resident early, it
    // waits for the launch before it
    if (run_if) {
        asm volatile("griddepcontrol.launch_dependents;\n\tgriddepcontrol.wait;" ::: "memory");
        if (__ldg(run_if) != run_if_value) return;
    }
    using G = rows::Geo<LT, R, V, R>;
    extern __shared__ __align__(16) unsigned char smem[];
    const int wi = threadIdx.x >> 5;
    const int warp = blockIdx.x * ROWS_WARPS + wi;
    int r_begin = 0, r_stop = 0;
    if (warp < nwarps) {
        r_begin = __ldg(wstart + warp);
        r_stop = __ldg(wstart + warp + 1);
    }
    const uint64_t pol_x = l2_evict_last_policy();

    unsigned char* wbuf = smem + wi * G::BUF_BYTES;
    rows::walk<LT, R, V, R>(brptr, headers, values, valptr, r_begin, r_stop, wbuf,
                            [&](const rows::Chunk& ch, const uint32_t* hw, const V* vbuf) {
                                chunk_spmv<LT, R, V, X, A, Y, FORM>(ch, hw, vbuf, x, y, nrows, pol_x);
                            });
}

// Calls f(std::integral_constant<int, R>{}) for r in {1, 2, 4, 8}.
template <class F>
void dispatch_r(int r, F&& f) {
    switch (r) {
        case 1: f(std::integral_constant<int, 1>{}); return;
        case 2: f(std::integral_constant<int, 2>{}); return;
        case 4: f(std::integral_constant<int, 4>{}); return;
        case 8: f(std::integral_constant<int, 8>{}); return;
    }
    throw Error(SPC5CUDA_ERR_FORMAT, "r must be 1, 2, 4 or 8");
}

// The kernel of a form (the deep one exists for 8 columns and r >= 4).
template <class LT, int R, class V, class X, class A, class Y>
auto rows_kernel(int form) {
    if constexpr (Layout<LT>::VS == 8 && R >= 4)
        if (form == DEEP) return k_rows<LT, R, V, X, A, Y, DEEP>;
    return form == NARROW ? k_rows<LT, R, V, X, A, Y, NARROW> : k_rows<LT, R, V, X, A, Y, WIDE>;
}

template <class LT, class V, class X, class A, class Y>
int rows_occupancy(int r, int form) {
    int n = 0;
    dispatch_r(r, [&](auto RC) {
        constexpr int R_ = decltype(RC)::value;
        using G = rows::Geo<LT, R_, V, R_>;
        auto kern = rows_kernel<LT, R_, V, X, A, Y>(form);
        set_smem(kern, G::SMEM);
        SPC5_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, ROWS_THREADS, G::SMEM));
    });
    return std::max(1, std::min(n, ROWS_CTAS_PER_SM));
}

template <class LT, class V, class X, class A, class Y>
void launch_rows_impl(const BetaView& m, const X* x, Y* y, cudaStream_t s) {
    if (m.nbr <= 0 || m.nwarps <= 0) return;
    const V* vals = static_cast<const V*>(m.values);
    const int ctas = (m.nwarps + ROWS_WARPS - 1) / ROWS_WARPS;
    dispatch_r(m.r, [&](auto RC) {
        constexpr int R_ = decltype(RC)::value;
        using G = rows::Geo<LT, R_, V, R_>;
        auto kern = rows_kernel<LT, R_, V, X, A, Y>(m.form);
        set_smem(kern, G::SMEM);
        launch_after(kern, dim3(unsigned(ctas)), ROWS_THREADS, G::SMEM, m.follows, s, m.nrows, m.brptr, m.headers, vals,
                     m.valptr, m.wstart, m.nwarps, x, y, m.run_if, m.run_if_value);
    });
    SPC5_CUDA(cudaGetLastError());
}

// Of at most SAMPLED blocks spread over the matrix: how many, and how many
// whose every sub-row mask spans at most NS columns.
constexpr int SAMPLED = 1 << 15;
template <class LT, int R>
__global__ void __launch_bounds__(256) k_narrow_sample(int nbr, const int* __restrict__ brptr,
                                                       const uint8_t* __restrict__ headers, int* __restrict__ out) {
    const long nblocks = brptr[nbr];
    const long step = max(1L, nblocks / SAMPLED);
    const long i = (long(blockIdx.x) * blockDim.x + threadIdx.x) * step;
    const bool in = i < nblocks && i / step < SAMPLED;
    bool narrow = in;
    if (in) {
        uint32_t mw[Header<LT, R>::MASK_WORDS];
        load_header<LT, R>(headers, i, mw);
#pragma unroll
        for (int s = 0; s < R; ++s) {
            const uint32_t m = mask_of<LT, R>(mw, s);
            narrow = narrow && (m == 0u || (m >> (__ffs(m) - 1)) < (1u << NS));
        }
    }
    const unsigned n = __popc(__ballot_sync(FULL, narrow)), all = __popc(__ballot_sync(FULL, in));
    if ((threadIdx.x & 31) == 0 && all) {
        atomicAdd(out, int(n));
        atomicAdd(out + 1, int(all));
    }
}

template <class LT>
void narrow_sample(int r, int nbr, const int* brptr, const uint8_t* headers, int* out, cudaStream_t s) {
    dispatch_r(r, [&](auto RC) {
        k_narrow_sample<LT, decltype(RC)::value><<<SAMPLED / 256, 256, 0, s>>>(nbr, brptr, headers, out);
    });
}

// Largest block count and value count of any block-row.
__global__ void k_blockrow_max(int nbr, const int* __restrict__ brptr, const int* __restrict__ valptr,
                               int* __restrict__ out) {
    int mb = 0, mv = 0;
    for (long i = long(blockIdx.x) * blockDim.x + threadIdx.x; i < nbr; i += long(gridDim.x) * blockDim.x) {
        mb = max(mb, brptr[i + 1] - brptr[i]);
        mv = max(mv, valptr[i + 1] - valptr[i]);
    }
    for (int d = 16; d >= 1; d >>= 1) {
        mb = max(mb, __shfl_xor_sync(FULL, mb, d));
        mv = max(mv, __shfl_xor_sync(FULL, mv, d));
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMax(out, mb);
        atomicMax(out + 1, mv);
    }
}

}  // namespace

int rows_warps(int vt, int r, int form) {
    // cached per (device, value type, r, instantiation): the drop-in symbols ask on every call
    static std::mutex mu;
    static std::map<std::tuple<int, int, int, int>, int> cache;
    int dev = 0;
    SPC5_CUDA(cudaGetDevice(&dev));
    const auto key = std::make_tuple(dev, vt, r, form);
    {
        std::lock_guard<std::mutex> lk(mu);
        auto it = cache.find(key);
        if (it != cache.end()) return it->second;
    }
    int per_sm;
    if (vt == SPC5CUDA_F64) {
        per_sm = rows_occupancy<double, double, double, double, double>(r, form);
    } else if (vt == SPC5CUDA_F32_V8) {
        per_sm = rows_occupancy<double, float, float, double, double>(r, form);
    } else {
        per_sm = std::min(rows_occupancy<float, float, float, float, float>(r, form),
                          rows_occupancy<float, float, float, double, double>(r, form));
    }
    const int n = sm_count() * per_sm * ROWS_WARPS;
    std::lock_guard<std::mutex> lk(mu);
    cache[key] = n;
    return n;
}

RowStats row_stats(int vt, int r, int nbr, const int* brptr, const int* valptr, const uint8_t* headers,
                   long nblocks, long nnz, cudaStream_t s) {
    // the largest block and value counts of any block-row; narrow and all sampled blocks
    PoolBuf d(4 * sizeof(int), s);
    int* stats = d.as<int>();
    SPC5_CUDA(cudaMemsetAsync(stats, 0, 4 * sizeof(int), s));
    if (nbr > 0) {
        const int threads = 256;
        const int blocks = std::max(1, std::min(div_up(nbr, threads), sm_count() * 4));
        k_blockrow_max<<<blocks, threads, 0, s>>>(nbr, brptr, valptr, stats);
        if (headers) {
            if (vt == SPC5CUDA_F32) narrow_sample<float>(r, nbr, brptr, headers, stats + 2, s);
            else narrow_sample<double>(r, nbr, brptr, headers, stats + 2, s);
        }
        SPC5_CUDA(cudaGetLastError());
    }
    int h[4] = {0, 0, 0, 0};
    SPC5_CUDA(cudaMemcpyAsync(h, d.p, sizeof(h), cudaMemcpyDeviceToHost, s));
    SPC5_CUDA(cudaStreamSynchronize(s));
    const bool is_narrow = rows::narrow(vt, r, nbr, nblocks, nnz, h[2], h[3]);
    const int form = is_narrow ? NARROW : (deep(vt, r, nbr, nblocks, nnz) ? DEEP : WIDE);
    return RowStats{rows::fit(vt, r, h[0], h[1]), form};
}

void launch_rows_kind(int kind, const BetaView& m, const void* x, void* y, cudaStream_t s) {
    switch (kind) {
        case 0: launch_rows_f64(m, static_cast<const double*>(x), static_cast<double*>(y), s); return;
        case 1: launch_rows_f32(m, static_cast<const float*>(x), static_cast<float*>(y), s); return;
        case 2: launch_rows_mixed(m, static_cast<const float*>(x), static_cast<double*>(y), s); return;
        default: launch_rows_mixed8(m, static_cast<const float*>(x), static_cast<double*>(y), s); return;
    }
}

void launch_rows_f64(const BetaView& m, const double* x, double* y, cudaStream_t s) {
    launch_rows_impl<double, double, double, double, double>(m, x, y, s);
}

void launch_rows_f32(const BetaView& m, const float* x, float* y, cudaStream_t s) {
    launch_rows_impl<float, float, float, float, float>(m, x, y, s);
}

void launch_rows_mixed(const BetaView& m, const float* x, double* y, cudaStream_t s) {
    launch_rows_impl<float, float, float, double, double>(m, x, y, s);
}

void launch_rows_mixed8(const BetaView& m, const float* x, double* y, cudaStream_t s) {
    launch_rows_impl<double, float, float, double, double>(m, x, y, s);
}

}  // namespace spc5cuda
