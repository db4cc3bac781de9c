// spmm_cols.cuh -- staged multi-RHS SpMM with a lane per column, for few
// right-hand sides on blocks of many rows and for long rows of full blocks
// (spmm_columns in spmm_rows.cu says which; that file has the other staged SpMM, and
// why it tests less).
//
// A warp walks its block-rows in chunks staged into shared memory; each
// block-row of a chunk is served by L lanes (mm_lanes), and lane q owns the
// columns q + L k of every block for all R sub-rows and KC right-hand sides
// (R * VS / L * KC accumulators, at most 32).  Per block a lane decodes the
// staged header once for all sub-rows -- what the lane-per-sub-row list of
// spmm_rows.cu does once per sub-row --, loads its KC x values per column (only
// where some sub-row has a value in that column: blocks at the right edge may
// reach past the last column), reads each of its values once from shared memory
// and issues KC multiply-adds with it.
//
// Arithmetic per right-hand side j is the SpMV's (src/spc5.hpp:2309-2715):
// accumulator (i, j) of column c receives fma(value, x[col + c][j], acc) for
// every block in order whose mask i has bit c; the row sum is the
// _mm512_reduce_add tree over the VS columns (XOR distances VS/2, ..., 1: in
// the lane, then across the L lanes); then
// Y[row][j] += sum (one rounding: red.add.f64 for double Y, load-add-store for
// float Y, exactly as the SpMV kernels).  Column j of the result is therefore
// bit-identical to an SpMV with column j of X.
//
// One source file per kind of values (spmm_cols_f64.cu, ...) instantiates these, so that
// each is a module of its own: a process loads a module at the first use of one of its
// kernels, and all kinds in one took 17 ms on a B200.
#pragma once

#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "kernels.h"
#include "rows_stage.cuh"

namespace spc5cuda {

namespace {

using rows::FULL;

// Registers limit this kernel to 4 CTAs per SM, so it stages larger chunks than
// the SpMV (every block-row that fits the SpMV's buffers fits these).
// One or two right-hand sides leave room for the SpMV's own chunks and 5 or 6
// CTAs, except with double values at r = 8, and where those chunks hold 32 sub-rows
// (stencil 64^3, k = 2 on a B200: mixed 77 us at 4 CTAs and larger chunks / 67 so, r =
// 4 46 / 38; FP64, r = 8 55 / 73; 32^3 grid of 3 unknowns, 81 values per row, FP64, r = 4
// 31 / 41).
constexpr bool cols_small(int value_bytes, int r, int kc, int chunk_rows) {
    return kc <= 2 && (r < 8 || value_bytes == 4) && chunk_rows >= 32;
}
template <bool SMALL>
constexpr int cols_hb = SMALL ? rows::HB : 2048;
template <bool SMALL>
constexpr int cols_vb = SMALL ? rows::VB : 8192;
template <bool SMALL>
constexpr int cols_ctas(int acc_bytes) { return SMALL ? (acc_bytes > 64 ? 5 : 6) : 1; }

// Union of the sub-row masks (bit c: some sub-row has a value in column c).
template <class LT, int R>
__device__ __forceinline__ uint32_t mask_union(const uint32_t (&mw)[Header<LT, R>::MASK_WORDS]) {
    uint32_t uni = 0;
#pragma unroll
    for (int w = 0; w < Header<LT, R>::MASK_WORDS; ++w) uni |= mw[w];
    if constexpr (Layout<LT>::MASK_BYTES == 1) return (uni | (uni >> 16)) | ((uni | (uni >> 16)) >> 8);
    else return uni | (uni >> 16);
}

// Per mask word: exclusive prefix of the sub-row value counts, one field per
// sub-row (pre); returns the block's value count.
template <class LT, int R>
__device__ __forceinline__ int subrow_prefix(const uint32_t (&mw)[Header<LT, R>::MASK_WORDS],
                                             uint32_t (&pre)[Header<LT, R>::MASK_WORDS]) {
    uint32_t carry = 0;
#pragma unroll
    for (int w = 0; w < Header<LT, R>::MASK_WORDS; ++w) {
        uint32_t cnt = mw[w] - ((mw[w] >> 1) & 0x55555555u);
        cnt = (cnt & 0x33333333u) + ((cnt >> 2) & 0x33333333u);
        cnt = (cnt + (cnt >> 4)) & 0x0F0F0F0Fu;
        if constexpr (Layout<LT>::MASK_BYTES == 1) {
            pre[w] = cnt * 0x01010100u + carry * 0x01010101u;
            carry += (cnt * 0x01010101u) >> 24;
        } else {
            cnt = (cnt + (cnt >> 8)) & 0x001F001Fu;
            pre[w] = (cnt << 16) + carry * 0x00010001u;
            carry += (cnt + (cnt >> 16)) & 0xFFFFu;
        }
    }
    return int(carry);
}

// Field f of the result: offset, from the block's first value, of the value
// of sub-row (w * fields per word + f) in the column whose lower columns are
// `below`, for mask word w with prefix pre_w.
template <class LT, int R>
__device__ __forceinline__ uint32_t column_offsets(uint32_t mw_w, uint32_t pre_w, uint32_t below) {
    if constexpr (R == 1) {
        return uint32_t(__popc(mw_w & below));
    } else if constexpr (Layout<LT>::MASK_BYTES == 1) {
        uint32_t t = mw_w & (below * 0x01010101u);
        t = t - ((t >> 1) & 0x55555555u);
        t = (t & 0x33333333u) + ((t >> 2) & 0x33333333u);
        return pre_w + ((t + (t >> 4)) & 0x0F0F0F0Fu);
    } else {
        uint32_t t = mw_w & (below * 0x00010001u);
        t = t - ((t >> 1) & 0x55555555u);
        t = (t & 0x33333333u) + ((t >> 2) & 0x33333333u);
        t = (t + (t >> 4)) & 0x0F0F0F0Fu;
        return pre_w + ((t + (t >> 8)) & 0x001F001Fu);
    }
}

// Lanes per block-row of the staged SpMM: one column per lane for double
// blocks (8 columns); for float blocks (16 columns) two per lane, except at
// r = 8 where one column per lane keeps four right-hand sides per pass.
template <class LT, int R>
constexpr int mm_lanes() {
    return (Layout<LT>::VS == 16 && R == 8) ? 16 : 8;
}

// Y += A X over block-rows [r_begin, r_stop) of one matrix for right-hand
// sides [0, KC) of xm / ym (already offset to the pass's first one).
template <class LT, int R, int KC, bool SMALL, class V, class X, class A, class Y>
__device__ __forceinline__ void mm_range(int nrows, const int* __restrict__ brptr,
                                         const uint8_t* __restrict__ headers, const V* __restrict__ values,
                                         const int* __restrict__ valptr, int r_begin, int r_stop,
                                         const X* __restrict__ xm, long ldx, long xcs, Y* __restrict__ ym,
                                         long ldy, long ycs, unsigned char* wbuf) {
    constexpr int VS = Layout<LT>::VS;
    constexpr int L = mm_lanes<LT, R>();  // lanes per block-row
    constexpr int CPL = VS / L;                // columns per lane: q + L k
    constexpr int LOGL = L == 16 ? 4 : (L == 8 ? 3 : (L == 4 ? 2 : (L == 2 ? 1 : 0)));
    using G = rows::Geo<LT, R, V, L, cols_hb<SMALL>, cols_vb<SMALL>>;
    constexpr int MB = G::MB, MW = G::MW;
    constexpr int FPW = 4 / MB;  // mask fields per 32-bit word
    constexpr int BITS = 8 * MB;
    constexpr uint32_t FMASK = MB == 1 ? 0xFFu : 0xFFFFu;
    constexpr bool Y_ATOMIC = sizeof(Y) == 8;
    static_assert(R * CPL * KC <= 32, "accumulators");
    // blocks per step: their x loads are issued before the FMAs, which still
    // run block by block (the chain order is kept)
    constexpr int XW = CPL * KC;  // x values of one block
    constexpr int U = XW >= 8 ? 1 : 8 / XW;
    const int lane = threadIdx.x & 31;
    const int slot = lane / L;  // block-row of the chunk
    const int q = lane % L;     // this lane's columns: q + L k
    const uint64_t pol_x = l2_evict_last_policy();

    A acc[R][CPL][KC];
    auto zero = [&]() {
#pragma unroll
        for (int i = 0; i < R; ++i)
#pragma unroll
            for (int k = 0; k < CPL; ++k)
#pragma unroll
                for (int j = 0; j < KC; ++j) acc[i][k][j] = A(0);
    };

    // ---- row sums: the _mm512_reduce_add tree (distance VS/2, ..., 1).
    // Levels of distance >= L pair columns of one lane.  The last log2(L)
    // levels pair the lanes of the block-row as a reduce-scatter of the
    // N = R KC sums: at distance d the lane with bit d set keeps the odd
    // entries and its partner the even ones, each adding the partner's
    // copy (the same pairs as the tree, so the same bits), until one sum
    // per entry is left; then the plain butterfly.  Lane q ends with the
    // entries t L + rev(q) (rev: q's log2(L) bits reversed), or, when
    // N < L, entry rev(q) mod N in the lanes whose low bits are zero.
    // Entries are ordered so that one store covers neighbouring
    // addresses: (i, j) at i KC + j for row-major Y (ycs == 1), at j R + i
    // otherwise (the R rows of consecutive block-rows are adjacent).  Then
    // Y[brow R + i][j] += sum (warp-uniform call).
    auto flush = [&](bool mine, int brow) {
        constexpr int N = R * KC;
#pragma unroll
        for (int i = 0; i < R; ++i) {
#pragma unroll
            for (int j = 0; j < KC; ++j) {
#pragma unroll
                for (int d = CPL / 2; d >= 1; d >>= 1) {
#pragma unroll
                    for (int k = 0; k < d; ++k) acc[i][k][j] = acc[i][k][j] + acc[i][k + d][j];
                }
            }
        }
        const bool row_major = ycs == 1;
        A sv[N];
#pragma unroll
        for (int e = 0; e < N; ++e) sv[e] = row_major ? acc[e / KC][0][e % KC] : acc[e % R][0][e / R];
#pragma unroll
        for (int lev = 0; lev < LOGL; ++lev) {
            const int d = L >> (lev + 1);
            const int n = N >> lev;  // entries still held
            const bool hi = (q & d) != 0;
            if (n >= 2) {
#pragma unroll
                for (int t = 0; t < n / 2; ++t) {
                    const A keep = hi ? sv[2 * t + 1] : sv[2 * t];
                    const A send = hi ? sv[2 * t] : sv[2 * t + 1];
                    sv[t] = keep + __shfl_xor_sync(FULL, send, d);
                }
            } else {
                sv[0] = sv[0] + __shfl_xor_sync(FULL, sv[0], d);
            }
        }
        const int rq = LOGL ? int(__brev(unsigned(q)) >> (32 - LOGL)) : 0;
        constexpr int PER = N >= L ? N / L : 1;
        const bool writer = mine && (N >= L || (q & (L / N - 1)) == 0);
        const long row0 = long(brow) * R;
#pragma unroll
        for (int t = 0; t < PER; ++t) {
            const int e = N >= L ? t * L + rq : (rq & (N - 1));
            const int i = row_major ? e / KC : e % R;
            const int j = row_major ? e % KC : e / R;
            const long yrow = row0 + i;
            if (writer && yrow < nrows) {
                Y* dst = ym + yrow * ldy + long(j) * ycs;
                if constexpr (Y_ATOMIC) atomicAdd(dst, Y(sv[t]));
                else *dst = *dst + Y(sv[t]);
            }
        }
    };

    auto compute = [&](const rows::Chunk& ch, const uint32_t* hw, const V* vbuf) {
        const int src = slot > 0 ? slot - 1 : 0;
        const int b_prev = __shfl_sync(FULL, ch.b_hi, src);
        const int v_prev = __shfl_sync(FULL, ch.v_hi, src);
        const int b_mine = __shfl_sync(FULL, ch.b_hi, slot);
        const bool mine = slot < ch.nrow;
        int b = mine ? (slot > 0 ? b_prev : ch.b_lo) : 0;
        const int b_stop = mine ? b_mine : 0;
        int v = (mine ? (slot > 0 ? v_prev : ch.v_lo) : 0) - ch.v_al;

        zero();
        while (__any_sync(FULL, b < b_stop)) {
            int col[U];
            uint32_t mw[U][MW];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                col[u] = 0;
#pragma unroll
                for (int w = 0; w < MW; ++w) mw[u][w] = 0u;
                if (b + u < b_stop) col[u] = rows::decode_staged<LT, R>(hw, long(b + u) * G::STRIDE - ch.h_al, mw[u]);
            }
            // x of this lane's columns where some sub-row has a value
            X xk[U][CPL][KC];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const uint32_t uni = mask_union<LT, R>(mw[u]);
#pragma unroll
                for (int k = 0; k < CPL; ++k) {
                    const bool has = (uni >> (q + L * k)) & 1u;
                    const X* xr = xm + long(col[u] + q + L * k) * ldx;
#pragma unroll
                    for (int j = 0; j < KC; ++j) xk[u][k][j] = has ? ld_x(xr + long(j) * xcs, pol_x) : X(0);
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                uint32_t pre[MW];
                const int tot = subrow_prefix<LT, R>(mw[u], pre);
#pragma unroll
                for (int k = 0; k < CPL; ++k) {
                    const int c = q + L * k;
                    const uint32_t below = (1u << c) - 1u;
#pragma unroll
                    for (int w = 0; w < MW; ++w) {
                        const uint32_t off = column_offsets<LT, R>(mw[u][w], pre[w], below);
#pragma unroll
                        for (int f = 0; f < FPW; ++f) {
                            const int i = w * FPW + f;
                            if (i < R && ((mw[u][w] >> (f * BITS + c)) & 1u)) {
                                const A e = A(vbuf[v + int((off >> (f * BITS)) & FMASK)]);
#pragma unroll
                                for (int j = 0; j < KC; ++j) acc[i][k][j] = fma(e, A(xk[u][k][j]), acc[i][k][j]);
                            }
                        }
                    }
                }
                v += tot;
            }
            b += U;
        }
        flush(mine, ch.r0 + slot);
    };
    rows::walk<LT, R, V, L, cols_hb<SMALL>, cols_vb<SMALL>>(brptr, headers, values, valptr, r_begin, r_stop, wbuf, compute);
}

// One matrix: the grid's warps, one resident wave, share its block-rows
// (part_start).  The SpMV's partition is for 5 to 7 CTAs per SM, of which 3 or 4
// fit here: stencil 64^3, r = 8, on a B200 FP64 k = 4 74 us, now 60; k = 2 55 / 45;
// mixed k = 5 148 / 121.
template <class LT, int R, int KC, bool SMALL, class V, class X, class A, class Y>
__global__ void __launch_bounds__(rows::THREADS, cols_ctas<SMALL>(Layout<LT>::VS * int(sizeof(A))))
    k_spmm_cols(int nrows, const int* __restrict__ brptr, const uint8_t* __restrict__ headers,
                const V* __restrict__ values, const int* __restrict__ valptr, const int* __restrict__ wstart,
                int nwarps, const X* __restrict__ xm, long ldx, long xcs, Y* __restrict__ ym, long ldy, long ycs) {
    using G = rows::Geo<LT, R, V, mm_lanes<LT, R>(), cols_hb<SMALL>, cols_vb<SMALL>>;
    extern __shared__ __align__(16) unsigned char smem[];
    const int wi = threadIdx.x >> 5;
    const int warp = blockIdx.x * rows::WARPS + wi;
    const int W = gridDim.x * rows::WARPS;
    const int r_begin = rows::part_start(wstart, nwarps, warp, W), r_stop = rows::part_start(wstart, nwarps, warp + 1, W);
    mm_range<LT, R, KC, SMALL, V, X, A, Y>(nrows, brptr, headers, values, valptr, r_begin, r_stop, xm, ldx, xcs, ym, ldy, ycs,
                                    smem + wi * G::BUF_BYTES);
}

// Batched: warps walk the job list with the grid's warp count as stride; job
// j is block-rows [r_begin, r_end) of mats[j.mat] for right-hand sides
// [kofs, kofs + KC).  X and Y of a batch are row-major (xcs = ycs = 1).
template <class LT, int R, int KC, bool SMALL, class V, class X, class A, class Y>
__global__ void __launch_bounds__(rows::THREADS, cols_ctas<SMALL>(Layout<LT>::VS * int(sizeof(A))))
    k_spmm_cols_batch(const BatchMat* __restrict__ mats, const BatchJob* __restrict__ jobs, int njobs) {
    using G = rows::Geo<LT, R, V, mm_lanes<LT, R>(), cols_hb<SMALL>, cols_vb<SMALL>>;
    extern __shared__ __align__(16) unsigned char smem[];
    const int wi = threadIdx.x >> 5;
    const int nw = gridDim.x * rows::WARPS;
    for (int j = blockIdx.x * rows::WARPS + wi; j < njobs; j += nw) {  // warp-uniform
        const BatchJob job = jobs[j];
        const BatchMat& m = mats[job.mat];
        mm_range<LT, R, KC, SMALL, V, X, A, Y>(m.nrows, m.brptr, m.headers, static_cast<const V*>(m.values), m.valptr,
                                        job.r_begin, job.r_end, static_cast<const X*>(m.x) + job.kofs, m.ldx, 1L,
                                        static_cast<Y*>(m.y) + job.kofs, m.ldy, 1L, smem + wi * G::BUF_BYTES);
    }
}

// Calls f(integral_constant<R>, integral_constant<KC>, bool_constant<SMALL>) for r in
// {1, 2, 4, 8} and kc a power of two up to mm_kc_limit of the kernel's lanes.
template <class LT, class V, class F>
void dispatch_rkc(int r, int kc, int chunk_rows, F&& f) {
    using std::integral_constant;
    auto with_r = [&](auto RC) {
        constexpr int R_ = decltype(RC)::value;
        constexpr int KMAX = mm_kc_limit(Layout<LT>::VS, R_, mm_lanes<LT, R_>());
        auto with_kc = [&](auto KCC) {
            constexpr int KC_ = decltype(KCC)::value;
            if constexpr (KC_ <= KMAX) {
                if constexpr (cols_small(int(sizeof(V)), R_, KC_, 32))
                    if (cols_small(int(sizeof(V)), R_, KC_, chunk_rows)) {
                        f(RC, KCC, std::true_type{});
                        return true;
                    }
                f(RC, KCC, std::false_type{});
                return true;
            }
            return false;
        };
        switch (kc) {
            case 1: return with_kc(integral_constant<int, 1>{});
            case 2: return with_kc(integral_constant<int, 2>{});
            case 4: return with_kc(integral_constant<int, 4>{});
            case 8: return with_kc(integral_constant<int, 8>{});
            case 16: return with_kc(integral_constant<int, 16>{});
        }
        return false;
    };
    bool done = false;
    switch (r) {
        case 1: done = with_r(integral_constant<int, 1>{}); break;
        case 2: done = with_r(integral_constant<int, 2>{}); break;
        case 4: done = with_r(integral_constant<int, 4>{}); break;
        case 8: done = with_r(integral_constant<int, 8>{}); break;
    }
    if (!done) throw Error(SPC5CUDA_ERR_INVALID, "unsupported (r, right-hand sides per pass)");
}

template <class LT, class V, class X, class A, class Y>
void cols_pass(const BetaView& m, int kc, const void* x, long ldx, long xcs, void* y, long ldy, long ycs,
               cudaStream_t s) {
    dispatch_rkc<LT, V>(m.r, kc, m.chunk_rows, [&](auto RC, auto KCC, auto SC) {
        constexpr int R_ = decltype(RC)::value, KC_ = decltype(KCC)::value;
        constexpr bool SMALL = decltype(SC)::value;
        constexpr int SMEM = rows::Geo<LT, R_, V, mm_lanes<LT, R_>(), cols_hb<SMALL>, cols_vb<SMALL>>::SMEM;
        auto kern = k_spmm_cols<LT, R_, KC_, SMALL, V, X, A, Y>;
        set_smem(kern, SMEM);
        static const int per_sm = resident_ctas(kern, rows::THREADS, SMEM);
        const int ctas = std::min((m.nwarps + rows::WARPS - 1) / rows::WARPS, sm_count() * per_sm);
        kern<<<ctas, rows::THREADS, SMEM, s>>>(m.nrows, m.brptr, m.headers, static_cast<const V*>(m.values), m.valptr,
                                               m.wstart, m.nwarps, static_cast<const X*>(x), ldx, xcs,
                                               static_cast<Y*>(y), ldy, ycs);
    });
    SPC5_CUDA(cudaGetLastError());
}

template <class LT, class V, class X, class A, class Y>
void cols_batch(int r, int kc, const BatchMat* mats, const BatchJob* jobs, int njobs, cudaStream_t s) {
    // (the chunks of a class of jobs: as for full ones)
    dispatch_rkc<LT, V>(r, kc, 32, [&](auto RC, auto KCC, auto SC) {
        constexpr int R_ = decltype(RC)::value, KC_ = decltype(KCC)::value;
        constexpr bool SMALL = decltype(SC)::value;
        constexpr int SMEM = rows::Geo<LT, R_, V, mm_lanes<LT, R_>(), cols_hb<SMALL>, cols_vb<SMALL>>::SMEM;
        auto kern = k_spmm_cols_batch<LT, R_, KC_, SMALL, V, X, A, Y>;
        set_smem(kern, SMEM);
        int per_sm = 0;
        SPC5_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, rows::THREADS, SMEM));
        const int grid = std::max(1, std::min(div_up(njobs, rows::WARPS), sm_count() * std::max(1, per_sm)));
        kern<<<grid, rows::THREADS, SMEM, s>>>(mats, jobs, njobs);
    });
    SPC5_CUDA(cudaGetLastError());
}

}  // namespace

#define SPC5_COLS_KIND(NAME, LT, V, X, A, Y)                                                                       \
    void launch_spmm_cols_##NAME(const BetaView& m, int kc, const void* x, long ldx, long xcs, void* y, long ldy,  \
                                 long ycs, cudaStream_t s) {                                                       \
        cols_pass<LT, V, X, A, Y>(m, kc, x, ldx, xcs, y, ldy, ycs, s);                                             \
    }                                                                                                              \
    void launch_batch_cols_##NAME(int r, int kc, const BatchMat* mats, const BatchJob* jobs, int njobs,            \
                                  cudaStream_t s) {                                                                \
        cols_batch<LT, V, X, A, Y>(r, kc, mats, jobs, njobs, s);                                                   \
    }

}  // namespace spc5cuda
