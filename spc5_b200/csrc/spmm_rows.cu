// spmm_rows.cu -- staged multi-RHS SpMM, Y += A X, for matrices whose every
// block-row fits the row kernels' staging buffers (rows_stage.cuh).
//
// A warp walks its block-rows in chunks of 32 sub-rows staged into shared
// memory.  One lane per sub-row first lists the sub-row's values in chain order
// -- column class 0 of its blocks in block order, then class 1, ... -- each
// with its x index and its place in the staged values (two walks over the
// staged headers: count, place).  Then KC / 2 lanes serve one sub-row, two
// neighbouring right-hand sides each, 64 / KC sub-rows at a time: per value a
// lane reads the list entry and the value (the same for the sub-row's lanes),
// loads its two x (16 or 8 bytes at once where X allows) and does two
// multiply-adds; where a chain ends it leaves the results in shared memory.
//
// What bounds it: instructions.  With a lane per column (before) each lane
// tested every sub-row's mask per block and issued KC multiply-adds for each,
// of which a matrix with 1 to 4 values per block uses a tenth: 16 instructions
// per value and 8 right-hand sides, now 9 to 10.  Measured on B200, before / now
// (us, FP64): banded n = 200,000, 21 values per row, r = 4, k = 8 140 / 76; r = 1, k
// = 16 330 / 137; r = 2, k = 4 100 / 57.  Where a lane per column is still the
// faster one (few right-hand sides on blocks of many rows) it stays:
// spmm_cols.cu.
//
// Arithmetic per right-hand side j is the SpMV's (src/spc5.hpp:2309-2715):
// the chain of (sub-row, column class c) receives fma(value, x[col + c][j],
// acc) for every block in order whose mask has bit c; the row sum is the
// _mm512_reduce_add tree over the VS chains (+0 for a class without values);
// then Y[row][j] += sum.  Column j of the result is therefore bit-identical to
// an SpMV with column j of X.
#include <algorithm>

#include "common.cuh"
#include "kernels.h"
#include "rows_blocks.cuh"

namespace spc5cuda {

namespace {

using rows::FULL;

constexpr uint32_t LAST = 1u << 31;  // list entry: the last one of its chain (x indices are below 2^31)
constexpr int MM_CTAS = 6;  // of 2 warps: the shared memory of 12 to 13 warps per SM
constexpr int MM_WARPS = 2;  // per CTA: finer steps of shared memory than 4
constexpr int MM_THREADS = MM_WARPS * 32;

// One warp's shared memory: the staged headers (later the chain results, one
// column per lane), the staged values, the list.
template <class LT, int R, class V, class A>
struct MMGeo {
    static constexpr int VS = Layout<LT>::VS;
    static constexpr int CHAIN = VS * 32 * 2 * int(sizeof(A));
    static constexpr int HB = CHAIN > rows::HB ? CHAIN : rows::HB;
    static constexpr int VB = rows::VB;
    static constexpr int VALUES = VB / int(sizeof(V));
    static constexpr int WARP = HB + VB + VALUES * 8;
    static constexpr int SMEM = MM_WARPS * WARP;
};

// Two neighbouring elements as one vector.
template <class T>
struct __align__(2 * sizeof(T)) Two {
    T a, b;
};

// x of two right-hand sides: one vector load (vec: unit stride, aligned) or two.
__device__ __forceinline__ Two<double> ld_two(const double* p) {
    const double2 t = __ldg(reinterpret_cast<const double2*>(p));
    return {t.x, t.y};
}
__device__ __forceinline__ Two<float> ld_two(const float* p) {
    const float2 t = __ldg(reinterpret_cast<const float2*>(p));
    return {t.x, t.y};
}

// A list entry in shared memory (on != 0; predicated without a branch), and LAST
// set in one.
__device__ __forceinline__ void st_entry_if(uint32_t saddr, uint32_t x, uint32_t v, uint32_t on) {
    asm volatile("{ .reg .pred q; setp.ne.u32 q, %3, 0; @q st.shared.v2.u32 [%0], {%1, %2}; }" ::"r"(saddr), "r"(x),
                 "r"(v), "r"(on)
                 : "memory");
}
__device__ __forceinline__ void mark_last(uint32_t saddr) {
    uint32_t x;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(x) : "r"(saddr) : "memory");
    asm volatile("st.shared.u32 [%0], %1;" ::"r"(saddr), "r"(x | LAST) : "memory");
}

// Y += A X over block-rows [r_begin, r_stop) of one matrix for the kc <= KC
// right-hand sides of xm / ym (already offset to the pass's first one).
template <class LT, int R, int KC, class V, class X, class A, class Y>
__device__ __forceinline__ void mm_range(int nrows, const int* __restrict__ brptr,
                                         const uint8_t* __restrict__ headers, const V* __restrict__ values,
                                         const int* __restrict__ valptr, int r_begin, int r_stop, int kc,
                                         const X* __restrict__ xm, long ldx, long xcs, Y* __restrict__ ym, long ldy,
                                         long ycs, unsigned char* wbuf) {
    using G = MMGeo<LT, R, V, A>;
    constexpr int VS = G::VS, STRIDE = Header<LT, R>::STRIDE;
    constexpr int LPS = KC / 2;    // lanes per sub-row
    constexpr int PAR = 32 / LPS;  // sub-rows at a time
    constexpr int U = 8;           // list entries at a time (4 / 6 / 8: r = 4, k = 8 90 / 82 / 80 us)
    const int lane = threadIdx.x & 31;
    const int q = lane % R;
    const int h = lane / LPS, j = 2 * (lane % LPS);
    const bool both = j + 1 < kc;
    const bool vec = xcs == 1 && ldx % 2 == 0 && (reinterpret_cast<uintptr_t>(xm) % (2 * sizeof(X))) == 0;
    Two<A>* chain = reinterpret_cast<Two<A>*>(wbuf) + lane;
    // list entry: x index (and LAST), byte offset of the value in the staged values
    unsigned char* list = wbuf + G::HB + G::VB;
    const rows::SubRowOf<LT, R> me(q);
    const X* xj = xm + long(j) * xcs;
    Y* yj = ym + long(j) * ycs;

    auto compute = [&](const rows::Chunk& ch, const uint32_t* hw, const V* vbuf) {
        // ---- the sub-row's values per column class
        const rows::SubRow at = rows::sub_row_at<LT, R>(ch, lane);
        const unsigned char* vb = reinterpret_cast<const unsigned char*>(vbuf);
        int cnt[VS];
        uint32_t chains = 0u;
        if (__any_sync(FULL, at.n > 255)) {
#pragma unroll
            for (int c = 0; c < VS; ++c) cnt[c] = 0;
            for (int k = 0; k < at.n; ++k) {
                rows::Block<LT, R> b;
                me.load(hw, at.hoff + k * STRIDE, true, b);
                chains |= b.m;
#pragma unroll
                for (int c = 0; c < VS; ++c) cnt[c] += int((b.m >> c) & 1u);
            }
        } else {  // four counts to a word
            uint32_t sum[VS / 4];
#pragma unroll
            for (int w = 0; w < VS / 4; ++w) sum[w] = 0u;
            for (int k = 0; k < at.n; ++k) {
                rows::Block<LT, R> b;
                me.load(hw, at.hoff + k * STRIDE, true, b);
                chains |= b.m;
#pragma unroll
                for (int w = 0; w < VS / 4; ++w) sum[w] += (((b.m >> (4 * w)) & 0xFu) * 0x00204081u) & 0x01010101u;
            }
#pragma unroll
            for (int c = 0; c < VS; ++c) cnt[c] = int((sum[c / 4] >> (8 * (c % 4))) & 0xFFu);
        }
        int len = 0;
#pragma unroll
        for (int c = 0; c < VS; ++c) {
            const int n = cnt[c];
            cnt[c] = 8 * len;  // from here on: byte offset of the class's next place
            len += n;
        }
        int first = len;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int t = __shfl_up_sync(FULL, first, d);
            if (lane >= d) first += t;
        }
        first = 8 * (first - len);
        // ---- the list
        {
            const uint32_t l = uint32_t(__cvta_generic_to_shared(list)) + unsigned(first);
#pragma unroll
            for (int c = 0; c < VS; ++c) cnt[c] += int(l);
            int v = at.v * int(sizeof(V));
            for (int k = 0; k < at.n; ++k) {
                rows::Block<LT, R> b;
                me.load(hw, at.hoff + k * STRIDE, true, b);
                int w = v + me.before(b) * int(sizeof(V));
#pragma unroll
                for (int c = 0; c < VS; ++c) {
                    const uint32_t on = b.m & (1u << c);
                    st_entry_if(uint32_t(cnt[c]), uint32_t(b.col + c), uint32_t(w), on);
                    cnt[c] += on ? 8 : 0;
                    w += on ? int(sizeof(V)) : 0;
                }
                v += me.values(b) * int(sizeof(V));
            }
#pragma unroll
            for (int c = 0; c < VS; ++c)
                if (chains & (1u << c)) mark_last(uint32_t(cnt[c]) - 8u);
        }
        __syncwarp();  // the list is complete, the headers are done with

        // ---- KC lanes per sub-row
        const long row0 = long(ch.r0) * R;
        const int live = int(std::min(long(ch.nrow) * R, nrows - row0));
        for (int i0 = 0; i0 < live; i0 += PAR) {
            const int i = i0 + h;
            const uint2* at0 = reinterpret_cast<const uint2*>(list + __shfl_sync(FULL, first, i));
            const int n = __shfl_sync(FULL, len, i);
            const uint32_t mask = __shfl_sync(FULL, chains, i);
            const bool mine = i < live && j < kc;
            const int stop = mine ? n : 0;
            A acc0 = A(0), acc1 = A(0);
            Two<A>* slot = chain;
            for (int k = 0; k < stop; k += U) {
                uint32_t e[U];
                V v[U];
                Two<X> x[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    e[u] = 0u;
                    if (k + u < stop) {
                        const uint2 t = at0[k + u];
                        e[u] = t.x;
                        v[u] = *reinterpret_cast<const V*>(vb + t.y);
                    }
                }
                if (vec && both) {
#pragma unroll
                    for (int u = 0; u < U; ++u)
                        if (k + u < stop) x[u] = ld_two(xj + long(e[u] & ~LAST) * ldx);
                } else {
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        if (k + u < stop) {
                            const X* xp = xj + long(e[u] & ~LAST) * ldx;
                            x[u].a = __ldg(xp);
                            x[u].b = both ? __ldg(xp + xcs) : X(0);
                        }
                    }
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    if (k + u < stop) {
                        acc0 = fma(A(v[u]), A(x[u].a), acc0);
                        acc1 = fma(A(v[u]), A(x[u].b), acc1);
                        if (e[u] & LAST) {
                            *slot = Two<A>{acc0, acc1};
                            slot += 32;
                            acc0 = acc1 = A(0);
                        }
                    }
                }
            }
            if (mine) {
                const Two<A>* from = chain;
                A a0[VS], a1[VS];
#pragma unroll
                for (int c = 0; c < VS; ++c) {
                    Two<A> t{A(0), A(0)};
                    if (mask & (1u << c)) {
                        t = *from;
                        from += 32;
                    }
                    a0[c] = t.a;
                    a1[c] = t.b;
                }
                Y* yp = yj + (row0 + i) * ldy;
                rows::add_to(yp, Y(rows::reduce_tree<A, VS>(a0)));
                if (both) rows::add_to(yp + ycs, Y(rows::reduce_tree<A, VS>(a1)));
            }
        }
    };
    rows::walk<LT, R, V, R, G::HB, G::VB>(brptr, headers, values, valptr, r_begin, r_stop, wbuf, compute);
}

// One matrix: the grid's warps, one resident wave, share its block-rows
// (part_start).  With the SpMV's partition, for 24 to 28 warps per SM, the last
// of its two or three waves was part empty: stencil 64^3, k = 16, FP64 on a B200
// 187 us at r = 2, now 149; r = 1 195 / 154; r = 4 181 / 146.
template <class LT, int R, int KC, class V, class X, class A, class Y>
__global__ void __launch_bounds__(MM_THREADS, MM_CTAS)
    k_spmm_rows(int nrows, const int* __restrict__ brptr, const uint8_t* __restrict__ headers,
                const V* __restrict__ values, const int* __restrict__ valptr, const int* __restrict__ wstart,
                int nwarps, int kc, const X* __restrict__ xm, long ldx, long xcs, Y* __restrict__ ym, long ldy,
                long ycs) {
    using G = MMGeo<LT, R, V, A>;
    extern __shared__ __align__(16) unsigned char smem[];
    const int wi = threadIdx.x >> 5;
    const int warp = blockIdx.x * MM_WARPS + wi;
    const int W = gridDim.x * MM_WARPS;
    mm_range<LT, R, KC, V, X, A, Y>(nrows, brptr, headers, values, valptr, rows::part_start(wstart, nwarps, warp, W),
                                    rows::part_start(wstart, nwarps, warp + 1, W), kc, xm, ldx, xcs, ym, ldy, ycs, smem + wi * G::WARP);
}

// Batched: warps walk the job list with the grid's warp count as stride; job
// j is block-rows [r_begin, r_end) of mats[j.mat] for the right-hand sides
// [kofs, kofs + kc).  X and Y of a batch are row-major (xcs = ycs = 1).
template <class LT, int R, int KC, class V, class X, class A, class Y>
__global__ void __launch_bounds__(MM_THREADS, MM_CTAS)
    k_spmm_rows_batch(const BatchMat* __restrict__ mats, const BatchJob* __restrict__ jobs, int njobs) {
    using G = MMGeo<LT, R, V, A>;
    extern __shared__ __align__(16) unsigned char smem[];
    const int wi = threadIdx.x >> 5;
    const int nw = gridDim.x * MM_WARPS;
    for (int j = blockIdx.x * MM_WARPS + wi; j < njobs; j += nw) {  // warp-uniform
        const BatchJob job = jobs[j];
        const BatchMat& m = mats[job.mat];
        mm_range<LT, R, KC, V, X, A, Y>(m.nrows, m.brptr, m.headers, static_cast<const V*>(m.values), m.valptr,
                                        job.r_begin, job.r_end, m.k - job.kofs, static_cast<const X*>(m.x) + job.kofs,
                                        m.ldx, 1L, static_cast<Y*>(m.y) + job.kofs, m.ldy, 1L, smem + wi * G::WARP);
    }
}

// The jobs of one right-hand side with contiguous x and y: the row SpMV's
// chunks.
template <class LT, int R, class V, class X, class A, class Y, int FORM>
__global__ void __launch_bounds__(rows::THREADS, 5)
    k_spmv_rows_batch(const BatchMat* __restrict__ mats, const BatchJob* __restrict__ jobs, int njobs) {
    using G = rows::Geo<LT, R, V, R>;
    extern __shared__ __align__(16) unsigned char smem[];
    const int wi = threadIdx.x >> 5;
    const int nw = gridDim.x * rows::WARPS;
    const uint64_t pol_x = l2_evict_last_policy();
    for (int j = blockIdx.x * rows::WARPS + wi; j < njobs; j += nw) {  // warp-uniform
        const BatchJob job = jobs[j];
        const BatchMat& m = mats[job.mat];
        const int nrows = m.nrows;
        const X* x = static_cast<const X*>(m.x);
        Y* y = static_cast<Y*>(m.y);
        rows::walk<LT, R, V, R>(m.brptr, m.headers, static_cast<const V*>(m.values), m.valptr, job.r_begin, job.r_end,
                                smem + wi * G::BUF_BYTES,
                                [&](const rows::Chunk& ch, const uint32_t* hw, const V* vbuf) {
                                    rows::chunk_spmv<LT, R, V, X, A, Y, FORM>(ch, hw, vbuf, x, y, nrows, pol_x);
                                });
    }
}

// Calls f(integral_constant<R>) for r in {1, 2, 4, 8}.
template <class F>
void dispatch_r(int r, F&& f) {
    using std::integral_constant;
    switch (r) {
        case 1: f(integral_constant<int, 1>{}); return;
        case 2: f(integral_constant<int, 2>{}); return;
        case 4: f(integral_constant<int, 4>{}); return;
        case 8: f(integral_constant<int, 8>{}); return;
    }
    throw Error(SPC5CUDA_ERR_FORMAT, "r must be 1, 2, 4 or 8");
}

// Calls f(integral_constant<R>, integral_constant<KC>) for kc in {2, 4, 8, 16}.
template <class F>
void dispatch_rkc(int r, int kc, F&& f) {
    using std::integral_constant;
    dispatch_r(r, [&](auto RC) {
        switch (kc) {
            case 2: f(RC, integral_constant<int, 2>{}); return;
            case 4: f(RC, integral_constant<int, 4>{}); return;
            case 8: f(RC, integral_constant<int, 8>{}); return;
            case 16: f(RC, integral_constant<int, 16>{}); return;
        }
        throw Error(SPC5CUDA_ERR_INVALID, "right-hand sides per pass");
    });
}

template <int KIND, class LT, class V, class X, class A, class Y>
void spmm_rows_impl(const BetaView& m, int k, const X* x, long ldx, long xcs, Y* y, long ldy, long ycs,
                    cudaStream_t s) {
    if (m.nbr <= 0 || k <= 0 || m.nwarps <= 0) return;
    const V* vals = static_cast<const V*>(m.values);
    for (int k0 = 0; k0 < k;) {
        const X* xp = x + long(k0) * xcs;
        Y* yp = y + long(k0) * ycs;
        const bool columns = spmm_columns(Layout<LT>::VS, int(sizeof(V)), m.r, m.fill, m.list_rows, k - k0);
        const bool one = k - k0 == 1 && ldx == 1 && ldy == 1;
        // one contiguous right-hand side: the SpMV
        if (one && !spmv_columns(Layout<LT>::VS, m.r, m.fill, m.chunk_rows)) {
            launch_rows_kind(KIND, m, xp, yp, s);
            return;
        }
        if (columns || one) {
            const int kc = spmm_cols_kc(Layout<LT>::VS, m.r, k - k0);
            launch_spmm_cols(KIND, m, kc, xp, ldx, xcs, yp, ldy, ycs, s);
            k0 += kc;
            continue;
        }
        const int kc = spmm_rows_kc(k - k0);
        dispatch_rkc(m.r, kc, [&](auto RC, auto KCC) {
            constexpr int R_ = decltype(RC)::value, KC_ = decltype(KCC)::value;
            constexpr int SMEM = MMGeo<LT, R_, V, A>::SMEM;
            auto kern = k_spmm_rows<LT, R_, KC_, V, X, A, Y>;
            set_smem(kern, SMEM);
            static const int per_sm = resident_ctas(kern, MM_THREADS, SMEM);
            const int ctas = std::min((m.nwarps + MM_WARPS - 1) / MM_WARPS, sm_count() * per_sm);
            kern<<<ctas, MM_THREADS, SMEM, s>>>(m.nrows, m.brptr, m.headers, vals, m.valptr, m.wstart, m.nwarps,
                                                   std::min(k - k0, KC_), xp, ldx, xcs, yp, ldy, ycs);
        });
        k0 += kc;
    }
    SPC5_CUDA(cudaGetLastError());
}

template <class K>
void launch_jobs(K kern, int threads, int smem, const BatchMat* mats, const BatchJob* jobs, int njobs, cudaStream_t s) {
    set_smem(kern, smem);
    int per_sm = 0;
    SPC5_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem));
    const int grid = std::max(1, std::min(div_up(njobs, threads / 32), sm_count() * std::max(1, per_sm)));
    kern<<<grid, threads, smem, s>>>(mats, jobs, njobs);
}

template <class LT, class V, class X, class A, class Y>
void batch_rows_impl(int r, int kc, bool narrow, const BatchMat* mats, const BatchJob* jobs, int njobs,
                     cudaStream_t s) {
    if (kc == 1) {
        dispatch_r(r, [&](auto RC) {
            constexpr int R_ = decltype(RC)::value, SMEM = rows::Geo<LT, R_, V, R_>::SMEM;
            if (narrow) launch_jobs(k_spmv_rows_batch<LT, R_, V, X, A, Y, rows::NARROW>, rows::THREADS, SMEM, mats, jobs, njobs, s);
            else launch_jobs(k_spmv_rows_batch<LT, R_, V, X, A, Y, rows::WIDE>, rows::THREADS, SMEM, mats, jobs, njobs, s);
        });
        return;
    }
    dispatch_rkc(r, kc, [&](auto RC, auto KCC) {
        constexpr int R_ = decltype(RC)::value, KC_ = decltype(KCC)::value;
        launch_jobs(k_spmm_rows_batch<LT, R_, KC_, V, X, A, Y>, MM_THREADS, MMGeo<LT, R_, V, A>::SMEM, mats, jobs, njobs, s);
    });
}

}  // namespace

// Measured on B200 (us, columns / lists; 27-point stencil 64^3, fill 3 per
// sub-row and block at r = 4, 1.5 at r = 8; banded n = 100,000, fill 1 and 0.9):
//   r = 8, FP64: k = 2 47 / 59 and 30 / 39, k = 3 90 / 92 and 55 / 53, k = 4 72 /
//     78 and 49 / 45, k = 8 (two passes of columns) 149 / 96 and 96 / 61;
//   r = 4, FP64: k = 2 42 / 55 and 31 / 29, k = 4 49 / 72 and 43 / 34, k = 8 98 /
//     107 and 84 / 45, k = 12 (two passes of columns) 145 / 172;
//   float layout, r = 4: k = 2 55 / 55 and 32 / 35, k = 3 111 / 86 and 61 / 49, k =
//     4 67 / 74 and 41 / 43, k = 5 126 / 135, k = 8 137 / 112 and 81 / 55; r = 8: k = 4 65 / 82 and
//     43 / 49, k = 8 133 / 119 and 84 / 61;
//   r = 1 and 2: lists (r = 2, k = 4 81 / 74 and 58 / 34), but for long rows (below).
//   8 columns of float values (mixed): as FP64, but the columns' x are half as
//     wide: r = 4, fill 3, k = 16 166 / 183; r = 8, k = 5 135 / 153.
//   Long rows of full blocks: a chunk holds fewer sub-rows than the lists have
//     lanes for, and each lists its values alone.  FP64, 32^3 grid of 3 unknowns (81
//     values per row, fill 4.5): r = 2, k = 2 39 / 90, k = 8 76 / 101; 20^3 of 6 (162,
//     fill 4.5 to 6): r = 1, k = 2 35 / 140, k = 8 82 / 144; blocks of 8 at random
//     columns, 480 per row: r = 1, k = 4 84 / 626.  Banded n = 60,000, 41 values per
//     row, fill 1, r = 4, FP64, k = 2 31 / 44.  From 9 right-hand sides on the rows of
//     X at random columns count for more: the blocks, 240 values per row, r = 1, k = 16,
//     FP64 549 / 232, mixed 305 / 270; 800 values per row, one sub-row per chunk, mixed
//     523 / 1361.
bool spmm_columns(int vs, int value_bytes, int r, float fill, int list_rows, int k) {
    const bool wide = value_bytes == 8;
    if (r <= 2) {
        const bool lists16 = list_rows > (wide ? 1 : 2) && (wide || list_rows < 8);  // from 9 right-hand sides on
        if (list_rows > (wide ? 16 : 24) || k > (lists16 ? 8 : 16)) return false;
        return fill >= (r == 2 ? 2.f : (vs == 16 ? 2.5f : 4.f));
    }
    if (vs == 16) return (k <= 5 && k != 3) || (k <= 8 && fill >= 2.5f && list_rows <= 24);
    if (r == 8) return k <= (wide ? 4 : 5);
    return (fill >= 2.f && k <= (wide ? 12 : 16)) || (k == 2 && fill >= 0.9f && list_rows < 24);
}

// Measured on B200 (us, SpMV / one column of columns): 40,000 rows of 100 random values,
// FP64, r = 1 150 / 115, 25,000 of 200 467 / 238; 60,000 of 40, r = 2 108 / 62; 20^3 grid
// of 6 unknowns, r = 2 47 / 33; of 3 unknowns 35 / 66 and 37 / 41; 30 blocks of 8 at
// random columns, r = 4, mixed 259 / 74, float layout 223 / 276.
bool spmv_columns(int vs, int r, float fill, int chunk_rows) {
    if (r > 1 && fill < 0.7f && chunk_rows < 24) return true;
    return r == 1 ? chunk_rows < 5 : (r == 2 ? chunk_rows < 8 : r == 4 && vs == 8 && chunk_rows <= 8);
}

int spmm_rows_kc(int k) { return k > 8 ? 16 : (k > 4 ? 8 : (k > 2 ? 4 : 2)); }

void launch_spmm_rows_f64(const BetaView& m, int k, const double* x, long ldx, long xcs, double* y, long ldy,
                          long ycs, cudaStream_t s) {
    spmm_rows_impl<0, double, double, double, double, double>(m, k, x, ldx, xcs, y, ldy, ycs, s);
}

void launch_spmm_rows_f32(const BetaView& m, int k, const float* x, long ldx, long xcs, float* y, long ldy,
                          long ycs, cudaStream_t s) {
    spmm_rows_impl<1, float, float, float, float, float>(m, k, x, ldx, xcs, y, ldy, ycs, s);
}

void launch_spmm_rows_mixed(const BetaView& m, int k, const float* x, long ldx, long xcs, double* y, long ldy,
                            long ycs, cudaStream_t s) {
    spmm_rows_impl<2, float, float, float, double, double>(m, k, x, ldx, xcs, y, ldy, ycs, s);
}

void launch_spmm_rows_mixed8(const BetaView& m, int k, const float* x, long ldx, long xcs, double* y, long ldy,
                             long ycs, cudaStream_t s) {
    spmm_rows_impl<3, double, float, float, double, double>(m, k, x, ldx, xcs, y, ldy, ycs, s);
}

void launch_batch_rows(int kind, int r, int kc, bool narrow, const BatchMat* mats, const BatchJob* jobs, int njobs,
                       cudaStream_t s) {
    if (njobs <= 0) return;
    if (kind == 0) batch_rows_impl<double, double, double, double, double>(r, kc, narrow, mats, jobs, njobs, s);
    else if (kind == 1) batch_rows_impl<float, float, float, float, float>(r, kc, narrow, mats, jobs, njobs, s);
    else if (kind == 2) batch_rows_impl<float, float, float, double, double>(r, kc, narrow, mats, jobs, njobs, s);
    else batch_rows_impl<double, float, float, double, double>(r, kc, narrow, mats, jobs, njobs, s);
    SPC5_CUDA(cudaGetLastError());
}

}  // namespace spc5cuda
