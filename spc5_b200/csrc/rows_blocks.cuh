// rows_blocks.cuh -- the blocks of a staged chunk (rows_stage.cuh) as the lane of
// one sub-row sees them, and its multiply-adds over all of them for one x: the
// body of the row SpMV kernel (spmv_rows.cu, where the two forms are described)
// and of the batched products with one right-hand side (spmm_rows.cu).
#pragma once

#include "rows_stage.cuh"

namespace spc5cuda {
namespace rows {

// The lane of sub-row q of its block-row: where it stands in the staged chunk.
struct SubRow {
    int n;      // blocks left
    int hoff;   // byte offset of the next block's header in the staged headers
    int v;      // index of its first value in the staged values
};

// One staged block as sub-row q sees it: first column, own mask, its values'
// place (from the block's first value) and the block's value count.
template <class LT, int R>
struct Block {
    static constexpr int MW = Header<LT, R>::MASK_WORDS;
    int col;
    uint32_t mw[MW], m;
};

template <class LT, int R>
struct SubRowOf {
    static constexpr int MB = Layout<LT>::MASK_BYTES, MW = Header<LT, R>::MASK_WORDS;
    static constexpr int FPW = 4 / MB, BITS = 8 * MB;
    int wq;            // mask word of sub-row q
    unsigned sh;       // its field in that word
    uint32_t low[MW];  // mask bits of the sub-rows below q
    __device__ __forceinline__ explicit SubRowOf(int q) : wq(q / FPW), sh(unsigned(q % FPW) * BITS) {
#pragma unroll
        for (int w = 0; w < MW; ++w) low[w] = w < wq ? 0xFFFFFFFFu : (w == wq ? (1u << sh) - 1u : 0u);
    }
    static_assert(MW == 1 || MW == 2 || MW == 4, "mask words of a block");
    // the block at header offset off, empty when !ok
    __device__ __forceinline__ void load(const uint32_t* hw, int off, bool ok, Block<LT, R>& b) const {
        constexpr uint32_t FMASK = MB == 1 ? 0xFFu : 0xFFFFu;
        b.col = 0;
#pragma unroll
        for (int w = 0; w < MW; ++w) b.mw[w] = 0u;
        if (ok) b.col = rows::decode_staged<LT, R>(hw, off, b.mw);
        // (a select per word: a loop of them became an array in local memory at four words)
        uint32_t word = b.mw[0];
        if constexpr (MW == 2) word = wq & 1 ? b.mw[1] : b.mw[0];
        if constexpr (MW == 4) {
            const uint32_t lo = wq & 1 ? b.mw[1] : b.mw[0], hi = wq & 1 ? b.mw[3] : b.mw[2];
            word = wq & 2 ? hi : lo;
        }
        b.m = R == 1 ? word : (word >> sh) & FMASK;
    }
    __device__ __forceinline__ int before(const Block<LT, R>& b) const {
        int n = 0;
        if constexpr (R > 1) {
#pragma unroll
            for (int w = 0; w < MW; ++w) n += __popc(b.mw[w] & low[w]);
        }
        return n;
    }
    static __device__ __forceinline__ int values(const Block<LT, R>& b) {
        int n = 0;
#pragma unroll
        for (int w = 0; w < MW; ++w) n += __popc(b.mw[w]);
        return n;
    }
};

// All VS columns of every block, UT blocks per step (their x loads are issued
// together).
template <class LT, int R, class V, class X, class A, int UT>
__device__ __forceinline__ void wide_blocks(const uint32_t* hw, const V* vbuf, const X* __restrict__ x, int q,
                                            SubRow at, uint64_t pol_x, A (&acc)[Layout<LT>::VS]) {
    constexpr int VS = Layout<LT>::VS, STRIDE = Header<LT, R>::STRIDE;
    const SubRowOf<LT, R> me(q);
    const int steps = (__reduce_max_sync(FULL, at.n) + UT - 1) / UT;
#pragma unroll 1
    for (int step = 0; step < steps; ++step) {
        Block<LT, R> b[UT];
        X xk[UT][VS];
#pragma unroll
        for (int u = 0; u < UT; ++u) me.load(hw, at.hoff + u * STRIDE, u < at.n, b[u]);
#pragma unroll
        for (int u = 0; u < UT; ++u) {
            const X* xp = x + b[u].col;
#pragma unroll
            for (int c = 0; c < VS; ++c) xk[u][c] = b[u].m & (1u << c) ? ld_x(xp + c, pol_x) : X(0);
        }
#pragma unroll
        for (int u = 0; u < UT; ++u) {
            const V* vp = vbuf + at.v + me.before(b[u]);
#pragma unroll
            for (int c = 0; c < VS; ++c) {
                if (b[u].m & (1u << c)) {
                    acc[c] = fma(A(*vp), A(xk[u][c]), acc[c]);
                    ++vp;
                }
            }
            at.v += me.values(b[u]);
        }
        at.n -= UT;
        at.hoff += UT * STRIDE;
    }
}

// A window of NS columns, from the first column of the sub-row's first
// non-empty mask on: accumulator a is column (rho + a) mod VS.
constexpr int NS = 3;

// Whether every block-row alone fits a warp's staging buffers, alignment included.
__host__ __device__ inline bool fit(int vt, int r, int max_blocks, int max_values) {
    const int stride = 4 + r * (vt == SPC5CUDA_F32 ? 2 : 1);
    const int vbytes = vt == SPC5CUDA_F64 ? 8 : 4;
    return long(max_blocks) * stride + 32 <= HB && (long(max_values) + 2 * (16 / vbytes)) * vbytes <= VB;
}

// Whether the narrow kernel runs: at least 7 of 8 of the blocks looked at keep
// every sub-row mask within NS columns, and at r > 1 a sub-row has at least 1.22
// values per block, since a lane steps over the blocks that hold nothing of its
// sub-row one by one (measured on B200, us, wide / narrow, a diagonal of 1,000,000
// rows: FP64 r = 4 18.1 / 21.4, float layout r = 8 21.0 / 25.2; two values per row,
// one of them far from the diagonal, FP64 r = 4 29.0 / 35.5; 5-point Poisson 900^2,
// 1.67 values, float layout r = 4 28.4 / 25.1).  Float values in 8 columns: only where
// block-rows are short (60,000 rows of 40 random values, 80 blocks per block-row, r = 2
// 168 / 147).  At r = VS its steps of 3 blocks pay
// for themselves only on block-rows of several steps (FP64: 27-point stencil 127^3,
// 18 blocks per block-row, 234 / 181; Poisson 900^2, 4 blocks, 25.7 / 28.2; float
// values 32.0 / 30.4).
__host__ __device__ inline bool narrow(int vt, int r, int nbr, long nblocks, long nnz, int narrow_blocks, int looked_at) {
    const int vs = vt == SPC5CUDA_F32 ? 16 : 8;
    const bool few_empty = r == 1 || 50 * nnz >= 61 * r * nblocks || (vt == SPC5CUDA_F32_V8 && nblocks >= 3L * nbr);
    return looked_at > 0 && long(narrow_blocks) * 8 >= long(looked_at) * 7 && few_empty &&
           (r < vs || vt == SPC5CUDA_F32_V8 || nblocks >= 6L * nbr);
}

template <class LT, int R, class V, class X, class A>
__device__ __forceinline__ void narrow_blocks(const uint32_t* hw, const V* vbuf, const X* __restrict__ x, int q,
                                              SubRow at, uint64_t pol_x, A (&acc)[Layout<LT>::VS]) {
    constexpr int VS = Layout<LT>::VS, STRIDE = Header<LT, R>::STRIDE;
    constexpr uint32_t VSMASK = (1u << VS) - 1u;
    constexpr bool WRAP = R == VS;  // the window may run over the last column into the next block
    // blocks per step: a 27-point stencil's row has 9 at r <= 4 (2 / 3 / 4 blocks
    // measured on B200: 160^3 r = 4 253 / 240 / 249 us, 101^3 r = 1 f32 52 / 48 / 50)
    constexpr int UT = 3;
    const SubRowOf<LT, R> me(q);
    int rho = 0;
    // the window's columns (bit[a]), the columns outside it (all of them until
    // the lane has met its first mask; at r = 1 a block starts at its first
    // column), and x there
    uint32_t bit[NS], outside;
    const X* xw[NS];
    auto window = [&]() {
        outside = VSMASK;
#pragma unroll
        for (int a = 0; a < NS; ++a) {
            const int c = WRAP ? (rho + a) & (VS - 1) : rho + a;
            bit[a] = 1u << c;
            outside &= ~bit[a];
            xw[a] = x + c;
        }
    };
    window();
    if constexpr (R > 1) outside = VSMASK;
    const int steps = (__reduce_max_sync(FULL, at.n) + UT - 1) / UT;
#pragma unroll 1
    for (int step = 0; step < steps; ++step) {
        Block<LT, R> b[UT];
        uint32_t some = 0u;
#pragma unroll
        for (int u = 0; u < UT; ++u) {
            me.load(hw, at.hoff + u * STRIDE, u < at.n, b[u]);
            some |= b[u].m;
        }
        if (__any_sync(FULL, (some & outside) != 0u)) {
            bool wide = true;
            if constexpr (R > 1) {
                if (some && outside == VSMASK) {  // the lane's first masks
                    uint32_t first = b[UT - 1].m;
#pragma unroll
                    for (int u = UT - 2; u >= 0; --u) first = b[u].m ? b[u].m : first;
                    rho = __ffs(first) - 1;
                    window();
                }
                wide = __any_sync(FULL, (some & outside) != 0u);
            }
            if (wide) {
                // a wide mask: the accumulators back at their columns, and the
                // rest of the chunk over all columns
                if constexpr (R > 1) {
#pragma unroll
                    for (int d = 1; d < VS; d <<= 1) {
                        A t[VS];
#pragma unroll
                        for (int c = 0; c < VS; ++c) t[c] = acc[c];
#pragma unroll
                        for (int c = 0; c < VS; ++c) acc[c] = (rho & d) ? t[(c - d) & (VS - 1)] : t[c];
                    }
                }
                wide_blocks<LT, R, V, X, A, 1>(hw, vbuf, x, q, at, pol_x, acc);
                return;
            }
        }
        X xk[UT][NS];
#pragma unroll
        for (int u = 0; u < UT; ++u) {
#pragma unroll
            for (int a = 0; a < NS; ++a) {
                xk[u][a] = b[u].m & bit[a] ? ld_x(xw[a] + b[u].col, pol_x) : X(0);
            }
        }
#pragma unroll
        for (int u = 0; u < UT; ++u) {
            // values are in column order: those of the window's columns
            // past the last one (its wrapped part) come first
            const V* v0 = vbuf + at.v + me.before(b[u]);
            const V* vp = v0;
            if constexpr (WRAP) vp += __popc(b[u].m & ((1u << rho) - 1u));
#pragma unroll
            for (int a = 0; a < NS; ++a) {
                if (WRAP && a > 0 && rho == VS - a) vp = v0;
                if (b[u].m & bit[a]) {
                    acc[a] = fma(A(*vp), A(xk[u][a]), acc[a]);
                    ++vp;
                }
            }
            at.v += me.values(b[u]);
        }
        at.n -= UT;
        at.hoff += UT * STRIDE;
    }
}

// Where lane `lane` (sub-row lane % R of block-row lane / R) stands at the start
// of a chunk.
template <class LT, int R>
__device__ __forceinline__ SubRow sub_row_at(const Chunk& ch, int lane) {
    constexpr int STRIDE = Header<LT, R>::STRIDE;
    const int slot = lane / R;
    const int src = slot > 0 ? slot - 1 : 0;
    const int b_prev = __shfl_sync(FULL, ch.b_hi, src);
    const int v_prev = __shfl_sync(FULL, ch.v_hi, src);
    const int b_mine = __shfl_sync(FULL, ch.b_hi, slot);
    const int b = slot > 0 ? b_prev : ch.b_lo;
    SubRow at;
    at.n = slot < ch.nrow ? b_mine - b : 0;
    at.hoff = int(long(b) * STRIDE - ch.h_al);
    at.v = (slot > 0 ? v_prev : ch.v_lo) - ch.v_al;
    return at;
}

// The forms of the row kernel: the wide and the narrow one (spmv_rows.cu), and the
// wide one with twice the blocks per step.
constexpr int WIDE = 0, NARROW = 1, DEEP = 2;

// The row sum of VS accumulators: the _mm512_reduce_add tree (distance VS/2,
// ..., 1).
template <class A, int VS>
__device__ __forceinline__ A reduce_tree(A (&acc)[VS]) {
#pragma unroll
    for (int d = VS / 2; d >= 1; d >>= 1) {
#pragma unroll
        for (int c = 0; c < d; ++c) acc[c] = acc[c] + acc[c + d];
    }
    return acc[0];
}

// y + v rounded once: red.add.f64, or load, add, store.
__device__ __forceinline__ void add_to(double* y, double v) { atomicAdd(y, v); }
__device__ __forceinline__ void add_to(float* y, float v) { *y = *y + v; }

// One chunk of block-rows for one x and y: the lane of every sub-row runs its
// blocks and adds the row sum to y.
template <class LT, int R, class V, class X, class A, class Y, int FORM>
__device__ __forceinline__ void chunk_spmv(const Chunk& ch, const uint32_t* hw, const V* vbuf,
                                           const X* __restrict__ x, Y* __restrict__ y, int nrows, uint64_t pol_x) {
    constexpr int VS = Layout<LT>::VS;
    const int lane = threadIdx.x & 31;
    const SubRow at = sub_row_at<LT, R>(ch, lane);
    A acc[VS];
#pragma unroll
    for (int c = 0; c < VS; ++c) acc[c] = A(0);
    constexpr int UT = 16 / VS > 1 ? 16 / VS : 1;
    if constexpr (FORM == NARROW)
        narrow_blocks<LT, R, V, X, A>(hw, vbuf, x, lane % R, at, pol_x, acc);
    else
        // 16 columns per step (r = 8, FP64, 2 blocks and 6 CTAs per SM against 4 and
        // 4 on B200: banded 150,000 44 / 42 us, 5-point Poisson 700^2 19.2 / 21.1;
        // mixed, banded 200,000 14.2 / 19.1)
        wide_blocks<LT, R, V, X, A, (FORM == DEEP ? 2 * UT : UT)>(hw, vbuf, x, lane % R, at, pol_x, acc);
    const A sum = reduce_tree<A, VS>(acc);
    const long yrow = long(ch.r0) * R + lane;  // sub-row `lane` of the chunk
    if (lane / R < ch.nrow && yrow < nrows) add_to(y + yrow, Y(sum));
}

}  // namespace rows
}  // namespace spc5cuda
