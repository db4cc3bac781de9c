// stream.cu -- SpMV and SpMM over the sorted plan (stream.cuh; plan.cu builds
// it; chain.cuh has the kernels of its chain part).
//
// Arithmetic (bit-identical to the reference kernels core_SPC5_{r}rVc_Spmv_*,
// src/spc5.hpp:2309-2715): every (row, column class c) chain is one
// accumulator, the reference's vector lane c, which receives fma(value,
// x[col + c], acc) for each block in order whose mask has bit c; a row's sum
// is the _mm512_reduce_add tree over its VS accumulators (+0 for a class
// without values) and y[row] += sum.
//
// What bounds it: latency.  In a window of steps the index loads, the x gathers and
// the multiply-adds follow one another, and the longest rows are the tail (power-law
// of 1,000,000 rows on a B200: L1 45%, issue 33%, 22% of the warps active).  An x
// gather costs one L2 -> L1 sector (32 bytes) per distinct sector that its
// instruction touches, about one per cycle and SM; the long rows' streams keep a
// row-block's columns side by side, so that n neighbouring columns cost 1 + (n - 1) /
// 4 sectors instead of n.
#include <algorithm>
#include <memory>
#include <type_traits>

#include "chain.cuh"
#include "stream.cuh"

namespace spc5cuda {

namespace {

using namespace stream;

constexpr int THREADS = 128;
constexpr int WARPS = THREADS / 32;

// The long rows' SpMV: steps per window, staged values (at least one step's 32),
// gathers in flight per lane, steps per multiply-add batch, CTAs per SM asked
// of the compiler.  A window of a power-law row's steps holds about 295 values:
// 320 take it in two passes of 160.  Measured on B200, power-law N = 4M, r = 1
// / N = 1M, r = 8, mixed (us per SpMV): 5 gathers, 7 CTAs 319 / 103; 5 and 6
// CTAs 331 / 101; 5 and 8 CTAs (64 registers, 2 steps per batch) 358 / 112; 8
// gathers and 7 CTAs (spills) 485 / 107.
constexpr int WIN = 32;
constexpr int BUF = 320;
constexpr int UG = 5;
constexpr int PH = 4;
constexpr int LONG_CTAS = 7;
// The short rows' SpMV: entries in flight per lane, CTAs per SM.  4 entries
// and 8 CTAs (54 registers) 328 us at N = 4M, 8 entries and no bound (84
// registers) 377.
constexpr int SU = 4;
constexpr int SHORT_CTAS = 8;

template <class V, class X>
struct __align__(16) WarpBuf {
    V val[BUF];
    X x[BUF];
    uint2 step[WIN + PH];  // mask, first value (from the window's); read, not used, past the window
};

// Asynchronous copy of one value to shared memory, streamed through L2.
template <class V>
__device__ __forceinline__ void cp_async_value(uint32_t saddr, const V* g, uint64_t pol) {
    if constexpr (sizeof(V) == 8)
        asm volatile("cp.async.ca.shared.global.L2::cache_hint [%0], [%1], 8, %2;\n" ::"r"(saddr), "l"(g), "l"(pol)
                     : "memory");
    else
        asm volatile("cp.async.ca.shared.global.L2::cache_hint [%0], [%1], 4, %2;\n" ::"r"(saddr), "l"(g), "l"(pol)
                     : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }
__device__ __forceinline__ void prefetch_l2(const void* p) {
    asm volatile("prefetch.global.L2 [%0];" ::"l"(p) : "memory");
}

// Loads of an active lane (on != 0), predicated without a branch, so that the
// loads of several steps are issued together; v is left as it is otherwise.
__device__ __forceinline__ void ld_if(double& v, const double* p, uint32_t on) {
    asm volatile("{ .reg .pred q; setp.ne.u32 q, %2, 0; @q ld.global.nc.f64 %0, [%1]; }"
                 : "+d"(v) : "l"(p), "r"(on));
}
__device__ __forceinline__ void ld_if(float& v, const float* p, uint32_t on) {
    asm volatile("{ .reg .pred q; setp.ne.u32 q, %2, 0; @q ld.global.nc.f32 %0, [%1]; }"
                 : "+f"(v) : "l"(p), "r"(on));
}
__device__ __forceinline__ void ld_if(int& v, const int* p, uint32_t on) {
    asm volatile("{ .reg .pred q; setp.ne.u32 q, %2, 0; @q ld.global.nc.s32 %0, [%1]; }"
                 : "+r"(v) : "l"(p), "r"(on));
}
__device__ __forceinline__ void ld_if(uint4& v, const void* p, uint32_t on) {
    asm volatile("{ .reg .pred q; setp.ne.u32 q, %5, 0; @q ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%4]; }"
                 : "+r"(v.x), "+r"(v.y), "+r"(v.z), "+r"(v.w) : "l"(p), "r"(on));
}

// (launch_after, with this file's CTA.)
template <class... P, class... Q>
void launch(void (*kern)(P...), dim3 grid, bool follows, cudaStream_t s, Q... args) {
    launch_after(kern, grid, THREADS, 0, follows, s, args...);
}

// The long rows: one warp per slab.  STRIDED: a column of row-major X and Y, element
// i at i ldx and i ldy.  FOLLOWS: after another launch of the product (a kernel of its
// own: with the wait at its end the 1,000,000-row power-law matrix, 8-column mixed
// layout, took 118 us instead of 109).
template <class V, class X, class A, class Y, int VS, bool STRIDED, bool FOLLOWS>
__global__ void __launch_bounds__(THREADS, LONG_CTAS)
    k_stream_spmv(const __grid_constant__ View p, const V* __restrict__ val, const X* __restrict__ x, long ldx,
                  Y* __restrict__ y, long ldy) {
    using Buf = WarpBuf<V, X>;
    griddep_launch();
    constexpr int G = 32 / VS;
    __shared__ Buf bufs[WARPS];
    const int lane = threadIdx.x & 31;
    Buf& buf = bufs[threadIdx.x >> 5];
    const int slab = blockIdx.x * WARPS + (threadIdx.x >> 5);
    if (slab >= p.long_slabs()) return;  // warp-uniform
    const int g = lane / VS, c = lane % VS;
    const uint32_t bit = 1u << lane, lt = bit - 1u;
    const SlabRows sr = slab_rows<G>(p, slab);
    const int nrows = sr.row_end - sr.row0;
    const int s0 = __ldg(p.sstep + slab);
    const int ns = __ldg(p.sstep + slab + 1) - s0;
    long base = __ldg(p.sval + slab);
    uint32_t mask = lane < ns ? __ldcs(p.mask + s0 + lane) : 0u;
    const long all = p.long_values();
    const uint64_t pol_x = l2_evict_last_policy(), pol_v = l2_evict_first_policy();
    const uint32_t s_val = uint32_t(__cvta_generic_to_shared(buf.val)) + unsigned(lane * sizeof(V));
    // ends of the rounds: lane q holds the row-blocks of round q
    const int nb = lane < sr.rounds && lane * G < nrows ? __ldg(p.key + sr.row0 + lane * G) - LONG_KEY : 0;
    int q = 0, end = __shfl_sync(FULL, nb, 0);
    int row = lane < nrows ? __ldg(p.perm + sr.row0 + lane) : 0;

    A acc = A(0);
    // the end of round q: the reduce tree over the lanes of each group
    auto end_round = [&]() {
#pragma unroll
        for (int d = VS / 2; d >= 1; d >>= 1) acc = acc + __shfl_xor_sync(FULL, acc, d);
        const int yrow = __shfl_sync(FULL, row, (q * G + g) & 31);
        if (c == 0 && q * G + g < nrows) add_to(STRIDED ? y + long(yrow) * ldy : y + yrow, Y(acc));
        acc = A(0);
        ++q;
        end += __shfl_sync(FULL, nb, q);
        // the next 32 rows of the slab
        if ((q * G) % 32 == 0 && q * G + lane < nrows) row = __ldg(p.perm + sr.row0 + q * G + lane);
    };

    for (int w = 0; w < ns; w += WIN) {  // warp-uniform
        // ---- the window's steps: masks and value offsets
        const int nsw = min(WIN, ns - w);
        int incl = __popc(mask);
#pragma unroll
        for (int d = 1; d < WIN; d <<= 1) {
            const int u = __shfl_up_sync(FULL, incl, d);
            if (lane >= d) incl += u;
        }
        buf.step[lane] = make_uint2(mask, unsigned(incl - __popc(mask)));
        const int total = __shfl_sync(FULL, incl, WIN - 1);
        mask = w + WIN + lane < ns ? __ldcs(p.mask + s0 + w + WIN + lane) : 0u;
        // the next window (about as large) into L2, one 128-byte line per lane
        if (w + WIN < ns) {
            const long at = base + total + lane * long(128 / sizeof(V));
            if (lane * (128 / int(sizeof(V))) < total && at < all) prefetch_l2(val + at);
            const long ac = base + total + lane * 32L;
            if (lane * 32 < total && ac < all) prefetch_l2(p.col + ac);
        }
        int vb = 0;
        for (int done = 0; done < nsw;) {
            // ---- as many steps as fit the buffer: their values and x, one
            // value per lane (neighbouring lanes read neighbouring columns)
            const uint32_t fit = __ballot_sync(FULL, lane >= done && lane < nsw && incl - vb <= BUF);
            const int stop = done + __popc(fit);
            const int nv = __shfl_sync(FULL, incl, stop - 1) - vb;
            const int* cp = p.col + base + vb;
            const V* vp = val + base + vb;
#pragma unroll 1
            for (int i0 = 0; i0 < nv; i0 += 32 * UG) {
                int col[UG];
                X xv[UG];
#pragma unroll
                for (int u = 0; u < UG; ++u) {
                    const int i = i0 + u * 32 + lane;
                    if (i < nv) col[u] = __ldcs(cp + i);
                }
#pragma unroll
                for (int u = 0; u < UG; ++u) {
                    const int i = i0 + u * 32;
                    if (i + lane < nv) cp_async_value(s_val + unsigned(i * sizeof(V)), vp + i + lane, pol_v);
                }
#pragma unroll
                for (int u = 0; u < UG; ++u)
                    if (i0 + u * 32 + lane < nv) xv[u] = ld_x(STRIDED ? x + long(col[u]) * ldx : x + col[u], pol_x);
#pragma unroll
                for (int u = 0; u < UG; ++u) {
                    const int i = i0 + u * 32 + lane;
                    if (i < nv) buf.x[i] = xv[u];
                }
            }
            cp_async_wait();
            __syncwarp();
            // ---- the multiply-adds, step by step, up to the end of the round
            for (int t = done; t < stop;) {
                const int upto = min(stop, end - w);
#pragma unroll 1
                for (; t < upto; t += PH) {
                    uint32_t m[PH];
                    A v[PH], xv[PH];
#pragma unroll
                    for (int u = 0; u < PH; ++u) {
                        const uint2 st = buf.step[t + u];
                        m[u] = t + u < upto ? st.x & bit : 0u;
                        const int i = int(st.y) - vb + __popc(st.x & lt);
                        if (m[u]) {
                            v[u] = A(buf.val[i]);
                            xv[u] = A(buf.x[i]);
                        }
                    }
#pragma unroll
                    for (int u = 0; u < PH; ++u)
                        if (m[u]) acc = fma(v[u], xv[u], acc);
                }
                t = upto;
                if (w + t == end) end_round();
            }
            __syncwarp();
            vb += nv;
            done = stop;
        }
        base += total;
    }
    if constexpr (FOLLOWS) end_launch(true);
}

// The short rows: one warp per slab, one lane per row.  A lane runs its chains
// one after the other and leaves their results in its own column of shared
// memory, in chain order (slot 0 takes what precedes the first chain).
template <class V, class X, class A, class Y, int VS, bool STRIDED>
__global__ void __launch_bounds__(THREADS, SHORT_CTAS)
    k_short_spmv(const __grid_constant__ View p, const V* __restrict__ val, const X* __restrict__ x, long ldx,
                 Y* __restrict__ y, long ldy, bool follows) {
    griddep_launch();
    __shared__ A chain[WARPS][VS + 1][32];
    const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
    const int slab = blockIdx.x * WARPS + wi;
    if (slab < p.short_slabs()) {  // warp-uniform
        const ShortRows sr = short_rows(p, slab);
        const bool live = lane < sr.rows;
        const int* cp = p.col + sr.at + lane;
        const V* vp = val + sr.at + lane;
        const uint32_t w = live ? uint32_t(__ldcs(p.chains + slab * 32L + lane)) : 0u;
        const int row = live ? __ldcs(p.perm + sr.row0 + lane) : 0;
        const uint64_t pol_x = l2_evict_last_policy();
        A acc = A(0);
        A* slot = &chain[wi][0][lane];
        for (int j0 = 0; j0 < sr.len; j0 += SU) {
            int col[SU];
            V v[SU];
            X xv[SU];
#pragma unroll
            for (int u = 0; u < SU; ++u) {
                if (live && j0 + u < sr.len) {
                    col[u] = __ldcs(cp + 32 * (j0 + u));
                    v[u] = __ldcs(vp + 32 * (j0 + u));
                }
            }
#pragma unroll
            for (int u = 0; u < SU; ++u)
                if (live && j0 + u < sr.len) {
                    const uint32_t xi = uint32_t(col[u]) & ~FIRST;
                    xv[u] = ld_x(STRIDED ? x + long(xi) * ldx : x + xi, pol_x);
                }
#pragma unroll
            for (int u = 0; u < SU; ++u) {
                if (live && j0 + u < sr.len) {
                    if (col[u] < 0) {
                        *slot = acc;
                        slot += 32;
                        acc = A(0);
                    }
                    acc = fma(A(v[u]), A(xv[u]), acc);
                }
            }
        }
        *slot = acc;
        A a[VS];
#pragma unroll
        for (int c = 0; c < VS; ++c)
            a[c] = (w >> c) & 1u ? chain[wi][1 + __popc(w & ((1u << c) - 1u))][lane] : A(0);
#pragma unroll
        for (int d = VS / 2; d >= 1; d >>= 1) {
#pragma unroll
            for (int k = 0; k < d; ++k) a[k] = a[k] + a[k + d];
        }
        if (live) add_to(STRIDED ? y + long(row) * ldy : y + row, Y(a[0]));
    }
    end_launch(follows);
}


// Y += A X over the long rows of the slabs [slab0, slab1) for kc <= KQ G
// right-hand sides.  Lane (c, jq) = (lane / G, lane % G) owns column c and the
// right-hand sides jq + G i (VEC: KQ jq + i, read as 16-byte vectors), with one
// accumulator per row and right-hand side.  GP = G: the warp takes the G
// row-blocks of a step one after the other; GP = 1: only those of one group, the
// G groups of a slab in neighbouring CTAs (the longest rows: more warps, fewer
// dependent steps each; the longest of all begin first: with the groups in
// blockIdx.y the last group's longest row began when the others were done, and the
// launch took 490 us instead of 306 on power-law N = 600,000, r = 2, k = 16, FP64,
// the SpMM 586 instead of 483 on a B200).  U
// steps at a time: their values and x indices, then their x, then the
// multiply-adds in order.
template <class V, class X, class A, class Y, int VS, int KQ, bool VEC, int U, int GP>
__global__ void __launch_bounds__(THREADS) k_stream_spmm(const __grid_constant__ View p, int slab0, int slab1, const V* __restrict__ val,
                                                         int kc, const X* __restrict__ x, long ldx, long xcs,
                                                         Y* __restrict__ y, long ldy, long ycs, bool follows) {
    constexpr int G = 32 / VS;
    static_assert(32 % U == 0, "whole batches per window");
    griddep_launch();
    const int lane = threadIdx.x & 31;
    constexpr int PARTS = G / GP;
    const int slab = slab0 + blockIdx.x / PARTS * WARPS + (threadIdx.x >> 5);
    if (slab >= slab1) return;  // warp-uniform
    const int g0 = GP == 1 ? blockIdx.x % PARTS : 0;
    const int c = lane / G, jq = lane % G;
    const SlabRows sr = slab_rows<G>(p, slab);
    const int nrows = sr.row_end - sr.row0;
    int row = lane < nrows ? __ldg(p.perm + sr.row0 + lane) : 0;
    const int nb = lane < sr.rounds && lane * G < nrows ? __ldg(p.key + sr.row0 + lane * G) - LONG_KEY : 0;
    const int s0 = __ldg(p.sstep + slab);
    const int ns = __ldg(p.sstep + slab + 1) - s0;
    long base = __ldg(p.sval + slab);
    uint32_t mask = lane < ns ? __ldg(p.mask + s0 + lane) : 0u;
    auto rhs = [&](int i) { return VEC ? jq * KQ + i : jq + G * i; };

    A acc[GP][KQ];
    auto zero = [&]() {
#pragma unroll
        for (int g = 0; g < GP; ++g)
#pragma unroll
            for (int i = 0; i < KQ; ++i) acc[g][i] = A(0);
    };
    // Row sums of round q: the reduce tree over the columns (lane distance G
    // VS / 2, ..., G) as a reduce-scatter of the N = GP KQ entries g KQ + i
    // while more than one is held: at each level the lane with the bit set
    // keeps the odd entries and its partner the even ones.
    auto flush = [&](int q) {
        constexpr int N = GP * KQ;
        A sv[N];
#pragma unroll
        for (int e = 0; e < N; ++e) sv[e] = acc[e / KQ][e % KQ];
        int ent = 0, held = 1;  // entry of sv[0], and the distance to the next
        bool own = true;
        int n = N;
#pragma unroll
        for (int d = VS / 2; d >= 1; d >>= 1) {
            const bool hi = (c & d) != 0;
            if (n >= 2) {
#pragma unroll
                for (int e = 0; e < N / 2; ++e) {
                    if (e < n / 2) {
                        const A keep = hi ? sv[2 * e + 1] : sv[2 * e];
                        const A send = hi ? sv[2 * e] : sv[2 * e + 1];
                        sv[e] = keep + __shfl_xor_sync(FULL, send, d * G);
                    }
                }
                if (hi) ent += held;
                held *= 2;
                n /= 2;
            } else {
                sv[0] = sv[0] + __shfl_xor_sync(FULL, sv[0], d * G);
                own = own && !hi;
            }
        }
#pragma unroll
        for (int e = 0; e < N; ++e) {
            if (e < n) {
                const int at = ent + e * held;
                const int g = g0 + at / KQ, j = rhs(at % KQ);
                const int yrow = __shfl_sync(FULL, row, (q * G + g) & 31);
                if (own && q * G + g < nrows && j < kc) add_to(y + long(yrow) * ldy + long(j) * ycs, Y(sv[e]));
            }
        }
        zero();
        // the next 32 rows of the slab
        if (((q + 1) * G) % 32 == 0 && (q + 1) * G + lane < nrows)
            row = __ldg(p.perm + sr.row0 + (q + 1) * G + lane);
    };

    zero();
    int q = 0, end = __shfl_sync(FULL, nb, 0);
    for (int w = 0; w < ns; w += 32) {  // warp-uniform
        int incl = __popc(mask);
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int t = __shfl_up_sync(FULL, incl, d);
            if (lane >= d) incl += t;
        }
        const uint32_t wmask = mask;
        const int excl = incl - __popc(mask);
        mask = w + 32 + lane < ns ? __ldg(p.mask + s0 + w + 32 + lane) : 0u;
        const int nsw = min(32, ns - w);
#pragma unroll 1
        for (int t0 = 0; t0 < nsw; t0 += U) {
            uint32_t on[U][GP];
            V v[U][GP];
            int col[U][GP];
            X xv[U][GP][KQ];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const uint32_t m = __shfl_sync(FULL, wmask, t0 + u);  // 0 past the window's steps
                const long at0 = base + __shfl_sync(FULL, excl, t0 + u);
#pragma unroll
                for (int g = 0; g < GP; ++g) {
                    const uint32_t b = 1u << ((g0 + g) * VS + c);
                    on[u][g] = m & b;
                    const long at = at0 + __popc(m & (b - 1u));
                    col[u][g] = 0;
                    ld_if(col[u][g], p.col + at, on[u][g]);
                    v[u][g] = V(0);
                    ld_if(v[u][g], val + at, on[u][g]);
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
#pragma unroll
                for (int g = 0; g < GP; ++g) {
                    const X* xr = x + long(col[u][g]) * ldx;
                    if constexpr (VEC) {
                        constexpr int PER = 16 / int(sizeof(X));
#pragma unroll
                        for (int i = 0; i < KQ; i += PER) {
                            uint4 t4 = make_uint4(0u, 0u, 0u, 0u);
                            ld_if(t4, xr + rhs(i), rhs(i) < kc ? on[u][g] : 0u);
                            const X* e = reinterpret_cast<const X*>(&t4);
#pragma unroll
                            for (int k = 0; k < PER; ++k) xv[u][g][i + k] = e[k];
                        }
                    } else {
#pragma unroll
                        for (int i = 0; i < KQ; ++i) {
                            xv[u][g][i] = X(0);
                            ld_if(xv[u][g][i], xr + long(rhs(i)) * xcs, rhs(i) < kc ? on[u][g] : 0u);
                        }
                    }
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
#pragma unroll
                for (int g = 0; g < GP; ++g)
                    if (on[u][g]) {
#pragma unroll
                        for (int i = 0; i < KQ; ++i) acc[g][i] = fma(A(v[u][g]), A(xv[u][g][i]), acc[g][i]);
                    }
                if (w + t0 + u + 1 == end) {  // the round's last step
                    flush(q);
                    ++q;
                    end += __shfl_sync(FULL, nb, q);
                }
            }
        }
        base += __shfl_sync(FULL, incl, 31);
    }
    end_launch(follows);
}

// Y += A X over the short rows for kc <= KC right-hand sides: KC lanes per
// row, one right-hand side each, 32 / KC rows of the slab at a time.
template <class V, class X, class A, class Y, int VS, int KC>
__global__ void __launch_bounds__(THREADS) k_short_spmm(const __grid_constant__ View p, const V* __restrict__ val, int kc,
                                                        const X* __restrict__ x, long ldx, long xcs,
                                                        Y* __restrict__ y, long ldy, long ycs, bool follows) {
    constexpr int U = 4;
    constexpr int PAR = 32 / KC;  // rows at a time
    __shared__ A chain[WARPS][VS + 1][32];
    griddep_launch();
    const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
    const int slab = blockIdx.x * WARPS + wi;
    if (slab >= p.short_slabs()) return;  // warp-uniform
    const ShortRows sr = short_rows(p, slab);
    const int h = lane / KC, j = lane % KC;
    const uint32_t words = __ldg(p.chains + slab * 32L + lane);
    const int rows = lane < sr.rows ? __ldg(p.perm + sr.row0 + lane) : 0;
    const uint64_t pol_x = l2_evict_last_policy();
    const X* xj = x + long(j) * xcs;
    for (int i0 = 0; i0 < sr.rows; i0 += PAR) {
        const uint32_t w = __shfl_sync(FULL, words, i0 + h);
        const int row = __shfl_sync(FULL, rows, i0 + h);
        const bool live = i0 + h < sr.rows && j < kc;
        const int len = live ? sr.len : 0;
        const int* cp = p.col + sr.at + i0 + h;
        const V* vp = val + sr.at + i0 + h;
        A acc = A(0);
        A* slot = &chain[wi][0][lane];
        for (int k0 = 0; k0 < len; k0 += U) {
            int col[U];
            V v[U];
            X xv[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (k0 + u < len) {
                    col[u] = __ldg(cp + 32 * (k0 + u));
                    v[u] = __ldg(vp + 32 * (k0 + u));
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (k0 + u < len) xv[u] = ld_x(xj + long(uint32_t(col[u]) & ~FIRST) * ldx, pol_x);
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (k0 + u < len) {
                    if (col[u] < 0) {
                        *slot = acc;
                        slot += 32;
                        acc = A(0);
                    }
                    acc = fma(A(v[u]), A(xv[u]), acc);
                }
            }
        }
        *slot = acc;
        A a[VS];
#pragma unroll
        for (int c = 0; c < VS; ++c)
            a[c] = (w >> c) & 1u ? chain[wi][1 + __popc(w & ((1u << c) - 1u))][lane] : A(0);
#pragma unroll
        for (int d = VS / 2; d >= 1; d >>= 1) {
#pragma unroll
            for (int k = 0; k < d; ++k) a[k] = a[k] + a[k + d];
        }
        if (live) add_to(y + long(row) * ldy + long(j) * ycs, Y(a[0]));
    }
    end_launch(follows);
}

// Two right-hand sides run as an SpMV each from this many values in the streams on
// (power-law on B200, FP64, r = 1, us: 300,000 rows, 3.2M values 152 together, 178 one
// after the other; 1,000,000 rows 440, 193).
constexpr long PAIR_VALUES = 4L << 20;

// The streams and the short rows for one x; follows: a launch of this product came before.
template <class V, class X, class A, class Y, int VS, bool STRIDED>
void run_rows(const SortedPlan& p, const X* x, long ldx, Y* y, long ldy, bool& follows, cudaStream_t s) {
    const View v = view_of(p);
    const V* val = p.val.as<V>();
    if (v.long_slabs() > 0) {
        auto kern = follows ? k_stream_spmv<V, X, A, Y, VS, STRIDED, true> : k_stream_spmv<V, X, A, Y, VS, STRIDED, false>;
        launch(kern, dim3(div_up(v.long_slabs(), WARPS)), follows, s, v, val, x, ldx, y, ldy);
        follows = true;
    }
    if (v.short_slabs() > 0) {
        launch(k_short_spmv<V, X, A, Y, VS, STRIDED>, dim3(div_up(v.short_slabs(), WARPS)), follows, s, v, val, x, ldx, y,
               ldy, follows);
        follows = true;
    }
}

template <class V, class X, class A, class Y, int VS>
void run_spmv(const spc5cuda_mat* m, const X* x, Y* y, cudaStream_t s) {
    const SortedPlan& p = *m->plan;
    bool follows = false;
    if (p.chain_rows == 0) {
        run_rows<V, X, A, Y, VS, false>(p, x, 1L, y, 1L, follows, s);
        return;
    }
    const ChainView c = chain_view_of(p);
    PoolBuf sums(sizeof(A) * size_t(c.rows) * VS, s);
    auto kern = c.slabs <= 8 * sm_count() ? k_chain_spmv<V, X, A, CHAIN_DEEP> : k_chain_spmv<V, X, A, CHAIN_U>;
    launch(kern, dim3(div_up(c.slabs, CHAIN_THREADS / 32)), false, s, c, static_cast<const V*>(p.cval), x, sums.as<A>());
    follows = true;
    run_rows<V, X, A, Y, VS, false>(p, x, 1L, y, 1L, follows, s);
    launch(k_chain_rows<A, Y, VS, 1>, dim3(div_up(c.rows, CHAIN_THREADS)), false, s, c, 1, sums.as<A>(), y, 1L, 1L);
}

template <class V, class X, class A, class Y, int VS>
void run_spmm(const spc5cuda_mat* m, int k, const X* x, long ldx, long xcs, Y* y, long ldy, long ycs,
              cudaStream_t s) {
    constexpr int G = 32 / VS;
    const SortedPlan& p = *m->plan;
    const View v = view_of(p);
    const V* val = p.val.as<V>();
    bool follows = false;  // a launch of this pass came before
    // slabs [a, b) of the long rows
    auto longs = [&](auto kq, auto u, auto gp, int a, int b, int kc, const X* xp, Y* yp) {
        constexpr int KQ = decltype(kq)::value, U = decltype(u)::value, GP = decltype(gp)::value;
        constexpr int PER = 16 / int(sizeof(X));
        if (a >= b) return;
        const dim3 grid(unsigned(div_up(b - a, WARPS) * (G / GP)));
        const bool after = follows;
        follows = true;
        if constexpr (KQ >= PER) {
            // rows of X as 16-byte vectors: unit stride, aligned, whole vectors
            if (xcs == 1 && ldx % PER == 0 && kc % PER == 0 && aligned(xp, 16)) {
                launch(k_stream_spmm<V, X, A, Y, VS, KQ, true, U, GP>, grid, after, s, v, a, b, val, kc, xp, ldx, xcs, yp,
                       ldy, ycs, after);
                return;
            }
        }
        launch(k_stream_spmm<V, X, A, Y, VS, KQ, false, U, GP>, grid, after, s, v, a, b, val, kc, xp, ldx, xcs, yp, ldy,
               ycs, after);
    };
    auto shorts = [&](auto kcc, int kc, const X* xp, Y* yp) {
        if (v.short_slabs() > 0)
            launch(k_short_spmm<V, X, A, Y, VS, decltype(kcc)::value>, dim3(div_up(v.short_slabs(), WARPS)), follows, s,
                   v, val, kc, xp, ldx, xcs, yp, ldy, ycs, follows);
    };
    // the chain part's launches, before and after the others
    std::unique_ptr<PoolBuf> sums;
    auto chains = [&](auto kcc, int kc, const X* xp) {
        constexpr int KC = decltype(kcc)::value;
        if (p.chain_rows == 0) return;
        const ChainView c = chain_view_of(p);
        const size_t bytes = sizeof(A) * size_t(c.rows) * VS * KC;
        if (!sums || sums->bytes < bytes) sums = std::make_unique<PoolBuf>(bytes, s);
        const int warps = div_up(c.chains, 32 * chain_w<KC> / KC);
        launch(k_chain_spmm<V, X, A, KC>, dim3(div_up(warps, CHAIN_THREADS / 32)), false, s, c,
               static_cast<const V*>(p.cval), kc, xp, ldx, xcs, sums->as<A>());
        follows = true;
    };
    auto chain_rows = [&](auto kcc, int kc, Y* yp) {
        constexpr int KC = decltype(kcc)::value;
        if (p.chain_rows == 0) return;
        launch(k_chain_rows<A, Y, VS, KC>, dim3(div_up(long(p.chain_rows) * KC, CHAIN_THREADS)), false, s,
               chain_view_of(p), kc, sums->as<A>(), yp, ldy, ycs);
    };
    using std::integral_constant;
    // right-hand sides per pass: 16, fewer where the chains' scratch would be more than 1 GiB
    int per = 16;
    while (per > 4 && sizeof(A) * size_t(p.chain_rows) * VS * size_t(per) > (size_t(1) << 30)) per /= 2;
    for (int q0 = 0; q0 < k;) {
        const int kc = std::min(per, k - q0);
        follows = false;
        const X* xp = x + long(q0) * xcs;
        Y* yp = y + long(q0) * ycs;
        if (k - q0 == 1 && ldx == 1 && ldy == 1) {  // one contiguous right-hand side
            run_spmv<V, X, A, Y, VS>(m, xp, yp, s);
            return;
        }
        const int a = v.slab_end[0], b = v.long_slabs();
        constexpr integral_constant<int, G> all{};
        constexpr integral_constant<int, 1> one{};
        constexpr integral_constant<int, 4> deep{};
        if (kc > 8) {
            chains(integral_constant<int, 16>{}, kc, xp);
            longs(integral_constant<int, 16 / G>{}, deep, one, 0, a, kc, xp, yp);
            longs(integral_constant<int, 16 / G>{}, one, all, a, b, kc, xp, yp);
            shorts(integral_constant<int, 16>{}, kc, xp, yp);
            chain_rows(integral_constant<int, 16>{}, kc, yp);
        } else if (kc > 4) {
            chains(integral_constant<int, 8>{}, kc, xp);
            longs(integral_constant<int, 8 / G>{}, deep, one, 0, a, kc, xp, yp);
            longs(integral_constant<int, 8 / G>{}, integral_constant<int, 2>{}, all, a, b, kc, xp, yp);
            shorts(integral_constant<int, 8>{}, kc, xp, yp);
            chain_rows(integral_constant<int, 8>{}, kc, yp);
        } else if (kc == 1 || (kc == 2 && p.long_values >= PAIR_VALUES)) {
            // an SpMV each
            chains(integral_constant<int, 2>{}, kc, xp);
            for (int j = 0; j < kc; ++j)
                run_rows<V, X, A, Y, VS, true>(p, xp + j * xcs, ldx, yp + j * ycs, ldy, follows, s);
            chain_rows(integral_constant<int, 2>{}, kc, yp);
        } else {
            chains(integral_constant<int, 4>{}, kc, xp);
            longs(integral_constant<int, 4 / G>{}, integral_constant<int, 8>{}, one, 0, a, kc, xp, yp);
            longs(integral_constant<int, 4 / G>{}, integral_constant<int, 2>{}, all, a, b, kc, xp, yp);
            shorts(integral_constant<int, 4>{}, kc, xp, yp);
            chain_rows(integral_constant<int, 4>{}, kc, yp);
        }
        q0 += kc;
    }
}

}  // namespace

void plan_spmv(const spc5cuda_mat* m, const void* x, void* y, bool mixed, cudaStream_t s) {
    if (m->value_type == SPC5CUDA_F64)
        run_spmv<double, double, double, double, 8>(m, static_cast<const double*>(x), static_cast<double*>(y), s);
    else if (m->value_type == SPC5CUDA_F32_V8)
        run_spmv<float, float, double, double, 8>(m, static_cast<const float*>(x), static_cast<double*>(y), s);
    else if (mixed)
        run_spmv<float, float, double, double, 16>(m, static_cast<const float*>(x), static_cast<double*>(y), s);
    else
        run_spmv<float, float, float, float, 16>(m, static_cast<const float*>(x), static_cast<float*>(y), s);
}

void plan_spmm(const spc5cuda_mat* m, int k, const void* x, long ldx, long xcs, void* y, long ldy, long ycs,
               bool mixed, cudaStream_t s) {
    if (m->value_type == SPC5CUDA_F64)
        run_spmm<double, double, double, double, 8>(m, k, static_cast<const double*>(x), ldx, xcs,
                                                    static_cast<double*>(y), ldy, ycs, s);
    else if (m->value_type == SPC5CUDA_F32_V8)
        run_spmm<float, float, double, double, 8>(m, k, static_cast<const float*>(x), ldx, xcs,
                                                  static_cast<double*>(y), ldy, ycs, s);
    else if (mixed)
        run_spmm<float, float, double, double, 16>(m, k, static_cast<const float*>(x), ldx, xcs,
                                                   static_cast<double*>(y), ldy, ycs, s);
    else
        run_spmm<float, float, float, float, 16>(m, k, static_cast<const float*>(x), ldx, xcs,
                                                 static_cast<float*>(y), ldy, ycs, s);
}

}  // namespace spc5cuda
