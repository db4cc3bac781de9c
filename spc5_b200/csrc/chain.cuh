// chain.cuh -- SpMV and SpMM over the chain part of the sorted plan (stream.cuh has
// its layout; plan.cu builds it): one lane runs one (row, column) chain of
// multiply-adds (SpMM: for one or two right-hand sides), and a last launch adds each
// row's VS chains by the reduce tree.
#pragma once

#include <type_traits>

#include "stream.cuh"

namespace spc5cuda {
namespace stream {

// The chains' results, chain (sorted row i, column c) of right-hand side j at
// (i VS + c) KC + j, go through scratch of the call.
// Entries per step of a lane: 8; 16 in the SpMV where the slabs are few and the
// longest chain's latency is the time.
constexpr int CHAIN_U = 8, CHAIN_DEEP = 16;
constexpr int CHAIN_THREADS = 128;

// The kernels of one SpMV or SpMM write disjoint rows of y: each lets the next
// one begin while its own last warps run (the longest rows decide when a
// kernel ends), and the last block of a kernel that follows another waits for
// the one before it, so that the end of the last launch is the end of all.
// (That block's first warp always has a slab and reaches end_launch.)
__device__ __forceinline__ void griddep_launch() { asm volatile("griddepcontrol.launch_dependents;"); }
__device__ __forceinline__ void end_launch(bool follows) {
    if (follows && blockIdx.x == gridDim.x - 1)
        asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Where a lane's chain q lies; a lane past the last chain runs the last one again
// and writes nothing.
struct Chain {
    int len, pitch;
    long at;  // first entry; the next ones pitch apart
};
__device__ __forceinline__ Chain chain_at(const ChainView& p, long q) {
    const long r = min(q, p.chains - 1);
    return Chain{__ldg(p.len + r), chains_of(p.chains, r / 32), __ldg(p.first + r / 32) + r % 32};
}

// f with the chain's pitch, a constant in all slabs but a last one of fewer chains
// (warp-uniform).
template <class F>
__device__ __forceinline__ void with_pitch(const Chain& c, F&& f) {
    if (c.pitch == 32) f(std::integral_constant<int, 32>{});
    else f(c.pitch);
}

// acc += the chain's multiply-adds of the entries from j0 on for W right-hand sides,
// x element i at x[i ldx + w xcs], U entries at a time: the next step's values and x
// indices load while this step's x are gathered.  Every load guarded: the chains of a
// slab differ in length.
template <int U, int W, class V, class X, class A, class P>
__device__ __forceinline__ void run_guarded(const Chain& c, int j0, P pitch, const V* __restrict__ val,
                                            const int* __restrict__ xcol, const X* __restrict__ x, long ldx, long xcs,
                                            A (&acc)[W]) {
    const V* vp = val + c.at;
    const int* cp = xcol + c.at;
    const int width = __reduce_max_sync(FULL, c.len);
    const uint64_t pol = l2_evict_last_policy();
    V v[U];
    int col[U];
    auto load = [&](int j, V (&v1)[U], int (&c1)[U]) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            v1[u] = V(0);
            c1[u] = 0;
            if (j + u < c.len) {
                v1[u] = __ldcs(vp + long(pitch) * (j + u));
                c1[u] = __ldcs(cp + long(pitch) * (j + u));
            }
        }
    };
    load(j0, v, col);
    for (; j0 < width; j0 += U) {
        X xv[U][W];
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int w = 0; w < W; ++w) xv[u][w] = j0 + u < c.len ? ld_x(x + long(col[u]) * ldx + w * xcs, pol) : X(0);
        V vn[U];
        int cn[U];
        load(j0 + U, vn, cn);
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (j0 + u < c.len) {
#pragma unroll
                for (int w = 0; w < W; ++w) acc[w] = fma(A(v[u]), A(xv[u][w]), acc[w]);
            }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            v[u] = vn[u];
            col[u] = cn[u];
        }
    }
}

// The same without guards up to the last whole step of the warp's shortest chain.
// Guarded, the compiler put the conversion of a float behind its own load, one
// load at a time (one row of 20,000 values, 8-column mixed layout 185 us, so 95;
// several right-hand sides, 50,000 rows of 400 values, k = 1, mixed 168 / 59);
// doubles with one x run faster guarded (97 / 154).
template <int U, int W, class V, class X, class A, class P>
__device__ __forceinline__ void run_whole(const Chain& c, P pitch, const V* __restrict__ val,
                                          const int* __restrict__ xcol, const X* __restrict__ x, long ldx, long xcs,
                                          A (&acc)[W]) {
    const V* vp = val + c.at;
    const int* cp = xcol + c.at;
    const int whole = __reduce_min_sync(FULL, c.len) / U * U;
    const uint64_t pol = l2_evict_last_policy();
    V v[U];
    int col[U];
    auto load = [&](int j, V (&v1)[U], int (&c1)[U]) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            v1[u] = __ldcs(vp + long(pitch) * (j + u));
            c1[u] = __ldcs(cp + long(pitch) * (j + u));
        }
    };
    if (whole > 0) load(0, v, col);
    for (int j0 = 0; j0 < whole; j0 += U) {
        X xv[U][W];
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int w = 0; w < W; ++w) xv[u][w] = ld_x(x + long(col[u]) * ldx + w * xcs, pol);
        V vn[U];
        int cn[U];
        load(min(j0 + U, whole - U), vn, cn);
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int w = 0; w < W; ++w) acc[w] = fma(A(v[u]), A(xv[u][w]), acc[w]);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            v[u] = vn[u];
            col[u] = cn[u];
        }
    }
    run_guarded<CHAIN_U, W, V, X, A>(c, whole, pitch, val, xcol, x, ldx, xcs, acc);
}

// One warp per slab, one lane per chain.
template <class V, class X, class A, int U>
__global__ void __launch_bounds__(CHAIN_THREADS) k_chain_spmv(const __grid_constant__ ChainView p, const V* __restrict__ val,
                                                              const X* __restrict__ x, A* __restrict__ out) {
    griddep_launch();
    const long q = long(blockIdx.x) * CHAIN_THREADS + threadIdx.x;
    if (q / 32 >= p.slabs) return;  // warp-uniform
    const Chain c = chain_at(p, q);
    A acc[1] = {A(0)};
    with_pitch(c, [&](auto pitch) {
        if constexpr (U == CHAIN_DEEP && sizeof(A) > sizeof(V)) run_whole<U, 1, V, X, A>(c, pitch, val, p.col, x, 1L, 0L, acc);
        else run_guarded<U, 1, V, X, A>(c, 0, pitch, val, p.col, x, 1L, 0L, acc);
    });
    if (q < p.chains) out[__ldg(p.id + q)] = acc[0];
}

// KC / W lanes per chain, W neighbouring right-hand sides each, 32 W / KC neighbouring
// chains of a slab per warp.  W = 2 from 8 right-hand sides on: half the loads of values
// and indices (20^3 grid of 6 unknowns, FP64, r = 8, k = 16 190 us, now 137).
template <int KC>
constexpr int chain_w = KC >= 8 ? 2 : 1;

template <class V, class X, class A, int KC>
__global__ void __launch_bounds__(CHAIN_THREADS) k_chain_spmm(const __grid_constant__ ChainView p, const V* __restrict__ val,
                                                              int kc, const X* __restrict__ x, long ldx, long xcs,
                                                              A* __restrict__ out) {
    griddep_launch();
    constexpr int W = chain_w<KC>, L = KC / W;  // lanes per chain
    const long t = long(blockIdx.x) * CHAIN_THREADS + threadIdx.x;
    const long q = t / L;
    const int j = int(t % L) * W;
    if (t / 32 * (32 / L) >= p.chains) return;  // warp-uniform
    const Chain c = chain_at(p, q);
    A acc[W];
#pragma unroll
    for (int w = 0; w < W; ++w) acc[w] = A(0);
    // lanes past the last right-hand side read the last one's again (an odd one's
    // second: the first again)
    const long x0 = long(min(j, kc - 1)) * xcs, step = j + 1 < kc ? xcs : 0L;
    with_pitch(c, [&](auto pitch) {
        run_whole<CHAIN_U, W, V, X, A>(c, pitch, val, p.col, x + x0, ldx, step, acc);
    });
    if (q < p.chains) {
        const long at = __ldg(p.id + q) * long(KC) + j;
#pragma unroll
        for (int w = 0; w < W; ++w)
            if (j + w < kc) out[at + w] = acc[w];
    }
}

// Y[row][j] += the reduce tree over the VS chains of every row of the chain part.
template <class A, class Y, int VS, int KC>
__global__ void __launch_bounds__(CHAIN_THREADS) k_chain_rows(const __grid_constant__ ChainView p, int kc,
                                                              const A* __restrict__ in, Y* __restrict__ y, long ldy,
                                                              long ycs) {
    const long t = long(blockIdx.x) * CHAIN_THREADS + threadIdx.x;
    const long i = t / KC;
    const int j = int(t % KC);
    if (i >= p.rows || j >= kc) return;
    const uint32_t mask = __ldg(p.mask + i);
    A a[VS];
#pragma unroll
    for (int c = 0; c < VS; ++c) a[c] = (mask >> c) & 1u ? in[(i * VS + c) * KC + j] : A(0);
#pragma unroll
    for (int d = VS / 2; d >= 1; d >>= 1) {
#pragma unroll
        for (int c = 0; c < d; ++c) a[c] = a[c] + a[c + d];
    }
    add_to(y + long(__ldg(p.perm + i)) * ldy + long(j) * ycs, Y(a[0]));
}

}  // namespace stream
}  // namespace spc5cuda
