// core_prep.cu -- what the drop-in symbols (core_SPC5_{r}rVc_Spmv_*) must know
// about bare beta(r,VS) arrays before their SpMV: the value offsets of the
// block-rows, the per-group and per-warp splits, and which kernel runs.
//
// Bound by launches and by one pass over the headers.  Two launches do it: the
// first counts values per block-row, a tile of block-rows per CTA, and leaves
// one sum and one set of maxima per tile; in the second every CTA adds the
// sums of the tiles before its own.  The second is resident while the first
// ends (its start-up is hidden) and waits for it.  A call on the 27-point stencil
// 100^3 at r = 4 takes 84 us on a B200, of which the product 54; with ten launches
// (a counting pass of one thread per block-row and one byte per load, three for
// the scan, two splits, a memset, the maxima, a sample, the flag) and the gated
// kernels one after the other it took 122.
#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "handle.h"
#include "rows_blocks.cuh"

namespace spc5cuda {

namespace {

using rows::NS;

constexpr int THREADS = 256;
constexpr int TILE = THREADS;  // block-rows per CTA of the second launch
// Lanes per block-row in the counting pass: a 27-point stencil's 9 blocks take
// three loads per lane.  The smallest parts have the threads for 16.
constexpr int L = 4, MOST_L = 16;
// Up to this many parts a CTA sums the parts before its own tile itself, 16 loads
// per thread at most; more are scanned by a launch between.
constexpr int MAX_DIRECT = 4096;
// Parts of a tile: 256, 64 or 16 block-rows, the largest with enough CTAs for the
// chip, since the threads of a CTA share its block-rows' headers and a few long
// block-rows are as much work as many short ones.  With whole tiles, 50,000 rows of
// 400 values at r = 8 (25 tiles) made a call of 3452 us on a B200, now 1227.
int part_rows(int nbr) {
    for (int part : {TILE, TILE / 4})
        if (div_up(long(nbr) + 1, part) >= 2 * sm_count()) return part;
    return TILE / MOST_L;
}

// Per part: values, most blocks and most values of a block-row, blocks whose
// every sub-row mask spans at most NS columns.
struct TileStats {
    int values, blocks, most_values, narrow;
};

__device__ __forceinline__ int warp_sum(int v) { return int(__reduce_add_sync(0xffffffffu, unsigned(v))); }
__device__ __forceinline__ int warp_max(int v) { return __reduce_max_sync(0xffffffffu, v); }

// counts[i] = values of block-row i (0 for i = nbr), and the stats of the part of
// ROWS block-rows; LANES lanes per block-row.
template <class LT, int R, int ROWS, int LANES>
__global__ void __launch_bounds__(THREADS) k_core_count(int nbr, const int* __restrict__ brptr,
                                                        const uint8_t* __restrict__ headers, int* __restrict__ counts,
                                                        TileStats* __restrict__ stats) {
    asm volatile("griddepcontrol.launch_dependents;");
    __shared__ TileStats part[THREADS / 32];
    const int q = threadIdx.x % LANES;
    const long base = long(blockIdx.x) * ROWS;
    TileStats t{0, 0, 0, 0};
    for (int i0 = threadIdx.x / LANES; i0 < ROWS; i0 += THREADS / LANES) {  // uniform
        const long i = base + i0;
        const long b0 = i < nbr ? __ldg(brptr + i) : 0, b1 = i < nbr ? __ldg(brptr + i + 1) : 0;
        int v = 0;
        for (long b = b0 + q; b < b1; b += LANES) {
            uint32_t mw[Header<LT, R>::MASK_WORDS];
            load_header<LT, R>(headers, b, mw);
            bool narrow = true;
#pragma unroll
            for (int s = 0; s < R; ++s) {
                const uint32_t m = mask_of<LT, R>(mw, s);
                v += __popc(m);
                narrow = narrow && (m == 0u || (m >> (__ffs(m) - 1)) < (1u << NS));
            }
            t.narrow += narrow ? 1 : 0;
        }
#pragma unroll
        for (int d = LANES / 2; d >= 1; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
        if (q == 0) {
            if (i <= nbr) counts[i] = v;
            t.values += v;
        }
        t.blocks = max(t.blocks, int(b1 - b0));
        t.most_values = max(t.most_values, v);
    }
    t = TileStats{warp_sum(t.values), warp_max(t.blocks), warp_max(t.most_values), warp_sum(t.narrow)};
    if (threadIdx.x % 32 == 0) part[threadIdx.x / 32] = t;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < THREADS / 32; ++w) {
            t.values += part[w].values;
            t.blocks = max(t.blocks, part[w].blocks);
            t.most_values = max(t.most_values, part[w].most_values);
            t.narrow += part[w].narrow;
        }
        stats[blockIdx.x] = t;
    }
}

// One CTA: before[t] = values of the parts before part t.
__global__ void __launch_bounds__(THREADS) k_core_parts(int nparts, const TileStats* __restrict__ stats,
                                                        int* __restrict__ before) {
    __shared__ int sums[THREADS / 32];
    int carry = 0;
    const int lane = threadIdx.x % 32, w = threadIdx.x / 32;
    for (int t0 = 0; t0 < nparts; t0 += THREADS) {  // uniform
        const int t = t0 + threadIdx.x;
        const int v = t < nparts ? stats[t].values : 0;
        int incl = v;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d) incl += u;
        }
        if (lane == 31) sums[w] = incl;
        __syncthreads();
        int at = carry + incl - v;
        for (int k = 0; k < THREADS / 32; ++k) {
            if (k < w) at += sums[k];
            carry += sums[k];
        }
        __syncthreads();
        if (t < nparts) before[t] = at;
    }
}

// valptr (in: counts) = value offset of every block-row, the splits, and (CTA
// 0) flag = 0 when some block-row does not fit the row kernel's buffers, else
// 1 for its wide, 2 for its narrow instantiation.  nparts stats, `per` of them to
// a tile; before: see k_core_parts, null when the CTA adds up the parts itself.
__global__ void __launch_bounds__(THREADS) k_core_split(int nbr, const int* __restrict__ brptr, int* valptr, int nparts,
                                                        int per, const TileStats* stats, const int* before, int ngroups,
                                                        int* __restrict__ gstart, int nwarps, int* __restrict__ wstart,
                                                        int value_type, int r, int* __restrict__ flag) {
    __shared__ TileStats part[THREADS / 32];
    __shared__ int sums[THREADS / 32];
    const int lane = threadIdx.x % 32, w = threadIdx.x / 32;
    const int nblocks = __ldg(brptr + nbr);
    const long i = long(blockIdx.x) * TILE + threadIdx.x;
    // ---- the splits (of the caller's arrays alone)
    if (i <= nbr) {
        split_at(int(i), nbr, brptr, nblocks, ngroups, gstart);
        split_at(int(i), nbr, brptr, nblocks, nwarps, wstart);
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");  // the counts
    // ---- values of the tiles before this one
    int carry = 0;
    const int first = int(blockIdx.x) * per;
    if (!before)
        for (int t = threadIdx.x; t < first; t += THREADS) carry += __ldcg(&stats[t].values);
    else if (threadIdx.x == 0)
        carry = __ldcg(before + first);
    carry = warp_sum(carry);
    // ---- the tile
    const int v = i <= nbr ? __ldcg(valptr + i) : 0;
    int incl = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += u;
    }
    if (lane == 31) {
        sums[w] = incl;
        part[w].values = carry;
    }
    __syncthreads();
    int before_me = incl - v;
#pragma unroll
    for (int k = 0; k < THREADS / 32; ++k) before_me += part[k].values + (k < w ? sums[k] : 0);
    if (i <= nbr) valptr[i] = before_me;
    if (blockIdx.x != 0) return;
    // ---- the kernel that runs
    __syncthreads();
    TileStats m{0, 0, 0, 0};
    for (int t = threadIdx.x; t < nparts; t += THREADS) {
        m.values += __ldcg(&stats[t].values);
        m.blocks = max(m.blocks, __ldcg(&stats[t].blocks));
        m.most_values = max(m.most_values, __ldcg(&stats[t].most_values));
        m.narrow += __ldcg(&stats[t].narrow);
    }
    m = TileStats{warp_sum(m.values), warp_max(m.blocks), warp_max(m.most_values), warp_sum(m.narrow)};
    if (lane == 0) part[w] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 1; k < THREADS / 32; ++k) {
            m.values += part[k].values;
            m.blocks = max(m.blocks, part[k].blocks);
            m.most_values = max(m.most_values, part[k].most_values);
            m.narrow += part[k].narrow;
        }
        const bool narrow = rows::narrow(value_type, r, nbr, nblocks, m.values, m.narrow, nblocks);
        *flag = rows::fit(value_type, r, m.blocks, m.most_values) ? (narrow ? 2 : 1) : 0;
    }
}

constexpr size_t round_up(size_t n) { return (n + 255) / 256 * 256; }  // whole 128-byte lines per array

}  // namespace

CoreScratch core_scratch(int nbr, int ngroups, int nwarps) {
    const size_t nparts = size_t(div_up(long(nbr) + 1, part_rows(nbr)));
    CoreScratch c;
    size_t at = 0;
    auto take = [&](size_t ints) {
        const size_t here = at;
        at += round_up(sizeof(int) * ints);
        return here;
    };
    c.valptr = take(size_t(nbr) + 1);
    c.stats = take(nparts * sizeof(TileStats) / sizeof(int));
    c.before = take(nparts > MAX_DIRECT ? nparts : 0);
    c.gstart = take(size_t(ngroups) + 1);
    c.wstart = take(size_t(nwarps) + 1);
    c.flag = take(1);
    c.bytes = at;
    return c;
}

void launch_core_prep(int value_type, int r, int nbr, const int* brptr, const uint8_t* headers, int ngroups, int nwarps,
                      const CoreScratch& c, unsigned char* mem, cudaStream_t s) {
    const int rows = part_rows(nbr), nparts = div_up(long(nbr) + 1, rows), ntiles = div_up(long(nbr) + 1, TILE);
    int* valptr = reinterpret_cast<int*>(mem + c.valptr);
    TileStats* stats = reinterpret_cast<TileStats*>(mem + c.stats);
    int* before = nparts > MAX_DIRECT ? reinterpret_cast<int*>(mem + c.before) : nullptr;
    auto count_r = [&](auto lt, auto RC) {
        using LT = decltype(lt);
        constexpr int R = decltype(RC)::value;
        auto kern = rows == TILE ? k_core_count<LT, R, TILE, L>
                                 : (rows == TILE / 4 ? k_core_count<LT, R, TILE / 4, L>
                                                     : k_core_count<LT, R, TILE / MOST_L, MOST_L>);
        kern<<<nparts, THREADS, 0, s>>>(nbr, brptr, headers, valptr, stats);
    };
    auto count = [&](auto lt) {
        using std::integral_constant;
        switch (r) {
            case 1: count_r(lt, integral_constant<int, 1>{}); return;
            case 2: count_r(lt, integral_constant<int, 2>{}); return;
            case 4: count_r(lt, integral_constant<int, 4>{}); return;
            case 8: count_r(lt, integral_constant<int, 8>{}); return;
        }
        throw Error(SPC5CUDA_ERR_FORMAT, "r must be 1, 2, 4 or 8");
    };
    if (value_type == SPC5CUDA_F32) count(float{});
    else count(double{});
    SPC5_CUDA(cudaGetLastError());
    if (before) {
        k_core_parts<<<1, THREADS, 0, s>>>(nparts, stats, before);
        SPC5_CUDA(cudaGetLastError());
    }
    launch_after(k_core_split, dim3(unsigned(ntiles)), THREADS, 0, !before, s, nbr, brptr, valptr, nparts, TILE / rows,
                 static_cast<const TileStats*>(stats), static_cast<const int*>(before), ngroups,
                 reinterpret_cast<int*>(mem + c.gstart), nwarps, reinterpret_cast<int*>(mem + c.wstart), value_type, r,
                 reinterpret_cast<int*>(mem + c.flag));
}

}  // namespace spc5cuda
