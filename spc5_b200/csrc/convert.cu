// convert.cu -- CSR -> beta(r,VS) conversion on the device, plus the scans
// and per-block-row offsets the SpMV kernels use.
//
// The conversion is the reference's greedy (core_CSR_to_SPC5_rVc,
// src/spc5.hpp:165-228; CSR_to_SPC5_1rVc 455-488) run as two passes over
// independent block-rows:
//   pass 1  counts[br]  = blocks of block-row br         (k_blockrow_counts)
//   scan    brptr       = exclusive scan of the counts   (== rowsSize after
//                                                         conversion, 220-227)
//   pass 2  headers + values of block-row br at brptr[br] and at the CSR
//           value offset rowptr[br*r]                    (k_emit)
// Inside a block-row the greedy is a sequential chain (the next block starts
// at the smallest unconsumed column of the r sub-rows); block-rows are
// independent.  At r = 1 a warp resolves 32 entries at a time (row_windows); at
// r > 1 one lane walks a short block-row and a warp a long one.  Values are
// copied bit for bit (at r = 1 they stay where they are), so the arrays equal
// the reference's exactly.
#include <climits>

#include "common.cuh"
#include "kernels.h"

namespace spc5cuda {

// ---------------------------------------------------------------------------
// exclusive scan (int32), three phases: tile sums, scan of tile sums, tiles
// ---------------------------------------------------------------------------

namespace {

constexpr int SCAN_THREADS = 256;
constexpr int SCAN_ITEMS = 8;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;

__device__ __forceinline__ int warp_inclusive_scan(int v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, v, d);
        if (lane >= d) v += t;
    }
    return v;
}

// Block-wide exclusive scan of one value per thread; returns the exclusive
// prefix and writes the block total to *total.
__device__ __forceinline__ int block_exclusive_scan(int v, int* total) {
    __shared__ int warp_sums[32];
    __shared__ int block_total;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nwarps = blockDim.x >> 5;
    const int inc = warp_inclusive_scan(v);
    if (lane == 31) warp_sums[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        const int w = lane < nwarps ? warp_sums[lane] : 0;
        const int wi = warp_inclusive_scan(w);
        if (lane < nwarps) warp_sums[lane] = wi - w;
        if (lane == 31) block_total = wi;
    }
    __syncthreads();
    const int res = inc - v + warp_sums[warp];
    if (total) *total = block_total;
    __syncthreads();
    return res;
}

__global__ void __launch_bounds__(SCAN_THREADS) k_tile_sums(const int* __restrict__ in, long n,
                                                            int* __restrict__ sums) {
    const long base = long(blockIdx.x) * SCAN_TILE;
    int s = 0;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        const long i = base + long(k) * SCAN_THREADS + threadIdx.x;
        if (i < n) s += in[i];
    }
    int total;
    block_exclusive_scan(s, &total);
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

// One CTA scans the tile sums in place (exclusive) and writes the grand
// total to sums[ntiles].
__global__ void __launch_bounds__(1024) k_scan_sums(int* __restrict__ sums, long ntiles) {
    __shared__ int carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (long b = 0; b < ntiles; b += blockDim.x) {
        const long i = b + threadIdx.x;
        const int v = i < ntiles ? sums[i] : 0;
        int total;
        const int ex = block_exclusive_scan(v, &total);
        const int c = carry;
        if (i < ntiles) sums[i] = c + ex;
        __syncthreads();
        if (threadIdx.x == 0) carry = c + total;
        __syncthreads();
    }
    if (threadIdx.x == 0) sums[ntiles] = carry;
}

__global__ void __launch_bounds__(SCAN_THREADS) k_scan_tiles(const int* in, int* out, long n,
                                                             const int* __restrict__ sums,
                                                             long ntiles) {
    const long base = long(blockIdx.x) * SCAN_TILE;
    // thread t owns items [base + t*ITEMS, +ITEMS): blocked arrangement
    int v[SCAN_ITEMS];
    int s = 0;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        const long i = base + long(threadIdx.x) * SCAN_ITEMS + k;
        v[k] = i < n ? in[i] : 0;
        s += v[k];
    }
    int running = block_exclusive_scan(s, nullptr) + sums[blockIdx.x];
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        const long i = base + long(threadIdx.x) * SCAN_ITEMS + k;
        if (i < n) out[i] = running;
        running += v[k];
    }
    if (blockIdx.x == ntiles - 1 && threadIdx.x == 0) out[n] = sums[ntiles];
}

}  // namespace

long scan_tmp_ints(long n) { return (n + SCAN_TILE - 1) / SCAN_TILE + 1; }

void exclusive_scan_i32(const int* in, int* out, long n, int* tmp, cudaStream_t s) {
    if (n <= 0) {
        SPC5_CUDA(cudaMemsetAsync(out, 0, sizeof(int), s));
        return;
    }
    const long ntiles = (n + SCAN_TILE - 1) / SCAN_TILE;
    k_tile_sums<<<unsigned(ntiles), SCAN_THREADS, 0, s>>>(in, n, tmp);
    k_scan_sums<<<1, 1024, 0, s>>>(tmp, ntiles);
    k_scan_tiles<<<unsigned(ntiles), SCAN_THREADS, 0, s>>>(in, out, n, tmp, ntiles);
    SPC5_CUDA(cudaGetLastError());
}

// ---------------------------------------------------------------------------
// CSR validation
// ---------------------------------------------------------------------------

namespace {

// Threads per CTA of the kernels that give a warp 32 rows: few, so that a CTA
// does not wait long for the warp with the most entries.
constexpr int ROW_THREADS = 64;

// Columns must ascend inside a row: of all entries whose column does not exceed
// the one before it (descents), each must be a row's first.  So the entries are
// streamed without regard to the rows, four per thread, and their descents
// counted; a thread per row then takes off the descents at rows' first entries.
// What is left is inside rows.  Bound by the stream of the columns.  (A warp per
// 32 rows, 32 entries at a time, waited for one load after the other: 116 us, now 23, on a
// power-law matrix of 15M entries, B200.)
//
// out[0] = largest error code, out[1] = descents inside rows (modulo 2^32; as
// many as entries at most, so 0 only without any).
__global__ void __launch_bounds__(256) k_validate_csr(int nrows, int ncols, long nnz, const int* __restrict__ rowptr,
                                                      const int* __restrict__ colidx, int* __restrict__ out) {
    const long tid = long(blockIdx.x) * blockDim.x + threadIdx.x;
    const long threads = long(gridDim.x) * blockDim.x;
    int worst = 0;
    unsigned descents = 0u;
    auto entry = [&](int c, int before) {
        if (unsigned(c) >= unsigned(ncols)) worst = max(worst, 2);
        descents += c <= before ? 1u : 0u;
    };
    if (tid == 0 && (rowptr[0] != 0 || long(rowptr[nrows]) != nnz)) worst = 1;
    const long quads = nnz / 4;
#pragma unroll 2
    for (long i = tid; i < quads; i += threads) {
        const int before = i > 0 ? __ldg(colidx + 4 * i - 1) : INT_MIN;
        const int4 c = __ldg(reinterpret_cast<const int4*>(colidx) + i);
        entry(c.x, before);
        entry(c.y, c.x);
        entry(c.z, c.y);
        entry(c.w, c.z);
    }
    if (tid < nnz % 4) {
        const long k = 4 * quads + tid;
        entry(colidx[k], k > 0 ? colidx[k - 1] : INT_MIN);
    }
#pragma unroll 4
    for (long row = tid; row < nrows; row += threads) {
        const int a = rowptr[row], b = rowptr[row + 1];
        if (b < a || a < 0 || long(b) > nnz) worst = max(worst, 1);
        else if (a < b && a > 0 && __ldg(colidx + a) <= __ldg(colidx + a - 1)) --descents;
    }
    worst = __reduce_max_sync(0xffffffffu, worst);
    descents = __reduce_add_sync(0xffffffffu, descents);
    if ((threadIdx.x & 31) == 0) {
        if (worst) atomicMax(out, worst);
        if (descents) atomicAdd(out + 1, int(descents));
    }
}

}  // namespace

void launch_validate_csr(int nrows, int ncols, long nnz, const int* rowptr, const int* colidx,
                         int* d_out, cudaStream_t s) {
    SPC5_CUDA(cudaMemsetAsync(d_out, 0, 2 * sizeof(int), s));
    const int blocks = std::max(1, std::min(div_up(std::max(nnz / 4, long(nrows)), 256), sm_count() * 8));
    k_validate_csr<<<blocks, 256, 0, s>>>(nrows, ncols, nnz, rowptr, colidx, d_out);
    SPC5_CUDA(cudaGetLastError());
}

// ---------------------------------------------------------------------------
// the greedy (spc5.hpp:186-218), one thread per block-row
// ---------------------------------------------------------------------------

namespace {

// A block-row of more than LONG_ENTRIES entries is walked by its whole warp
// (long_blocks), a shorter one by its own lane.  Headers and values on a B200,
// by lanes / by warps: stencil 100^3, r = 4 (108 entries) 1328 us / 361, r = 2 (54)
// 1216 / 622; Poisson 64^2, r = 8 (40, with few warps to share them) 26 / 79.
constexpr int LONG_ENTRIES = 48;

// The greedy over block-row br by one warp: L = 32 / R lanes per sub-row hold
// its next L columns.  Calls block(index, first column) per block, and per
// step put(sub-row's entry, bit, lane takes part) for the entries that go to
// that block; the lanes of a sub-row advance together.
template <int VS, int R, class B, class P>
__device__ __forceinline__ void long_blocks(int nrows, long br, const int* __restrict__ rowptr,
                                            const int* __restrict__ colidx, B&& block, P&& put) {
    constexpr int L = 32 / R;
    constexpr unsigned LMASK = (1u << L) - 1u;
    const int lane = threadIdx.x & 31;
    const int s = lane / L, t = lane % L;
    const long row = br * R + s;
    int head = row < nrows ? rowptr[row] : 0;
    const int end = row < nrows ? rowptr[row + 1] : 0;
    int c = t < end - head ? __ldg(colidx + head + t) : INT_MAX;
    for (int n = 0;; ++n) {
        const int idx = __reduce_min_sync(0xffffffffu, c);  // a sub-row's columns ascend: its lane 0 has its least
        if (idx == INT_MAX) break;
        block(n, idx);
        for (;;) {
            const bool take = c != INT_MAX && c - idx < VS;
            const unsigned all = __ballot_sync(0xffffffffu, take);
            if (all == 0u) break;
            const int k = __popc((all >> (s * L)) & LMASK);  // a prefix of the sub-row's lanes
            put(head + t, c - idx, take, s);
            if (k > 0) {
                head += k;
                c = t < end - head ? __ldg(colidx + head + t) : INT_MAX;
            }
        }
    }
}

// per (a power of two up to 32): block-rows that a warp takes at a time, so that
// few long block-rows do not queue up behind one another in few warps
// (block_rows_per_warp).
template <int VS, int R>
__global__ void __launch_bounds__(256) k_blockrow_counts(int nrows, int nbr, int per,
                                                         const int* __restrict__ rowptr,
                                                         const int* __restrict__ colidx,
                                                         int* __restrict__ counts) {
    const int lane = threadIdx.x & 31;
    const long warps = long(gridDim.x) * blockDim.x / 32;
    for (long b0 = (long(blockIdx.x) * blockDim.x + threadIdx.x) / 32 * per; b0 < nbr; b0 += warps * per) {  // warp-uniform
        const long br = b0 + lane;
        const bool mine = lane < per && br < nbr;
        const long row0 = br * R;
        int head[R], end[R];
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const bool ok = mine && row0 + i < nrows;
            head[i] = ok ? rowptr[row0 + i] : 0;
            end[i] = ok ? rowptr[row0 + i + 1] : 0;
        }
        int entries = 0;
#pragma unroll
        for (int i = 0; i < R; ++i) entries += end[i] - head[i];
        const bool by_warp = entries > LONG_ENTRIES;
        int cnt = 0;
        if (!by_warp) {
            for (;;) {
                bool have = false;
                int idx = INT_MAX;
#pragma unroll
                for (int i = 0; i < R; ++i) {
                    if (head[i] < end[i]) {
                        have = true;
                        idx = min(idx, __ldg(colidx + head[i]));
                    }
                }
                if (!have) break;
                ++cnt;
#pragma unroll
                for (int i = 0; i < R; ++i) {
                    // columns inside a row ascend, so col >= idx: col < idx + VS
                    // is col - idx < VS without the int overflow of idx + VS
                    while (head[i] < end[i] && __ldg(colidx + head[i]) - idx < VS) ++head[i];
                }
            }
        }
        unsigned todo = __ballot_sync(0xffffffffu, by_warp);
        while (todo) {
            const int l = __ffs(todo) - 1;
            todo &= todo - 1u;
            int n = 0;
            long_blocks<VS, R>(nrows, b0 + l, rowptr, colidx, [&](int k, int) { n = k + 1; },
                               [](int, int, bool, int) {});
            if (lane == l) cnt = n;
        }
        if (mine) counts[br] = cnt;
    }
}

// Headers of every block-row, and its values in block order.
template <int VS, int R, class V>
__global__ void __launch_bounds__(256) k_emit(int nrows, int nbr, int per, const int* __restrict__ rowptr,
                                              const int* __restrict__ colidx,
                                              const V* __restrict__ vin,
                                              const int* __restrict__ brptr,
                                              uint8_t* __restrict__ headers, V* __restrict__ vout) {
    constexpr int MB = VS == 8 ? 1 : 2;
    constexpr int STRIDE = 4 + R * MB;
    constexpr int L = 32 / R;
    const int lane = threadIdx.x & 31;
    const long warps = long(gridDim.x) * blockDim.x / 32;
    for (long b0 = (long(blockIdx.x) * blockDim.x + threadIdx.x) / 32 * per; b0 < nbr; b0 += warps * per) {  // warp-uniform
        const long br = b0 + lane;
        const bool mine = lane < per && br < nbr;
        const long row0 = br * R;
        int head[R], end[R];
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const bool ok = mine && row0 + i < nrows;
            head[i] = ok ? rowptr[row0 + i] : 0;
            end[i] = ok ? rowptr[row0 + i + 1] : 0;
        }
        int entries = 0;
#pragma unroll
        for (int i = 0; i < R; ++i) entries += end[i] - head[i];
        const bool by_warp = entries > LONG_ENTRIES;
        if (!by_warp && entries > 0) {
            long vo = head[0];
            uint8_t* h = headers + long(brptr[br]) * STRIDE;
            for (;;) {
                bool have = false;
                int idx = INT_MAX;
#pragma unroll
                for (int i = 0; i < R; ++i) {
                    if (head[i] < end[i]) {
                        have = true;
                        idx = min(idx, __ldg(colidx + head[i]));
                    }
                }
                if (!have) break;
                h[0] = uint8_t(idx);
                h[1] = uint8_t(idx >> 8);
                h[2] = uint8_t(idx >> 16);
                h[3] = uint8_t(idx >> 24);
#pragma unroll
                for (int i = 0; i < R; ++i) {
                    uint32_t m = 0;
                    while (head[i] < end[i]) {
                        const int d = __ldg(colidx + head[i]) - idx;
                        if (d >= VS) break;
                        vout[vo++] = vin[head[i]];
                        m |= 1u << d;
                        ++head[i];
                    }
                    h[4 + i * MB] = uint8_t(m);
                    if (MB == 2) h[5 + i * MB] = uint8_t(m >> 8);
                }
                h += STRIDE;
            }
        }
        unsigned todo = __ballot_sync(0xffffffffu, by_warp);
        while (todo) {
            const int l = __ffs(todo) - 1;
            todo &= todo - 1u;
            const long b = b0 + l;
            uint8_t* h = headers + long(brptr[b]) * STRIDE;
            // a block's masks are complete when the next block begins; the
            // values of its sub-rows follow one another
            const int s = lane / L;
            long vo = rowptr[b * R];  // the block's first value
            uint32_t mask = 0u;       // of the lane's sub-row
            int first = 0;            // the sub-row's first entry in this block
            auto close = [&]() {
                if (lane % L == 0) {
                    h[4 + s * MB] = uint8_t(mask);
                    if (MB == 2) h[5 + s * MB] = uint8_t(mask >> 8);
                }
                // values of the sub-rows up to this one, of the whole block
                const int n = __popc(mask);
                int upto = n;
#pragma unroll
                for (int d = L; d < 32; d <<= 1) {
                    const int u = __shfl_up_sync(0xffffffffu, upto, d);
                    if (lane >= d) upto += u;
                }
                for (int k = lane % L; k < n; k += L) vout[vo + upto - n + k] = vin[first + k];
                vo += __shfl_sync(0xffffffffu, upto, 31);
                h += STRIDE;
                mask = 0u;
            };
            bool open = false;
            long_blocks<VS, R>(nrows, b, rowptr, colidx,
                               [&](int, int idx) {
                                   if (open) close();
                                   open = true;
                                   if (lane < 4) h[lane] = uint8_t(uint32_t(idx) >> (8 * lane));
                               },
                               [&](int entry, int d, bool take, int) {
                                   // the sub-row's lanes agree on its mask; its first entry
                                   // is the one its lane 0 takes first
                                   const int e0 = __shfl_sync(0xffffffffu, entry, lane / L * L);
                                   if (mask == 0u) first = e0;
                                   uint32_t m = take ? 1u << d : 0u;
#pragma unroll
                                   for (int x = L / 2; x >= 1; x >>= 1) m |= __shfl_xor_sync(0xffffffffu, m, x);
                                   mask |= m;
                               });
            if (open) close();
        }
    }
}

// r = 1: a warp takes 32 rows, whose entries are one range, 32 at a time.
// Every row's first entry starts a block; from there block starts follow from
// one another, entry p's next block being at the first entry of the row past
// column + VS.  All 32 successors are found at once, and the starts reachable
// from the window's (its first entry, the rows' first ones, entries VS or more
// past the one before) by doubling.  A
// window ends before its last block unless nothing follows, so that its blocks
// are complete.  Calls put(window's first entry, its blocks, the starts, the
// lane's column, one past the entries of the block that the lane's entry would
// start).
//
// One lane per row (and a warp per long row) was bound by the chain of one
// row's loads: power-law, 1M rows, 15M entries, counts 538 us and headers
// 910 us on a B200; now 191 and 238.
template <int VS, class P>
__device__ __forceinline__ void row_windows(int a, int b, bool in, long k0, long k1, const int* __restrict__ colidx,
                                            P&& put) {
    constexpr unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    // columns of entries [q, q + 32), the next 32 and the 32 after those
    long q = k0;
    auto load = [&](long at) { return at + lane < k1 ? __ldg(colidx + at + lane) : 0; };
    int c0 = load(q), c1 = load(q + 32), c2 = load(q + 64);
    for (long k = k0; k < k1;) {
        const int n = int(min(32L, k1 - k));
        if (k - q >= 32) {
            q += 32;
            c0 = c1;
            c1 = c2;
            c2 = load(q + 64);
        }
        const int off = int(k - q) + lane;
        const int lo = __shfl_sync(FULL, c0, off & 31), hi = __shfl_sync(FULL, c1, off & 31);
        const int c = off < 32 ? lo : hi;
        const unsigned row_starts = __reduce_or_sync(FULL, in && a < b && a >= k && a - k < n ? 1u << (a - k) : 0u);
        const unsigned above = lane == 31 ? 0u : row_starts & (FULL << (lane + 1));
        const int row_end = above ? __ffs(above) - 1 : n;  // of the lane's row, in this window
        int last = lane;                                   // the block's last entry
#pragma unroll
        for (int d = VS / 2; d >= 1; d >>= 1) {
            const int cc = __shfl_sync(FULL, c, (last + d) & 31);
            if (last + d < row_end && cc - c < VS) last += d;
        }
        const int before = __shfl_up_sync(FULL, c, 1);
        unsigned starts = row_starts | 1u | __ballot_sync(FULL, lane > 0 && lane < row_end && c - before >= VS);
        int jump = last + 1;
#pragma unroll
        for (int i = 0; i < 5; ++i) {
            const unsigned more =
                starts | __reduce_or_sync(FULL, ((starts >> lane) & 1u) && jump < n ? 1u << jump : 0u);
            if (more == starts) break;  // closed under this many steps and so under all
            starts = more;
            const int next = __shfl_sync(FULL, jump, jump & 31);
            jump = jump < n ? next : 32;
        }
        int used = n;
        if (k + n < k1) {  // a full window: its last start is not its first
            used = 31 - __clz(starts);
            starts ^= 1u << used;
        }
        put(k, starts, c, last + 1);
        k += used;
    }
}

__device__ __forceinline__ unsigned bits_below(long n) {
    return n <= 0 ? 0u : (n >= 32 ? 0xffffffffu : (1u << int(n)) - 1u);
}

// EMIT: the headers at brptr, else the blocks per row.
template <int VS, bool EMIT>
__global__ void __launch_bounds__(ROW_THREADS) k_rows1(int nrows, const int* __restrict__ rowptr,
                                               const int* __restrict__ colidx, const int* __restrict__ brptr,
                                               int* __restrict__ counts, uint8_t* __restrict__ headers) {
    constexpr int MB = VS == 8 ? 1 : 2;
    constexpr int STRIDE = 4 + MB;
    const int lane = threadIdx.x & 31;
    const long warps = long(gridDim.x) * blockDim.x / 32;
    for (long r0 = (long(blockIdx.x) * blockDim.x + threadIdx.x) / 32 * 32; r0 < nrows; r0 += warps * 32) {
        const long row = r0 + lane;
        const bool in = row < nrows;
        const int a = in ? rowptr[row] : 0, b = in ? rowptr[row + 1] : 0;
        const int last = int(min(31L, nrows - 1 - r0));
        const long k0 = __shfl_sync(0xffffffffu, a, 0), k1 = __shfl_sync(0xffffffffu, b, last);
        if constexpr (EMIT) {
            long at = brptr[r0];
            row_windows<VS>(a, b, in, k0, k1, colidx, [&](long, unsigned starts, int c, int end) {
                const bool mine = (starts >> lane) & 1u;
                const int len = mine ? end - lane : 0;
                const int longest = __reduce_max_sync(0xffffffffu, len);
                uint32_t m = 1u;
                for (int d = 1; d < longest; ++d) {
                    const int cc = __shfl_down_sync(0xffffffffu, c, d);
                    if (d < len) m |= 1u << (cc - c);
                }
                if (mine) {
                    uint8_t* h = headers + (at + __popc(starts & bits_below(lane))) * STRIDE;
                    h[0] = uint8_t(c);
                    h[1] = uint8_t(c >> 8);
                    h[2] = uint8_t(c >> 16);
                    h[3] = uint8_t(c >> 24);
                    h[4] = uint8_t(m);
                    if (MB == 2) h[5] = uint8_t(m >> 8);
                }
                at += __popc(starts);
            });
        } else {
            int cnt = 0;
            row_windows<VS>(a, b, in, k0, k1, colidx, [&](long k, unsigned starts, int, int) {
                cnt += __popc(starts & bits_below(b - k) & ~bits_below(a - k));
            });
            if (in) counts[row] = cnt;
        }
    }
}

__global__ void k_valptr_from_csr(int r, int nrows, int nbr, const int* __restrict__ rowptr,
                                  int* __restrict__ valptr) {
    for (long br = long(blockIdx.x) * blockDim.x + threadIdx.x; br <= nbr;
         br += long(gridDim.x) * blockDim.x) {
        const long row = br * r < nrows ? br * r : nrows;
        valptr[br] = rowptr[row];
    }
}

template <int MB>
__global__ void __launch_bounds__(256) k_value_counts(int r, int nbr, const int* __restrict__ brptr,
                                                      const uint8_t* __restrict__ headers,
                                                      int* __restrict__ counts) {
    const int stride = 4 + r * MB;
    for (long br = long(blockIdx.x) * blockDim.x + threadIdx.x; br < nbr;
         br += long(gridDim.x) * blockDim.x) {
        int s = 0;
        for (long b = brptr[br]; b < brptr[br + 1]; ++b) {
            const uint8_t* h = headers + b * stride + 4;
            for (int k = 0; k < r * MB; ++k) s += __popc(uint32_t(h[k]));
        }
        counts[br] = s;
    }
}

// Block-rows per warp of the passes over block-rows: 32, fewer until there are 32
// warps per SM.  With 32 always, 50,000 rows of 400 values at r = 4 (391 warps)
// took 28.1 ms to convert on a B200.
int block_rows_per_warp(int nbr) {
    int per = 32;
    while (per > 1 && nbr / per < sm_count() * 32) per /= 2;
    return per;
}

template <int VS, int R>
void counts_r(int nrows, const int* rowptr, const int* colidx, int* counts, cudaStream_t s) {
    const int nbr = div_up(nrows, R);
    const int threads = 256, per = block_rows_per_warp(nbr);
    const int blocks = std::max(1, std::min(div_up(nbr, threads / 32 * per), sm_count() * 16));
    if constexpr (R == 1)
        k_rows1<VS, false><<<div_up(nrows, ROW_THREADS), ROW_THREADS, 0, s>>>(nrows, rowptr, colidx, nullptr, counts, nullptr);
    else
        k_blockrow_counts<VS, R><<<blocks, threads, 0, s>>>(nrows, nbr, per, rowptr, colidx, counts);
}

template <int VS, int R, class V>
void emit_r(int nrows, const int* rowptr, const int* colidx, const void* vin, const int* brptr,
            uint8_t* headers, void* vout, cudaStream_t s) {
    const int nbr = div_up(nrows, R);
    const int threads = 256, per = block_rows_per_warp(nbr);
    const int blocks = std::max(1, std::min(div_up(nbr, threads / 32 * per), sm_count() * 16));
    if constexpr (R == 1)
        k_rows1<VS, true><<<div_up(nrows, ROW_THREADS), ROW_THREADS, 0, s>>>(nrows, rowptr, colidx, brptr, nullptr, headers);
    else
        k_emit<VS, R, V><<<blocks, threads, 0, s>>>(nrows, nbr, per, rowptr, colidx, static_cast<const V*>(vin), brptr,
                                                    headers, static_cast<V*>(vout));
}

}  // namespace

void launch_blockrow_counts(int vs, int r, int nrows, const int* rowptr, const int* colidx,
                            int* counts, cudaStream_t s) {
    if (nrows <= 0) return;
#define SPC5_COUNTS(VS_, R_) \
    if (vs == VS_ && r == R_) { counts_r<VS_, R_>(nrows, rowptr, colidx, counts, s); }
    SPC5_COUNTS(8, 1) else SPC5_COUNTS(8, 2) else SPC5_COUNTS(8, 4) else SPC5_COUNTS(8, 8)
    else SPC5_COUNTS(16, 1) else SPC5_COUNTS(16, 2) else SPC5_COUNTS(16, 4) else SPC5_COUNTS(16, 8)
    else throw Error(SPC5CUDA_ERR_FORMAT, "unsupported (VS, r)");
#undef SPC5_COUNTS
    SPC5_CUDA(cudaGetLastError());
}

void launch_emit(int vs, int r, int nrows, const int* rowptr, const int* colidx, const void* vin,
                 int value_bytes, const int* brptr, uint8_t* headers, void* vout, cudaStream_t s) {
    if (nrows <= 0) return;
    if (value_bytes == 8) {
#define SPC5_EMIT(VS_, R_) \
    if (vs == VS_ && r == R_) { emit_r<VS_, R_, double>(nrows, rowptr, colidx, vin, brptr, headers, vout, s); }
        SPC5_EMIT(8, 1) else SPC5_EMIT(8, 2) else SPC5_EMIT(8, 4) else SPC5_EMIT(8, 8)
        else SPC5_EMIT(16, 1) else SPC5_EMIT(16, 2) else SPC5_EMIT(16, 4) else SPC5_EMIT(16, 8)
        else throw Error(SPC5CUDA_ERR_FORMAT, "unsupported (VS, r)");
#undef SPC5_EMIT
    } else if (value_bytes == 4) {
#define SPC5_EMIT(VS_, R_) \
    if (vs == VS_ && r == R_) { emit_r<VS_, R_, float>(nrows, rowptr, colidx, vin, brptr, headers, vout, s); }
        SPC5_EMIT(8, 1) else SPC5_EMIT(8, 2) else SPC5_EMIT(8, 4) else SPC5_EMIT(8, 8)
        else SPC5_EMIT(16, 1) else SPC5_EMIT(16, 2) else SPC5_EMIT(16, 4) else SPC5_EMIT(16, 8)
        else throw Error(SPC5CUDA_ERR_FORMAT, "unsupported (VS, r)");
#undef SPC5_EMIT
    } else {
        throw Error(SPC5CUDA_ERR_INVALID, "value size must be 4 or 8");
    }
    SPC5_CUDA(cudaGetLastError());
}

void launch_valptr_from_csr(int r, int nrows, const int* rowptr, int* valptr, cudaStream_t s) {
    const int nbr = div_up(nrows, r);
    const int threads = 256;
    const int blocks = std::max(1, std::min(div_up(long(nbr) + 1, threads), sm_count() * 16));
    k_valptr_from_csr<<<blocks, threads, 0, s>>>(r, nrows, nbr, rowptr, valptr);
    SPC5_CUDA(cudaGetLastError());
}

void launch_blockrow_value_counts(int mask_bytes, int r, int nbr, const int* brptr,
                                  const uint8_t* headers, int* counts, cudaStream_t s) {
    if (nbr <= 0) return;
    const int threads = 256;
    const int blocks = std::max(1, std::min(div_up(nbr, threads), sm_count() * 16));
    if (mask_bytes == 1)
        k_value_counts<1><<<blocks, threads, 0, s>>>(r, nbr, brptr, headers, counts);
    else
        k_value_counts<2><<<blocks, threads, 0, s>>>(r, nbr, brptr, headers, counts);
    SPC5_CUDA(cudaGetLastError());
}

}  // namespace spc5cuda
