// plan.cu -- the sorted SpMV plan of a matrix with irregular block-rows.
//
// Power-law and other irregular matrices mix block-rows of one block with
// block-rows of hundreds; no single work split suits both.  The plan sorts the
// rows of the matrix by size and stores the long ones as warp streams or as chains
// (chain_rows says which) and the short ones one per lane (stream.cuh): every chain
// of multiply-adds keeps its values in block order, so y is bit-identical.  The plan
// holds the only copy of the values; the handle keeps the reference-order headers, from
// which the values can be put back in the reference order (rebuild_values).
//
// Build, all on the device: row-blocks and values of every row (k_row_stats),
// a radix sort of the rows by size, the sizes of the long rows' slabs
// (k_slab_size) and their scans, then one warp per slab writes its masks, x
// indices and values (k_stream_fill, k_short_fill).  The chains: their lengths
// (k_chain_len), a radix sort by length class, the slabs (k_chain_slabs), then one
// warp per row writes its entries (k_chain_fill).
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include <algorithm>

#include "stream.cuh"

namespace spc5cuda {

namespace {

using namespace stream;

int grid_for(long n, int threads, int per_sm = 16) {
    return std::max(1, std::min(div_up(n, threads), sm_count() * per_sm));
}

// Sort key and values of every row (0 .. nrows), and the row ids: VS lanes per
// block-row, lane j takes the blocks j, j + VS, ...
template <class LT, int R>
__global__ void __launch_bounds__(256) k_row_stats(int nrows, int nbr, const int* __restrict__ brptr,
                                                   const uint8_t* __restrict__ hdr, int* __restrict__ key,
                                                   int* __restrict__ rv, int* __restrict__ ids) {
    constexpr int VS = Layout<LT>::VS;
    const int c = threadIdx.x & (VS - 1);
    const long step = long(gridDim.x) * blockDim.x / VS;
    const long first = (long(blockIdx.x) * blockDim.x + threadIdx.x) / VS;
    for (long i0 = first - first % (32 / VS); i0 < nbr; i0 += step) {  // warp-uniform
        const long i = i0 + first % (32 / VS);
        const bool has = i < nbr;
        const long b0 = has ? brptr[i] : 0, b1 = has ? brptr[i + 1] : 0;
        int n[R], v[R];
#pragma unroll
        for (int s = 0; s < R; ++s) n[s] = v[s] = 0;
        for (long b = b0 + c; b < b1; b += VS) {
            uint32_t mw[Header<LT, R>::MASK_WORDS];
            load_header<LT, R>(hdr, b, mw);
#pragma unroll
            for (int s = 0; s < R; ++s) {
                const uint32_t m = mask_of<LT, R>(mw, s);
                n[s] += m ? 1 : 0;
                v[s] += __popc(m);
            }
        }
#pragma unroll
        for (int s = 0; s < R; ++s) {
#pragma unroll
            for (int d = VS / 2; d >= 1; d >>= 1) {
                n[s] += __shfl_xor_sync(FULL, n[s], d);
                v[s] += __shfl_xor_sync(FULL, v[s], d);
            }
            const long row = i * R + s;
            if (has && c == s % VS && row < nrows) {
                key[row] = v[s] <= SHORT_VALUES ? v[s] : LONG_KEY + n[s];
                rv[row] = v[s];
                ids[row] = int(row);
            }
        }
    }
}

constexpr int OCTAVES = CLASSES + SHORT_VALUES + 1;
struct Counts {
    int rows[OCTAVES + 31];
    int longest;                // row-blocks of the longest row
    unsigned long long blocks;  // of all long rows
};

// rows[j] = sorted rows of more than class_min(j) row-blocks (the last class
// takes the long rows' rest); rows[CLASSES + n] = sorted rows of at least n
// values (all long rows among them); rows[OCTAVES + b] = sorted rows of at least
// 2^b row-blocks.
__global__ void k_class_counts(int nrows, const int* __restrict__ key, Counts* __restrict__ out) {
    unsigned long long blocks = 0;
    for (long i = long(blockIdx.x) * blockDim.x + threadIdx.x; i < nrows; i += long(gridDim.x) * blockDim.x) {
        const int k = key[i], next = i + 1 < nrows ? key[i + 1] : -1;
        blocks += static_cast<unsigned long long>(max(k - LONG_KEY, 0));
        if (i == 0) out->longest = max(k - LONG_KEY, 0);
        if (k == next) continue;
#pragma unroll
        for (int j = 0; j < CLASSES; ++j) {
            const int least = LONG_KEY + class_min(j);
            if (k > least && next <= least) out->rows[j] = int(i + 1);
        }
        for (int b = 0; b < 31; ++b) {
            const long least = LONG_KEY + (1L << b);
            if (k >= least && next < least) out->rows[OCTAVES + b] = int(i + 1);
        }
        for (int n = max(next + 1, 0); n <= min(k, SHORT_VALUES); ++n) out->rows[CLASSES + n] = int(i + 1);
    }
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1) blocks += __shfl_xor_sync(FULL, blocks, d);
    if ((threadIdx.x & 31) == 0 && blocks) atomicAdd(&out->blocks, blocks);
}

// Steps and values of every slab.
template <int G>
__global__ void k_slab_size(View p, int nslabs, const int* __restrict__ rv, int* __restrict__ nstep,
                            int* __restrict__ nval) {
    for (long s = long(blockIdx.x) * blockDim.x + threadIdx.x; s < nslabs; s += long(gridDim.x) * blockDim.x) {
        const SlabRows sr = slab_rows<G>(p, int(s));
        int steps = 0, vals = 0;
        for (int i = sr.row0; i < sr.row_end; ++i) {
            if ((i - sr.row0) % G == 0) steps += p.key[i] - LONG_KEY;  // the round's longest row
            vals += rv[p.perm[i]];
        }
        nstep[s] = steps;
        nval[s] = vals;
    }
}

constexpr int FILL_THREADS = 64;

// One warp per slab, in step order, VS steps at a time.  A group decodes its
// row's next VS blocks (lane j block j: its column, the row's mask and the
// offset of the row's first value in it, by a scan of the blocks' value counts)
// and queues its row-blocks until it has VS of them; lane c of every group then
// places row-block c of the queue.  Step by step, with a value's latency in each,
// a power-law matrix (1M rows, 15M values, r = 1) took 467 us on a B200, now
// 243.  BACK: the values only, from the streams back to the reference order
// (out), else the slab's masks, x indices and values.
template <class LT, int R, class V, bool BACK>
__global__ void __launch_bounds__(FILL_THREADS) k_stream_fill(View p, int nslabs, const int* __restrict__ brptr,
                                                     const int* __restrict__ valptr,
                                                     const uint8_t* __restrict__ hdr, const V* __restrict__ in,
                                                     V* __restrict__ out, uint32_t* __restrict__ mask,
                                                     int* __restrict__ xcol) {
    constexpr int VS = Layout<LT>::VS, G = 32 / VS, Q = 2 * VS;
    constexpr int MW = Header<LT, R>::MASK_WORDS;
    constexpr uint32_t VSMASK = (1u << VS) - 1u;
    constexpr int U = 4;  // values in flight per lane
    struct Entry {
        int col, v;
        uint32_t m;
    };
    __shared__ Entry queue[FILL_THREADS / 32][G][Q];
    const int lane = threadIdx.x & 31;
    const int g = lane / VS, c = lane % VS;
    Entry* const mine = queue[threadIdx.x >> 5][g];
    const uint32_t below = (1u << c) - 1u, groups_below = (1u << (g * VS)) - 1u;
    const long warps = long(gridDim.x) * blockDim.x / 32;
    for (long slab = (long(blockIdx.x) * blockDim.x + threadIdx.x) / 32; slab < nslabs; slab += warps) {
        const SlabRows sr = slab_rows<G>(p, int(slab));
        long step = p.sstep[slab], base = p.sval[slab];  // the next step, its first value
        for (int q = 0; sr.row0 + q * G < sr.row_end; ++q) {
            const int at = sr.row0 + q * G + g;
            const bool valid = at < sr.row_end;
            const int nb = p.key[sr.row0 + q * G] - LONG_KEY;
            const int row = valid ? p.perm[at] : 0;
            const int br = row / R, s = row % R;
            int b = valid ? brptr[br] : 0;
            const int b_end = valid ? brptr[br + 1] : 0;
            int v_next = valid ? valptr[br] : 0;
            int head = 0, have = 0;  // the queue: have entries from head
            for (int k = 0; k < nb; k += VS) {
                while (__any_sync(FULL, have < VS && b < b_end)) {
                    const bool need = have < VS && b < b_end;
                    int col = 0, tot = 0, low = 0;
                    uint32_t m = 0u;
                    if (need && b + c < b_end) {
                        uint32_t mw[MW];
                        col = load_header<LT, R>(hdr, long(b) + c, mw);
#pragma unroll
                        for (int i = 0; i < R; ++i) {
                            const uint32_t mi = mask_of<LT, R>(mw, i);
                            tot += __popc(mi);
                            low += i < s ? __popc(mi) : 0;
                            m = i == s ? mi : m;
                        }
                    }
                    int incl = tot;
#pragma unroll
                    for (int d = 1; d < VS; d <<= 1) {
                        const int t = __shfl_up_sync(FULL, incl, d, VS);
                        if (c >= d) incl += t;
                    }
                    const int all = __shfl_sync(FULL, incl, VS - 1, VS);
                    const uint32_t some = (__ballot_sync(FULL, m != 0u) >> (g * VS)) & VSMASK;
                    if (m != 0u)
                        mine[(head + have + __popc(some & below)) % Q] = Entry{col, v_next + incl - tot + low, m};
                    if (need) {
                        have += __popc(some);
                        v_next += all;
                        b += VS;
                    }
                }
                __syncwarp();
                Entry e{0, 0, 0u};
                if (c < have) e = mine[(head + c) % Q];
                __syncwarp();  // read before the next entries are queued
                head = (head + min(have, VS)) % Q;
                have -= min(have, VS);
                uint32_t M = 0u;  // of step k + c; 0 past the round's last step
#pragma unroll
                for (int i = 0; i < G; ++i) M |= __shfl_sync(FULL, e.m, i * VS + c) << (i * VS);
                int incl = __popc(M);
#pragma unroll
                for (int d = 1; d < VS; d <<= 1) {
                    const int t = __shfl_up_sync(FULL, incl, d, VS);
                    if (c >= d) incl += t;
                }
                long to = base + incl - __popc(M) + __popc(M & groups_below), from = e.v;
                if (!BACK && g == 0 && c < nb - k) mask[step + c] = M;
                base += __shfl_sync(FULL, incl, VS - 1);
                step += min(VS, nb - k);
                for (uint32_t left = e.m; left != 0u;) {
                    const int n = __popc(left);
                    V v[U];
#pragma unroll
                    for (int u = 0; u < U; ++u)
                        if (u < n) v[u] = in[(BACK ? to : from) + u];
#pragma unroll
                    for (int u = 0; u < U; ++u)
                        if (u < n) {
                            out[(BACK ? from : to) + u] = v[u];
                            if (!BACK) xcol[to + u] = e.col + __ffs(left) - 1;
                            left &= left - 1u;
                        }
                    to += U;
                    from += U;
                }
                __syncwarp();
            }
        }
    }
}

// One warp per slab of short rows, one lane per row: a first walk over the
// row's blocks counts its chains, a second one places its values in chain
// order.  BACK: the values only, back to the reference order.
template <class LT, int R, class V, bool BACK>
__global__ void __launch_bounds__(256) k_short_fill(View p, const int* __restrict__ brptr,
                                                    const int* __restrict__ valptr, const uint8_t* __restrict__ hdr,
                                                    const V* __restrict__ in, V* __restrict__ out,
                                                    uint16_t* __restrict__ chains_of, int* __restrict__ xcol) {
    constexpr int VS = Layout<LT>::VS;
    constexpr int MW = Header<LT, R>::MASK_WORDS;
    const int lane = threadIdx.x & 31;
    const long warps = long(gridDim.x) * blockDim.x / 32;
    for (long slab = (long(blockIdx.x) * blockDim.x + threadIdx.x) / 32; slab < p.short_slabs(); slab += warps) {
        const ShortRows sr = short_rows(p, int(slab));
        const int at = sr.row0 + lane;
        const long e0 = sr.at + lane;
        uint32_t chains = 0u;
        int len = 0;
        if (lane < sr.rows) {
            const int row = p.perm[at];
            const int br = row / R, s = row % R;
            const int b0 = brptr[br], b1 = brptr[br + 1];
            int pos[VS], first[VS];
#pragma unroll
            for (int c = 0; c < VS; ++c) pos[c] = 0;
            for (int b = b0; b < b1; ++b) {
                uint32_t mw[MW];
                load_header<LT, R>(hdr, b, mw);
                uint32_t m = 0u;
#pragma unroll
                for (int i = 0; i < R; ++i) m = i == s ? mask_of<LT, R>(mw, i) : m;
#pragma unroll
                for (int c = 0; c < VS; ++c) pos[c] += int((m >> c) & 1u);
            }
#pragma unroll
            for (int c = 0; c < VS; ++c) {
                chains |= pos[c] ? 1u << c : 0u;
                const int n = pos[c];
                first[c] = pos[c] = len;
                len += n;
            }
            long v = valptr[br];
            for (int b = b0; b < b1; ++b) {
                uint32_t mw[MW];
                const int col = load_header<LT, R>(hdr, b, mw);
                uint32_t m = 0u;
                int tot = 0, low = 0;
#pragma unroll
                for (int i = 0; i < R; ++i) {
                    const uint32_t mi = mask_of<LT, R>(mw, i);
                    tot += __popc(mi);
                    low += i < s ? __popc(mi) : 0;
                    m = i == s ? mi : m;
                }
                long ref = v + low;
#pragma unroll
                for (int c = 0; c < VS; ++c) {
                    if ((m >> c) & 1u) {
                        const long e = e0 + 32L * pos[c];
                        if constexpr (BACK) {
                            out[ref] = in[e];
                        } else {
                            out[e] = in[ref];
                            xcol[e] = int(uint32_t(col + c) | (pos[c] == first[c] ? FIRST : 0u));
                        }
                        ++pos[c];
                        ++ref;
                    }
                }
                v += tot;
            }
        }
        if constexpr (!BACK) chains_of[slab * 32 + lane] = uint16_t(chains);
    }
}

// Length class of a chain of n entries: n itself below 8, then eight classes per
// octave (monotone in n; the lengths of one class differ by an eighth at most).
__device__ __forceinline__ int length_class(int n) {
    if (n < 8) return n;
    const int b = 31 - __clz(n);
    return 8 * (b - 2) + ((n >> (b - 3)) & 7);
}
constexpr int CLASS_BITS = 8;  // of a class: below 8 * 29

// Chain ids i VS + c, their entries and length classes, and the rows' masks of
// non-empty chains, for the first nrows sorted rows, a warp per row; totals: their
// values, the non-empty chains.
template <class LT, int R>
__global__ void __launch_bounds__(256) k_chain_len(int nrows, const int* __restrict__ perm, const int* __restrict__ brptr,
                                                   const uint8_t* __restrict__ hdr, int* __restrict__ len,
                                                   int* __restrict__ cls, int* __restrict__ ids,
                                                   uint16_t* __restrict__ mask, unsigned long long* __restrict__ totals) {
    constexpr int VS = Layout<LT>::VS;
    const int lane = threadIdx.x & 31;
    const long warps = long(gridDim.x) * blockDim.x / 32;
    for (long i = (long(blockIdx.x) * blockDim.x + threadIdx.x) / 32; i < nrows; i += warps) {
        const int row = perm[i], br = row / R, s = row % R;
        const long b1 = brptr[br + 1];
        int n[VS];
#pragma unroll
        for (int c = 0; c < VS; ++c) n[c] = 0;
        for (long b = brptr[br] + lane; b < b1; b += 32) {
            uint32_t mw[Header<LT, R>::MASK_WORDS];
            load_header<LT, R>(hdr, b, mw);
            uint32_t m = 0u;
#pragma unroll
            for (int q = 0; q < R; ++q) m = q == s ? mask_of<LT, R>(mw, q) : m;
#pragma unroll
            for (int c = 0; c < VS; ++c) n[c] += int((m >> c) & 1u);
        }
        int mine = 0, all = 0;  // lane c: chain c
#pragma unroll
        for (int c = 0; c < VS; ++c) {
            const int t = int(__reduce_add_sync(FULL, unsigned(n[c])));
            mine = lane == c ? t : mine;
            all += t;
        }
        const uint32_t some = __ballot_sync(FULL, lane < VS && mine > 0);
        if (lane < VS) {
            len[i * VS + lane] = mine;
            cls[i * VS + lane] = length_class(mine);
            ids[i * VS + lane] = int(i * VS + lane);
        }
        if (lane == 0) {
            mask[i] = uint16_t(some);
            atomicAdd(totals, static_cast<unsigned long long>(all));
            atomicAdd(totals + 1, static_cast<unsigned long long>(__popc(some)));
        }
    }
}

// A warp per slab of sorted chains: their lengths, and the slab's entries (0 for
// slab = nslabs).
__global__ void __launch_bounds__(256) k_chain_slabs(long nchains, int nslabs, const int* __restrict__ id,
                                                     const int* __restrict__ len_of, int* __restrict__ len,
                                                     long* __restrict__ entries) {
    const int lane = threadIdx.x & 31;
    const long warps = long(gridDim.x) * blockDim.x / 32;
    for (long slab = (long(blockIdx.x) * blockDim.x + threadIdx.x) / 32; slab <= nslabs; slab += warps) {
        const long q = slab * 32 + lane;
        const int n = q < nchains ? len_of[id[q]] : 0;
        if (q < nchains) len[q] = n;
        const int most = __reduce_max_sync(FULL, n);
        if (lane == 0) entries[slab] = slab < nslabs ? long(chains_of(nchains, slab)) * most : 0L;
    }
}

// place[id] = sorted place of every non-empty chain.
__global__ void __launch_bounds__(256) k_chain_places(long nchains, const int* __restrict__ id, int* __restrict__ place) {
    for (long q = long(blockIdx.x) * blockDim.x + threadIdx.x; q < nchains; q += long(gridDim.x) * blockDim.x)
        place[id[q]] = int(q);
}

// The chains' entries, a warp per row, 32 blocks at a time (a value's entry is its
// chain's entries in the blocks before).  BACK: the values only, back to the
// reference order.
template <class LT, int R, class V, bool BACK>
__global__ void __launch_bounds__(256) k_chain_fill(int nrows, long nchains, const int* __restrict__ perm, const int* __restrict__ brptr,
                                                    const int* __restrict__ valptr, const uint8_t* __restrict__ hdr,
                                                    const uint16_t* __restrict__ mask, const int* __restrict__ place,
                                                    const long* __restrict__ first, const V* __restrict__ in,
                                                    V* __restrict__ out, int* __restrict__ xcol) {
    constexpr int VS = Layout<LT>::VS;
    const int lane = threadIdx.x & 31;
    const uint32_t before = (1u << lane) - 1u;
    const long warps = long(gridDim.x) * blockDim.x / 32;
    for (long i = (long(blockIdx.x) * blockDim.x + threadIdx.x) / 32; i < nrows; i += warps) {
        const int row = perm[i], br = row / R, s = row % R;
        const int b1 = brptr[br + 1];
        long v0 = valptr[br];
        long next = 0;  // lane c: chain c's next entry, and the distance to the one after it
        int pitch = 0;
        if (lane < VS && (mask[i] >> lane) & 1u) {
            const int q = place[i * VS + lane];
            next = first[q / 32] + q % 32;
            pitch = chains_of(nchains, q / 32);
        }
        for (int b0 = brptr[br]; b0 < b1; b0 += 32) {
            int col = 0, tot = 0, low = 0;
            uint32_t m = 0u;
            if (b0 + lane < b1) {
                uint32_t mw[Header<LT, R>::MASK_WORDS];
                col = load_header<LT, R>(hdr, long(b0) + lane, mw);
#pragma unroll
                for (int q = 0; q < R; ++q) {
                    const uint32_t mq = mask_of<LT, R>(mw, q);
                    tot += __popc(mq);
                    low += q < s ? __popc(mq) : 0;
                    m = q == s ? mq : m;
                }
            }
            int incl = tot;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int t = __shfl_up_sync(FULL, incl, d);
                if (lane >= d) incl += t;
            }
            long ref = v0 + incl - tot + low;
            int steps = 0;
#pragma unroll
            for (int c = 0; c < VS; ++c) {
                const uint32_t has = __ballot_sync(FULL, (m >> c) & 1u);
                const long e = __shfl_sync(FULL, next, c) + long(__shfl_sync(FULL, pitch, c)) * __popc(has & before);
                if ((m >> c) & 1u) {
                    if constexpr (BACK) {
                        out[ref] = in[e];
                    } else {
                        out[e] = in[ref];
                        xcol[e] = col + c;
                    }
                    ++ref;
                }
                steps = lane == c ? __popc(has) : steps;
            }
            next += long(pitch) * steps;
            v0 += __shfl_sync(FULL, incl, 31);
        }
    }
}

// Calls f(layout tag, std::integral_constant<int, R>, value tag) for a handle.
template <class F>
void dispatch_layout(const spc5cuda_mat* m, F&& f) {
    auto with = [&](auto lt, auto v) {
        switch (m->r) {
            case 1: f(lt, std::integral_constant<int, 1>{}, v); return;
            case 2: f(lt, std::integral_constant<int, 2>{}, v); return;
            case 4: f(lt, std::integral_constant<int, 4>{}, v); return;
            case 8: f(lt, std::integral_constant<int, 8>{}, v); return;
        }
        throw Error(SPC5CUDA_ERR_FORMAT, "r must be 1, 2, 4 or 8");
    };
    switch (m->value_type) {
        case SPC5CUDA_F64: with(double{}, double{}); return;
        case SPC5CUDA_F32: with(float{}, float{}); return;
        default: with(double{}, float{}); return;  // F32_V8: float values, the 8-column layout
    }
}

// Sorted rows of the chain part.  All long rows where they are about as long as one
// another: a stream's step has a lane per column of a row-block, most of them
// idle at few values per row-block, and a chain's lanes idle only where chains
// differ.  Else the streams share a row-block's sectors, and the few longest rows
// are chains if their steps, one after the other, would outlast the rest.
// Measured on B200 (us per SpMV, FP64, streams / chains): 50,000 rows of 400 random
// values 157 / 63, 1,000,000 of 40 400 / 178, 20,000 of 100 runs of 8 64 / 39;
// longest row at 24 (1M power-law) and 50 times (log-normal) the mean, all long rows
// as chains 111 / 138 and 312 / 520.
int chain_rows(const spc5cuda_mat* m, const Counts& c) {
    const int rows = c.rows[CLASSES - 1], vs = vs_of(m->value_type);
    if (rows == 0 || long(rows) * vs >= 1L << 31) return 0;  // (chain ids are int)
    if (c.longest <= 8.0 * double(c.blocks) / rows) return rows;
    // about 31 ps per warp step (of G row-blocks) and 3.2 ps per value for all rows;
    // 50 ns per step of one row, of which all above half that time go to the chains.
    // Power-law of 20,000 rows, rows of more than 32 row-blocks: 45 us, now 31; 100,000
    // rows, 128: 64 / 50; 300,000, 512: 84 / 84
    const int G = 32 / vs;
    const double rest_us = 31e-6 * double(c.blocks) / G + 3.2e-6 * double(m->nnz);
    if (50e-3 * c.longest < 2.0 * rest_us) return 0;
    for (int b = 4; b < 31; ++b)
        if (2.0 * 50e-3 * double(1L << b) >= rest_us) return c.rows[OCTAVES + b];
    return 0;
}

int warps_for(long n) { return grid_for(n * 32, 256); }

// The chain part of the first p.chain_rows sorted rows (synchronises s).
void build_chains(const spc5cuda_mat* m, SortedPlan& p, cudaStream_t s) {
    const int vs = vs_of(m->value_type), rows = p.chain_rows;
    const long nids = long(rows) * vs;
    const size_t id_ints = sizeof(int) * size_t(nids);
    DevBuf len(id_ints, s), cls(id_ints, s), ids(id_ints, s), sorted(id_ints, s), order(id_ints, s),
        totals(2 * sizeof(long), s), mask(sizeof(uint16_t) * size_t(rows), s);
    SPC5_CUDA(cudaMemsetAsync(totals.p, 0, totals.bytes, s));
    dispatch_layout(m, [&](auto lt, auto RC, auto) {
        k_chain_len<decltype(lt), decltype(RC)::value><<<warps_for(rows), 256, 0, s>>>(
            rows, p.perm.as<int>(), m->brptr.as<int>(), m->headers.as<uint8_t>(), len.as<int>(), cls.as<int>(),
            ids.as<int>(), mask.as<uint16_t>(), totals.as<unsigned long long>());
    });
    SPC5_CUDA(cudaGetLastError());
    size_t temp = 0;
    SPC5_CUDA(cub::DeviceRadixSort::SortPairsDescending(nullptr, temp, cls.as<int>(), sorted.as<int>(), ids.as<int>(),
                                                        order.as<int>(), int(nids), 0, CLASS_BITS, s));
    DevBuf tmp(temp, s);
    SPC5_CUDA(cub::DeviceRadixSort::SortPairsDescending(tmp.p, temp, cls.as<int>(), sorted.as<int>(), ids.as<int>(),
                                                        order.as<int>(), int(nids), 0, CLASS_BITS, s));
    long sums[2] = {0, 0};
    SPC5_CUDA(cudaMemcpyAsync(sums, totals.p, sizeof(sums), cudaMemcpyDeviceToHost, s));
    SPC5_CUDA(cudaStreamSynchronize(s));
    p.chain_values = sums[0];
    p.nchains = sums[1];
    const int slabs = div_up(p.nchains, 32);
    DevBuf entries(sizeof(long) * size_t(slabs + 1), s), first(sizeof(long) * size_t(slabs + 1), s);
    k_chain_slabs<<<warps_for(slabs + 1L), 256, 0, s>>>(p.nchains, slabs, order.as<int>(), len.as<int>(),
                                                        sorted.as<int>(), entries.as<long>());
    SPC5_CUDA(cudaGetLastError());
    SPC5_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, temp, entries.as<long>(), first.as<long>(), slabs + 1, s));
    DevBuf scan(temp, s);
    SPC5_CUDA(cub::DeviceScan::ExclusiveSum(scan.p, temp, entries.as<long>(), first.as<long>(), slabs + 1, s));
    long total = 0;
    SPC5_CUDA(cudaMemcpyAsync(&total, first.as<long>() + slabs, sizeof(long), cudaMemcpyDeviceToHost, s));
    SPC5_CUDA(cudaStreamSynchronize(s));
    // ---- the buffer and what is known of it (the entries: fill_chains)
    size_t at = 0;
    auto take = [&](size_t bytes) {
        const size_t here = at;
        at += (bytes + 255) / 256 * 256;
        return here;
    };
    const size_t chain_ints = sizeof(int) * size_t(p.nchains);
    const size_t a_first = take(first.bytes), a_val = take(size_t(value_bytes_of(m->value_type)) * size_t(total)),
                 a_col = take(sizeof(int) * size_t(total)), a_len = take(chain_ints), a_id = take(chain_ints),
                 a_mask = take(mask.bytes);
    p.chain.alloc(at);
    unsigned char* base = p.chain.as<unsigned char>();
    p.cfirst = reinterpret_cast<long*>(base + a_first);
    p.cval = base + a_val;
    p.ccol = reinterpret_cast<int*>(base + a_col);
    p.clen = reinterpret_cast<int*>(base + a_len);
    p.cid = reinterpret_cast<int*>(base + a_id);
    p.cmask = reinterpret_cast<uint16_t*>(base + a_mask);
    SPC5_CUDA(cudaMemcpyAsync(p.cfirst, first.p, first.bytes, cudaMemcpyDeviceToDevice, s));
    SPC5_CUDA(cudaMemcpyAsync(p.clen, sorted.p, chain_ints, cudaMemcpyDeviceToDevice, s));
    SPC5_CUDA(cudaMemcpyAsync(p.cid, order.p, chain_ints, cudaMemcpyDeviceToDevice, s));
    SPC5_CUDA(cudaMemcpyAsync(p.cmask, mask.p, mask.bytes, cudaMemcpyDeviceToDevice, s));
}

// The chains' values: from the reference order (in) to the chains and their x
// indices, or (BACK) from the chains to the reference order (out).
template <bool BACK>
void fill_chains(const spc5cuda_mat* m, const SortedPlan& p, const void* in, void* out, cudaStream_t s) {
    DevBuf place(sizeof(int) * size_t(p.chain_rows) * size_t(vs_of(m->value_type)), s);
    k_chain_places<<<grid_for(p.nchains, 256), 256, 0, s>>>(p.nchains, p.cid, place.as<int>());
    dispatch_layout(m, [&](auto lt, auto RC, auto val) {
        using V = decltype(val);
        k_chain_fill<decltype(lt), decltype(RC)::value, V, BACK><<<warps_for(p.chain_rows), 256, 0, s>>>(
            p.chain_rows, p.nchains, p.perm.as<int>(), m->brptr.as<int>(), m->valptr.as<int>(),
            m->headers.as<uint8_t>(), p.cmask, place.as<int>(), p.cfirst, static_cast<const V*>(in), static_cast<V*>(out),
            BACK ? nullptr : p.ccol);
    });
    SPC5_CUDA(cudaGetLastError());
}

}  // namespace

void build_sorted_plan(spc5cuda_mat* m, cudaStream_t s) {
    const int nrows = m->nrows, nbr = m->nbr();
    auto plan = std::make_unique<SortedPlan>();
    if (nrows <= 0) {
        m->plan = std::move(plan);
        return;
    }
    SortedPlan& p = *plan;
    const int G = 32 / vs_of(m->value_type);
    const size_t row_ints = sizeof(int) * size_t(nrows);
    p.perm.alloc(row_ints);
    p.key.alloc(row_ints);
    DevBuf rv(row_ints, s);
    Counts found{};
    const int* counts = found.rows;
    {
        // ---- the rows by size, largest first (stable)
        DevBuf key(row_ints, s), ids(row_ints, s), dc(sizeof(Counts), s);
        dispatch_layout(m, [&](auto lt, auto RC, auto) {
            using LT = decltype(lt);
            constexpr int VS = Layout<LT>::VS;
            k_row_stats<LT, decltype(RC)::value><<<grid_for(long(nbr) * VS, 256), 256, 0, s>>>(
                nrows, nbr, m->brptr.as<int>(), m->headers.as<uint8_t>(), key.as<int>(), rv.as<int>(), ids.as<int>());
        });
        SPC5_CUDA(cudaGetLastError());
        size_t temp = 0;
        SPC5_CUDA(cub::DeviceRadixSort::SortPairsDescending(nullptr, temp, key.as<int>(), p.key.as<int>(),
                                                            ids.as<int>(), p.perm.as<int>(), nrows, 0, 31, s));
        DevBuf tmp(temp, s);
        SPC5_CUDA(cub::DeviceRadixSort::SortPairsDescending(tmp.p, temp, key.as<int>(), p.key.as<int>(),
                                                            ids.as<int>(), p.perm.as<int>(), nrows, 0, 31, s));
        SPC5_CUDA(cudaMemsetAsync(dc.p, 0, dc.bytes, s));
        k_class_counts<<<grid_for(nrows, 256), 256, 0, s>>>(nrows, p.key.as<int>(), dc.as<Counts>());
        SPC5_CUDA(cudaGetLastError());
        SPC5_CUDA(cudaMemcpyAsync(&found, dc.p, sizeof(found), cudaMemcpyDeviceToHost, s));
        SPC5_CUDA(cudaStreamSynchronize(s));
    }
    p.chain_rows = chain_rows(m, found);
    if (p.chain_rows > 0) build_chains(m, p, s);
    // ---- classes (a class without rows ends where the one before it ends)
    int rows = p.chain_rows, slabs = 0;
    for (int j = 0; j < CLASSES; ++j) {
        const int end = std::max(rows, counts[j]);
        slabs += div_up(end - rows, G * class_rounds(j));
        rows = end;
        p.row_end[j] = rows;
        p.slab_end[j] = slabs;
    }
    for (int n = SHORT_VALUES; n >= 0; --n) {
        const int end = std::max(rows, counts[CLASSES + n]);
        p.short_rows[n] = end - rows;
        p.short_slabs += div_up(end - rows, 32);
        rows = end;
    }
    // ---- slab sizes and offsets
    p.sstep.alloc(sizeof(int) * size_t(slabs + 1));
    p.sval.alloc(sizeof(int) * size_t(slabs + 1));
    int sizes[2] = {0, 0};  // steps and values of the long rows
    if (slabs > 0) {
        const View v = view_of(p);
        DevBuf tmp(sizeof(int) * size_t(scan_tmp_ints(slabs)), s);
        const int blocks = grid_for(slabs, 128);
        if (G == 4)
            k_slab_size<4><<<blocks, 128, 0, s>>>(v, slabs, rv.as<int>(), p.sstep.as<int>(), p.sval.as<int>());
        else
            k_slab_size<2><<<blocks, 128, 0, s>>>(v, slabs, rv.as<int>(), p.sstep.as<int>(), p.sval.as<int>());
        SPC5_CUDA(cudaGetLastError());
        exclusive_scan_i32(p.sstep.as<int>(), p.sstep.as<int>(), slabs, tmp.as<int>(), s);
        exclusive_scan_i32(p.sval.as<int>(), p.sval.as<int>(), slabs, tmp.as<int>(), s);
        SPC5_CUDA(cudaMemcpyAsync(&sizes[0], p.sstep.as<int>() + slabs, sizeof(int), cudaMemcpyDeviceToHost, s));
        SPC5_CUDA(cudaMemcpyAsync(&sizes[1], p.sval.as<int>() + slabs, sizeof(int), cudaMemcpyDeviceToHost, s));
        SPC5_CUDA(cudaStreamSynchronize(s));
    }
    p.long_values = sizes[1];
    long entries = sizes[1];
    for (int n = 0; n <= SHORT_VALUES; ++n) entries += 32L * n * div_up(p.short_rows[n], 32);
    // ---- masks, x indices and values
    p.mask.alloc(sizeof(uint32_t) * size_t(std::max(sizes[0], 1)));
    p.chains.alloc(sizeof(uint16_t) * 32 * size_t(std::max(p.short_slabs, 1)));
    p.col.alloc(sizeof(int) * size_t(std::max(entries, 1L)));
    p.val.alloc(size_t(value_bytes_of(m->value_type)) * size_t(std::max(entries, 2L)));
    const View v = view_of(p);
    dispatch_layout(m, [&](auto lt, auto RC, auto val) {
        using LT = decltype(lt);
        using V = decltype(val);
        constexpr int R = decltype(RC)::value;
        if (slabs > 0)
            k_stream_fill<LT, R, V, false><<<grid_for(long(slabs) * 32, FILL_THREADS), FILL_THREADS, 0, s>>>(
                v, slabs, m->brptr.as<int>(), m->valptr.as<int>(), m->headers.as<uint8_t>(), m->values.as<V>(),
                p.val.as<V>(), p.mask.as<uint32_t>(), p.col.as<int>());
        if (p.short_slabs > 0)
            k_short_fill<LT, R, V, false><<<grid_for(long(p.short_slabs) * 32, 256), 256, 0, s>>>(
                v, m->brptr.as<int>(), m->valptr.as<int>(), m->headers.as<uint8_t>(), m->values.as<V>(),
                p.val.as<V>(), p.chains.as<uint16_t>(), p.col.as<int>());
    });
    SPC5_CUDA(cudaGetLastError());
    if (p.chain_rows > 0) fill_chains<false>(m, p, m->values.p, p.cval, s);
    SPC5_CUDA(cudaStreamSynchronize(s));
    m->plan = std::move(plan);
    // the streams serve every SpMV now: the reference-order values are put
    // back together when a call needs them (restore_values), if the rows hold
    // all of them (the caller's arrays may hold more: values of the rows past
    // the last one of a block-row that is not full, or past the masks')
    long held = m->plan->chain_values + m->plan->long_values;
    for (int n = 0; n <= SHORT_VALUES; ++n) held += long(n) * m->plan->short_rows[n];
    if (m->use_plan() && held == m->nnz) {
        m->values.release();
        m->values_dropped = true;
    }
}

void rebuild_values(const spc5cuda_mat* m, void* values, cudaStream_t s) {
    const SortedPlan& p = *m->plan;
    const View v = view_of(p);
    dispatch_layout(m, [&](auto lt, auto RC, auto val) {
        using LT = decltype(lt);
        using V = decltype(val);
        constexpr int R = decltype(RC)::value;
        if (v.long_slabs() > 0)
            k_stream_fill<LT, R, V, true><<<grid_for(long(v.long_slabs()) * 32, FILL_THREADS), FILL_THREADS, 0, s>>>(
                v, v.long_slabs(), m->brptr.as<int>(), m->valptr.as<int>(), m->headers.as<uint8_t>(), p.val.as<V>(),
                static_cast<V*>(values), nullptr, nullptr);
        if (v.short_slabs() > 0)
            k_short_fill<LT, R, V, true><<<grid_for(long(v.short_slabs()) * 32, 256), 256, 0, s>>>(
                v, m->brptr.as<int>(), m->valptr.as<int>(), m->headers.as<uint8_t>(), p.val.as<V>(),
                static_cast<V*>(values), nullptr, nullptr);
    });
    SPC5_CUDA(cudaGetLastError());
    if (p.chain_rows > 0) fill_chains<true>(m, p, p.cval, values, s);
}

}  // namespace spc5cuda
