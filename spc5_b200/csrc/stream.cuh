// stream.cuh -- the layout of the sorted plan (plan.cu builds it, stream.cu
// runs SpMV and SpMM over it).
//
// A row's row-blocks are the blocks of its block-row in which its own
// sub-row mask is not empty, in block order.  The rows are sorted by size,
// largest first (stable): the long rows (more than SHORT_VALUES values) by
// their number of row-blocks, then the short rows by their number of values.
//
// Long rows: warp streams.  The rows are dealt to the G = 32 / VS lane groups
// of a warp: group g runs the sorted rows row0 + q G + g, round after round q,
// one row-block per step, in lockstep (the rows of a round have about the same
// number of row-blocks; the shorter ones idle at the end).  Lane c of a group
// owns column c of every row-block, so at a step the masks of the G groups
// side by side are the warp's 32-bit active-lane mask M, and lane l's value is
// number popc(M & lanes below l) of the step's values, which are stored
// densely, step after step, each with its x index: a row-block's neighbouring
// columns are neighbours in memory too.  A slab is one warp's work: `rounds`
// rounds of G rows.  Rows of more than 32 row-blocks run one round per slab;
// shorter ones 2, 4, 8 or 16 rounds, so that a slab has about 32 to 64 steps.
//
// Chain part: the first sorted rows of a plan may be stored as their (row, column)
// chains instead: chain (sorted row i, column c) has id i VS + c and holds the
// row's values in column c of its blocks, in block order, each with its x index.
// The non-empty chains are sorted by length class (length_class, longest first,
// stable, so that neighbouring lanes often run neighbouring columns of a row) and
// cut into slabs of 32 (the last one of n), one lane per chain: entry j of lane l is
// at the slab's first entry + 32 j + l (n j + l), with room for the longest chain.
//
// Short rows: one lane per row, 32 rows of the same number of values per slab
// (the last slab of a length has fewer); entry j of lane l is at the slab's
// first entry + 32 j + l.  A row's entries are in chain order -- column class 0
// of its blocks in block order, then class 1, ... -- and the first entry of a
// chain has FIRST set in its x index; `chains` holds the mask of the row's
// non-empty chains.
#pragma once

#include "common.cuh"
#include "handle.h"

namespace spc5cuda {
namespace stream {

constexpr unsigned FULL = 0xFFFFFFFFu;
constexpr int SHORT_VALUES = SortedPlan::SHORT_VALUES;  // short rows: at most this many values
constexpr int LONG_KEY = 64;          // sort key: values of a short row, LONG_KEY + row-blocks of a long row
constexpr uint32_t FIRST = 1u << 31;  // x indices are below 2^31
constexpr int CLASSES = SortedPlan::CLASSES;  // long rows of > 32, > 16, > 8, > 4, <= 4 row-blocks ...
__host__ __device__ constexpr int class_rounds(int j) { return 1 << j; }  // ... run 1, 2, 4, 8, 16 rounds per slab
__host__ __device__ constexpr int class_min(int j) { return j < CLASSES - 1 ? 32 >> j : 0; }  // class j: more than this

// Device pointers of a plan without its chain part (sorted rows are counted from the
// first one after that).
struct View {
    const uint32_t* mask;
    const int* col;
    const int* sstep;
    const int* sval;
    const int* key;
    const int* perm;
    const uint16_t* chains;
    int row_end[CLASSES];
    int slab_end[CLASSES];
    int short_row[SHORT_VALUES + 2];   // short rows of n values: [short_row[n], short_row[n - 1])
    int short_slab[SHORT_VALUES + 2];  // and their slabs; [0]: all short slabs
    long short_val[SHORT_VALUES + 1];  // first entry of the first of them
    __host__ __device__ int long_rows() const { return row_end[CLASSES - 1]; }
    __host__ __device__ int long_slabs() const { return slab_end[CLASSES - 1]; }
    __host__ __device__ long long_values() const { return short_val[SHORT_VALUES]; }
    __host__ __device__ int short_slabs() const { return short_slab[0]; }
};

inline View view_of(const SortedPlan& p) {
    View v;
    v.mask = p.mask.as<uint32_t>();
    v.col = p.col.as<int>();
    v.sstep = p.sstep.as<int>();
    v.sval = p.sval.as<int>();
    v.key = p.key.as<int>() + p.chain_rows;
    v.perm = p.perm.as<int>() + p.chain_rows;
    v.chains = p.chains.as<uint16_t>();
    for (int j = 0; j < CLASSES; ++j) {
        v.row_end[j] = p.row_end[j] - p.chain_rows;
        v.slab_end[j] = p.slab_end[j];
    }
    int row = v.long_rows(), slab = 0;
    long at = p.long_values;
    v.short_row[SHORT_VALUES + 1] = row;
    for (int n = SHORT_VALUES; n >= 0; --n) {  // longest first
        v.short_slab[n + 1] = slab;
        v.short_val[n] = at;
        const int rows = p.short_rows[n], slabs = div_up(rows, 32);
        slab += slabs;
        row += rows;
        at += 32L * n * slabs;
        v.short_row[n] = row;
    }
    v.short_slab[0] = slab;
    return v;
}

// Chains of a slab.
__host__ __device__ inline int chains_of(long nchains, long slab) {
    const long left = nchains - slab * 32;
    return left < 32 ? int(left) : 32;
}

// Device pointers of the chain part.
struct ChainView {
    const int* len;       // entries of every chain
    const int* id;        // its id
    const long* first;    // first entry of every slab
    const int* col;       // x indices
    const uint16_t* mask; // non-empty chains of every row
    const int* perm;
    int rows, slabs;
    long chains;
};

inline ChainView chain_view_of(const SortedPlan& p) {
    ChainView v;
    v.len = p.clen;
    v.id = p.cid;
    v.first = p.cfirst;
    v.col = p.ccol;
    v.mask = p.cmask;
    v.perm = p.perm.as<int>();
    v.rows = p.chain_rows;
    v.slabs = div_up(p.nchains, 32);
    v.chains = p.nchains;
    return v;
}

// y[row] += sum: red.add.f64 (y + sum rounded once) or load, add, store.
__device__ __forceinline__ void add_to(double* y, double v) { atomicAdd(y, v); }
__device__ __forceinline__ void add_to(float* y, float v) { *y = *y + v; }

// First sorted row, end of the sorted rows and rounds of a slab of long rows.
struct SlabRows {
    int row0, row_end, rounds;
};

template <int G>
__device__ __forceinline__ SlabRows slab_rows(const View& v, int slab) {
    SlabRows s;
    int row_a = 0, slab_a = 0;
    s.rounds = class_rounds(0);
    s.row_end = v.row_end[0];
#pragma unroll
    for (int j = 1; j < CLASSES; ++j) {
        if (slab >= v.slab_end[j - 1]) {
            row_a = v.row_end[j - 1];
            slab_a = v.slab_end[j - 1];
            s.rounds = class_rounds(j);
            s.row_end = v.row_end[j];
        }
    }
    s.row0 = row_a + (slab - slab_a) * s.rounds * G;
    s.row_end = min(s.row_end, s.row0 + s.rounds * G);
    return s;
}

// A slab of short rows: their number of values, first sorted row, rows and
// first entry.
struct ShortRows {
    int len, row0, rows;
    long at;
};

__device__ __forceinline__ ShortRows short_rows(const View& v, int slab) {
    // rows of n values: slabs [short_slab[n + 1], next shorter length's first)
    ShortRows s{0, 0, 0, 0};
#pragma unroll
    for (int n = SHORT_VALUES; n >= 0; --n) {
        if (slab >= v.short_slab[n + 1]) {
            const int k = slab - v.short_slab[n + 1];
            s.len = n;
            s.row0 = v.short_row[n + 1] + 32 * k;
            s.rows = min(32, v.short_row[n] - s.row0);
            s.at = v.short_val[n] + 32L * n * k;
        }
    }
    return s;
}

}  // namespace stream
}  // namespace spc5cuda
