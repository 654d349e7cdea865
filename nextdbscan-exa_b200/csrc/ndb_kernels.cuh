// ndb_kernels.cuh -- the DBSCAN hot-path kernels (sm_100a), templated on the
// dimensionality D and, for the grid, on the cell-key type K.
//
// Pipeline (one job):
//   bbox      per-dimension min/max of the grid-eligible points        (HBM bound)
//   keys      per-point cell key, invalid points get the all-ones key  (HBM bound)
//   sort      stable LSD radix sort of (key, point id)                  (ndb_prims.cu)
//   cells     cell boundaries, cell keys, point -> cell                 (HBM bound)
//   gather    coordinates in cell order, padded stride                  (HBM bound)
//   rows      per (cell, stencil row): range of neighbour cells         (L2 binary search)
//   count     per-point neighbour count / core flag                     (FP32 pipe)
//   union     core-core connectivity, lock-free union-find              (FP32 pipe + L2 atomics)
//   labels    canonical cluster ids (rank of the smallest core)          (HBM bound)
//   border    border points take the minimum adjacent cluster id        (FP32 pipe)
//
// Replaces data_process::process_points (data_process.cpp:395-458) and
// data_process::process_cores (data_process.cpp:93-266): the reference tests every
// pair of points; here only pairs whose cells are within the stencil are tested,
// with the identical FP32 predicate, so every accepted pair is the same.
#pragma once

#include <float.h>

#include <type_traits>

#include "ndb_common.cuh"

namespace ndb {

// Grid description passed by value to the kernels.
constexpr int kMaxGridDims = 4;

struct GridDev {
    int k;                                  // gridded dimensions (1..4)
    int dim[kMaxGridDims];                  // input dimension of each gridded dimension
    double lo[kMaxGridDims];                // origin per gridded dimension
    double inv_w[kMaxGridDims];             // 1 / cell width
    long long g[kMaxGridDims];              // cells per gridded dimension
    unsigned long long stride[kMaxGridDims];  // key strides (1, g0, g0*g1, g0*g1*g2)
};

// Neighbour rows of a cell.  Row r covers the cells at offsets (x in
// [-xr, +xr], o1, o2, o3) in gridded dimensions (0, 1, 2, 3); those cells have
// consecutive keys, hence form one contiguous run of the sorted cell list.
struct Stencil {
    int n_rows;
    int4 rows[kMaxRows];  // (o1, o2, o3, xr), nearest rows first
};

// Per-job parameters of a batched run (independent DBSCAN jobs concatenated into
// one pipeline).  Kernels take a null table in a single-job run.  Cell keys of
// job j are key_base + the job's own cell key, so jobs never share a cell.
struct JobDev {
    long long off;                 // first point of the job in the concatenated input
    long long n;                   // points of the job
    float e2;                      // eps * eps (FP32)
    int min_pts;
    int list_cap;                  // neighbour-list entries recorded (min_pts - 1, 0 = none)
    int linked;                    // same-cell-linked grid (cell units)
    unsigned long long key_base;   // first composite cell key of the job
    long long col_base;            // first entry of the job's columns in the column table
    GridDev g;
    const float *src;              // the job's coordinates (device), gathered into the batch
    int32_t *nn_out;               // caller's outputs (device; may be null)
    int32_t *ci_out;
};

// job of a point in concatenated input order (jobs sorted by offset)
__device__ __forceinline__ int job_of_point(const JobDev *__restrict__ jobs, int n_jobs, long long o) {
    int lo = 0, hi = n_jobs - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (jobs[mid].off <= o) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

constexpr int kBlock = 256;
constexpr int kMaxRowCells = 5;
constexpr int kMaxListCap = 64;  // largest min_pts - 1 for which neighbour lists are kept
constexpr int kWarpsPerBlock = kBlock / kWarp;
// The count runs two warps per block: an item's candidate list can be thousands of
// points long, and small blocks free their slot as soon as both items are done.
constexpr int kCountWarps = 2;

// ---------------------------------------------------------------------------
// point validity: a point takes part in the grid iff all coordinates are finite
// and its first coordinate is not FLT_MAX.  With a finite e2 any other point is in
// range of nothing: NaN/inf coordinates make a squared difference NaN or inf, and
// FLT_MAX in coordinate 0 is the reference's padding marker
// (data_process.cpp:196, :440) whose distance to any other first coordinate
// squares to inf.
// ---------------------------------------------------------------------------
__device__ __forceinline__ int ordered_int(float f) {
    const int i = __float_as_int(f);
    return i >= 0 ? i : i ^ 0x7fffffff;
}

__global__ void set_int_kernel(int *p, int v) { *p = v; }

// Bounds as unsigned words whose identity is 0, so that zeroed memory starts a reduction:
// the maximum as its ordered unsigned value, the minimum as the complement of its own.
__host__ __device__ __forceinline__ uint32_t encode_hi(int ordered) { return (uint32_t)ordered ^ 0x80000000u; }
__host__ __device__ __forceinline__ uint32_t encode_lo(int ordered) { return ~encode_hi(ordered); }
__host__ __device__ __forceinline__ int decode_hi(uint32_t v) { return (int)(v ^ 0x80000000u); }
__host__ __device__ __forceinline__ int decode_lo(uint32_t v) { return decode_hi(~v); }

// The last block of a grid to come here (its earlier atomics are visible to it) copies
// `words` words from src to mail (mapped host memory): the host reads a kernel's result
// without a copy behind it.  done starts at zero and is left so.
__device__ __forceinline__ void mail_last_block(uint32_t *done, const uint32_t *src, int words,
                                                volatile uint32_t *mail) {
    __shared__ int s_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    for (int i = threadIdx.x; i < words; i += blockDim.x) mail[i] = __ldcg(src + i);
    if (threadIdx.x == 0) *done = 0;  // for the next launch
}

// The block's bounds and invalid points, added to lo_hi (encoded minima, then maxima)
// and n_invalid.
template <int D>
__device__ __forceinline__ void bbox_reduce(int (&lo)[D], int (&hi)[D], unsigned bad, int (*s_lh)[2 * D],
                                            unsigned *s_bad, uint32_t *lh, unsigned long long *n_invalid) {
    constexpr int W = kBlock / kWarp;
#pragma unroll
    for (int k = 0; k < D; ++k) {
        lo[k] = __reduce_min_sync(kFull, lo[k]);
        hi[k] = __reduce_max_sync(kFull, hi[k]);
    }
    bad = __reduce_add_sync(kFull, bad);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) {
#pragma unroll
        for (int k = 0; k < D; ++k) {
            s_lh[w][k] = lo[k];
            s_lh[w][D + k] = hi[k];
        }
        s_bad[w] = bad;
    }
    __syncthreads();
    if (threadIdx.x < 2 * D) {
        const int t = threadIdx.x;
        int v = s_lh[0][t];
        for (int q = 1; q < W; ++q) v = t < D ? min(v, s_lh[q][t]) : max(v, s_lh[q][t]);
        if (t < D) {
            if (v != 0x7fffffff) atomicMax(lh + t, encode_lo(v));
        } else {
            if (v != (int)0x80000000) atomicMax(lh + t, encode_hi(v));
        }
    }
    if (threadIdx.x == 0) {
        unsigned b = 0;
        for (int q = 0; q < W; ++q) b += s_bad[q];
        if (b) atomicAdd(n_invalid, (unsigned long long)b);
    }
}

// One point's coordinates: 16-byte vector loads when a point's row is a multiple of
// 16 bytes (d % 4 == 0; rows then start 16-byte aligned), 8-byte ones at d = 2.
template <int D>
__device__ __forceinline__ void load_row(const float *__restrict__ p, float (&x)[D]) {
    if constexpr (D % 4 == 0) {
#pragma unroll
        for (int q = 0; q < D / 4; ++q) {
            const float4 v = __ldg(reinterpret_cast<const float4 *>(p) + q);
            x[4 * q + 0] = v.x;
            x[4 * q + 1] = v.y;
            x[4 * q + 2] = v.z;
            x[4 * q + 3] = v.w;
        }
    } else if constexpr (D == 2) {
        const float2 v = __ldg(reinterpret_cast<const float2 *>(p));
        x[0] = v.x;
        x[1] = v.y;
    } else {
#pragma unroll
        for (int k = 0; k < D; ++k) x[k] = __ldg(p + k);
    }
}

// The same for a caller's array, which may be aligned to 4 bytes only: vec says whether
// its rows take the vector loads (rows_aligned).
template <int D>
__device__ __forceinline__ void load_row(const float *__restrict__ p, float (&x)[D], bool vec) {
    if ((D % 4 == 0 || D == 2) && vec) {
        load_row<D>(p, x);
    } else {
#pragma unroll
        for (int k = 0; k < D; ++k) x[k] = __ldg(p + k);
    }
}
template <int D>
inline bool rows_aligned(const float *p) {
    return ((uintptr_t)p & (D % 4 == 0 ? 15 : 7)) == 0;
}

// lo_hi[0..D) = encoded minima, lo_hi[D..2D) = encoded maxima.  Warps reduce by
// shuffles, the block through shared memory, and one thread per dimension and bound
// issues the block's atomic: with one atomic per warp the kernel's time was the queue of
// atomics on 2 D addresses (16-D 200k 128 -> 7 us, 8-D 2M 110 -> 15 us).  With mail the
// bounds and the invalid count (mail_words from lo_hi on) go to the host.
template <int D>
__global__ void __launch_bounds__(kBlock) bbox_kernel(const float *__restrict__ coords, int64_t n, bool vec,
                                                      uint32_t *lo_hi, unsigned long long *n_invalid,
                                                      uint32_t *done, int mail_words, volatile uint32_t *mail) {
    __shared__ int s_lh[kBlock / kWarp][2 * D];
    __shared__ unsigned s_bad[kBlock / kWarp];
    int lo[D], hi[D];
#pragma unroll
    for (int k = 0; k < D; ++k) {
        lo[k] = 0x7fffffff;
        hi[k] = (int)0x80000000;
    }
    unsigned bad = 0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        float x[D];
        load_row<D>(coords + i * D, x, vec);
        bool ok = x[0] != FLT_MAX;
#pragma unroll
        for (int k = 0; k < D; ++k) ok = ok && isfinite(x[k]);
        if (!ok) {
            ++bad;
            continue;
        }
#pragma unroll
        for (int k = 0; k < D; ++k) {
            const int v = ordered_int(x[k]);
            lo[k] = min(lo[k], v);
            hi[k] = max(hi[k], v);
        }
    }
    bbox_reduce<D>(lo, hi, bad, s_lh, s_bad, lo_hi, n_invalid);
    if (mail) mail_last_block(done, lo_hi, mail_words, mail);
}

// Cell coordinate along gridded dimension a.  Computed in double: with at most
// 2^30 cells per dimension the result is within 2^-21 cells of the exact value,
// which the host's stencil and same-cell margins absorb.
__device__ __forceinline__ long long cell_coord(const GridDev &g, int a, float x) {
    const double t = ((double)x - g.lo[a]) * g.inv_w[a];
    long long c = (long long)floor(t);
    c = c < 0 ? 0 : c;
    c = c > g.g[a] - 1 ? g.g[a] - 1 : c;
    return c;
}

// Memory the later grid kernels expect zeroed (the sort's and the chained scans' state,
// the column table), zeroed by the key kernels' threads; t of `threads` takes its share.
struct ZeroJob {
    uint4 *a, *b;
    int64_t na, nb;
    __device__ void run(int64_t t, int64_t threads) const {
        const uint4 z = make_uint4(0, 0, 0, 0);
        for (int64_t i = t; i < na; i += threads) a[i] = z;
        for (int64_t i = t; i < nb; i += threads) b[i] = z;
    }
};

template <int D, typename K>
__global__ void __launch_bounds__(kBlock) key_kernel(const float *__restrict__ coords, int64_t n, bool vec,
                                                     GridDev g, K invalid_key, K *__restrict__ keys,
                                                     uint32_t *__restrict__ core_bits, ZeroJob zero) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    zero.run(i, (int64_t)gridDim.x * blockDim.x);
    if (i >= n) return;
    if ((i & 31) == 0) core_bits[i >> 5] = 0;  // for core_flags_kernel
    const float *p = coords + i * D;
    K key = invalid_key;
    float x[D];  // validity from one load of the row; the gridded coordinates are re-read (L1)
    load_row<D>(p, x, vec);
    bool ok = x[0] != FLT_MAX;
#pragma unroll
    for (int k = 0; k < D; ++k) ok = ok && isfinite(x[k]);
    if (ok) {
        unsigned long long kk = 0;
#pragma unroll
        for (int a = 0; a < kMaxGridDims; ++a)
            if (a < g.k) kk += (unsigned long long)cell_coord(g, a, p[g.dim[a]]) * g.stride[a];
        key = (K)kk;
    }
    keys[i] = key;
}

// Cells from the sorted keys (chain_scan_kernel): the prefix of the "first point of a
// cell" flags numbers the cells; meanwhile every point's coordinates are gathered into
// cell order.
template <int D, typename K>
struct CellsOp {
    const K *keys;
    const int32_t *perm;
    const float *coords;
    bool vec;
    int64_t nv;
    float *xs;
    int32_t *cell_start;
    K *cell_key;
    int32_t *pcell;
    int32_t *nn_sorted;  // zeroed for full counts (null: early exit)
    __device__ uint32_t value(int64_t e) const { return e == 0 || keys[e] != keys[e - 1] ? 1u : 0u; }
    __device__ void early(int64_t e) const {
        if (nn_sorted) nn_sorted[e] = 0;
        constexpr int P = Stride<D>::P;
        float x[D], v[P];
        load_row<D>(coords + (int64_t)perm[e] * D, x, vec);
#pragma unroll
        for (int k = 0; k < P; ++k) v[k] = k < D ? x[k] : 0.0f;
        float *q = xs + e * P;
        if constexpr (P % 4 == 0) {
#pragma unroll
            for (int k = 0; k < P / 4; ++k)
                reinterpret_cast<float4 *>(q)[k] = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
        } else if constexpr (P == 2) {
            *reinterpret_cast<float2 *>(q) = make_float2(v[0], v[1]);
        } else {
            q[0] = v[0];
        }
    }
    __device__ void emit(int64_t e, uint32_t first, uint32_t before) const {
        const uint32_t c = before + first - 1;
        if (first) {
            cell_start[c] = (int32_t)e;
            cell_key[c] = keys[e];
        }
        pcell[e] = (int32_t)c;
        if (e == nv - 1) cell_start[c + 1] = (int32_t)nv;
    }
};

// Open-addressing hash table of the non-empty cells: key -> cell index.  Empty
// slots hold the all-ones key, which no cell has (it marks invalid points).
__device__ __forceinline__ unsigned long long hash_slot(unsigned long long key, unsigned long long mask) {
    return ((key + 1ull) * 0x9E3779B97F4A7C15ull >> 17) & mask;
}

template <typename K>
__global__ void hash_clear_kernel(K *__restrict__ hkeys, int64_t size) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < size) hkeys[i] = ~(K)0;
}

__device__ __forceinline__ uint32_t key_cas(uint32_t *a, uint32_t cmp, uint32_t val) { return atomicCAS(a, cmp, val); }
__device__ __forceinline__ uint64_t key_cas(uint64_t *a, uint64_t cmp, uint64_t val) {
    return (uint64_t)atomicCAS(reinterpret_cast<unsigned long long *>(a), (unsigned long long)cmp,
                               (unsigned long long)val);
}

template <typename K>
__global__ void hash_insert_kernel(const K *__restrict__ cell_key, const uint32_t *__restrict__ n_cells, K *hkeys,
                                   int32_t *__restrict__ hvals, unsigned long long mask) {
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= *n_cells) return;
    const K key = cell_key[c];
    unsigned long long h = hash_slot((unsigned long long)key, mask);
    for (unsigned long long probe = 0; probe <= mask; ++probe) {
        const K prev = key_cas(hkeys + h, ~(K)0, key);
        if (prev == ~(K)0 || prev == key) {
            hvals[h] = (int32_t)c;
            return;
        }
        h = (h + 1) & mask;
    }
}

template <typename K>
__device__ __forceinline__ int hash_find(const K *__restrict__ hkeys, const int32_t *__restrict__ hvals,
                                         unsigned long long mask, unsigned long long key) {
    unsigned long long h = hash_slot(key, mask);
    for (unsigned long long probe = 0; probe <= mask; ++probe) {
        const K k = __ldg(hkeys + h);
        if ((unsigned long long)k == key) return __ldg(hvals + h);
        if (k == ~(K)0) return -1;
        h = (h + 1) & mask;
    }
    return -1;
}

// ---------------------------------------------------------------------------
// How cells are found by key.  A column is the run of cells that differ only in
// gridded dimension 0; sorted by key, a column's cells are contiguous and ordered
// by x.  When the grid's columns are few enough (their count depends on the
// bounding box, not on n), a dense table holds each column's [first, end) range
// of cell indices, so a stencil row is one table load plus a search inside one
// short column.  Otherwise the open-addressing hash table of the cell keys is
// probed per x position.
// ---------------------------------------------------------------------------
template <typename K>
struct CellIndex {
    const int2 *col;      // column table (null: use the hash table)
    const K *hkeys;
    const int32_t *hvals;
    unsigned long long mask;
};

// Column of every cell: the table entry of its column gets the first cell (the
// column's first in key order) and the end (one past its last).  The table starts
// zeroed (empty columns read [0, 0)).
template <typename K>
__device__ __forceinline__ long long global_column(const K *__restrict__ cell_key, int64_t c, const GridDev &g_one,
                                                   const JobDev *__restrict__ jobs,
                                                   const int32_t *__restrict__ cell_job) {
    unsigned long long key_base = 0;
    long long col_base = 0, g0 = g_one.g[0];
    if (jobs) {
        const JobDev &J = jobs[cell_job[c]];
        key_base = J.key_base;
        col_base = J.col_base;
        g0 = J.g.g[0];
    }
    const unsigned long long local = (unsigned long long)cell_key[c] - key_base;
    if constexpr (sizeof(K) == 4) return col_base + (long long)((uint32_t)local / (uint32_t)g0);
    else return col_base + (long long)(local / (unsigned long long)g0);
}

template <typename K>
__global__ void col_range_kernel(const K *__restrict__ cell_key, const uint32_t *__restrict__ n_cells_dev,
                                 GridDev g_one, const JobDev *__restrict__ jobs,
                                 const int32_t *__restrict__ cell_job, int2 *__restrict__ col) {
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, n_cells = *n_cells_dev;
    if (c >= n_cells) return;
    const long long mine = global_column(cell_key, c, g_one, jobs, cell_job);
    if (c == 0 || global_column(cell_key, c - 1, g_one, jobs, cell_job) != mine) col[mine].x = (int)c;
    if (c == n_cells - 1 || global_column(cell_key, c + 1, g_one, jobs, cell_job) != mine) col[mine].y = (int)(c + 1);
}

// First cell of column range cr whose key is >= key (cr.y when none); the column's cells
// have strictly increasing keys.  A column without gaps places it directly: first +
// (key - first key).
template <typename K>
__device__ __forceinline__ int col_lower(const K *__restrict__ cell_key, int2 cr, K key) {
    if (cr.x >= cr.y) return cr.y;
    const K kf = __ldg(cell_key + cr.x);
    if (key <= kf) return cr.x;
    const K d = key - kf;  // keys grow by >= 1 per cell: cell_key[cr.x + d] >= key
    int hi = cr.y;
    if (d < (K)(cr.y - cr.x)) {
        hi = cr.x + (int)d;
        if (__ldg(cell_key + hi) == key) return hi;
    }
    int lo = cr.x + 1;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(cell_key + mid) < key) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// Cell index of the cell with key rowkey + x in column ncol, or -1.
template <typename K>
__device__ __forceinline__ int find_cell(const CellIndex<K> &L, const K *__restrict__ cell_key, long long ncol,
                                         unsigned long long rowkey, long long x) {
    const unsigned long long key = rowkey + (unsigned long long)x;
    if (!L.col) return hash_find(L.hkeys, L.hvals, L.mask, key);
    const int2 cr = __ldg(L.col + ncol);
    const int a = col_lower(cell_key, cr, (K)key);
    return a < cr.y && __ldg(cell_key + a) == (K)key ? a : -1;
}

// Cell coordinates from a key (x fastest); 32-bit arithmetic for 32-bit keys.
template <typename K>
__device__ __forceinline__ void decode_key(K key, const GridDev &g, long long (&c)[kMaxGridDims]) {
    using U = typename std::conditional<sizeof(K) == 4, uint32_t, unsigned long long>::type;
    U rest = (U)key;
#pragma unroll
    for (int a = 0; a < kMaxGridDims; ++a) {
        if (a < g.k - 1) {
            const U ga = (U)g.g[a];
            const U q = rest / ga;
            c[a] = (long long)(rest - q * ga);
            rest = q;
        } else if (a == g.k - 1) {
            c[a] = (long long)rest;
        } else {
            c[a] = 0;
        }
    }
}

// nbr[c * n_rows + r] = [first, last) cell index of row r around cell c: the cells
// of a row have consecutive keys, so the existing ones are consecutive in the
// sorted cell list and the range runs from the smallest to the largest found.
// One lane per (cell, row): 2^group_log2 lanes (>= n_rows) per cell, so a cell's rows
// are looked up in parallel and its row table is written at once.  Bound: instruction
// issue, so keys, coordinates and columns are computed in the key's own width (a row's
// key and column are the cell's plus the row's offsets; a coordinate below zero wraps
// and fails the bound): against 64-bit arithmetic throughout the grid phase of 3-D 10M
// takes 1.10 instead of 1.24 ms, of the 4,096-job batch 20.4 instead of 23.4 ms.
template <typename K>
__global__ void __launch_bounds__(kBlock) rows_kernel(const K *__restrict__ cell_key,
                                                      const uint32_t *__restrict__ n_cells_dev, GridDev g_one,
                                                      Stencil stencil, int group_log2, CellIndex<K> L,
                                                      int2 *__restrict__ nbr, const JobDev *__restrict__ jobs,
                                                      const int32_t *__restrict__ cell_job) {
    __shared__ int4 s_rows[kMaxRows];
    const int n_rows = stencil.n_rows;
    for (int r = threadIdx.x; r < n_rows; r += blockDim.x) s_rows[r] = stencil.rows[r];
    __syncthreads();
    const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t c = gid >> group_log2, n_cells = *n_cells_dev;
    const int r = (int)(gid & ((1 << group_log2) - 1));
    if (c >= n_cells || r >= n_rows) return;
    const JobDev *J = jobs ? jobs + cell_job[c] : nullptr;
    const GridDev &g = J ? J->g : g_one;
    const K key_base = J ? (K)J->key_base : (K)0;
    const long long col_base = J ? J->col_base : 0;
    const int4 row = s_rows[r];
    const int off[kMaxGridDims] = {0, row.x, row.y, row.z};
    const K local = cell_key[c] - key_base, g0 = (K)g.g[0];
    K rest = local / g0;
    const K x = local - rest * g0;
    K base = cell_key[c] - x;  // key of x = 0 in the row's column
    K col = rest, cstride = 1;
    bool in = true;
#pragma unroll
    for (int a = 1; a < kMaxGridDims; ++a) {
        if (a < g.k) {
            const K ga = (K)g.g[a];
            K q = 0, v = rest;
            if (a < g.k - 1) {
                q = rest / ga;
                v = rest - q * ga;
            }
            rest = q;
            const K o = (K)(long long)off[a];
            in = in && (K)(v + o) < ga;
            base += o * (K)g.stride[a];
            col += o * cstride;
            cstride *= ga;
        }
    }
    int2 res = make_int2(0, 0);
    if (in) {
        const K w = (K)row.w;
        const K x0 = x < w ? (K)0 : x - w, x1 = x + w > g0 - 1 ? g0 - 1 : x + w;
        const K kmax = base + x1;
        // the row's existing cells are consecutive in the sorted cell list: find the
        // first one (a column-table search, or hashing from x0 on), then count the
        // keys that follow it within the row (independent loads, at most 2 row.w)
        int ca = -1;
        if (L.col) {
            const int2 cr = __ldg(L.col + col_base + (long long)col);
            const int a = col_lower(cell_key, cr, (K)(base + x0));
            if (a < cr.y && __ldg(cell_key + a) <= kmax) ca = a;
        } else {
            for (K xx = x0; xx <= x1 && ca < 0; ++xx)
                ca = hash_find(L.hkeys, L.hvals, L.mask, (unsigned long long)(K)(base + xx));
        }
        if (ca >= 0) {
            // keys are sorted and unique: the row's cells after ca are a prefix of the
            // next keys; four independent loads cover rows of up to 5 cells
            const int n = (int)n_cells;
            int cb = ca + 1;
            bool more = true;
            K nk[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) nk[q] = ca + 1 + q < n ? __ldg(cell_key + ca + 1 + q) : (K)0;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                more = more && ca + 1 + q < n && nk[q] <= kmax;
                cb += more ? 1 : 0;
            }
            if (more)
                while (cb < n && __ldg(cell_key + cb) <= kmax) ++cb;
            res = make_int2(ca, cb);
        }
    }
    nbr[c * n_rows + r] = res;
}

// Work items (cell, first point), chunks of up to 32 points of a cell, in cell order
// (chain_scan_kernel over the cells); also clears the cells' core flags.
struct ItemsOp {
    const int32_t *cell_start;
    int2 *items;
    uint8_t *cell_has_core;
    __device__ uint32_t value(int64_t c) const {
        return (uint32_t)((cell_start[c + 1] - cell_start[c] + kTile - 1) / kTile);
    }
    __device__ void early(int64_t c) const { cell_has_core[c] = 0; }
    __device__ void emit(int64_t c, uint32_t cnt, uint32_t before) const {
        const int32_t s0 = cell_start[c];
        for (uint32_t q = 0; q < cnt; ++q) items[before + q] = make_int2((int)c, s0 + (int)q * kTile);
    }
};

// ---------------------------------------------------------------------------
// Row table: the candidate ranges of one cell's stencil rows, gathered by the
// warp in one round (lane r loads row r) and flattened, so that the lanes walk the
// candidates of all rows 32 at a time instead of row by row.  Host planning keeps
// the number of rows <= 32.
// ---------------------------------------------------------------------------
struct RowTable {
    int start[kWarp];    // first candidate (point index, or cell index for CELLS) of each row
    int off[kWarp + 1];  // exclusive prefix of the row lengths; off[n_rows] = total
};

// Row table from one (start, len) range per lane (lanes >= n_rows hold len 0).
__device__ __forceinline__ int build_rows(int start, int len, int n_rows, RowTable &rt, int lane) {
    int incl = len;
#pragma unroll
    for (int o = 1; o < kWarp; o <<= 1) {
        const int y = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane < n_rows) {
        rt.start[lane] = start;
        rt.off[lane] = incl - len;
    }
    const int total = __shfl_sync(kFull, incl, kWarp - 1);
    if (lane == 0) rt.off[n_rows] = total;
    __syncwarp();
    return total;
}

// CELLS: ranges of cell indices >= min_cell; otherwise ranges of point indices.
template <bool CELLS>
__device__ __forceinline__ int gather_rows(const int2 *__restrict__ nbr_row, int n_rows,
                                           const int32_t *__restrict__ cell_start, int min_cell,
                                           RowTable &rt, int lane) {
    int start = 0, len = 0;
    if (lane < n_rows) {
        const int2 cr = nbr_row[lane];
        if (CELLS) {
            start = max(cr.x, min_cell);
            len = max(cr.y - start, 0);
        } else if (cr.x < cr.y) {
            start = cell_start[cr.x];
            len = cell_start[cr.y] - start;
        }
    }
    return build_rows(start, len, n_rows, rt, lane);
}

// Candidate t (0 <= t < total) of the flattened rows: the last row whose offset is
// <= t.  For rows of cells (at most a few entries each).
__device__ __forceinline__ int row_lookup(const RowTable &rt, int n_rows, int t) {
    int lo = 0, hi = n_rows - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (rt.off[mid] <= t) lo = mid;
        else hi = mid - 1;
    }
    return rt.start[lo] + (t - rt.off[lo]);
}

// Candidate t for a lane whose t only grows (by a warp per step): advance the
// lane's row cursor over the row offsets (empty rows skipped) instead of searching.
__device__ __forceinline__ int row_next(const RowTable &rt, int &row, int t) {
    while (rt.off[row + 1] <= t) ++row;
    return rt.start[row] + (t - rt.off[row]);
}

// ---------------------------------------------------------------------------
// Neighbour count.  One warp per item (up to 32 points i of one cell).  The i
// points sit in shared memory; lanes walk the flattened candidates of the
// stencil rows 32 at a time (coalesced loads), every lane tests its candidate j
// against each i (broadcast reads), and transposed hit masks give that i's count.
// Rows are ordered nearest first.
// It stops once every i of the item has reached min_pts (exact counts below min_pts, so
// exact core flags), or with `all` at the end of the candidates (exact counts).  dense_skip: with same-cell-linked cells a cell
// of >= min_pts points is all cores (every pair inside it is in range), so its
// points need no test at all; they report the cell size.
// ---------------------------------------------------------------------------
//
// GRAM (d >= 8): a pair is first decided from centred FP32 dot products.  With
// a = x_i - o and b = x_j - o (o the item's first point), D~ = |a|^2 + |b|^2 - 2 a.b
// costs d FMAs per pair, against the 3d separately rounded operations of the
// reference's sum.  A pair is a hit when D~ is below e2 by more than a bound on its
// error, a miss when above by more than it; the pairs in between (the guard band)
// are decided by the reference's own FP32 sum.  Counts, lists and core flags are
// therefore the exact kernel's.  Error bound (u = 2^-24, K = d): centring in FP32
// moves |a - b|^2 off |x_i - x_j|^2 by at most 4u (n_a + n_b); the FMA chains give
// |a|^2, |b|^2 and a.b within K u of n_a, n_b and |a||b| <= (n_a + n_b) / 2; forming
// v = n_a - 2 a.b and v + n_b adds 2u (n_a + n_b).  So |D~ - |x_i - x_j|^2| <=
// (3K + 6) u (n_a + n_b), and gram_kappa is twice that.  The reference's sum is
// within (K + 2) u of |x_i - x_j|^2 (gram_gamma covers 2 (K + 8) u), and the
// thresholds carry the rounding of their own arithmetic (kGramSigma e2).
// ---------------------------------------------------------------------------
template <int K>
__host__ __device__ constexpr float gram_kappa() {
    return 2.0f * (3.0f * K + 6.0f) * (1.0f / 16777216.0f);
}
template <int K>
__host__ __device__ constexpr float gram_gamma() {
    return 2.0f * (K + 8) * (1.0f / 16777216.0f);
}
constexpr float kGramSigma = 8.0f / 16777216.0f;

// ---------------------------------------------------------------------------
// Hit masks: lane l holds, per candidate it owns, one bit per owned point (bit k =
// point k is in range of the candidate).  A pair's bit is the sign of a difference,
// appended by one funnel shift, so the pair loop has no vote, no compare and no
// branch; a 32x32 bit transpose per 32 candidates then hands lane k the candidates
// that hit point k, and lane k counts them and writes point k's list entries.  Steps
// without any hit skip the transpose.
// Packing: points that reached min_pts leave the item.  The remaining ones move to the
// first slots (coordinates in shared memory, count and index with their lane), so the
// pair loop always runs over a dense range of slots.
// Bound: instruction issue and the FMA pipe (8-D early exit: 23 thread instructions per
// pair, issue 60 %, FMA pipe 54 %).  The form before this one voted and updated counts and lists per
// pair and step (58 instructions per pair).  Measured on B200, before and after: 8-D 2M
// early exit 4.47 -> 2.69 ms, 2-D 100k full counts 0.565 -> 0.213 ms, 3-D 1M full
// counts 1.63 -> 0.89 ms, 5-D 300k full counts 2.84 -> 1.56 ms.
// ---------------------------------------------------------------------------
// (acc << 1) | sign bit of x
__device__ __forceinline__ unsigned push_sign(unsigned acc, float x) {
    unsigned r;
    asm("shf.l.wrap.b32 %0, %1, %2, 1;" : "=r"(r) : "r"(__float_as_uint(x)), "r"(acc));
    return r;
}

// The reference's sum with b given negated: x + (-b) is the reference's difference (or
// its negative), so every square is the same.  Two dimensions go through one packed
// subtraction and one packed multiplication; the additions stay scalar and in order
// (a packed addition after a packed multiplication would be contracted).
template <int D>
__device__ __forceinline__ float dist_negated(const float (&x)[D], const float (&nb)[D]) {
    float len = 0.0f;
#pragma unroll
    for (int k = 0; k + 1 < D; k += 2) {
        const float2 t = __fadd2_rn(make_float2(x[k], x[k + 1]), make_float2(nb[k], nb[k + 1]));
        const float2 q = __fmul2_rn(t, t);
        len = k ? __fadd_rn(len, q.x) : q.x;
        len = __fadd_rn(len, q.y);
    }
    if constexpr (D & 1) {
        const float t = __fadd_rn(x[D - 1], nb[D - 1]);
        len = D > 1 ? __fadd_rn(len, __fmul_rn(t, t)) : __fmul_rn(t, t);
    }
    return len;
}

// The squared distance by FMAs (b negated), two chains joined by one addition: within
// (D + 2) u of the real one, like the reference's sum, so the two decide a pair alike
// unless |e2 - dist_fma| <= direct_gamma e2 (u = 2^-24; derivation at count_kernel).
template <int D>
__device__ __forceinline__ float dist_fma(const float (&x)[D], const float (&nb)[D]) {
    float2 acc = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int k = 0; k + 1 < D; k += 2) {
        const float2 t = __fadd2_rn(make_float2(x[k], x[k + 1]), make_float2(nb[k], nb[k + 1]));
        acc = k ? __ffma2_rn(t, t, acc) : __fmul2_rn(t, t);
    }
    if constexpr (D & 1) {
        const float t = __fadd_rn(x[D - 1], nb[D - 1]);
        acc.x = __fmaf_rn(t, t, acc.x);
    }
    return __fadd_rn(acc.x, acc.y);
}
template <int D>
__host__ __device__ constexpr float direct_gamma() {
    return 2.0f * (D + 8) * (1.0f / 16777216.0f);
}

// 32x32 bit-matrix transpose across a warp: lane l holds row l (bit c = column
// c) on entry and column l (bit r = row r) on return.  Step j exchanges the
// off-diagonal j x j blocks.  ROTATE: a lane takes its partner's word rotated by j
// towards its own half (the bits a rotation wraps around are outside the mask), three
// instructions a step but ten lane constants in registers; otherwise both halves are
// formed and one is selected.  The registers cost the early exit at d <= 3, whose short
// items live on resident warps, more than the instructions (3-D 10M 0.55 against 0.67
// ms); everywhere else rotating is faster (5-D 300k full counts 1.38 against 1.56 ms).
template <bool ROTATE = true>
__device__ __forceinline__ unsigned transpose32(unsigned x, int lane) {
    const unsigned masks[5] = {0x0000FFFFu, 0x00FF00FFu, 0x0F0F0F0Fu, 0x33333333u, 0x55555555u};
#pragma unroll
    for (int s = 0; s < 5; ++s) {
        const int j = 16 >> s;
        const unsigned m = masks[s];
        const bool upper = lane & j;
        const unsigned y = __shfl_xor_sync(kFull, x, j);
        if constexpr (ROTATE) {
            const unsigned keep = upper ? ~m : m;
            x = (x & keep) | (__funnelshift_l(y, y, upper ? kWarp - j : j) & ~keep);
        } else {
            x = upper ? ((x & ~m) | ((y >> j) & m)) : ((x & m) | ((y << j) & ~m));
        }
    }
    return x;
}

// Two FMA chains over the even and the odd dimensions, one starting at |a|^2 (within the
// bound's share for forming v), joined by one addition: v = |a|^2 - 2 a.b, with b2 = -2 b.
template <int D>
__device__ __forceinline__ float gram_value(const float (&a)[D], float na, const float (&b2)[D]) {
    float2 v2 = make_float2(na, 0.0f);
#pragma unroll
    for (int q = 0; q + 1 < D; q += 2)
        v2 = __ffma2_rn(make_float2(a[q], a[q + 1]), make_float2(b2[q], b2[q + 1]), v2);
    if constexpr (D & 1) v2.x = __fmaf_rn(a[D - 1], b2[D - 1], v2.x);
    return __fadd_rn(v2.x, v2.y);
}

// kDirect: the out-of-range bits of a lane's candidates by the reference's sum (rare).
template <int D, int CH>
__device__ __forceinline__ void recheck_exact(const float *si, int nk, const float (&xj)[CH][D], float e2,
                                           unsigned (&miss)[CH]) {
    constexpr int P = Stride<D>::P;
    for (int c = 0; c < CH; ++c) miss[c] = 0;
    for (int k = nk - 1; k >= 0; --k) {
        float xi[D];
        load_point_smem<D>(si + k * P, xi);
#pragma unroll
        for (int c = 0; c < CH; ++c) miss[c] = push_sign(miss[c], __fsub_rn(e2, dist_negated<D>(xj[c], xi)));
    }
}

// Full counts: adds the hits in m to point p's count; with `list`, the old count owns the
// list slots from there on, and those below list_cap are written (other(bit): the point
// at the other end).  Returns the count after the addition when it was asked for.
template <typename F>
__device__ __forceinline__ int add_hits(int32_t *nn_sorted, int32_t *__restrict__ nbr_list, int list_cap,
                                        int list_stride, int p, bool list, unsigned m, F other) {
    const int h = __popc(m);
    if (!list) {
        atomicAdd(nn_sorted + p, h);
        return list_cap;
    }
    const int old = atomicAdd(nn_sorted + p, h);
    for (int slot = old; m && slot < list_cap; m &= m - 1, ++slot)
        nbr_list[(int64_t)p * list_stride + slot] = other(__ffs(m) - 1);
    return old + h;
}

// Row table of the candidate points at and behind point p0 (sorted order).
__device__ __forceinline__ int gather_points_from(const int2 *__restrict__ nbr_row, int n_rows,
                                                  const int32_t *__restrict__ cell_start, int p0, RowTable &rt,
                                                  int lane) {
    int start = 0, len = 0;
    if (lane < n_rows) {
        const int2 cr = nbr_row[lane];
        if (cr.x < cr.y) {
            start = max(cell_start[cr.x], p0);
            len = max(cell_start[cr.y] - start, 0);
        }
    }
    return build_rows(start, len, n_rows, rt, lane);
}

// How a pair is decided (results never depend on it):
//   kExact   the reference's sum
//   kDirect  dist_fma against e2; when one of a lane's pairs of the step falls within
//            direct_gamma e2 of e2, the lane decides the step's pairs by the reference's sum
//   kGram    centred dot products with a guard band (d >= 8, see above)
// kDirect: let S be the real squared distance of the FP32 points.  Both sums consist of
// rounded differences, squares and at most D additions of non-negative terms, so both are
// within (D + 2) u S of S (and of underflow, below 2^-140, which e2 >= 2^-100 hides; a sum
// that overflows belongs to a pair whose other sum is above e2 as well, since e2 <= 2^100).
// If the FMA sum is below e2 - w or above e2 + w with w >= 2 (D + 3) u e2 / (1 - 2 (D + 3) u),
// the reference's sum lies on the same side; direct_gamma is 2 (D + 8) u.  It costs 2 d + 1
// operations on the FMA pipe against 3 d (8-D 2M early exit 2.63 -> 2.29 ms, 16-D 200k 1.38
// -> 1.28 ms).  Used for d >= 4; below, the sum is short.
constexpr int kExact = 0, kDirect = 1, kGram = 2;

// Handing items on (d >= kDeferDim, early exit, with defer): an item whose points are not
// done early costs less in the tensor-core count, which a caller's launch over the list in
// defer provides; an item whose points are done soon costs less here.  Which it is depends
// on the data, so items vote: after 1/64 of its candidates an item says whether its points
// would reach min_pts at the rate of hits so far (n_defer: 0 items handed on, 1 votes, 2
// votes against).  Once there are kDeferVotes votes, two per CTA of the tensor-core count, and
// at least half of them are against, items hand themselves on at that look; an item that
// looks before there are as many looks again at 1/32, 1/16 and 1/8.  Only items of at least
// kDeferCandidates candidates and kDeferPoints unfinished points take part: below, a tile of
// the tensor cores is not filled.  An item handed on is counted again from its first
// candidate.  Measured on B200 (count phase: always here, always handed on, this): 16-D 1M of
// which 9 % are core (minPts 64) 37.4, 30.9 and 30.3 ms, 16-D 200k without a core 26.7, 25.2
// and 20.7 ms; where most points are done early 16-D 1M 12.6, 20.2 and 12.3 ms, 13-D 400k 9.2,
// 17.7 and 9.3 ms.  With fewer votes (128), or by each item's own forecast, the few that hand
// on make a tail of their own (16-D 200k 1.57 against 1.24 ms, 1M 13.9 against 12.3).
constexpr int kDeferDim = 12, kDeferPoints = 16, kDeferCandidates = 8192, kDeferVotes = 1480;

template <int D, int MODE>
__global__ void __launch_bounds__(kCountWarps * kWarp) count_kernel(
    const int2 *__restrict__ items, const uint32_t *__restrict__ n_items, const int32_t *__restrict__ cell_start,
    const int2 *__restrict__ nbr, int n_rows, const float *__restrict__ xs, float e2, int min_pts,
    int dense_skip, int all, int32_t *__restrict__ nn_sorted, int32_t *__restrict__ nbr_list, int list_cap,
    int list_stride, unsigned long long *__restrict__ pair_counter, const JobDev *__restrict__ jobs,
    const int32_t *__restrict__ cell_job, unsigned long long *__restrict__ band_counter, int2 *__restrict__ defer,
    uint32_t *n_defer) {
    constexpr int P = Stride<D>::P;
    constexpr bool GRAM = MODE == kGram;
    static_assert(!GRAM || D >= 8, "the Gram filter is built for d >= 8");
    // d >= 8: each lane holds two candidates per step (64 per warp), so an owned
    // point is read from shared memory once per two pairs and the two distance sums
    // (each in the reference's order) are independent chains for the scheduler
    constexpr int CH = D >= 8 ? 2 : 1;
    __shared__ __align__(16) float s_i[kCountWarps][kTile * P];
    __shared__ __align__(16) float s_a[kCountWarps][GRAM ? kTile * P : 4];  // centred points
    __shared__ float s_n[kCountWarps][GRAM ? kTile : 1];                     // their squared norms
    __shared__ RowTable s_rows[kCountWarps];
    __shared__ int s_j[kCountWarps][CH * kWarp];  // the step's candidates
    __shared__ int2 s_move[kCountWarps][kTile];   // (index, count) of the points a packing moves
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int64_t item_id = (int64_t)blockIdx.x * kCountWarps + wib;
    if (item_id >= *n_items) return;
    const int2 item = items[item_id];
    const int cell = item.x, p0 = item.y;
    const int cs = cell_start[cell], ce = cell_start[cell + 1];
    const int cnt = min(kTile, ce - p0);
    if (jobs) {
        const JobDev &J = jobs[cell_job[cell]];
        e2 = J.e2;
        min_pts = J.min_pts;
        dense_skip = J.linked;
        list_cap = J.list_cap;
    }
    if (all) {  // exact counts (sparse cells): no point leaves
        min_pts = 0x7fffffff;
        dense_skip = 0;
    }
    if (dense_skip && ce - cs >= min_pts) {
        if (lane < cnt) nn_sorted[p0 + lane] = ce - cs;
        return;
    }
    if (!nbr_list) list_cap = 0;
    float *si = s_i[wib];
    float *sa = s_a[wib];
    int *sj = s_j[wib];
    RowTable &rt = s_rows[wib];
    float o[GRAM ? D : 1];  // GRAM: the item's first point, the origin of the centring
    float nmax = 0.0f;      // GRAM: largest |a|^2 of the item
    if constexpr (GRAM) load_point<D>(xs, p0, o);
    if (lane < cnt) {
        float x[D];
        load_point<D>(xs, p0 + lane, x);
        if constexpr (!GRAM) {
#pragma unroll
            for (int k = 0; k < D; ++k) x[k] = -x[k];  // for dist_negated
        }
        store_point_smem<D>(si + lane * P, x);
        if constexpr (GRAM) {
            float a[D];
            float n = 0.0f;
#pragma unroll
            for (int k = 0; k < D; ++k) {
                a[k] = __fsub_rn(x[k], o[k]);
                n = __fmaf_rn(a[k], a[k], n);
            }
            store_point_smem<D>(sa + lane * P, a);
            s_n[wib][lane] = n;
            nmax = n;
        }
    }
    if constexpr (GRAM) {
#pragma unroll
        for (int sft = 16; sft > 0; sft >>= 1) nmax = fmaxf(nmax, __shfl_xor_sync(kFull, nmax, sft));
    }
    const int total = gather_rows<false>(nbr + (int64_t)cell * n_rows, n_rows, cell_start, 0, rt, lane);
    __syncwarp();
    // slot k < nk holds point p0 + pid of lane k, whose count is lane k's mycnt
    int nk = cnt, pid = lane, mycnt = 0;
    unsigned long long pairs = 0;
    unsigned band = 0;  // GRAM: pairs rechecked in the guard band
    int row = 0;        // this lane's stencil row: its candidate index only grows
    // the candidate at which the item looks at the votes (see kDeferDim), -1: at none
    int look = D >= kDeferDim && defer && total >= kDeferCandidates ? ((total >> 6) + 63) & ~63 : -1;
    for (int tb = 0; tb < total; tb += kWarp * CH) {
        if constexpr (D >= kDeferDim) {
            if (tb == look) {
                if (look == (((total >> 6) + 63) & ~63)) {
                    // hits so far, without the points themselves
                    const int hits = __reduce_add_sync(kFull, lane < nk && mycnt > 1 ? mycnt - 1 : 0);
                    if (lane == 0) {
                        atomicAdd(n_defer + 1, 1u);
                        if (nk >= kDeferPoints && (float)hits * (float)total <= (float)nk * (float)min_pts * (float)tb)
                            atomicAdd(n_defer + 2, 1u);
                    }
                }
                int go = 0;  // 1: hand on, -1: too few votes yet
                if (lane == 0 && nk >= kDeferPoints) {
                    const uint32_t votes = __ldcg(n_defer + 1), no = __ldcg(n_defer + 2);
                    go = votes < kDeferVotes ? -1 : 2 * no >= votes;
                    if (go > 0) {
                        defer[atomicAdd(n_defer, 1u)] = item;
                        atomicAdd(pair_counter, pairs);
                    }
                }
                go = __shfl_sync(kFull, go, 0);
                if (go > 0) {
                    if constexpr (GRAM) {
                        band = __reduce_add_sync(kFull, band);
                        if (lane == 0 && band) atomicAdd(band_counter, (unsigned long long)band);
                    }
                    return;
                }
                look = go < 0 && look < (total >> 3) ? 2 * look : -1;
            }
        }
        int j[CH];
        float xj[CH][D];  // GRAM: -2 times the centred candidate b = x_j - o
        float tlo[CH], thi[CH];
        unsigned miss[CH], over[CH];  // bit k: out of range; GRAM: above the hit bound, above the miss bound
        float near = INFINITY;        // kDirect: smallest distance of a pair's sum from e2
#pragma unroll
        for (int c = 0; c < CH; ++c) {
            const int t = tb + c * kWarp + lane;
            j[c] = t < total ? row_next(rt, row, t) : -1;
            load_point<D>(xs, max(j[c], 0), xj[c]);  // lanes past the end read a valid point and are masked below
            miss[c] = over[c] = 0;
            if constexpr (GRAM) {
                float nb = 0.0f;
#pragma unroll
                for (int k = 0; k < D; ++k) {
                    const float b = __fsub_rn(xj[c][k], o[k]);
                    nb = __fmaf_rn(b, b, nb);
                    xj[c][k] = __fmul_rn(-2.0f, b);
                }
                // hit when v = |a|^2 - 2 a.b <= tlo, miss when v > thi (see the bound above)
                const float slack = __fadd_rn(__fmul_rn(gram_kappa<D>(), __fadd_rn(nmax, nb)),
                                              __fmul_rn(kGramSigma, e2));
                tlo[c] = __fsub_rn(__fsub_rn(__fmul_rn(e2, 1.0f - gram_gamma<D>()), nb), slack);
                thi[c] = __fadd_rn(__fsub_rn(__fmul_rn(e2, 1.0f + gram_gamma<D>()), nb), slack);
            }
        }
#pragma unroll 2
        for (int k = nk - 1; k >= 0; --k) {
            if constexpr (GRAM) {
                float a[D];
                load_point_smem<D>(sa + k * P, a);
                const float na = s_n[wib][k];
#pragma unroll
                for (int c = 0; c < CH; ++c) {
                    const float v = gram_value<D>(a, na, xj[c]);
                    miss[c] = push_sign(miss[c], __fsub_rn(tlo[c], v));
                    over[c] = push_sign(over[c], __fsub_rn(thi[c], v));
                }
            } else {
                float xi[D];
                load_point_smem<D>(si + k * P, xi);
                // the reference's sum; e2 - len is negative exactly when len > e2 (the
                // difference of two different floats never rounds to zero, and
                // coordinates in the grid are finite, so len is never NaN)
#pragma unroll
                for (int c = 0; c < CH; ++c) {
                    const float len = MODE == kDirect ? dist_fma<D>(xj[c], xi) : dist_negated<D>(xj[c], xi);
                    const float d = __fsub_rn(e2, len);
                    miss[c] = push_sign(miss[c], d);
                    if constexpr (MODE == kDirect) near = fminf(near, fabsf(d));
                }
            }
        }
        if constexpr (MODE == kDirect) {
            if (near <= __fmul_rn(e2, direct_gamma<D>())) recheck_exact<D, CH>(si, nk, xj, e2, miss);
        }
        pairs += (unsigned long long)nk * (unsigned long long)min(kWarp * CH, total - tb);
        const unsigned slots = kFull >> (kWarp - nk);  // nk >= 1
        unsigned hb[CH];
#pragma unroll
        for (int c = 0; c < CH; ++c) {
            hb[c] = j[c] >= 0 ? ~miss[c] & slots : 0u;
            if constexpr (GRAM) {
                // the guard band (rare): the reference's own sum decides
                unsigned bb = j[c] >= 0 ? miss[c] & ~over[c] & slots : 0u;
                if (bb) {
                    band += __popc(bb);
                    float xr[D];
                    load_point<D>(xs, j[c], xr);
                    for (; bb; bb &= bb - 1) {
                        const int k = __ffs(bb) - 1;
                        float xi[D];
                        load_point_smem<D>(si + k * P, xi);
                        if (in_range<D>(xi, xr, e2)) hb[c] |= 1u << k;
                    }
                }
            }
        }
        if (!__any_sync(kFull, (hb[0] | hb[CH - 1]) != 0)) continue;
        if (list_cap > 0) {
#pragma unroll
            for (int c = 0; c < CH; ++c) sj[c * kWarp + lane] = j[c];
            __syncwarp();
        }
#pragma unroll
        for (int c = 0; c < CH; ++c) {
            unsigned m = transpose32<(D > 3)>(hb[c], lane);  // the candidates that hit this lane's point
            int slot = mycnt;
            mycnt += __popc(m);
            // the first list_cap neighbours of each point; complete for every point
            // whose count stays below min_pts (list_cap = min_pts - 1)
            for (; m && slot < list_cap; m &= m - 1, ++slot)
                nbr_list[(int64_t)(p0 + pid) * list_stride + slot] = sj[c * kWarp + __ffs(m) - 1];
        }
        __syncwarp();
        const bool stay = lane < nk && mycnt < min_pts;
        const unsigned act = __ballot_sync(kFull, stay);
        const int left = __popc(act);
        if (left == nk) continue;
        if (lane < nk && !stay) nn_sorted[p0 + pid] = mycnt;
        nk = left;
        if (nk == 0) break;
        const int dst = __popc(act & lanemask_lt());
        float x[P], a[GRAM ? P : 1];
        float n = 0.0f;
        if (stay) {
#pragma unroll
            for (int q = 0; q < P; ++q) x[q] = si[lane * P + q];
            if constexpr (GRAM) {
#pragma unroll
                for (int q = 0; q < P; ++q) a[q] = sa[lane * P + q];
                n = s_n[wib][lane];
            }
        }
        __syncwarp();
        if (stay) {
#pragma unroll
            for (int q = 0; q < P; ++q) si[dst * P + q] = x[q];
            if constexpr (GRAM) {
#pragma unroll
                for (int q = 0; q < P; ++q) sa[dst * P + q] = a[q];
                s_n[wib][dst] = n;
            }
            s_move[wib][dst] = make_int2(pid, mycnt);
        }
        __syncwarp();
        if (lane < nk) {
            const int2 mv = s_move[wib][lane];
            pid = mv.x;
            mycnt = mv.y;
        } else {
            mycnt = 0;
        }
        __syncwarp();
    }
    if (lane < nk) nn_sorted[p0 + pid] = mycnt;
    if (lane == 0 && pairs) atomicAdd(pair_counter, pairs);
    if constexpr (GRAM) {
        band = __reduce_add_sync(kFull, band);
        if (lane == 0 && band) atomicAdd(band_counter, (unsigned long long)band);
    }
}

// ---------------------------------------------------------------------------
// Exact counts for every point.  No point leaves early, so every pair is tested once: an
// item meets only the candidates at and behind its first point in sorted order, and a
// hit counts for both ends.  The owned side is counted as in count_kernel; the candidate
// side is the population count of the lane's hit mask, added to the candidate's count
// with one atomic per step and lane (32 consecutive counts, one transaction).  Pairs inside
// the item are met from both sides and counted on the owned side only.
// nn_sorted (zeroed before) is also the cursor of a point's neighbour list: whoever adds
// hits owns the slots from the old count on, and writes those below list_cap.  Once a
// count has reached list_cap it only grows, so from then on owned hits stay in a
// register until the end and candidate hits need no answer from the atomic.
// Measured on B200 against the form that tested both directions: 5-D 300k 1.42 -> 0.75
// ms, 3-D 1M 0.88 -> 0.51 ms, 2-D 100k 0.19 -> 0.11 ms; with the tensor-core count
// (count_tc_kernel<D, true>, the same rule) 8-D 2M 9.1 -> 5.0 ms.
// ---------------------------------------------------------------------------
template <int D, int MODE>
__global__ void __launch_bounds__(kCountWarps * kWarp) count_full_kernel(
    const int2 *__restrict__ items, const uint32_t *__restrict__ n_items, const int32_t *__restrict__ cell_start,
    const int2 *__restrict__ nbr, int n_rows, const float *__restrict__ xs, float e2, int32_t *nn_sorted,
    int32_t *__restrict__ nbr_list, int list_cap, int list_stride, unsigned long long *__restrict__ pair_counter,
    const JobDev *__restrict__ jobs, const int32_t *__restrict__ cell_job,
    unsigned long long *__restrict__ band_counter) {
    constexpr int P = Stride<D>::P;
    constexpr bool GRAM = MODE == kGram;
    static_assert(!GRAM || D >= 8, "the Gram filter is built for d >= 8");
    constexpr int CH = 2;  // candidates per lane and step: an owned point is read once per two pairs
    __shared__ __align__(16) float s_i[kCountWarps][kTile * P];
    __shared__ __align__(16) float s_a[kCountWarps][GRAM ? kTile * P : 4];  // centred points
    __shared__ float s_n[kCountWarps][GRAM ? kTile : 1];                     // their squared norms
    __shared__ RowTable s_rows[kCountWarps];
    __shared__ int s_j[kCountWarps][CH * kWarp];  // the step's candidates
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int64_t item_id = (int64_t)blockIdx.x * kCountWarps + wib;
    if (item_id >= *n_items) return;
    const int2 item = items[item_id];
    const int cell = item.x, p0 = item.y;
    const int cnt = min(kTile, cell_start[cell + 1] - p0);
    if (jobs) {
        const JobDev &J = jobs[cell_job[cell]];
        e2 = J.e2;
        list_cap = J.list_cap;
    }
    if (!nbr_list) list_cap = 0;
    float *si = s_i[wib];
    float *sa = s_a[wib];
    int *sj = s_j[wib];
    RowTable &rt = s_rows[wib];
    float o[GRAM ? D : 1];  // GRAM: the item's first point, the origin of the centring
    float nmax = 0.0f;      // GRAM: largest |a|^2 of the item
    if constexpr (GRAM) load_point<D>(xs, p0, o);
    if (lane < cnt) {
        float x[D];
        load_point<D>(xs, p0 + lane, x);
        if constexpr (!GRAM) {
#pragma unroll
            for (int k = 0; k < D; ++k) x[k] = -x[k];  // for dist_negated
        }
        store_point_smem<D>(si + lane * P, x);
        if constexpr (GRAM) {
            float a[D];
            float n = 0.0f;
#pragma unroll
            for (int k = 0; k < D; ++k) {
                a[k] = __fsub_rn(x[k], o[k]);
                n = __fmaf_rn(a[k], a[k], n);
            }
            store_point_smem<D>(sa + lane * P, a);
            s_n[wib][lane] = n;
            nmax = n;
        }
    }
    if constexpr (GRAM) {
#pragma unroll
        for (int sft = 16; sft > 0; sft >>= 1) nmax = fmaxf(nmax, __shfl_xor_sync(kFull, nmax, sft));
    }
    const int total = gather_points_from(nbr + (int64_t)cell * n_rows, n_rows, cell_start, p0, rt, lane);
    __syncwarp();
    const int me = p0 + lane;
    bool open = lane < cnt && list_cap > 0;  // this lane's point may still take list entries
    int mine = 0;              // hits of this lane's point not yet added to nn_sorted
    unsigned long long pairs = 0;
    unsigned band = 0;  // GRAM: pairs rechecked in the guard band
    const unsigned slots = kFull >> (kWarp - cnt);
    int row = 0;  // this lane's stencil row: its candidate index only grows
    for (int tb = 0; tb < total; tb += kWarp * CH) {
        int j[CH], nj[CH];
        float xj[CH][D];  // GRAM: -2 times the centred candidate b = x_j - o
        float tlo[CH], thi[CH];
        unsigned miss[CH], over[CH];  // bit k: out of range; GRAM: above the hit bound, above the miss bound
        float near = INFINITY;        // kDirect: smallest distance of a pair's sum from e2
#pragma unroll
        for (int c = 0; c < CH; ++c) {
            const int t = tb + c * kWarp + lane;
            j[c] = t < total ? row_next(rt, row, t) : -1;
            load_point<D>(xs, max(j[c], 0), xj[c]);  // lanes past the end read a valid point and are masked below
            nj[c] = list_cap > 0 && j[c] >= 0 ? __ldcg(nn_sorted + j[c]) : list_cap;
            miss[c] = over[c] = 0;
            if constexpr (GRAM) {
                float nb = 0.0f;
#pragma unroll
                for (int k = 0; k < D; ++k) {
                    const float b = __fsub_rn(xj[c][k], o[k]);
                    nb = __fmaf_rn(b, b, nb);
                    xj[c][k] = __fmul_rn(-2.0f, b);
                }
                // hit when v = |a|^2 - 2 a.b <= tlo, miss when v > thi (see the bound above)
                const float slack = __fadd_rn(__fmul_rn(gram_kappa<D>(), __fadd_rn(nmax, nb)),
                                              __fmul_rn(kGramSigma, e2));
                tlo[c] = __fsub_rn(__fsub_rn(__fmul_rn(e2, 1.0f - gram_gamma<D>()), nb), slack);
                thi[c] = __fadd_rn(__fsub_rn(__fmul_rn(e2, 1.0f + gram_gamma<D>()), nb), slack);
            }
        }
#pragma unroll 2
        for (int k = cnt - 1; k >= 0; --k) {
            if constexpr (GRAM) {
                float a[D];
                load_point_smem<D>(sa + k * P, a);
                const float na = s_n[wib][k];
#pragma unroll
                for (int c = 0; c < CH; ++c) {
                    const float v = gram_value<D>(a, na, xj[c]);
                    miss[c] = push_sign(miss[c], __fsub_rn(tlo[c], v));
                    over[c] = push_sign(over[c], __fsub_rn(thi[c], v));
                }
            } else {
                float xi[D];
                load_point_smem<D>(si + k * P, xi);
#pragma unroll
                for (int c = 0; c < CH; ++c) {
                    const float len = MODE == kDirect ? dist_fma<D>(xj[c], xi) : dist_negated<D>(xj[c], xi);
                    const float d = __fsub_rn(e2, len);
                    miss[c] = push_sign(miss[c], d);
                    if constexpr (MODE == kDirect) near = fminf(near, fabsf(d));
                }
            }
        }
        if constexpr (MODE == kDirect) {
            if (near <= __fmul_rn(e2, direct_gamma<D>())) recheck_exact<D, CH>(si, cnt, xj, e2, miss);
        }
        pairs += (unsigned long long)cnt * (unsigned long long)min(kWarp * CH, total - tb);
        unsigned hb[CH];
#pragma unroll
        for (int c = 0; c < CH; ++c) {
            hb[c] = j[c] >= 0 ? ~miss[c] & slots : 0u;
            if constexpr (GRAM) {
                // the guard band (rare): the reference's own sum decides
                unsigned bb = j[c] >= 0 ? miss[c] & ~over[c] & slots : 0u;
                if (bb) {
                    band += __popc(bb);
                    float xr[D];
                    load_point<D>(xs, j[c], xr);
                    for (; bb; bb &= bb - 1) {
                        const int k = __ffs(bb) - 1;
                        float xi[D];
                        load_point_smem<D>(si + k * P, xi);
                        if (in_range<D>(xi, xr, e2)) hb[c] |= 1u << k;
                    }
                }
            }
        }
        if (!__any_sync(kFull, (hb[0] | hb[CH - 1]) != 0)) continue;
        const bool lists = __any_sync(kFull, open);
        if (lists) {
#pragma unroll
            for (int c = 0; c < CH; ++c) sj[c * kWarp + lane] = j[c];
            __syncwarp();
        }
#pragma unroll
        for (int c = 0; c < CH; ++c) {
            if (hb[c] && j[c] >= p0 + cnt)
                add_hits(nn_sorted, nbr_list, list_cap, list_stride, j[c], nj[c] < list_cap, hb[c],
                         [&](int k) { return p0 + k; });
            const unsigned m = transpose32(hb[c], lane);  // the candidates that hit this lane's point
            if (m && open) {
                const int got = add_hits(nn_sorted, nbr_list, list_cap, list_stride, me, true, m,
                                         [&](int k) { return sj[c * kWarp + k]; });
                open = got < list_cap;
            } else {
                mine += __popc(m);
            }
        }
        __syncwarp();
    }
    if (mine) atomicAdd(nn_sorted + me, mine);
    if (lane == 0 && pairs) atomicAdd(pair_counter, pairs);
    if constexpr (GRAM) {
        band = __reduce_add_sync(kFull, band);
        if (lane == 0 && band) atomicAdd(band_counter, (unsigned long long)band);
    }
}

// Core flags: per sorted point (u8), and a bitmap in input order (one bit per
// point, atomicOr; 12.5 MB for 10^8 points, so it stays in L2).  With the
// per-word prefix of its popcounts the bitmap gives every point's rank among the
// cores in input order (data_process.cpp:276-283, :153) without a per-point scan.
__global__ void core_flags_kernel(const int32_t *__restrict__ nn_sorted, int64_t nv, int64_t n, int min_pts,
                                  const int32_t *__restrict__ perm, const int32_t *__restrict__ pcell,
                                  uint8_t *__restrict__ core_sorted, uint8_t *__restrict__ cell_has_core,
                                  uint32_t *__restrict__ core_bits, const JobDev *__restrict__ jobs,
                                  const int32_t *__restrict__ cell_job, int n_jobs) {
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    if (jobs) min_pts = jobs[s < nv ? cell_job[pcell[s]] : job_of_point(jobs, n_jobs, perm[s])].min_pts;
    bool core;
    if (s < nv) {
        core = nn_sorted[s] >= min_pts;
        core_sorted[s] = core ? 1 : 0;
        if (core) cell_has_core[pcell[s]] = 1;
    } else {
        core = 0 >= min_pts;  // points outside the grid have no neighbour, not even themselves
    }
    if (core) {
        const int32_t o = perm[s];
        atomicOr(core_bits + (o >> 5), 1u << (o & 31));
    }
}

// Cores before each word of the bitmap (chain_scan_kernel over the words).
struct CorePrefixOp {
    const uint32_t *bits;
    uint32_t *prefix;
    __device__ uint32_t value(int64_t w) const { return (uint32_t)__popc(bits[w]); }
    __device__ void early(int64_t) const {}
    __device__ void emit(int64_t w, uint32_t, uint32_t before) const { prefix[w] = before; }
};

__device__ __forceinline__ bool is_core_o(const uint32_t *__restrict__ bits, int32_t o) {
    return (bits[o >> 5] >> (o & 31)) & 1u;
}

// rank of point o among the cores, in input order
__device__ __forceinline__ int32_t core_rank(const uint32_t *__restrict__ bits, const uint32_t *__restrict__ prefix,
                                             int32_t o) {
    return (int32_t)(prefix[o >> 5] + __popc(bits[o >> 5] & ((1u << (o & 31)) - 1u)));
}

// nn in input order (the caller's nn output)
// Input-order outputs are random 4-byte writes.  When the output is much larger
// than L2 the host runs the scatter in destination windows [win_lo, win_hi): each
// pass streams the sorted arrays (evict-first loads) and writes only the points
// whose destination falls in its window, so the partial-sector writes stay in L2.
__global__ void scatter_nn_kernel(const int32_t *__restrict__ nn_sorted, int64_t nv, int64_t n,
                                  const int32_t *__restrict__ perm, int32_t *__restrict__ out, int64_t win_lo,
                                  int64_t win_hi) {
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const int32_t o = __ldcs(perm + s);
    if (o < win_lo || o >= win_hi) return;
    out[o] = s < nv ? __ldcs(nn_sorted + s) : 0;
}

// Start of the label phase: every unit its own root, no component minimum yet; point
// units: no cell root yet (cell_root, null for cell units) and no union segment.
__global__ void init_units_kernel(int32_t *__restrict__ parent, int32_t *__restrict__ comp_min, int64_t bound,
                                  const uint32_t *__restrict__ n_cells, int32_t *__restrict__ cell_root,
                                  unsigned long long *__restrict__ n_seg) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < bound) {
        parent[i] = (int32_t)i;
        comp_min[i] = kNoCluster;
        if (cell_root && i < *n_cells) cell_root[i] = -1;
    }
    if (i == 0 && cell_root) *n_seg = 0;
}

// bytes [0, bytes) of p set to v: n16 16-byte stores (p 16-byte aligned; 0 when it
// is not), then the tail byte by byte
__global__ void fill_bytes_kernel(uint8_t *__restrict__ p, size_t bytes, int64_t n16, uint8_t v) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t w = 0x01010101u * v;
    for (int64_t i = t; i < n16; i += stride) reinterpret_cast<uint4 *>(p)[i] = make_uint4(w, w, w, w);
    for (int64_t i = n16 * 16 + t; i < (int64_t)bytes; i += stride) p[i] = v;
}

// n words from src to dst (either may be mapped host memory)
__global__ void copy_words_kernel(const uint32_t *__restrict__ src, uint32_t *__restrict__ dst, int64_t n) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) dst[i] = src[i];
}

// Loads the core points of an item into shared memory (compacted); returns how many.
template <int D>
__device__ __forceinline__ int load_item_cores(const float *__restrict__ xs, const uint8_t *__restrict__ core_sorted,
                                               int p0, int cnt, bool want_core, float *si, int *sidx, int lane) {
    constexpr int P = Stride<D>::P;
    const bool ok = lane < cnt && ((core_sorted[p0 + lane] != 0) == want_core);
    const unsigned mask = __ballot_sync(kFull, ok);
    if (ok) {
        const int slot = __popc(mask & lanemask_lt());
        float x[D];
        load_point<D>(xs, p0 + lane, x);
        store_point_smem<D>(si + slot * P, x);
        sidx[slot] = p0 + lane;
    }
    __syncwarp();
    return __popc(mask);
}

// Is any core among points [a0, a1) of a cell in range of any core of cell B?  The first
// go through shared memory 32 at a time; lanes hold B's points.  Stops at the first hit.
template <int D>
__device__ __forceinline__ bool cells_touch(int a0, int a1, int B, const int32_t *__restrict__ cell_start,
                                            const float *__restrict__ xs, const uint8_t *__restrict__ core_sorted,
                                            float e2, float *si, int lane, unsigned long long &pairs) {
    constexpr int P = Stride<D>::P;
    const int b0 = cell_start[B], b1 = cell_start[B + 1];
    for (int ab = a0; ab < a1; ab += kWarp) {
        const int i = ab + lane;
        const bool ok = i < a1 && core_sorted[i];
        const unsigned mask = __ballot_sync(kFull, ok);
        if (ok) {
            float x[D];
            load_point<D>(xs, i, x);
            store_point_smem<D>(si + __popc(mask & lanemask_lt()) * P, x);
        }
        __syncwarp();
        const int nc = __popc(mask);
        if (nc == 0) continue;
        for (int bb = b0; bb < b1; bb += kWarp) {
            const int j = bb + lane;
            float xj[D];
            if (j < b1 && core_sorted[j]) load_point<D>(xs, j, xj);
            else fill_nan<D>(xj);
            bool hit = false;
            for (int k = 0; k < nc; ++k) {
                float xi[D];
                load_point_smem<D>(si + k * P, xi);
                hit = hit || in_range<D>(xi, xj, e2);
            }
            pairs += (unsigned long long)nc * (unsigned long long)min(kWarp, b1 - bb);
            if (__any_sync(kFull, hit)) return true;
        }
        __syncwarp();
    }
    return false;
}

// ---------------------------------------------------------------------------
// First union pass over cells: one thread per cell A and forward face (x+1, y+1, z+1;
// the neighbour B is found through the key order and the cell index), or per cell with
// the faces one after the other (gridDim.y).  It tests the first kNearProbe cores of A
// against the first kNearProbe cores of B (independent loads, 16 predicates) and links A
// and B on a hit.  Face adjacency already connects every cell of a dense region, so this
// merges dense clusters with one cheap thread per cell; the full pass then sees
// them as one root.
// ---------------------------------------------------------------------------
constexpr int kNearProbe = 4;

template <int D>
__device__ __forceinline__ void load_first_cores(const float *__restrict__ xs, const uint8_t *__restrict__ core_sorted,
                                                 int c0, int c1, float (&x)[kNearProbe][D]) {
#pragma unroll
    for (int q = 0; q < kNearProbe; ++q) {
        const int i = c0 + q;
        if (i < c1 && core_sorted[i]) load_point<D>(xs, i, x[q]);
        else fill_nan<D>(x[q]);
    }
}

template <int D, typename K>
__global__ void __launch_bounds__(kBlock) union_near_kernel(
    const uint32_t *__restrict__ n_cells_dev, GridDev g_one, const K *__restrict__ cell_key, const int32_t *__restrict__ cell_start,
    CellIndex<K> L, const float *__restrict__ xs, float e2, const uint8_t *__restrict__ core_sorted,
    const uint8_t *__restrict__ cell_has_core, int32_t *parent, unsigned long long *__restrict__ pair_counter,
    int *err, const JobDev *__restrict__ jobs, const int32_t *__restrict__ cell_job) {
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, n_cells = *n_cells_dev;
    const int only = gridDim.y > 1 ? (int)blockIdx.y : -1;  // this thread's face, -1: all of them
    unsigned pairs = 0;
    if (idx < n_cells && cell_has_core[idx]) {
        const int A = (int)idx;
        const unsigned long long key = (unsigned long long)cell_key[A];
        GridDev g = g_one;
        unsigned long long key_base = 0;
        long long col_base = 0;
        if (jobs) {
            const JobDev &J = jobs[cell_job[A]];
            g = J.g;
            e2 = J.e2;
            key_base = J.key_base;
            col_base = J.col_base;
        }
        long long cc[kMaxGridDims];
        decode_key<K>((K)(key - key_base), g, cc);
        // the cell's column, and the keys of x = 0 in the columns one step up in y and z
        const long long col = col_base + cc[1] + (g.k >= 3 ? cc[2] * g.g[1] : 0);
        const unsigned long long row0 = key - (unsigned long long)cc[0];
        int nb[3] = {-1, -1, -1};
        if (only <= 0 && cc[0] + 1 < g.g[0] && A + 1 < n_cells && (unsigned long long)cell_key[A + 1] == key + 1ull)
            nb[0] = A + 1;
        if ((only < 0 || only == 1) && g.k >= 2 && cc[1] + 1 < g.g[1])
            nb[1] = find_cell(L, cell_key, col + 1, row0 + g.stride[1], cc[0]);
        if ((only < 0 || only == 2) && g.k >= 3 && cc[2] + 1 < g.g[2])
            nb[2] = find_cell(L, cell_key, col + g.g[1], row0 + g.stride[2], cc[0]);
        bool any = false;
#pragma unroll
        for (int f = 0; f < 3; ++f) {
            if (nb[f] >= 0 && !cell_has_core[nb[f]]) nb[f] = -1;
            any = any || nb[f] >= 0;
        }
        if (any) {
            float xa[kNearProbe][D];
            load_first_cores<D>(xs, core_sorted, cell_start[A], cell_start[A + 1], xa);
#pragma unroll
            for (int f = 0; f < 3; ++f) {
                if (nb[f] < 0) continue;
                const int B = nb[f];
                float xb[kNearProbe][D];
                load_first_cores<D>(xs, core_sorted, cell_start[B], cell_start[B + 1], xb);
                bool hit = false;
#pragma unroll
                for (int p = 0; p < kNearProbe; ++p)
#pragma unroll
                    for (int q = 0; q < kNearProbe; ++q) hit = hit || in_range<D>(xa[p], xb[q], e2);
                pairs += kNearProbe * kNearProbe;
                if (hit) uf_union(parent, A, B, err);
            }
        }
    }
    pairs = __reduce_add_sync(kFull, pairs);
    if ((threadIdx.x & 31) == 0 && pairs) atomicAdd(pair_counter, (unsigned long long)pairs);
}

// ---------------------------------------------------------------------------
// Union-find over cells (same-cell-linked grids): every pair inside a cell is in
// range, so all cores of a cell belong to one component and the cell is the
// union-find element.  One warp per cell A: the lanes gather A's half stencil
// (cells B > A holding cores), find every B's root in parallel, keep the B whose
// root differs from A's, then link A and B as soon as one core pair is in range.
// ---------------------------------------------------------------------------
constexpr int kMaxCandCells = 128;
constexpr int kProbe = 4;  // points of a candidate cell tested by the probe
// Points of A tested against a candidate cell between two looks at the roots.  Two dense
// cells that no pair links can meanwhile be joined through others, and the full test is
// the product of their sizes: 25 cells of 5,200 points in a row, one link found late, took
// 12.3 ms with one look per candidate cell, 0.15 ms with one per 64 points.
constexpr int kTouchPoints = 64;

//
// Runs after union_near_kernel has linked the adjacent dense cells, so the root
// filter removes most candidates before any point test.
// snap: every cell's root after the near pass (flatten_snap_kernel), -1 for cells
// without cores; one load per candidate tells both.  A root since hooked elsewhere
// only costs a needless probe below, never a missed union.
template <int D>
__global__ void __launch_bounds__(kBlock) union_cells_kernel(
    const uint32_t *__restrict__ n_cells, const int32_t *__restrict__ cell_start, const int2 *__restrict__ nbr, int n_rows,
    const float *__restrict__ xs, float e2, const uint8_t *__restrict__ core_sorted,
    const uint8_t *__restrict__ cell_has_core, int32_t *parent, unsigned long long *__restrict__ pair_counter,
    int *err, const JobDev *__restrict__ jobs, const int32_t *__restrict__ cell_job,
    const int32_t *__restrict__ snap) {
    constexpr int P = Stride<D>::P;
    __shared__ __align__(16) float s_i[kWarpsPerBlock][kTile * P];
    __shared__ RowTable s_rows[kWarpsPerBlock];
    __shared__ int s_b[kWarpsPerBlock][kMaxCandCells];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int64_t A64 = (int64_t)blockIdx.x * kWarpsPerBlock + wib;
    if (A64 >= *n_cells) return;
    const int A = (int)A64;
    if (!cell_has_core[A]) return;
    if (jobs) e2 = jobs[cell_job[A]].e2;
    RowTable &rt = s_rows[wib];
    int *sb = s_b[wib];
    const int total = gather_rows<true>(nbr + (int64_t)A * n_rows, n_rows, cell_start, A + 1, rt, lane);
    if (total == 0) return;
    const int rootA = __ldg(snap + A);
    // Candidate cells, four per lane per step so that their loads overlap: a cell with
    // cores whose snapshot root differs from A's is a candidate
    constexpr int U = 4;
    int nb = 0;
    for (int tb = 0; tb < total; tb += kWarp * U) {
        int B[U], p[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int t = tb + u * kWarp + lane;
            B[u] = t < total ? row_lookup(rt, n_rows, t) : -1;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) p[u] = B[u] >= 0 ? __ldg(snap + B[u]) : -1;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const bool ok = p[u] >= 0 && p[u] != rootA;
            const unsigned mask = __ballot_sync(kFull, ok);
            if (ok) {
                const int slot = nb + __popc(mask & lanemask_lt());
                if (slot < kMaxCandCells) sb[slot] = B[u];
            }
            nb += __popc(mask);
        }
    }
    __syncwarp();
    nb = min(nb, kMaxCandCells);
    unsigned long long pairs = 0;
    // Probe: A's first cores go to shared memory; each lane takes one candidate B
    // and tests B's first kProbe points against them.  Adjacent dense cells are
    // almost always settled here, in one lane-parallel round.
    {
        constexpr int P = Stride<D>::P;
        float *si = s_i[wib];
        const int a0 = cell_start[A], a1 = min(cell_start[A + 1], a0 + kWarp);
        const bool ok = a0 + lane < a1 && core_sorted[a0 + lane];
        const unsigned mask = __ballot_sync(kFull, ok);
        if (ok) {
            float x[D];
            load_point<D>(xs, a0 + lane, x);
            store_point_smem<D>(si + __popc(mask & lanemask_lt()) * P, x);
        }
        __syncwarp();
        const int nc0 = __popc(mask);
        for (int q = lane; q < nb; q += kWarp) {
            const int B = sb[q];
            const int b0 = cell_start[B], b1 = min(cell_start[B + 1], b0 + kProbe);
            bool hit = false;
            for (int j = b0; j < b1 && !hit; ++j) {
                if (!core_sorted[j]) continue;
                float xj[D];
                load_point<D>(xs, j, xj);
                for (int k = 0; k < nc0 && !hit; ++k) {
                    float xi[D];
                    load_point_smem<D>(si + k * P, xi);
                    hit = in_range<D>(xi, xj, e2);
                }
                pairs += (unsigned long long)nc0;
            }
            if (hit) {
                uf_union(parent, A, B, err);
                sb[q] = -1;
            }
        }
        __syncwarp();
    }
    for (int q = 0; q < nb; ++q) {
        const int B = sb[q];
        if (B < 0) continue;
        const int a1 = cell_start[A + 1];
        for (int a = cell_start[A]; a < a1; a += kTouchPoints) {
            int same = 0;
            if (lane == 0) same = uf_find(parent, A, err) == uf_find(parent, B, err);
            if (__shfl_sync(kFull, same, 0)) break;
            if (cells_touch<D>(a, min(a + kTouchPoints, a1), B, cell_start, xs, core_sorted, e2, s_i[wib], lane, pairs)) {
                if (lane == 0) uf_union(parent, A, B, err);
                break;
            }
        }
        __syncwarp();
    }
    if (lane == 0 && pairs) atomicAdd(pair_counter, pairs);
}

// ---------------------------------------------------------------------------
// Union-find over core points (general grids), after the list unions and a flatten
// that left every core's root in a snapshot (snap: root, -1 for non-cores; cell_root:
// the one root of each cell's cores, -1 without cores, -2 when they differ).  Pairs
// are visited once (the candidate behind the item's point in sorted order).
//
// Two kernels.  union_select_kernel, one warp per item, finds the candidates that can
// still matter: when the item's cores share one root, only the cells that are not
// wholly under that root; else every stencil row.  It cuts them into segments of
// kUnionSegment candidates and lists those; union_scan_kernel walks the listed
// segments, one warp each.  Most items need nothing and a few need their whole
// stencil, so one warp per item left the GPU idle behind the longest items
// (5 % of warps resident at d = 16).  A stale snapshot root only makes a candidate
// looked at, never skipped.
//
// Bound: latency of the snapshot loads; a step whose candidates all hang under the
// item's root costs one coalesced load per lane.  Segment length: long enough that the
// rebuilt row table (about a microsecond) does not show, short enough to fill the GPU.
// Measured on B200 against one kernel with a warp per item, which read core flag,
// parent and grandparent of every candidate: 16-D 200k 1.71 -> 0.22 ms, 8-D 2M 1.84 ->
// 0.36 ms, 5-D 300k 0.36 -> 0.10 ms.  Segments of 1,024 candidates: 0.28, 0.51 ms; of 512:
// 0.18, 0.44 ms, but 5-D 2M (dense, many components at first) 9.8 instead of 8.1 ms.
// ---------------------------------------------------------------------------
constexpr int kUnionSegment = 768;

// Candidate ranges of an item at and behind its first point p0; returns their total.
// root: the snapshot root of this lane's point (-1 without one).  Depends on the
// snapshot only, so both kernels build the same table.
__device__ __forceinline__ int union_rows(int A, int p0, int root, const int32_t *__restrict__ cell_start,
                                          const int2 *__restrict__ nbr, int n_rows,
                                          const int32_t *__restrict__ cell_root, RowTable &rt, RowTable &rc,
                                          int *need_cells, int lane) {
    const int2 *nbr_row = nbr + (int64_t)A * n_rows;
    const unsigned cores = __ballot_sync(kFull, root >= 0);
    if (!cores) return 0;
    const int root0 = __shfl_sync(kFull, root, __ffs(cores) - 1);
    if (__all_sync(kFull, root < 0 || root == root0)) {
        const int tcells = gather_rows<true>(nbr_row, n_rows, cell_start, A, rc, lane);
        int n_need = 0;
        for (int cb = 0; cb < tcells; cb += kWarp) {
            const int t = cb + lane;
            const int c = t < tcells ? row_lookup(rc, n_rows, t) : -1;
            const int r = c >= 0 ? __ldg(cell_root + c) : -1;
            const bool need = r != -1 && r != root0;
            const unsigned m = __ballot_sync(kFull, need);
            const int slot = n_need + __popc(m & lanemask_lt());
            if (need && slot < kWarp) need_cells[slot] = c;
            n_need += __popc(m);
        }
        __syncwarp();
        if (n_need <= kWarp) {
            int start = 0, len = 0;
            if (lane < n_need) {
                const int c = need_cells[lane];
                start = max(cell_start[c], p0);
                len = max(cell_start[c + 1] - start, 0);
            }
            return build_rows(start, len, n_need, rt, lane);
        }
    }
    return gather_points_from(nbr_row, n_rows, cell_start, p0, rt, lane);
}

__global__ void __launch_bounds__(kBlock) union_select_kernel(
    const int2 *__restrict__ items, const uint32_t *__restrict__ n_items, const int32_t *__restrict__ cell_start,
    const int2 *__restrict__ nbr, int n_rows, const int32_t *__restrict__ cell_root,
    const int32_t *__restrict__ snap, uint32_t *__restrict__ seg_item, uint32_t *__restrict__ seg_part,
    uint32_t seg_cap, unsigned long long *__restrict__ n_seg) {
    __shared__ RowTable s_rows[kWarpsPerBlock];
    __shared__ RowTable s_cells[kWarpsPerBlock];
    __shared__ int s_need[kWarpsPerBlock][kWarp];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int64_t item_id = (int64_t)blockIdx.x * kWarpsPerBlock + wib;
    if (item_id >= *n_items) return;
    const int2 item = items[item_id];
    const int A = item.x, p0 = item.y;
    if (__ldg(cell_root + A) == -1) return;
    const int cnt = min(kTile, cell_start[A + 1] - p0);
    const int root = lane < cnt ? __ldg(snap + p0 + lane) : -1;
    const int total = union_rows(A, p0, root, cell_start, nbr, n_rows, cell_root, s_rows[wib], s_cells[wib],
                                 s_need[wib], lane);
    const int parts = (int)(((unsigned)total + kUnionSegment - 1) / kUnionSegment);
    unsigned long long base = 0;  // 64 bits: the sum must not wrap where it overruns the list
    if (lane == 0 && parts) base = atomicAdd(n_seg, (unsigned long long)parts);
    base = __shfl_sync(kFull, base, 0);
    for (int q = lane; q < parts; q += kWarp) {
        const unsigned long long at = base + (unsigned long long)q;
        if (at < seg_cap) {
            seg_item[at] = (uint32_t)item_id;
            seg_part[at] = (uint32_t)q;
        }
    }
}

// When the segments overran their list (possible only without neighbour lists, on
// dense data), or when there is no list (seg_item null: without neighbour lists, on sparse
// data, where a second pass over the stencils cost more than it settled: minPts 1, 4-D 1M
// points in 0.96M cells, union phase 1.80 -> 0.95 ms), every item is walked whole instead.
template <int D>
__global__ void __launch_bounds__(kCountWarps * kWarp) union_scan_kernel(
    const int2 *__restrict__ items, const uint32_t *__restrict__ n_items, const int32_t *__restrict__ cell_start,
    const int2 *__restrict__ nbr, int n_rows, const float *__restrict__ xs, float e2,
    const int32_t *__restrict__ cell_root, const int32_t *__restrict__ snap, int32_t *parent,
    const uint32_t *__restrict__ seg_item, const uint32_t *__restrict__ seg_part, uint32_t seg_cap,
    const unsigned long long *__restrict__ n_seg, unsigned long long *__restrict__ pair_counter, int *err,
    const JobDev *__restrict__ jobs, const int32_t *__restrict__ cell_job) {
    constexpr int P = Stride<D>::P;
    __shared__ __align__(16) float s_i[kCountWarps][kTile * P];
    __shared__ int s_idx[kCountWarps][kTile];
    __shared__ int s_root[kCountWarps][kTile];
    __shared__ RowTable s_rows[kCountWarps];
    __shared__ RowTable s_cells[kCountWarps];
    __shared__ int s_need[kCountWarps][kWarp];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    float *si = s_i[wib];
    int *sidx = s_idx[wib];
    int *sroot = s_root[wib];
    RowTable &rt = s_rows[wib];
    unsigned long long pairs = 0;
    const bool listed = seg_item && *n_seg <= seg_cap;
    const uint32_t n_work = listed ? (uint32_t)*n_seg : *n_items;
    for (uint32_t w = blockIdx.x * kCountWarps + wib; w < n_work; w += gridDim.x * kCountWarps) {
        const int2 item = items[listed ? seg_item[w] : w];
        const int A = item.x, p0 = item.y;
        if (jobs) e2 = jobs[cell_job[A]].e2;
        const int cnt = min(kTile, cell_start[A + 1] - p0);
        const int mine = lane < cnt ? __ldg(snap + p0 + lane) : -1;
        // items walked whole: no lists, so the snapshot holds no joined cells to leave out
        int total = 0;
        if (listed) {
            total = union_rows(A, p0, mine, cell_start, nbr, n_rows, cell_root, rt, s_cells[wib], s_need[wib], lane);
        } else if (__any_sync(kFull, mine >= 0)) {
            total = gather_points_from(nbr + (int64_t)A * n_rows, n_rows, cell_start, p0, rt, lane);
            if (total == 1) continue;  // the item's own point
        }
        if (total == 0) continue;
        const int first = listed ? (int)seg_part[w] * kUnionSegment : 0;
        const int end = listed ? min(total - first, kUnionSegment) + first : total;
        // the item's cores, compacted: slot k holds its coordinates, index and root
        const unsigned cores = __ballot_sync(kFull, mine >= 0);
        const int nc = __popc(cores);
        if (mine >= 0) {
            const int slot = __popc(cores & lanemask_lt());
            float x[D];
            load_point<D>(xs, p0 + lane, x);
            store_point_smem<D>(si + slot * P, x);
            sidx[slot] = p0 + lane;
            sroot[slot] = mine;
        }
        __syncwarp();
        // cur0: the current root of the largest group of the item's cores, whose
        // snapshot root is snap0; diff: the slots under another root
        const int r_first = lane < nc ? sroot[lane] : -1 - lane;
        const unsigned peers = __match_any_sync(kFull, r_first);
        const int most = __reduce_max_sync(kFull, lane < nc ? __popc(peers) * kWarp + lane : -1) & (kWarp - 1);
        const int snap0 = __shfl_sync(kFull, r_first, most);
        int cur0 = 0;
        unsigned diff = 0;
        bool refresh = true;
        int row = 0;
        int j = first + lane < end ? row_next(rt, row, first + lane) : -1;
        int r = j >= 0 ? __ldg(snap + j) : -1;
        for (int tb = first; tb < end; tb += kWarp) {
            // the next step's candidate is loaded one step ahead
            const int jc = j, rc = r;
            const int t = tb + kWarp + lane;
            j = t < end ? row_next(rt, row, t) : -1;
            r = j >= 0 ? __ldg(snap + j) : -1;
            if (refresh) {
                const int now = lane < nc ? uf_find(parent, sroot[lane], err) : -1;
                cur0 = __shfl_sync(kFull, now, most);
                if (lane < nc) sroot[lane] = now;
                diff = __ballot_sync(kFull, lane < nc && now != cur0);
                refresh = false;
                __syncwarp();
            }
            const bool valid = rc >= 0;
            int rj = cur0;
            if (valid && rc != snap0) rj = uf_find(parent, rc, err);
            // candidates under another root meet every core, the others only the cores in diff
            const unsigned other = __ballot_sync(kFull, valid && rj != cur0);
            const unsigned test = other ? kFull >> (kWarp - nc) : diff;
            if (!test) continue;
            float xj[D];
            if (valid) load_point<D>(xs, jc, xj);
            else fill_nan<D>(xj);
            int tested = 0;
            bool joined = false;
            for (unsigned it = test; it; it &= it - 1) {
                const int k = __ffs(it) - 1;
                const int rk = sroot[k];
                const bool want = valid && jc > sidx[k] && rk != rj;
                if (!__any_sync(kFull, want)) continue;
                float xi[D];
                load_point_smem<D>(si + k * P, xi);
                bool hit = false;
                if constexpr (D >= 8) {
                    // the second half of the sum only when some lane's first half is
                    // still within e2 (exact: partial sums only grow)
                    constexpr int H = D / 2;
                    const float len = dist_part<D, 0, H>(xi, xj, 0.0f);
                    if (__any_sync(kFull, want && len <= e2)) hit = want && dist_part<D, H, D>(xi, xj, len) <= e2;
                } else {
                    hit = want && in_range<D>(xi, xj, e2);
                }
                tested += want ? 1 : 0;
                // finds from known ancestors; the shared root that comes back is again
                // an ancestor of the candidate
                if (hit) {
                    rj = uf_union_root(parent, rk, rj, err);
                    joined = true;
                }
            }
            pairs += (unsigned long long)__reduce_add_sync(kFull, (unsigned)tested);
            refresh = __any_sync(kFull, joined);
        }
        __syncwarp();
    }
    if (lane == 0 && pairs) atomicAdd(pair_counter, pairs);
}

// Lanes that share a root combine their core rank r, and one lane per root adds it to
// the component's minimum (clusters have millions of cores).
__device__ __forceinline__ void add_comp_min(bool ok, int root, int r, int32_t *__restrict__ comp_min) {
    unsigned pending = __ballot_sync(kFull, ok);
    const int lane = threadIdx.x & 31;
    while (pending) {
        const int leader = __ffs(pending) - 1;
        const int lroot = __shfl_sync(kFull, root, leader);
        const bool mine = ok && root == lroot;
        const int m = (int)__reduce_min_sync(kFull, mine ? (unsigned)r : (unsigned)kNoCluster);
        if (lane == leader) atomicMin(comp_min + lroot, m);
        pending &= ~__ballot_sync(kFull, mine);
    }
}

// Point units: parent[s] = root of s for every core, comp_min[root] = smallest core rank
// of the component.  Thread s is the only writer of parent[s] (read-only finds).
__global__ void flatten_min_points_kernel(int32_t *parent, int64_t nv, int *err, const uint8_t *__restrict__ core_sorted,
                                          const int32_t *__restrict__ perm, const uint32_t *__restrict__ core_bits,
                                          const uint32_t *__restrict__ core_prefix, int32_t *__restrict__ comp_min) {
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const bool ok = s < nv && core_sorted[s];
    int root = -1, r = kNoCluster;
    if (ok) {
        root = uf_find_ro(parent, (int)s, err);
        parent[s] = root;
        r = core_rank(core_bits, core_prefix, perm[s]);
    }
    add_comp_min(ok, root, r, comp_min);
}

// Cell units: the same per cell.  The smallest core rank of a cell is its first core's,
// because the stable radix sort (of points in input order) keeps the points of a cell in
// input order: one thread per cell instead of one per point.
__global__ void flatten_min_cells_kernel(int32_t *parent, const uint32_t *__restrict__ n_cells, int *err,
                                         const int32_t *__restrict__ cell_start,
                                         const uint8_t *__restrict__ cell_has_core,
                                         const uint8_t *__restrict__ core_sorted, const int32_t *__restrict__ perm,
                                         const uint32_t *__restrict__ core_bits,
                                         const uint32_t *__restrict__ core_prefix, int32_t *__restrict__ comp_min) {
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const bool ok = c < *n_cells && cell_has_core[c];
    int root = -1, r = kNoCluster;
    if (ok) {
        root = uf_find_ro(parent, (int)c, err);
        parent[c] = root;
        int p = cell_start[c];
        while (!core_sorted[p]) ++p;  // the cell has a core
        r = core_rank(core_bits, core_prefix, perm[p]);
    }
    add_comp_min(ok, root, r, comp_min);
}

// Point units, after the list unions: parent flattened, every
// core's root in snap (-1 for non-cores), and the one root of each cell's cores in
// cell_root: -1 without cores, -2 when they do not all share it.  One thread per
// point: the first core of a cell to arrive installs its root, any core with another
// root marks the cell mixed; a core whose root is already there skips the atomic.
// cell_root starts at -1.
__global__ void flatten_points_kernel(int32_t *parent, int64_t nv, int *err, const int32_t *__restrict__ pcell,
                                      const uint8_t *__restrict__ core_sorted, int32_t *__restrict__ snap,
                                      int32_t *cell_root) {
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nv) return;
    if (!core_sorted[s]) {
        snap[s] = -1;  // never an end of a union: parent[s] is s
        return;
    }
    const int r = uf_find_ro(parent, (int)s, err);
    parent[s] = r;
    snap[s] = r;
    const int c = pcell[s];
    const int cur = __ldcg(cell_root + c);
    if (cur == r || cur == -2) return;
    const int old = cur == -1 ? atomicCAS(cell_root + c, -1, r) : cur;
    if (old != -1 && old != r) atomicExch(cell_root + c, -2);
}

// First step of the union: every core is joined to the cores among the first
// neighbours the count recorded for it (at most kListUnions of them; no distance
// test, each listed point is in range).  Point units join the points, cell units
// their cells.  Clusters are then nearly all linked, and the candidate scans that
// follow skip every candidate already under the same root.  The points of a same-cell-
// linked grid's cells of >= min_pts points take no part: with the early exit the count
// records no list there, and with full counts their lists lead all over the stencil
// (2-D 3M: 0.49 ms of unions against 1.08 with them); the near and cell passes join
// those cells.  2^split_log2 threads share a core's list: a thread's unions follow each
// other, so few points are done sooner by more threads (100k points 2-D: 22 -> 9 us), many
// points by fewer, whose finds start from the previous union's root (8-D 2M: one thread
// 0.35 ms, two 0.53, four 1.0).
#ifndef NDB_LIST_UNIONS
#define NDB_LIST_UNIONS 16
#endif
constexpr int kListUnions = NDB_LIST_UNIONS;  // a build-time choice
__global__ void union_lists_kernel(int64_t nv, const int32_t *__restrict__ nn_sorted,
                                   const int32_t *__restrict__ nbr_list, int list_cap, int list_stride,
                                   const uint8_t *__restrict__ core_sorted, int32_t *parent, int *err,
                                   const JobDev *__restrict__ jobs, const int32_t *__restrict__ cell_job,
                                   const int32_t *__restrict__ pcell, int cell_units,
                                   const int32_t *__restrict__ cell_start, int min_pts, int split_log2) {
    const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t s = gid >> split_log2;
    if (s >= nv || !core_sorted[s]) return;
    int cap = list_cap;
    if (jobs) {
        const JobDev &J = jobs[cell_job[pcell[s]]];
        cap = J.list_cap;
        min_pts = J.min_pts;
    }
    const int a = cell_units ? pcell[s] : (int)s;
    if (cell_units && cell_start[a + 1] - cell_start[a] >= min_pts) return;
    const int len = min(min(nn_sorted[s], cap), kListUnions);
    const int32_t *l = nbr_list + s * list_stride;
    // every union starts its find from the root the previous one left (an ancestor
    // of a), not from a itself
    int ra = a;
    for (int q = (int)(gid & ((1 << split_log2) - 1)); q < len; q += 1 << split_log2) {
        const int j = l[q];
        if (j == (int)s || !core_sorted[j]) continue;
        const int b = cell_units ? pcell[j] : j;
        if (a != b) ra = uf_union_root(parent, ra, b, err);
    }
}

// Exact counts over points (and short lists), after the list unions: a core joins the middle core of its cell
// when that is in range.  Such a count fills a list with hits around the item it came
// from (every pair is met once, from the item that comes first), so on data that fill a cell
// densely the lists leave one component per item, and every item then walks its whole
// stencil: 9-D 66,000 uniform points, all near, union phase 1.47 -> 0.14 ms; 5-D 300k clustered
// 0.18 -> 0.15 ms, 8-D 2M 1.47 -> 1.51 ms.  One distance per core that is not joined yet.
// With the early exit, whose lists begin with the first hits of the nearest row and so meet
// in the same points, only lists of fewer than kShortLists entries need it: minPts 2, 13-D
// 300k uniform points 47.6 -> 4.4 ms, 8-D 200k 9.8 -> 3.7 ms, 8-D 300k clustered 0.44 both ways.
template <int D>
__global__ void union_middle_kernel(int64_t nv, const int32_t *__restrict__ pcell,
                                    const int32_t *__restrict__ cell_start, const float *__restrict__ xs, float e2,
                                    const uint8_t *__restrict__ core_sorted, int32_t *parent, int *err,
                                    const JobDev *__restrict__ jobs, const int32_t *__restrict__ cell_job) {
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nv || !core_sorted[s]) return;
    const int c = pcell[s], cs = cell_start[c], mid = cs + (cell_start[c + 1] - cs) / 2;
    if (mid == (int)s || !core_sorted[mid]) return;
    const int ra = uf_find(parent, (int)s, err), rm = uf_find(parent, mid, err);
    if (ra == rm) return;
    if (jobs) e2 = jobs[cell_job[c]].e2;
    float xa[D], xm[D];
    load_point<D>(xs, (int)s, xa);
    load_point<D>(xs, mid, xm);
    if (in_range<D>(xa, xm, e2)) uf_union_root(parent, ra, rm, err);
}

// After the list and near unions of cell units: parent[u] = root of u (thread u is its
// only writer, with read-only finds), and each cell's root in snap (-1 for a cell
// without cores) for the candidate filter of union_cells_kernel.
__global__ void flatten_snap_kernel(int32_t *parent, const uint32_t *__restrict__ n_cells, int *err,
                                    const uint8_t *__restrict__ has_core, int32_t *__restrict__ snap) {
    const int64_t u = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (u >= *n_cells) return;
    const int r = uf_find_ro(parent, (int)u, err);
    parent[u] = r;
    snap[u] = has_core[u] ? r : -1;
}

// Ids of the cores in sorted order, and for cell units the id of every cell's component;
// counters[0] += component roots.
__global__ void ids_kernel(int64_t nv, const uint32_t *__restrict__ n_cells, const uint8_t *__restrict__ core_sorted,
                           const int32_t *__restrict__ pcell, const uint8_t *__restrict__ cell_has_core,
                           int cell_units, const int32_t *__restrict__ parent, const int32_t *__restrict__ comp_min,
                           int32_t *__restrict__ ci_sorted, int32_t *__restrict__ cell_cid,
                           unsigned long long *__restrict__ counters, const int32_t *__restrict__ cell_job,
                           unsigned long long *__restrict__ job_counters) {
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    unsigned roots = 0;
    if (s < nv) {
        int id = kNoCluster;
        if (core_sorted[s]) {
            const int cell = pcell[s], root = parent[cell_units ? cell : (int)s];
            id = comp_min[root];
            if (!cell_units && root == (int)s) {
                if (job_counters) atomicAdd(job_counters + 4 * cell_job[cell], 1ull);
                else roots = 1;
            }
        }
        ci_sorted[s] = id;
    }
    if (cell_units && s < *n_cells) {
        int id = kNoCluster;
        if (cell_has_core[s]) {
            const int root = parent[s];
            id = comp_min[root];
            if (root == (int)s) {
                if (job_counters) atomicAdd(job_counters + 4 * cell_job[s], 1ull);
                else roots = 1;
            }
        }
        cell_cid[s] = id;
    }
    roots = __reduce_add_sync(kFull, roots);
    if ((threadIdx.x & 31) == 0 && roots) atomicAdd(counters + 0, (unsigned long long)roots);
}

// ---------------------------------------------------------------------------
// Border points: every non-core point takes the minimum cluster id over the
// cores in range (data_process.cpp:204-209), NO_CLUSTER when there is none.
// Cell units: all cores of a cell share one id, so the warp lists the stencil's
// core cells with their ids, sorts them by id, and walks them in that order; a
// point is settled by the first cell that has a core in range, and the walk ends
// once every point of the item is settled or no cell can lower its minimum.
// Point units: the flattened candidates carry their own ids; the warp takes the
// minimum over the candidates in range.
// ---------------------------------------------------------------------------
template <int D>
__global__ void __launch_bounds__(kBlock) border_kernel(
    const int2 *__restrict__ items, const uint32_t *__restrict__ n_items, const int32_t *__restrict__ cell_start,
    const int2 *__restrict__ nbr, int n_rows, const float *__restrict__ xs, float e2,
    const uint8_t *__restrict__ core_sorted, const uint8_t *__restrict__ cell_has_core, int cell_units,
    const int32_t *__restrict__ cell_cid, int32_t *__restrict__ ci_sorted,
    unsigned long long *__restrict__ pair_counter) {
    constexpr int P = Stride<D>::P;
    __shared__ __align__(16) float s_i[kWarpsPerBlock][kTile * P];
    __shared__ int s_idx[kWarpsPerBlock][kTile];
    __shared__ RowTable s_rows[kWarpsPerBlock];
    __shared__ int2 s_cand[kWarpsPerBlock][kMaxCandCells];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int64_t item_id = (int64_t)blockIdx.x * kWarpsPerBlock + wib;
    if (item_id >= *n_items) return;
    const int2 item = items[item_id];
    const int A = item.x, p0 = item.y;
    const int cnt = min(kTile, cell_start[A + 1] - p0);
    float *si = s_i[wib];
    int *sidx = s_idx[wib];
    RowTable &rt = s_rows[wib];
    const int nb = load_item_cores<D>(xs, core_sorted, p0, cnt, false, si, sidx, lane);
    if (nb == 0) return;
    int best[kTile];
#pragma unroll
    for (int k = 0; k < kTile; ++k) best[k] = kNoCluster;
    unsigned long long pairs = 0;
    if (cell_units) {
        int2 *cand = s_cand[wib];
        const int total = gather_rows<true>(nbr + (int64_t)A * n_rows, n_rows, cell_start, 0, rt, lane);
        int nc = 0;
        for (int tb = 0; tb < total; tb += kWarp) {
            const int t = tb + lane;
            int B = 0;
            bool ok = false;
            if (t < total) {
                B = row_lookup(rt, n_rows, t);
                ok = cell_has_core[B] != 0;
            }
            const unsigned mask = __ballot_sync(kFull, ok);
            if (ok) {
                const int slot = nc + __popc(mask & lanemask_lt());
                if (slot < kMaxCandCells) cand[slot] = make_int2(cell_cid[B], B);
            }
            nc += __popc(mask);
        }
        __syncwarp();
        nc = min(nc, kMaxCandCells);
        // Visit the candidate cells in increasing id order, lazily: each round takes
        // the smallest remaining id (warp min), and the walk ends once no pending
        // point can be lowered by it.  Lane l holds candidates l, l+32, ...
        constexpr int kPer = kMaxCandCells / kWarp;
        int lcid[kPer];
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
            const int e = q * kWarp + lane;
            lcid[q] = e < nc ? cand[e].x : kNoCluster;
        }
        while (true) {
            int mloc = kNoCluster, qloc = kPer;
#pragma unroll
            for (int q = 0; q < kPer; ++q)
                if (lcid[q] < mloc) {
                    mloc = lcid[q];
                    qloc = q;
                }
            const int cid = (int)__reduce_min_sync(kFull, (unsigned)mloc);
            if (cid == kNoCluster) break;
            bool useful = false;
#pragma unroll
            for (int k = 0; k < kTile; ++k) useful = useful || (k < nb && cid < best[k]);
            if (!useful) break;  // ids only grow from here
            const int owner = __ffs(__ballot_sync(kFull, mloc == cid)) - 1;
            int B = 0;
            if (lane == owner) {
#pragma unroll
                for (int q = 0; q < kPer; ++q)
                    if (q == qloc) {
                        B = cand[q * kWarp + lane].y;
                        lcid[q] = kNoCluster;
                    }
            }
            B = __shfl_sync(kFull, B, owner);
            const int j0 = cell_start[B], j1 = cell_start[B + 1];
            for (int jb = j0; jb < j1; jb += kWarp) {
                const int j = jb + lane;
                float xj[D];
                if (j < j1 && core_sorted[j]) load_point<D>(xs, j, xj);
                else fill_nan<D>(xj);
                bool pending = false;
#pragma unroll
                for (int k = 0; k < kTile; ++k) {
                    if (k < nb && cid < best[k]) {
                        float xi[D];
                        load_point_smem<D>(si + k * P, xi);
                        if (__any_sync(kFull, in_range<D>(xi, xj, e2))) best[k] = cid;
                        else pending = true;
                    }
                }
                pairs += (unsigned long long)nb * (unsigned long long)min(kWarp, j1 - jb);
                if (!pending) break;
            }
        }
    } else {
        const int total = gather_rows<false>(nbr + (int64_t)A * n_rows, n_rows, cell_start, 0, rt, lane);
        int cur = 0;
        for (int tb = 0; tb < total; tb += kWarp) {
            const int t = tb + lane;
            int j = -1;
            if (t < total) j = row_next(rt, cur, t);
            const bool valid = j >= 0 && core_sorted[j];
            float xj[D];
            int cj = kNoCluster;
            if (valid) {
                load_point<D>(xs, j, xj);
                cj = ci_sorted[j];
            } else {
                fill_nan<D>(xj);
            }
#pragma unroll
            for (int k = 0; k < kTile; ++k) {
                if (k < nb) {
                    float xi[D];
                    load_point_smem<D>(si + k * P, xi);
                    const int v = (cj < best[k] && in_range<D>(xi, xj, e2)) ? cj : kNoCluster;
                    best[k] = min(best[k], (int)__reduce_min_sync(kFull, (unsigned)v));
                }
            }
            pairs += (unsigned long long)nb * (unsigned long long)min(kWarp, total - tb);
        }
    }
    int mine_best = kNoCluster;
#pragma unroll
    for (int k = 0; k < kTile; ++k)
        if (k == lane) mine_best = best[k];
    if (lane < nb) ci_sorted[sidx[lane]] = mine_best;
    if (lane == 0 && pairs) atomicAdd(pair_counter, pairs);
}

// ---------------------------------------------------------------------------
// Border points from the count's neighbour lists: a non-core point has fewer than
// min_pts points in range, all of them recorded by count_kernel, so its id is the
// minimum id over the cores among them -- no second stencil scan.
// ---------------------------------------------------------------------------
__global__ void border_list_kernel(int64_t nv, const int32_t *__restrict__ nn_sorted,
                                   const int32_t *__restrict__ nbr_list, int list_stride,
                                   const uint8_t *__restrict__ core_sorted, int cell_units,
                                   const int32_t *__restrict__ pcell, const int32_t *__restrict__ cell_cid,
                                   int32_t *__restrict__ ci_sorted, unsigned long long *__restrict__ pair_counter) {
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    unsigned looked = 0;
    if (s < nv && !core_sorted[s]) {
        const int cnt = min(nn_sorted[s], list_stride);
        int best = kNoCluster;
        for (int q = 0; q < cnt; ++q) {
            const int j = nbr_list[s * list_stride + q];
            if (core_sorted[j]) best = min(best, cell_units ? cell_cid[pcell[j]] : ci_sorted[j]);
        }
        looked = (unsigned)cnt;
        ci_sorted[s] = best;
    }
    looked = __reduce_add_sync(kFull, looked);
    if ((threadIdx.x & 31) == 0 && looked) atomicAdd(pair_counter, (unsigned long long)looked);
}

// Cluster ids in input order (the caller's output; out may be null) and the
// counts that need them: counters[1] += noise, counters[0] += cores outside the
// grid (possible only with min_pts <= 0: in range of nothing, each is a cluster
// of its own, numbered by its rank).
__global__ void output_ci_kernel(const int32_t *__restrict__ ci_sorted, int64_t nv, int64_t n,
                                 const int32_t *__restrict__ perm, const uint32_t *__restrict__ core_bits,
                                 const uint32_t *__restrict__ core_prefix, int32_t *__restrict__ out,
                                 unsigned long long *__restrict__ counters, int64_t win_lo, int64_t win_hi) {
    // windows as in scatter_nn_kernel; every point is counted in its own window only
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    unsigned noise = 0, roots = 0;
    const int32_t o = s < n ? __ldcs(perm + s) : 0;
    if (s < n && o >= win_lo && o < win_hi) {
        int32_t v;
        if (s < nv) {
            v = __ldcs(ci_sorted + s);
        } else if (is_core_o(core_bits, o)) {
            v = core_rank(core_bits, core_prefix, o);
            roots = 1;
        } else {
            v = kNoCluster;
        }
        noise = v == kNoCluster;
        if (out) out[o] = v;
    }
    noise = __reduce_add_sync(kFull, noise);
    roots = __reduce_add_sync(kFull, roots);
    if ((threadIdx.x & 31) == 0) {
        if (noise) atomicAdd(counters + 1, (unsigned long long)noise);
        if (roots) atomicAdd(counters + 0, (unsigned long long)roots);
    }
}

// The border step from the count's lists (border_list_kernel), the counts (scatter_nn_kernel)
// and the ids (output_ci_kernel) in one pass over the points, for outputs that stay in
// L2: the permutation is read once and nothing is launched in between.  nn_out may be
// null; use_lists 0: a border kernel has run before.  With mail the run's counters
// (mail_words from counters on) go to the host.
__global__ void finish_kernel(int64_t nv, int64_t n, const int32_t *__restrict__ nn_sorted,
                              const int32_t *__restrict__ nbr_list, int list_stride, int use_lists,
                              const uint8_t *__restrict__ core_sorted, int cell_units,
                              const int32_t *__restrict__ pcell, const int32_t *__restrict__ cell_cid,
                              int32_t *ci_sorted, const int32_t *__restrict__ perm,
                              const uint32_t *__restrict__ core_bits, const uint32_t *__restrict__ core_prefix,
                              int32_t *__restrict__ nn_out, int32_t *__restrict__ ci_out,
                              unsigned long long *__restrict__ counters, const JobDev *__restrict__ jobs, int n_jobs,
                              unsigned long long *__restrict__ job_counters, uint32_t *done, int mail_words,
                              volatile uint32_t *mail) {
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    unsigned noise = 0, roots = 0, looked = 0;
    int job = -1;  // batched runs: the point's job, whose counters take its noise and roots
    if (s < n) {
        const int32_t o = perm[s];
        int32_t v, nn = 0;
        if (s < nv) {
            nn = nn_sorted[s];
            if (use_lists && !core_sorted[s]) {
                looked = (unsigned)min(nn, list_stride);
                v = kNoCluster;
                const int32_t *l = nbr_list + s * list_stride;
                for (unsigned q = 0; q < looked; ++q) {
                    const int j = l[q];
                    if (core_sorted[j]) v = min(v, cell_units ? cell_cid[pcell[j]] : ci_sorted[j]);
                }
                ci_sorted[s] = v;
            } else {
                v = ci_sorted[s];
            }
        } else if (is_core_o(core_bits, o)) {
            v = core_rank(core_bits, core_prefix, o);
            roots = 1;
        } else {
            v = kNoCluster;
        }
        noise = v == kNoCluster;
        if (jobs) {
            // ids are ranks among all cores of the batch: make them ranks within the job
            job = job_of_point(jobs, n_jobs, o);
            const JobDev &J = jobs[job];
            if (v != kNoCluster) v -= core_rank(core_bits, core_prefix, (int32_t)J.off);
            if (J.ci_out) J.ci_out[o - J.off] = v;
            if (J.nn_out) J.nn_out[o - J.off] = nn;
        } else {
            if (ci_out) ci_out[o] = v;
            if (nn_out) nn_out[o] = nn;
        }
    }
    if (jobs) {
        // per-job counters: the lanes of one job (sorted points are grouped by job,
        // so usually the whole warp) add their noise and roots with one atomic each
        const unsigned peers = __match_any_sync(kFull, job);
        const unsigned nm = __ballot_sync(kFull, noise != 0) & peers, rm = __ballot_sync(kFull, roots != 0) & peers;
        if (job >= 0 && (int)(threadIdx.x & 31) == __ffs(peers) - 1) {
            if (nm) atomicAdd(job_counters + 4 * job + 1, (unsigned long long)__popc(nm));
            if (rm) atomicAdd(job_counters + 4 * job, (unsigned long long)__popc(rm));
        }
        noise = 0;
        roots = 0;
    }
    noise = __reduce_add_sync(kFull, noise);
    roots = __reduce_add_sync(kFull, roots);
    looked = __reduce_add_sync(kFull, looked);
    if ((threadIdx.x & 31) == 0) {
        if (noise) atomicAdd(counters + 1, (unsigned long long)noise);
        if (roots) atomicAdd(counters + 0, (unsigned long long)roots);
        if (looked) atomicAdd(counters + 4, (unsigned long long)looked);
    }
    if (mail) mail_last_block(done, reinterpret_cast<const uint32_t *>(counters), mail_words, mail);
}

// ndb_b200_assign_border: the caller's id of every core (input order) into the
// sorted ids and the cells' ids, which the border kernels read; non-cores start
// over at NO_CLUSTER.  The cores of one cell are one component, so they carry one id.
__global__ void set_core_ids_kernel(int64_t nv, const uint8_t *__restrict__ core_sorted,
                                    const int32_t *__restrict__ perm, const int32_t *__restrict__ ids,
                                    const int32_t *__restrict__ pcell, int cell_units, int32_t *__restrict__ ci_sorted,
                                    int32_t *__restrict__ cell_cid) {
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nv) return;
    if (core_sorted[s]) {
        const int32_t v = ids[perm[s]];
        ci_sorted[s] = v;
        if (cell_units) cell_cid[pcell[s]] = v;
    } else {
        ci_sorted[s] = kNoCluster;
    }
}

// Ids in input order after ndb_b200_assign_border: the border pass's ids, and the
// caller's for cores outside the grid.
__global__ void output_ids_kernel(const int32_t *__restrict__ ci_sorted, int64_t nv, int64_t n,
                                  const int32_t *__restrict__ perm, const uint32_t *__restrict__ core_bits,
                                  const int32_t *__restrict__ ids, int32_t *__restrict__ out) {
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const int32_t o = perm[s];
    out[o] = s < nv ? ci_sorted[s] : (is_core_o(core_bits, o) ? ids[o] : kNoCluster);
}

// v_cluster_label in canonical form, on request: labels[rank(o)] = id of core o.
__global__ void labels_kernel(const int32_t *__restrict__ ci_sorted, int64_t nv, int64_t n,
                              const int32_t *__restrict__ perm, const uint32_t *__restrict__ core_bits,
                              const uint32_t *__restrict__ core_prefix, int32_t *__restrict__ labels) {
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const int32_t o = perm[s];
    if (!is_core_o(core_bits, o)) return;
    const int32_t r = core_rank(core_bits, core_prefix, o);
    labels[r] = s < nv ? ci_sorted[s] : r;
}


// ---------------------------------------------------------------------------
// Batched runs: per-job bounding boxes, the concatenation of the jobs'
// coordinates, composite cell keys and the cell -> job map.  blockIdx.y is the job.
// ---------------------------------------------------------------------------
template <int D>
__global__ void __launch_bounds__(kBlock) gather_jobs_kernel(const JobDev *__restrict__ jobs,
                                                             float *__restrict__ coords) {
    const JobDev &J = jobs[blockIdx.y];
    const int64_t total = J.n * D;
    float *dst = coords + J.off * D;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x)
        dst[i] = J.src[i];
}

// Per-job bounding boxes (encoded bounds) and invalid-point counts
// of a batch: blocks (x, job).
template <int D>
__global__ void __launch_bounds__(kBlock) bbox_batch_kernel(const float *__restrict__ coords,
                                                            const JobDev *__restrict__ jobs, uint32_t *lo_hi,
                                                            unsigned long long *n_invalid) {
    constexpr int W = kBlock / 32;
    __shared__ int s_lh[W][2 * D];
    __shared__ unsigned s_bad[W];
    const int j = blockIdx.y;
    const JobDev &J = jobs[j];
    int lo[D], hi[D];
#pragma unroll
    for (int k = 0; k < D; ++k) {
        lo[k] = 0x7fffffff;
        hi[k] = (int)0x80000000;
    }
    unsigned bad = 0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < J.n; i += (int64_t)gridDim.x * blockDim.x) {
        float x[D];
        load_row<D>(coords + (J.off + i) * D, x);
        bool ok = x[0] != FLT_MAX;
#pragma unroll
        for (int k = 0; k < D; ++k) ok = ok && isfinite(x[k]);
        if (!ok) {
            ++bad;
            continue;
        }
#pragma unroll
        for (int k = 0; k < D; ++k) {
            const int v = ordered_int(x[k]);
            lo[k] = min(lo[k], v);
            hi[k] = max(hi[k], v);
        }
    }
    bbox_reduce<D>(lo, hi, bad, s_lh, s_bad, lo_hi + (int64_t)j * 2 * D, n_invalid + j);
}

template <int D, typename K>
__global__ void __launch_bounds__(kBlock) key_batch_kernel(const float *__restrict__ coords,
                                                           const JobDev *__restrict__ jobs, K invalid_key,
                                                           K *__restrict__ keys, uint32_t *__restrict__ core_bits,
                                                           ZeroJob zero) {
    zero.run(((int64_t)blockIdx.y * gridDim.x + blockIdx.x) * blockDim.x + threadIdx.x,
             (int64_t)gridDim.y * gridDim.x * blockDim.x);
    const JobDev &J = jobs[blockIdx.y];
    const GridDev g = J.g;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < J.n; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t o = J.off + i;
        if ((o & 31) == 0) core_bits[o >> 5] = 0;  // for core_flags_kernel
        const float *p = coords + o * D;
        K key = invalid_key;
        float x[D];  // validity from one vector load of the row; the gridded coordinates are re-read (L1)
        load_row<D>(p, x);
        bool ok = x[0] != FLT_MAX;
#pragma unroll
        for (int k = 0; k < D; ++k) ok = ok && isfinite(x[k]);
        if (ok) {
            unsigned long long kk = J.key_base;
#pragma unroll
            for (int a = 0; a < kMaxGridDims; ++a)
                if (a < g.k) kk += (unsigned long long)cell_coord(g, a, p[g.dim[a]]) * g.stride[a];
            key = (K)kk;
        }
        keys[o] = key;
    }
}

// job of every cell: the last job whose key range starts at or below the cell key
// (every job of a pipeline owns a non-empty key range, so the bases increase)
template <typename K>
__global__ void cell_job_kernel(const K *__restrict__ cell_key, int64_t n_cells, const JobDev *__restrict__ jobs,
                                int n_jobs, int32_t *__restrict__ cell_job) {
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n_cells) return;
    const unsigned long long key = (unsigned long long)cell_key[c];
    int lo = 0, hi = n_jobs - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (jobs[mid].key_base <= key) lo = mid;
        else hi = mid - 1;
    }
    cell_job[c] = lo;
}

// cores of every job: rank of the job's end minus rank of its start
__global__ void job_cores_kernel(const JobDev *__restrict__ jobs, int n_jobs, const uint32_t *__restrict__ core_bits,
                                 const uint32_t *__restrict__ core_prefix, int64_t n_total,
                                 unsigned long long *__restrict__ job_counters) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n_jobs) return;
    const JobDev &J = jobs[j];
    const int64_t end = J.off + J.n;
    const int32_t r0 = core_rank(core_bits, core_prefix, (int32_t)J.off);
    const int32_t r1 = end < n_total ? core_rank(core_bits, core_prefix, (int32_t)end)
                                     : (int32_t)(core_prefix[(n_total - 1) >> 5] +
                                                 __popc(core_bits[(n_total - 1) >> 5] &
                                                        (0xffffffffu >> (31 - ((n_total - 1) & 31)))));
    job_counters[4 * j + 2] = (unsigned long long)(r1 - r0);
}

}  // namespace ndb
