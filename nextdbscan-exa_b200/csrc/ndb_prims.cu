// ndb_prims.cu -- stable LSD radix sort (key, value).
//
// With chain_scan_kernel (ndb_common.cuh) it replaces the reference's generic parallel
// primitives on the hot path (exa::exclusive_scan magma_exa_omp.h:92-129, exa::copy_if
// :131-162, and the sample sort :282-364 that the reference ships but never calls).
#include "ndb_common.cuh"
#include "ndb_internal.h"

namespace ndb {

namespace {

// ---------------------------------------------------------------------------
// radix sort: 8-bit digits, least significant first, one kernel per pass.
//
// A pass reads and writes every (key, value) once; the position of a tile's digits
// among all tiles comes from the tiles before it while they run (decoupled look-back),
// so there is no separate histogram read and digit-major scan per pass (five launches
// and 4 more bytes per key and pass).  Bound: instruction issue and shared memory in the
// ranking (about 190 instructions per warp and 32 elements), then the look-back; the
// payload alone would take a quarter of the time.  Tiles of 4,096 elements keep the
// tiles' digit states (2 KB each) at 1/16 of the payload; 4 blocks per SM (64 registers)
// against 2 at 128 registers: 100 against 134 us a pass at 10M.  Measured on B200 against
// histogram, scan and scatter per pass: 100M 30-bit keys 4.00 -> 3.33 ms, 10M 31-bit keys
// 0.49 -> 0.40 ms, 100k 15-bit keys 0.055 -> 0.033 ms.
// ---------------------------------------------------------------------------
constexpr int kSortThreads = 256;
constexpr int kSortWarps = kSortThreads / kWarp;           // 8
constexpr int kRadix = kSortRadix;
constexpr uint32_t kLookBackLimit = 1u << 16;  // polls of one predecessor before the prefix is recounted

// Histograms of all passes in one read of the keys.
template <typename K>
__global__ void __launch_bounds__(kSortThreads) sort_hist_kernel(const K *__restrict__ keys, int64_t n, int passes,
                                                                 uint32_t *__restrict__ hist) {
    __shared__ uint32_t s_h[kSortMaxPasses * kRadix];
    const int t = threadIdx.x, lane = t & 31;
    for (int i = t; i < passes * kRadix; i += kSortThreads) s_h[i] = 0;
    __syncthreads();
    constexpr int U = 8;  // independent loads per thread
    const int64_t step = (int64_t)kSortThreads * U;
    for (int64_t b = (int64_t)blockIdx.x * step; b < n; b += (int64_t)gridDim.x * step) {
        K key[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int64_t e = b + u * kSortThreads + t;
            key[u] = e < n ? keys[e] : (K)0;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const bool valid = b + u * kSortThreads + t < n;
            const unsigned active = __ballot_sync(kFull, valid);
            for (int p = 0; p < passes; ++p) {
                const uint32_t d = (uint32_t)(key[u] >> (8 * p)) & 0xffu;
                // a digit the whole warp shares (the high digits of clustered keys): one addition
                const uint32_t d0 = __shfl_sync(kFull, d, 0);
                if (p >= 2 && __all_sync(kFull, !valid || d == d0)) {
                    if (lane == 0 && active) atomicAdd(&s_h[p * kRadix + d0], (uint32_t)__popc(active));
                } else if (valid) {
                    atomicAdd(&s_h[p * kRadix + d], 1u);
                }
            }
        }
    }
    __syncthreads();
    for (int i = t; i < passes * kRadix; i += kSortThreads)
        if (s_h[i]) atomicAdd(hist + i, s_h[i]);
}

// Exclusive scan over the block's 256 threads; s_w: one word per warp.
__device__ __forceinline__ uint32_t block_scan256(uint32_t v, uint32_t *s_w, int lane, int warp) {
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(kFull, x, o);
        if (lane >= o) x += y;
    }
    __syncthreads();  // s_w may still be read by the previous scan
    if (lane == 31) s_w[warp] = x;
    __syncthreads();
    uint32_t before = 0;
#pragma unroll
    for (int w = 0; w < kSortWarps; ++w)
        if (w < warp) before += s_w[w];
    return before + x - v;
}

// One pass.  Element order inside a tile: warp w owns elements [w*512, w*512+512), item j
// of lane l is element w*512 + j*32 + l.  Ranks follow that order (items in order, lanes
// in order within an item), warps follow each other, and tiles follow each other
// through the look-back, so the sort is stable.  The tile is reordered by digit in
// shared memory, so the global writes go out as contiguous runs per digit.  FIRST: the
// values are the element indices.
//
// Look-back: a tile's state word per digit holds the pass (tag), whether the count is
// the tile's own or includes all tiles before it, and the count, so a word is complete
// when its tag is this pass's.  Tiles are taken in order from a ticket, so a tile's
// predecessors are running or done.  Every poll is bounded: past the limit the block
// counts the digits of the keys before its tile itself, which needs no other block.
template <typename K, bool FIRST>
__global__ void __launch_bounds__(kSortThreads, 4) sort_pass_kernel(const K *__restrict__ kin, const int32_t *__restrict__ vin,
                                                                 K *__restrict__ kout, int32_t *__restrict__ vout,
                                                                 int64_t n, int pass, const uint32_t *__restrict__ hist,
                                                                 uint32_t *__restrict__ ticket,
                                                                 unsigned long long *state) {
    constexpr int kSortTile = SortTile<K>::v, kSortItems = kSortTile / kSortThreads;
    __shared__ uint32_t s_cnt[kSortWarps][kRadix];
    __shared__ uint32_t s_base[kRadix];  // global position of tile slot 0 if it held the digit
    __shared__ uint32_t s_local[kRadix];  // first tile slot of each digit
    __shared__ uint32_t s_w[kSortWarps];
    __shared__ K s_key[kSortTile];
    __shared__ int32_t s_val[kSortTile];
    __shared__ uint32_t s_tile;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, shift = 8 * pass;
    if (t == 0) s_tile = atomicAdd(ticket, 1u);
    for (int i = t; i < kSortWarps * kRadix; i += kSortThreads) (&s_cnt[0][0])[i] = 0;
    __syncthreads();
    const int64_t tile = s_tile, tile0 = tile * kSortTile;
    const int held = (int)min((int64_t)kSortTile, n - tile0);  // elements of the tile
    const int first = warp * (kSortItems * kWarp) + lane;      // this thread's: first + 32 j
    const K *tin = kin + tile0 + first;
    const unsigned lt = lanemask_lt();
    K key[kSortItems];
    uint32_t rank[kSortItems];
#pragma unroll
    for (int j = 0; j < kSortItems; ++j) key[j] = first + j * kWarp < held ? tin[j * kWarp] : (K)0;
    uint32_t *cnt = s_cnt[warp];
#pragma unroll
    for (int j = 0; j < kSortItems; ++j) {
        const uint32_t d = (uint32_t)(key[j] >> shift) & 0xffu;
        // lanes with the same digit: eight votes (the match instruction shares its unit
        // with shared memory, which this kernel waits for).  Past the tile's end only
        // whole suffixes of a warp's elements are missing, so the last lanes drop out.
        const bool valid = first + j * kWarp < held;
        unsigned peers = __ballot_sync(kFull, valid);
#pragma unroll
        for (int bit = 0; bit < 8; ++bit) {
            const bool one = (d >> bit) & 1u;
            const unsigned ones = __ballot_sync(kFull, one);
            peers &= ones ^ (one ? 0u : ~0u);
        }
        const uint32_t old = cnt[d], below = (uint32_t)__popc(peers & lt);
        __syncwarp();
        if (valid && below == 0) cnt[d] = old + __popc(peers);
        rank[j] = old + below;
        __syncwarp();
    }
    __syncthreads();
    // digit t: exclusive prefix over the warps, and the tile's total
    uint32_t tot = 0;
#pragma unroll
    for (int w = 0; w < kSortWarps; ++w) {
        const uint32_t c = s_cnt[w][t];
        s_cnt[w][t] = tot;
        tot += c;
    }
    const unsigned long long tag = (unsigned long long)(pass + 1) << 56, whole = 1ull << 55, count = whole - 1;
    volatile unsigned long long *mine = state + tile * kRadix + t;
    *mine = tag | (tile == 0 ? whole : 0ull) | tot;
    const uint32_t local = block_scan256(tot, s_w, lane, warp);
    const uint32_t digit0 = block_scan256(hist[pass * kRadix + t], s_w, lane, warp);
    s_local[t] = local;
    __syncthreads();
    // the tile in digit order; the values' loads overlap the look-back
#pragma unroll
    for (int j = 0; j < kSortItems; ++j) {
        if (first + j * kWarp < held) {
            const uint32_t d = (uint32_t)(key[j] >> shift) & 0xffu;
            const uint32_t slot = s_local[d] + cnt[d] + rank[j];
            s_key[slot] = key[j];
            s_val[slot] = FIRST ? (int32_t)tile0 + first + j * kWarp : vin[tile0 + first + j * kWarp];
        }
    }
    // elements of digit t in the tiles before this one, four predecessors per round
    unsigned long long before = 0;
    bool lost = false;
    for (int64_t p = tile - 1; p >= 0 && !lost;) {
        unsigned long long w[4];
#pragma unroll
        for (int q = 0; q < 4; ++q)
            w[q] = p >= q ? *(volatile unsigned long long *)(state + (p - q) * kRadix + t) : 0ull;
        bool end = false;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (end || lost || p < 0) continue;
            unsigned long long v = w[q];
            for (uint32_t it = 0; (v >> 56) != (tag >> 56) && !lost; ++it) {
                v = *(volatile unsigned long long *)(state + p * kRadix + t);
                lost = it >= kLookBackLimit;
            }
            if (lost) continue;
            before += v & count;
            end = (v & whole) != 0;
            --p;
        }
        if (end) break;
    }
    if (__syncthreads_or(lost)) {
        // a predecessor did not answer: count the keys before this tile (s_base as bins)
        s_base[t] = 0;
        __syncthreads();
        for (int64_t e = t; e < tile0; e += kSortThreads) atomicAdd(&s_base[(uint32_t)(kin[e] >> shift) & 0xffu], 1u);
        __syncthreads();
        before = s_base[t];
        __syncthreads();
    }
    *mine = tag | whole | (before + tot);
    s_base[t] = digit0 + (uint32_t)before - local;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kSortItems; ++i) {
        const int e = i * kSortThreads + t;
        if (e < held) {
            const K k = s_key[e];
            const uint32_t pos = s_base[(uint32_t)(k >> shift) & 0xffu] + (uint32_t)e;
            kout[pos] = k;
            vout[pos] = s_val[e];
        }
    }
}

template <typename K>
cudaError_t radix_sort_pairs(K *k0, int32_t *v0, K *k1, int32_t *v1, int64_t n, int bits, uint32_t *scratch,
                             bool *result_in_first, cudaStream_t st) {
    *result_in_first = true;
    if (n <= 0) return cudaSuccess;
    const int64_t tiles = (n + SortTile<K>::v - 1) / SortTile<K>::v;
    const int passes = bits <= 0 ? 1 : (bits + 7) / 8;
    uint32_t *hist = scratch, *tickets = scratch + kSortHistWords;
    unsigned long long *state = reinterpret_cast<unsigned long long *>(tickets + kSortTicketWords);
    const int64_t hist_blocks = (n + kSortThreads * 8 - 1) / (kSortThreads * 8);
    ++launch_counter(), sort_hist_kernel<K><<<(unsigned)(hist_blocks < 148 * 6 ? hist_blocks : 148 * 6), kSortThreads, 0, st>>>(
        k0, n, passes, hist);
    K *ka = k0, *kb = k1;
    int32_t *va = v0, *vb = v1;
    for (int pass = 0; pass < passes; ++pass) {
        if (pass == 0)
            ++launch_counter(), sort_pass_kernel<K, true><<<(unsigned)tiles, kSortThreads, 0, st>>>(
                ka, va, kb, vb, n, pass, hist, tickets + pass, state);
        else
            ++launch_counter(), sort_pass_kernel<K, false><<<(unsigned)tiles, kSortThreads, 0, st>>>(
                ka, va, kb, vb, n, pass, hist, tickets + pass, state);
        K *tk = ka;
        ka = kb;
        kb = tk;
        int32_t *tv = va;
        va = vb;
        vb = tv;
        *result_in_first = !*result_in_first;
    }
    return cudaGetLastError();
}

}  // namespace

int &launch_counter() {
    static thread_local int count = 0;
    return count;
}

cudaError_t radix_sort_pairs_u32(uint32_t *k0, int32_t *v0, uint32_t *k1, int32_t *v1, int64_t n,
                                 int bits, uint32_t *scratch, bool *result_in_first, cudaStream_t st) {
    return radix_sort_pairs<uint32_t>(k0, v0, k1, v1, n, bits, scratch, result_in_first, st);
}

cudaError_t radix_sort_pairs_u64(uint64_t *k0, int32_t *v0, uint64_t *k1, int32_t *v1, int64_t n,
                                 int bits, uint32_t *scratch, bool *result_in_first, cudaStream_t st) {
    return radix_sort_pairs<uint64_t>(k0, v0, k1, v1, n, bits, scratch, result_in_first, st);
}

}  // namespace ndb
