// ndb_internal.h -- host-side declarations shared by the library's translation units.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <string>

namespace ndb {

// A device buffer that only grows.
struct DevBuf {
    void *ptr = nullptr;
    size_t bytes = 0;
    cudaError_t ensure(size_t want) {
        if (want <= bytes) return cudaSuccess;
        if (ptr) cudaFree(ptr);
        ptr = nullptr;
        bytes = 0;
        size_t rounded = (want + 4095) & ~size_t(4095);
        cudaError_t e = cudaMalloc(&ptr, rounded);
        if (e == cudaSuccess) bytes = rounded;
        return e;
    }
    void release() {
        if (ptr) cudaFree(ptr);
        ptr = nullptr;
        bytes = 0;
    }
    template <typename T>
    T *as() const { return static_cast<T *>(ptr); }
};

// Kernels launched by the calling thread since the last reset (a context is used
// by one host thread at a time, so this counts the launches of one job).
int &launch_counter();

// ---- primitives (ndb_prims.cu) ----
// Elements of one sort tile, by key size.
template <typename K>
struct SortTile {
    static constexpr int v = sizeof(K) == 4 ? 4096 : 2048;
};
constexpr int kSortRadix = 256, kSortMaxPasses = 8;
// Scratch (in uint32 words, 16-byte aligned) of a sort of n pairs: the digit
// histograms of all passes, one ticket per pass (64-bit slots), and one 64-bit state
// word per digit and tile.
constexpr int kSortHistWords = kSortMaxPasses * kSortRadix;
constexpr int kSortTicketWords = 2 * kSortMaxPasses;
template <typename K>
constexpr size_t sort_scratch_words(int64_t n) {
    return kSortHistWords + kSortTicketWords +
           2 * (size_t)kSortRadix * (size_t)((n + SortTile<K>::v - 1) / SortTile<K>::v + (n <= 0));
}
// Stable LSD radix sort of (key, element index) pairs on the low `bits` bits of the
// keys in k0: sorts between (k0, v0) and (k1, v1) and returns via *result_in_first
// whether the sorted keys and indices ended in (k0, v0).  v0 need not be set.  The
// caller has zeroed the scratch.
cudaError_t radix_sort_pairs_u32(uint32_t *k0, int32_t *v0, uint32_t *k1, int32_t *v1, int64_t n,
                                 int bits, uint32_t *scratch, bool *result_in_first, cudaStream_t st);
cudaError_t radix_sort_pairs_u64(uint64_t *k0, int32_t *v0, uint64_t *k1, int32_t *v1, int64_t n,
                                 int bits, uint32_t *scratch, bool *result_in_first, cudaStream_t st);

}  // namespace ndb
