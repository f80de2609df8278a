// Onesweep LSD radix sort of (uint32 key, uint32 index) pairs.
//
// One histogram kernel counts the 8-bit digits of every pass in a single read
// of the keys; each digit pass is then ONE kernel: a tile of 2048 keys is
// ranked in shared memory (warp multisplit with __match_any_sync, stable in
// input order), the tile's per-digit counts are chained to the preceding
// tiles by decoupled look-back, and the tile is written out through shared
// memory so that each digit run is stored contiguously.
//
// The sort is stable, so ties keep input order: sorting cell keys of
// particles 0..n-1 yields, inside each cell, ascending particle index, which
// is the order the reference's hash buckets hold (neighbor_search.cpp:14-22).
#pragma once

#include <cstddef>
#include <cstdint>

#include <cuda_runtime.h>

namespace pbf {

constexpr int kSortThreads = 256;
constexpr int kSortItems = 8;
constexpr int kSortTile = kSortThreads * kSortItems;  // 2048 keys per tile
constexpr int kSortMaxPasses = 4;

// Device scratch of one sorter, sized for `capacity` keys.
struct SortScratch {
    uint32_t* keys_alt = nullptr;  // ping-pong buffers
    uint32_t* vals_alt = nullptr;
    uint32_t* err = nullptr;       // bit 0: look-back wait gave up
    // One range, zeroed by a sort: hist | tile counters | look-back.
    uint32_t* hist = nullptr;      // [kSortMaxPasses][256]
    uint32_t* tile_ctr = nullptr;  // [kSortMaxPasses]
    uint32_t* lookback = nullptr;  // [passes][tiles of the sort][256]
    int capacity = 0;
    int tiles = 0;
};

// Bytes of one device allocation that sort_scratch_bind() carves into a
// sorter's scratch for `capacity` keys; each part starts on a 256-byte
// boundary.  constexpr, so a static array can be sized with it.
constexpr size_t sort_scratch_round(size_t b) { return (b + 255) / 256 * 256; }
constexpr size_t sort_scratch_bytes(int capacity) {
    const size_t cap = capacity > 0 ? (size_t)capacity : 1;
    const size_t tiles = (cap + kSortTile - 1) / kSortTile;
    return 2 * sort_scratch_round(cap * 4)                  // alt keys and values
           + 64                                             // error word
           + (size_t)kSortMaxPasses * 256 * 4               // hist
           + 64                                             // tile counters
           + (size_t)kSortMaxPasses * tiles * 256 * 4;      // look-back
}
// Carves the scratch out of one device allocation of sort_scratch_bytes().
void sort_scratch_bind(SortScratch& s, void* base, int capacity);

inline int sort_passes(int key_bits) { return key_bits <= 8 ? 1 : (key_bits + 7) / 8; }

// Up to this many keys one block does every pass in shared memory (a chain of
// launches over one to four tiles took 24 us for 8,000 keys).
constexpr int kSmallSort = 8192;

// A range to be set to `value` before a sort, or another build (k_clear).
struct ClearRange {
    uint32_t* p = nullptr;  // 16-byte aligned
    size_t words = 0;
    uint32_t value = 0;
};

// The sort's histograms, tile counters and look-back words (empty for a small
// sort).  The error word is cleared by its owner.
inline ClearRange sort_clear(const SortScratch& s, int n, int key_bits) {
    if (n <= kSmallSort) return ClearRange{};
    const size_t tiles = ((size_t)n + kSortTile - 1) / kSortTile;
    return ClearRange{s.hist, (size_t)kSortMaxPasses * 256 + 16 + (size_t)sort_passes(key_bits) * tiles * 256, 0u};
}

// Sets up to three ranges, in one launch.
cudaError_t clear_ranges(const ClearRange& a, const ClearRange& b, const ClearRange& c, cudaStream_t st);

// Where a kernel that makes the keys counts their digits (null for a small
// sort), and the counting: every thread of the block calls count for each of
// its keys between begin and end.
struct SortCounts {
    uint32_t* hist;
    int passes;
};
inline SortCounts sort_counts(const SortScratch& s, int n, int key_bits) {
    return SortCounts{n <= kSmallSort ? nullptr : s.hist, sort_passes(key_bits)};
}
// Blocks of kCountThreads for a kernel over n particles that counts: a few
// keys per thread at most, so that a block's counts are worth their adding.
constexpr int kCountThreads = 256;
inline int count_blocks(int n) {
    const int b = (n + kCountThreads - 1) / kCountThreads;
    return b < 152 * 8 ? b : 152 * 8;
}
#ifdef __CUDACC__
struct BlockCounts {
    uint32_t c[kSortMaxPasses][256];
    __device__ __forceinline__ void begin(const SortCounts& S) {
        if (!S.hist) return;
        for (int i = threadIdx.x; i < S.passes * 256; i += blockDim.x) (&c[0][0])[i] = 0u;
        __syncthreads();
    }
    __device__ __forceinline__ void count(const SortCounts& S, uint32_t key) {
        if (!S.hist) return;
        for (int p = 0; p < S.passes; ++p) atomicAdd(&c[p][(key >> (8 * p)) & 255u], 1u);
    }
    __device__ __forceinline__ void end(const SortCounts& S) {
        if (!S.hist) return;
        __syncthreads();
        for (int i = threadIdx.x; i < S.passes * 256; i += blockDim.x) {
            const uint32_t n = (&c[0][0])[i];
            if (n) atomicAdd(S.hist + i, n);
        }
    }
};
#endif

// Sorts keys_in[0..n) (each < 2^key_bits) whose scratch was cleared (sort_clear)
// and whose digits were counted (sort_counts); otherwise as radix_sort_pairs.
cudaError_t radix_sort_counted(const uint32_t* keys_in, uint32_t* keys_out, uint32_t* vals_out, int n,
                               int key_bits, SortScratch& s, cudaStream_t stream);

// Sorts keys_in[0..n) (each < 2^key_bits).  Values are the input positions.
// Results land in keys_out / vals_out.  keys_in is not modified and may not
// alias the outputs.  Returns a CUDA error code (cudaSuccess on success).
cudaError_t radix_sort_pairs(const uint32_t* keys_in, uint32_t* keys_out, uint32_t* vals_out,
                             int n, int key_bits, SortScratch& s, cudaStream_t stream);

}  // namespace pbf
