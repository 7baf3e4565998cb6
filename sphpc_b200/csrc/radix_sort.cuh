// radix_sort.cuh -- stable LSD radix sort of u32 keys with u32 values.
//
// Replaces thrust::sort_by_key (thrust_c.cu:86-91).  One "onesweep" kernel
// per 8-bit digit: every tile of 1024 to 4096 pairs ranks its keys stably inside the
// tile (warp match + per-warp digit counters, in input order), publishes its
// per-digit counts, resolves the per-digit prefix of all earlier tiles with a
// decoupled look-back, stages the tile in shared memory in digit order and
// writes each digit run contiguously.  HBM traffic per digit pass is one read
// and one write of the pairs (16 B per pair); the digit histograms of all
// passes come from one extra read of the keys (or from the hash kernel that
// produced them).  A digit that all keys share costs its pass a copy.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace sphpc {

constexpr int kRadixBits = 8;
constexpr int kRadix = 1 << kRadixBits;
constexpr int kSortThreads = 256;
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kMaxPasses = 4;

constexpr uint32_t kLbAgg = 1u << 30;   // look-back: tile aggregate available
constexpr uint32_t kLbInc = 2u << 30;   // look-back: inclusive prefix available
constexpr uint32_t kLbValue = (1u << 30) - 1u;
constexpr int kSpinLimit = 1 << 22;     // bounded waits: ~0.1-1 s, then error
constexpr int kLookBack = 4;            // look-back flags read per poll

// Pairs per thread of a tile.  A tile's latency grows with its items, and small
// sets cannot hide it behind other tiles: they take small tiles, which also
// spread over more SMs.  Measured per pass, us with 4 / 8 / 16 items: 4,096 keys
// 3.7 / 5.4 / 7.0; 97,785: 5.4 / 6.9 / 10.2; 290,177: 6.8 / 7.6 / 10.5; 524,288:
// 10.7 / 10.7 / 13.4; 1,048,573: 15.9 / 14.3 / 15.7; 2.1M: 25.9 / 21.0 / 20.1;
// 16.7M: 181 / 129 / 127.
constexpr int kSortSmall = 3 << 17, kSortMedium = 3 << 19;
inline constexpr int sort_items(int n) { return n <= kSortSmall ? 4 : n <= kSortMedium ? 8 : 16; }
inline constexpr int sort_tiles(int n) {
  const int tile = kSortThreads * sort_items(n);
  return (n + tile - 1) / tile;
}
// Most tiles of any n up to cap.
inline constexpr int sort_max_tiles(int cap) {
  int m = sort_tiles(cap);
  for (int step : {kSortSmall, kSortMedium})
    if (cap > step && sort_tiles(step) > m) m = sort_tiles(step);
  return m;
}

// Scratch needed by one sort of n pairs with `passes` digit passes.
struct SortScratch {
  uint32_t* keys_alt;     // n
  uint32_t* vals_alt;     // n
  uint32_t* err;          // error bits
  uint32_t* hist;         // kMaxPasses * kRadix digit counts, and right after them:
  uint32_t* counters;     // kMaxPasses tile counters
  uint32_t* lookback;     // kMaxPasses * tiles * kRadix
};

// Words of scratch excluding the two alternate buffers, and its layout.
inline constexpr size_t sort_aux_words(int cap) {
  return 4 + (size_t)kMaxPasses * kRadix + kMaxPasses +
         (size_t)kMaxPasses * sort_max_tiles(cap) * kRadix;
}
inline void sort_layout(SortScratch& s, uint32_t* aux) {
  s.err = aux;
  s.hist = aux + 4;
  s.counters = s.hist + (size_t)kMaxPasses * kRadix;
  s.lookback = s.counters + kMaxPasses;
}

// Clears the histograms, tile counters and look-back flags of a sort of n
// pairs (one memset).
cudaError_t sort_clear(const SortScratch& s, int n, int passes, cudaStream_t stream);

// Host: enqueue the whole sort on `stream`.  Sorts (keys, vals) by the low
// 8*passes bits of the keys.  With vals_iota the input values are taken to be
// 0..n-1 and vals is only an output buffer.  If hist_ready is true, the caller
// has called sort_clear and scratch.hist holds the digit counts of all passes
// (from a fused producer).  An odd pass count leaves the result in the scratch alternates:
// copy_back copies it into keys/vals, otherwise keys_res/vals_res say where
// it is.
cudaError_t radix_sort_pairs(uint32_t* keys, uint32_t* vals, int n, int passes,
                             const SortScratch& s, cudaStream_t stream, bool hist_ready,
                             bool vals_iota, bool copy_back, uint32_t** keys_res,
                             uint32_t** vals_res);

// Histogram of all `passes` digits, accumulated into hist (must be zeroed).
void launch_digit_histogram(const uint32_t* keys, int n, int passes, uint32_t* hist,
                            cudaStream_t stream);

// Device helper for fused producers: count the digits of one key into
// shared-memory histograms s_hist[passes][kRadix].
__device__ __forceinline__ void count_key_digits(uint32_t* s_hist, uint32_t key, int passes) {
  for (int p = 0; p < passes; ++p)
    atomicAdd(&s_hist[p * kRadix + ((key >> (p * kRadixBits)) & (kRadix - 1))], 1u);
}

// Failure-detection check of the look-back wait: one onesweep CTA waits on a
// flag that no CTA ever writes, with a poll limit of spin_limit; returns the
// error bits it raised (kErrSortSpin when the bounded wait gave up).
cudaError_t lookback_wait_probe(int spin_limit, uint32_t* err_bits);

// lower_bound / upper_bound of every c in [0, count) over sorted keys
// (FindLowerBounds / FindUpperBounds, thrust_c.cu:93-120).  err: the table of
// all cells, ended by c = count - 1; keys not below that raise kErrCellRange.
cudaError_t launch_bounds(const uint32_t* keys, int n, int count, uint32_t* out, bool upper,
                          cudaStream_t stream, uint32_t* err = nullptr);

}  // namespace sphpc
