// radix_sort.cu -- onesweep LSD radix sort and the cell-bounds seam kernels.
#include "radix_sort.cuh"

#include <climits>
#include <vector>

namespace sphpc {

namespace {

__device__ __forceinline__ uint32_t ld_volatile(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.volatile.global.u32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}

__device__ __forceinline__ void st_volatile(uint32_t* p, uint32_t v) {
  asm volatile("st.volatile.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__device__ __forceinline__ uint32_t lanemask_lt() {
  uint32_t m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

__global__ void __launch_bounds__(256) k_digit_histogram(const uint32_t* __restrict__ keys,
                                                         int n, int passes,
                                                         uint32_t* __restrict__ hist) {
  __shared__ uint32_t s_hist[kMaxPasses * kRadix];
  for (int i = threadIdx.x; i < kMaxPasses * kRadix; i += blockDim.x) s_hist[i] = 0;
  __syncthreads();
  const int step = gridDim.x * blockDim.x;
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  for (; i < n - 3 * step; i += 4 * step) {
    uint32_t k[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) k[u] = __ldg(keys + i + u * step);
#pragma unroll
    for (int u = 0; u < 4; ++u) count_key_digits(s_hist, k[u], passes);
  }
  for (; i < n; i += step) count_key_digits(s_hist, __ldg(keys + i), passes);
  __syncthreads();
  for (int i = threadIdx.x; i < passes * kRadix; i += blockDim.x)
    if (s_hist[i]) atomicAdd(hist + i, s_hist[i]);
}

// One digit pass.  vals_in == nullptr means the values are the input
// indices (iota), which is how SortHash calls SortByKey (neighbors.c:123).
// Five blocks per SM (48 registers, no spills; 43 KB of shared memory
// each) rather than the two that the compiler's own choice of 128
// registers leaves room for: the passes wait on loads and on the
// look-back, so resident warps are what hides it.  The values are loaded
// only when the tile is staged, which is what lets the ranking fit.  The
// smaller tiles take eight blocks.  The digits' offsets are scanned from the
// counts in every block (256 values: less than a launch), and a digit that
// all keys share leaves the order as it is: its tiles are copied.
template <int ITEMS>
__global__ void __launch_bounds__(kSortThreads, ITEMS == 16 ? 5 : 8)
    k_onesweep(const uint32_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in,
               uint32_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out, int n,
               int shift, const uint32_t* __restrict__ digit_count,
               uint32_t* __restrict__ lookback, uint32_t* __restrict__ tile_counter,
               uint32_t* __restrict__ err, int spin_limit) {
  constexpr int kSortTile = kSortThreads * ITEMS;
  __shared__ uint32_t s_tile;
  __shared__ uint32_t s_whist[kSortWarps][kRadix + 1];
  __shared__ uint32_t s_dstart[kRadix];
  __shared__ uint32_t s_gbase[kRadix];
  __shared__ uint32_t s_wsum[kRadix / 32], s_gsum[kRadix / 32];
  __shared__ uint32_t s_keys[kSortTile];
  __shared__ uint32_t s_vals[kSortTile];

  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const uint32_t all = __ldg(digit_count + t);
  if (t == 0) s_tile = atomicAdd(tile_counter, 1u);
  for (int i = t; i < kSortWarps * (kRadix + 1); i += kSortThreads)
    (&s_whist[0][0])[i] = 0;
  const bool one_digit = __syncthreads_or(all == (uint32_t)n) != 0;
  const uint32_t tile = s_tile;
  // n <= kLbValue < 2^30, so every index fits 32 bits
  const int tile_base = (int)tile * kSortTile;
  if (one_digit) {
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
      const int idx = tile_base + i * kSortThreads + t;
      if (idx < n) {
        keys_out[idx] = __ldg(keys_in + idx);
        vals_out[idx] = vals_in ? __ldg(vals_in + idx) : (uint32_t)idx;
      }
    }
    return;
  }
  const int wbase = tile_base + warp * 32 * ITEMS;

  // the values are loaded only when the tile is staged, so that the ranking
  // holds two arrays of registers, not three
  uint32_t key[ITEMS], rank[ITEMS];
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    const int idx = wbase + i * 32 + lane;
    key[i] = idx < n ? __ldg(keys_in + idx) : 0xffffffffu;
  }
  const uint32_t lt = lanemask_lt();
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    const int idx = wbase + i * 32 + lane;
    const uint32_t d = idx < n ? ((key[i] >> shift) & (kRadix - 1)) : (uint32_t)kRadix;
    const uint32_t peers = __match_any_sync(0xffffffffu, d);
    const int leader = __ffs(peers) - 1;
    uint32_t prev = 0;
    if (lane == leader) {
      prev = s_whist[warp][d];
      s_whist[warp][d] = prev + __popc(peers);
    }
    prev = __shfl_sync(0xffffffffu, prev, leader);
    rank[i] = prev + __popc(peers & lt);
    __syncwarp();
  }
  __syncthreads();

  // Per digit: exclusive prefix over warps, the tile count, look-back.
  {
    const int d = t;  // kSortThreads == kRadix
    uint32_t sum = 0;
#pragma unroll
    for (int w = 0; w < kSortWarps; ++w) {
      const uint32_t c = s_whist[w][d];
      s_whist[w][d] = sum;
      sum += c;
    }
    const uint32_t cnt = sum;
    uint32_t* my = lookback + (size_t)tile * kRadix + d;
    if (tile == 0) {
      st_volatile(my, kLbInc | cnt);
    } else {
      st_volatile(my, kLbAgg | cnt);
    }
    uint32_t excl = 0;
    if (tile > 0) {
      // kLookBack predecessors' flags per poll, consumed in order down to the
      // first inclusive one; a poll that finds the nearest one not yet
      // published waits and polls again from there
      int64_t pt = (int64_t)tile - 1;
      int spins = 0;
      for (;;) {
        uint32_t v[kLookBack];
#pragma unroll
        for (int k = 0; k < kLookBack; ++k)
          v[k] = pt - k >= 0 ? ld_volatile(lookback + (size_t)(pt - k) * kRadix + d) : 0u;
        int k = 0;
        bool done = false;
#pragma unroll
        for (; k < kLookBack; ++k) {
          if ((v[k] & (kLbAgg | kLbInc)) == 0) break;
          excl += v[k] & kLbValue;
          if (v[k] & kLbInc) {
            done = true;
            break;
          }
        }
        if (done) break;
        pt -= k;
        if (k == 0) {
          if (++spins > spin_limit) {
            atomicOr(err, 2u);  // kErrSortSpin
            break;
          }
          __nanosleep(32);
        }
      }
      st_volatile(my, kLbInc | (excl + cnt));
    }
    // exclusive scans over the digits: of the tile's counts, and of the counts
    // of all keys
    uint32_t x = cnt, g = all;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
      const uint32_t z = __shfl_up_sync(0xffffffffu, g, o);
      if (lane >= o) {
        x += y;
        g += z;
      }
    }
    if (lane == 31) {
      s_wsum[warp] = x;
      s_gsum[warp] = g;
    }
    __syncthreads();
    uint32_t wsum = 0, gsum = 0;
    for (int w = 0; w < warp; ++w) {
      wsum += s_wsum[w];
      gsum += s_gsum[w];
    }
    s_dstart[d] = wsum + x - cnt;
    s_gbase[d] = gsum + g - all + excl;
  }
  __syncthreads();

  // Stage the tile in digit order.
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    const int idx = wbase + i * 32 + lane;
    if (idx < n) {
      const uint32_t d = (key[i] >> shift) & (kRadix - 1);
      const uint32_t lp = s_dstart[d] + s_whist[warp][d] + rank[i];
      s_keys[lp] = key[i];
      s_vals[lp] = vals_in ? __ldg(vals_in + idx) : (uint32_t)idx;
    }
  }
  __syncthreads();
  const int valid = min(kSortTile, n - tile_base);
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    const int k = t + i * kSortThreads;
    if (k < valid) {
      const uint32_t kk = s_keys[k];
      const uint32_t d = (kk >> shift) & (kRadix - 1);
      const uint32_t g = s_gbase[d] + (uint32_t)k - s_dstart[d];
      if (g < (uint32_t)n) {
        keys_out[g] = kk;
        vals_out[g] = s_vals[k];
      } else {
        atomicOr(err, 4u);  // inconsistent digit counts: never write out of range
      }
    }
  }
}

// First position of sorted keys[0, n) whose key is >= v, by the whole warp: 32
// probes per step.
__device__ int warp_lower_bound(const uint32_t* __restrict__ keys, int n, int64_t v) {
  const int lane = threadIdx.x & 31;
  int lo = 0, hi = n;  // keys before lo are < v, keys from hi on are >= v
  while (lo < hi) {
    const int step = (hi - lo + 31) / 32;
    const int at = lo + lane * step;
    const bool less = at < hi && (int64_t)__ldg(keys + at) < v;
    const int below = __popc(__ballot_sync(0xffffffffu, less));
    if (below == 0) break;
    const int last = lo + (below - 1) * step;  // the last probe below v
    hi = min(hi, last + step);
    lo = last + 1;
  }
  return lo;
}

// start[c] = lower_bound(keys, first + c) of cells c in [0, count).  A block
// takes kBoundCells cells: two warps find where their keys begin and end, the
// block reads those keys once, marks the first key of each cell, and a suffix
// minimum over the cells gives the starts of the empty ones.  A run of more than
// kBoundRange keys is searched cell by cell instead.  Bounds: the latency of the
// two searches (four dependent loads at 1M keys).  1.8M cells over 1M keys, cold
// caches: 38 us with a binary search of all keys per cell, 20 us so.
// Keys that are out of order give wrong starts, all of them in [0, n].  With err,
// the cells are all that there are (the last one ends the table), and a key beyond
// them or out of its block's cells raises its bit.
constexpr int kBoundPer = 8;
constexpr int kBoundCells = 256 * kBoundPer;
constexpr int kBoundRange = 1 << 15;
__global__ void __launch_bounds__(256)
    k_bounds(const uint32_t* __restrict__ keys, int n, int count, int first,
             uint32_t* __restrict__ out, uint32_t* __restrict__ err) {
  __shared__ int s_first[kBoundCells];
  __shared__ int s_range[2], s_min[8];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int c0 = blockIdx.x * kBoundCells;
  const int nc = min(kBoundCells, count - c0);
  const int64_t v0 = (int64_t)c0 + first;
  if (warp < 2) {
    const int b = warp_lower_bound(keys, n, v0 + (warp ? nc : 0));
    if (lane == 0) s_range[warp] = b;
  }
  for (int i = t; i < kBoundCells; i += 256) s_first[i] = INT_MAX;
  __syncthreads();
  const int lo = s_range[0], hi = s_range[1];
  // (the start of the table's last cell)
  if (err && t == 0 && c0 + nc == count && n > 0 && (int64_t)__ldg(keys + n - 1) >= count - 1)
    atomicOr(err, 4u);  // kErrCellRange
  if (hi - lo > kBoundRange) {
    for (int i = t; i < nc; i += 256) {
      int a = lo, b = hi;
      while (a < b) {
        const int mid = (a + b) >> 1;
        if ((int64_t)__ldg(keys + mid) < v0 + i) a = mid + 1; else b = mid;
      }
      out[c0 + i] = (uint32_t)a;
    }
    return;
  }
  for (int j = lo + t; j < hi; j += 256) {
    const uint32_t k = __ldg(keys + j);
    if (j == lo || __ldg(keys + j - 1) != k) {
      const uint32_t c = k - (uint32_t)v0;
      if (c < (uint32_t)nc) s_first[c] = j;
      else if (err) atomicOr(err, 4u);  // kErrCellRange
    }
  }
  __syncthreads();
  // suffix minimum: kBoundPer cells per thread, then over the lanes and the warps
  int m[kBoundPer];
#pragma unroll
  for (int u = 0; u < kBoundPer; ++u) m[u] = s_first[kBoundPer * t + u];
#pragma unroll
  for (int u = kBoundPer - 2; u >= 0; --u) m[u] = min(m[u], m[u + 1]);
  int x = m[0];
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_down_sync(0xffffffffu, x, o);
    if (lane + o < 32) x = min(x, y);
  }
  if (lane == 0) s_min[warp] = x;
  int after = __shfl_down_sync(0xffffffffu, x, 1);
  if (lane == 31) after = INT_MAX;
  __syncthreads();
  for (int w = warp + 1; w < 8; ++w) after = min(after, s_min[w]);
  after = min(after, hi);
#pragma unroll
  for (int u = 0; u < kBoundPer; ++u)
    if (kBoundPer * t + u < nc) out[c0 + kBoundPer * t + u] = (uint32_t)min(m[u], after);
}

}  // namespace

void launch_digit_histogram(const uint32_t* keys, int n, int passes, uint32_t* hist,
                            cudaStream_t stream) {
  if (n <= 0) return;
  // 4096 keys a block: fewer would spend their time adding 256 counts per
  // digit to the totals (1M keys: 12 us with 256 threads per 885 keys)
  int blocks = (n + 4095) / 4096;
  if (blocks > 148 * 8) blocks = 148 * 8;
  k_digit_histogram<<<blocks, 256, 0, stream>>>(keys, n, passes, hist);
}

cudaError_t sort_clear(const SortScratch& s, int n, int passes, cudaStream_t stream) {
  const size_t words = (size_t)kMaxPasses * kRadix + kMaxPasses +
                       (size_t)passes * sort_tiles(n > 0 ? n : 1) * kRadix;
  return cudaMemsetAsync(s.hist, 0, sizeof(uint32_t) * words, stream);
}

cudaError_t radix_sort_pairs(uint32_t* keys, uint32_t* vals, int n, int passes,
                             const SortScratch& s, cudaStream_t stream, bool hist_ready,
                             bool vals_iota, bool copy_back, uint32_t** keys_res,
                             uint32_t** vals_res) {
  if (passes < 1 || passes > kMaxPasses) return cudaErrorInvalidValue;
  if (n < 0 || (uint64_t)n > kLbValue || vals == nullptr) return cudaErrorInvalidValue;
  cudaError_t e;
  if (n <= 1) {
    if (n == 1 && vals_iota) {
      e = cudaMemsetAsync(vals, 0, sizeof(uint32_t), stream);
      if (e != cudaSuccess) return e;
    }
    if (keys_res) *keys_res = keys;
    if (vals_res) *vals_res = vals;
    return cudaSuccess;
  }
  const int tiles = sort_tiles(n);
  if (!hist_ready) {
    e = sort_clear(s, n, passes, stream);
    if (e != cudaSuccess) return e;
    launch_digit_histogram(keys, n, passes, s.hist, stream);
  }
  // Pass p reads the previous output and writes buffer set (p & 1):
  // set 0 = scratch alternates, set 1 = the caller's arrays.
  uint32_t* const bk[2] = {s.keys_alt, keys};
  uint32_t* const bv[2] = {s.vals_alt, vals};
  const uint32_t* kin = keys;
  const uint32_t* vin = vals_iota ? nullptr : vals;
  const int items = sort_items(n);
  for (int p = 0; p < passes; ++p) {
    uint32_t* kout = bk[p & 1];
    uint32_t* vout = bv[p & 1];
    auto kernel = items == 4 ? k_onesweep<4> : items == 8 ? k_onesweep<8> : k_onesweep<16>;
    kernel<<<tiles, kSortThreads, 0, stream>>>(
        kin, vin, kout, vout, n, p * kRadixBits, s.hist + p * kRadix,
        s.lookback + (size_t)p * tiles * kRadix, s.counters + p, s.err, kSpinLimit);
    kin = kout;
    vin = vout;
  }
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  uint32_t* kres = const_cast<uint32_t*>(kin);
  uint32_t* vres = const_cast<uint32_t*>(vin);
  if (copy_back && kres != keys) {
    e = cudaMemcpyAsync(keys, kres, sizeof(uint32_t) * n, cudaMemcpyDeviceToDevice, stream);
    if (e != cudaSuccess) return e;
    e = cudaMemcpyAsync(vals, vres, sizeof(uint32_t) * n, cudaMemcpyDeviceToDevice, stream);
    if (e != cudaSuccess) return e;
    kres = keys;
    vres = vals;
  }
  if (keys_res) *keys_res = kres;
  if (vals_res) *vals_res = vres;
  return cudaSuccess;
}

cudaError_t lookback_wait_probe(int spin_limit, uint32_t* err_bits) {
  // Two tiles of keys; the tile counter starts at 1, so the one CTA
  // launched ranks tile 1 and looks back at tile 0, whose flag no CTA ever
  // writes.  Its wait gives up after spin_limit polls and sets kErrSortSpin;
  // the digit counts are those of both tiles, so every scatter the CTA
  // then makes stays below n.
  constexpr int kItems = 16, n = 2 * kSortThreads * kItems;
  std::vector<uint32_t> hk(n);
  uint32_t hist[kRadix] = {};
  for (int i = 0; i < n; ++i) {
    hk[i] = (uint32_t)i * 2654435761u;
    ++hist[hk[i] & (kRadix - 1)];
  }
  uint32_t* buf = nullptr;
  const size_t words = 4 * (size_t)n + kRadix + 2 * kRadix + 2;
  cudaError_t e = cudaMalloc(&buf, words * sizeof(uint32_t));
  if (e != cudaSuccess) return e;
  uint32_t* keys = buf;
  uint32_t* vals = buf + n;
  uint32_t* kout = buf + 2 * (size_t)n;
  uint32_t* vout = buf + 3 * (size_t)n;
  uint32_t* doff = buf + 4 * (size_t)n;
  uint32_t* lookback = doff + kRadix;
  uint32_t* counter = lookback + 2 * kRadix;
  uint32_t* err = counter + 1;
  const uint32_t one = 1u;
  e = cudaMemset(buf, 0, words * sizeof(uint32_t));
  if (e == cudaSuccess)
    e = cudaMemcpy(keys, hk.data(), sizeof(uint32_t) * n, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(doff, hist, sizeof(hist), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(counter, &one, sizeof(one), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    k_onesweep<kItems><<<1, kSortThreads>>>(keys, vals, kout, vout, n, 0, doff, lookback, counter, err,
                                    spin_limit);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaDeviceSynchronize();
  if (e == cudaSuccess) e = cudaMemcpy(err_bits, err, sizeof(uint32_t), cudaMemcpyDeviceToHost);
  cudaFree(buf);
  return e;
}

cudaError_t launch_bounds(const uint32_t* keys, int n, int count, uint32_t* out, bool upper,
                          cudaStream_t stream, uint32_t* err) {
  if (count <= 0) return cudaSuccess;
  // the upper bound of c is the lower bound of c + 1
  const int blocks = (int)(((int64_t)count + kBoundCells - 1) / kBoundCells);
  k_bounds<<<blocks, 256, 0, stream>>>(keys, n, count, upper ? 1 : 0, out, err);
  return cudaGetLastError();
}

}  // namespace sphpc
