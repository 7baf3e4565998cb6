// grid.cu -- uniform-grid hashing, particle reorder, cell-start table and the
// neighbour build of the PBF pipeline.
#include "kernels.cuh"

namespace sphpc {

namespace {

// x* as absolute FP32 for the neighbour build's candidate test, in pair
// blocks: slots 2b and 2b+1 share the 32 bytes {x0, x1, y0, y1, z0, z1, 0,
// 0} at float4 index 2b, so that the coordinates of a slot pair load as the
// 64-bit operands of the packed FP32x2 arithmetic of sm_100.
__device__ __forceinline__ void xsa_store(float4* xsa, int j, float x, float y, float z) {
  float* f = reinterpret_cast<float*>(xsa + (j & ~1)) + (j & 1);
  f[0] = x;
  f[2] = y;
  f[4] = z;
  f[6] = 0.0f;
}

__device__ __forceinline__ float4 xsa_load(const float4* __restrict__ xsa, int j) {
  const float* f = reinterpret_cast<const float*>(xsa + (j & ~1)) + (j & 1);
  return make_float4(__ldg(f), __ldg(f + 2), __ldg(f + 4), 0.0f);
}

// The pair block of even slot j as three 64-bit pairs {x_j, x_j+1}, {y..},
// {z..}: one 256-bit read-only load (sm_100).
__device__ __forceinline__ void ld_pair(const float4* __restrict__ xsa, int j, uint64_t& xx,
                                        uint64_t& yy, uint64_t& zz) {
  asm("{\n\t.reg .b64 pad;\n\t"
      "ld.global.nc.v4.u64 {%0,%1,%2,pad}, [%3];\n\t}"
      : "=l"(xx), "=l"(yy), "=l"(zz)
      : "l"(xsa + j));
}

// Canonical predicted position of one particle.  predict: ApplyGravity then
// PredictPositions (particles.c:516-527, 766-782) evaluated in FP64 exactly
// as the reference does, then the box clamp (particles.c:842-867); the
// displacement d = x* - x is rounded to FP32 and x* := fl64(x + d).
__device__ __forceinline__ void canonical_xstar(const DevParams& P, const float4 x,
                                                const float4 v, const float4 dgiven,
                                                bool predict, float4& d, double& xs,
                                                double& ys, double& zs) {
  if (predict) {
    double vx = (double)v.x, vy = (double)v.y, vz = (double)v.z;
    if (P.gaxis == 0) vx = __dadd_rn(vx, P.gdt_d);
    else if (P.gaxis == 1) vy = __dadd_rn(vy, P.gdt_d);
    else vz = __dadd_rn(vz, P.gdt_d);
    xs = __dadd_rn((double)x.x, __dmul_rn(vx, P.dt_d));
    ys = __dadd_rn((double)x.y, __dmul_rn(vy, P.dt_d));
    zs = __dadd_rn((double)x.z, __dmul_rn(vz, P.dt_d));
    xs = clamp_axis(xs, P.bmin[0], P.bmax[0], P.bmax_eps[0]);
    ys = clamp_axis(ys, P.bmin[1], P.bmax[1], P.bmax_eps[1]);
    zs = clamp_axis(zs, P.bmin[2], P.bmax[2], P.bmax_eps[2]);
    d = make_float4(__double2float_rn(__dsub_rn(xs, (double)x.x)),
                    __double2float_rn(__dsub_rn(ys, (double)x.y)),
                    __double2float_rn(__dsub_rn(zs, (double)x.z)), 0.0f);
  } else {
    d = dgiven;
  }
  xs = xstar_d(x.x, d.x);
  ys = xstar_d(x.y, d.y);
  zs = xstar_d(x.z, d.z);
}

__device__ __forceinline__ void grid_cell(const DevParams& P, double xs, double ys, double zs,
                                          int& cx, int& cy, int& cz) {
  cx = grid_coord(xs, P.hd);
  cy = grid_coord(ys, P.hd);
  cz = grid_coord(zs, P.hd);
}

// HashVal, neighbors.c:94-95 (unsigned arithmetic)
__device__ __forceinline__ uint32_t cell_key(const DevParams& P, int cx, int cy, int cz) {
  return (uint32_t)P.nx * (uint32_t)P.ny * (uint32_t)cz +
         ((uint32_t)cy * (uint32_t)P.nx + (uint32_t)cx);
}

__device__ __forceinline__ uint32_t pack_cell(const DevParams& P, int cx, int cy, int cz) {
  return (uint32_t)cx | ((uint32_t)cy << P.bx) | ((uint32_t)cz << (P.bx + P.by));
}

// Cell key of the particle in slot i (launch_hash).
__device__ __forceinline__ uint32_t key_of(const DevParams& P, const PD* __restrict__ pd,
                                           const float4* __restrict__ vel, int i, bool predict,
                                           uint32_t* __restrict__ err) {
  float4 x, dg;
  ld_pd(pd, i, x, dg);
  const float4 v = predict ? __ldg(vel + i) : make_float4(0.f, 0.f, 0.f, 0.f);
  float4 d;
  double xs, ys, zs;
  canonical_xstar(P, x, v, dg, predict, d, xs, ys, zs);
  int cx, cy, cz;
  grid_cell(P, xs, ys, zs, cx, cy, cz);
  const uint32_t key = cell_key(P, cx, cy, cz);
  if (key >= P.ncells || cx >= P.nx || cy >= P.ny || cz >= P.nz) {
    atomicOr(err, kErrCellRange);
    return P.ncells - 1;
  }
  return key;
}

__global__ void __launch_bounds__(kBlock)
    k_hash(const DevParams P, const PD* __restrict__ pd, const float4* __restrict__ vel,
           const uint32_t* __restrict__ ids,
           uint32_t* __restrict__ keys_by_id, uint32_t* __restrict__ loc_by_id,
           uint32_t* __restrict__ hist, int passes, int predict, uint32_t* __restrict__ err) {
  __shared__ uint32_t s_hist[kMaxPasses * kRadix];
  for (int i = threadIdx.x; i < kMaxPasses * kRadix; i += blockDim.x) s_hist[i] = 0;
  __syncthreads();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < P.n) {
    const uint32_t key = key_of(P, pd, vel, i, predict != 0, err);
    const uint32_t id = __ldg(ids + i);
    keys_by_id[id] = key;
    loc_by_id[id] = (uint32_t)i;
    count_key_digits(s_hist, key, passes);
  }
  __syncthreads();
  for (int k = threadIdx.x; k < passes * kRadix; k += blockDim.x)
    if (s_hist[k]) atomicAdd(hist + k, s_hist[k]);
}

// ---------------------------------------------------------------------------
// Slots by counting: count the particles of every cell, scan the counts to the
// cell starts, put every particle's id somewhere in its cell's range, and take
// its slot from the ids of the range (a cell's particles stand in ascending id).
//
// The state lies in the slots of the step before, so everything here runs nearly
// in order; the digit passes start from the order of the ids, which takes a
// scattered write and a scattered read of every particle besides.
// One step of 1,048,576 particles: hash, three digit passes, bounds and reorder
// 143 us, these and the reorder 74 us; 4.2M: 353 and 221 us; 290k: 83 and 39;
// 4096: 42 and 27.  Empty cells cost 12 bytes each here and 4 there: at 27 cells a
// particle 182 us against 229 (1M particles), 64 against 98 (262k).
//
// The rank by comparing takes time with the square of a cell's particles, so a
// cell of more than kCrowded is put in order instead, by the block that places its
// last particle (order_cell), and sets *crowded, host memory: digit passes are faster for
// such a set, and it goes over to them when the host sees it; the slots are the
// same either way.  Where the line lies, us from hash to reorder with 256 / 512 / 1000
// particles a cell, ranked by comparing and by digit passes: 32,768 particles 31 / 32 /
// 41 and 74 / 69 / 69; 262,144 48 / 59 / 83 and 96 / 96 / 80; 1,048,576 111 / 153 / 222 and
// 161 / 141 / 141; 4.2M 348 / 507 by comparing, 359 by digits (their build takes 8 ms).
// ---------------------------------------------------------------------------
constexpr uint32_t kCrowded = 512;

// keys[i] of slot i, and its rank among its cell's particles in the order that
// the atomics happen to take.  The lanes of a cell share one atomic: eight
// particles a cell stand side by side.
__global__ void __launch_bounds__(kBlock)
    k_count(const DevParams P, const PD* __restrict__ pd, const float4* __restrict__ vel,
            uint32_t* __restrict__ keys, uint32_t* __restrict__ rank, uint32_t* __restrict__ count,
            int predict, uint32_t* __restrict__ err) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned on = __ballot_sync(0xffffffffu, i < P.n);
  if (i >= P.n) return;
  const uint32_t key = key_of(P, pd, vel, i, predict != 0, err);
  const unsigned same = __match_any_sync(on, key);
  const int lane = threadIdx.x & 31, first = __ffs((int)same) - 1;
  uint32_t base = 0;
  if (lane == first) base = atomicAdd(count + key, (uint32_t)__popc(same));
  base = __shfl_sync(same, base, first);
  keys[i] = key;
  rank[i] = base + (uint32_t)__popc(same & ((1u << lane) - 1u));
}

// Exclusive scan of cells[0..m) in place: blocks of kScanItems cells in the
// order of a ticket, each adding what the blocks before it hold (state: one word
// a block, its own sum or the sum up to it).  state[0] is the ticket.
constexpr int kScanThreads = 256;
constexpr int kScanPer = 16;
constexpr int kScanItems = kScanThreads * kScanPer;
constexpr unsigned long long kScanSum = 1ull << 62, kScanPrefix = 2ull << 62;

__device__ __forceinline__ unsigned long long ld_state(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_state(unsigned long long* p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

__global__ void __launch_bounds__(kScanThreads)
    k_scan_counts(uint32_t* __restrict__ cells, uint32_t m, unsigned long long* __restrict__ state,
                  volatile uint32_t* crowded, uint32_t* __restrict__ any_crowded,
                  uint32_t* __restrict__ err) {
  __shared__ uint32_t s_warp[kScanThreads / 32];
  __shared__ uint32_t s_block, s_before;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) s_block = (uint32_t)atomicAdd(state, 1ull);
  __syncthreads();
  const uint32_t block = s_block;
  unsigned long long* mine = state + 1 + block;
  const uint64_t c0 = (uint64_t)block * kScanItems + (uint64_t)threadIdx.x * kScanPer;
  uint32_t v[kScanPer];
  if (c0 + kScanPer <= m) {
#pragma unroll
    for (int u = 0; u < kScanPer; u += 4) {
      const uint4 q = *reinterpret_cast<const uint4*>(cells + c0 + u);
      v[u] = q.x;
      v[u + 1] = q.y;
      v[u + 2] = q.z;
      v[u + 3] = q.w;
    }
  } else {
#pragma unroll
    for (int u = 0; u < kScanPer; ++u) v[u] = c0 + u < m ? cells[c0 + u] : 0u;
  }
  uint32_t sum = 0, most = 0;
#pragma unroll
  for (int u = 0; u < kScanPer; ++u) {
    const uint32_t x = v[u];
    most = max(most, x);
    v[u] = sum;
    sum += x;
  }
  if (most > kCrowded) *any_crowded = *crowded = 1u;
  uint32_t upto = sum;
#pragma unroll
  for (int k = 1; k < 32; k <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, upto, k);
    if (lane >= k) upto += y;
  }
  if (lane == 31) s_warp[warp] = upto;
  __syncthreads();
  uint32_t before = upto - sum, total = 0;
#pragma unroll
  for (int w = 0; w < kScanThreads / 32; ++w) {
    if (w < warp) before += s_warp[w];
    total += s_warp[w];
  }
  if (warp == 0) {
    uint32_t ahead = 0;
    if (block > 0) {
      if (lane == 0) st_state(mine, kScanSum | total);
      // 32 blocks back at a time until one that knows its prefix
      for (int64_t b = (int64_t)block - 1 - lane, spins = 0;;) {
        const unsigned long long q = b >= 0 ? ld_state(state + 1 + b) : kScanPrefix;
        const unsigned unknown = __ballot_sync(0xffffffffu, q < kScanSum);
        const unsigned prefix = __ballot_sync(0xffffffffu, q >= kScanPrefix);
        // lanes up to the nearest prefix count; all of them must be known
        const int last = prefix ? __ffs((int)prefix) - 1 : 31;
        if (unknown & (0xffffffffu >> (31 - last))) {
          if (++spins > (1 << 22)) {
            if (lane == 0) atomicOr(err, kErrScanSpin);
            break;
          }
          continue;
        }
        uint32_t x = lane <= last ? (uint32_t)q : 0u;
#pragma unroll
        for (int k = 16; k; k >>= 1) x += __shfl_xor_sync(0xffffffffu, x, k);
        ahead += x;
        if (prefix) break;
        b -= 32;
      }
    }
    if (lane == 0) {
      st_state(mine, kScanPrefix | (uint32_t)(ahead + total));
      s_before = ahead;
    }
  }
  __syncthreads();
  before += s_before;
  if (c0 + kScanPer <= m) {
#pragma unroll
    for (int u = 0; u < kScanPer; u += 4)
      *reinterpret_cast<uint4*>(cells + c0 + u) =
          make_uint4(before + v[u], before + v[u + 1], before + v[u + 2], before + v[u + 3]);
  } else {
#pragma unroll
    for (int u = 0; u < kScanPer; ++u)
      if (c0 + u < m) cells[c0 + u] = before + v[u];
  }
}

// The m ids of one cell into ascending order, their old slots with them, by one
// block: digit passes from the lowest digit on, between the cell's range of ids and
// src and that of ids2 and src2 (an even number, so that they end in the first).
// One block takes about 3 ns a pair and pass: 3.1 ms for 262,144 particles in one
// cell, 55 ms for 4.2M (by comparing 12.7 ms, and 256 times that).  Steps that were
// launched before the host saw the cell pay it, those after it go by digit passes.
constexpr int kOrderItems = 8;
__device__ __noinline__ void order_cell(uint32_t* ids, uint32_t* src, uint32_t* ids2,
                                        uint32_t* src2, uint32_t m, int passes) {
  __shared__ uint32_t s_base[kRadix], s_sum[kBlock / 32];
  __shared__ uint32_t s_warp[kBlock / 32][kRadix + 1];
  static_assert(kBlock == kRadix, "a thread a digit");
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  for (int pass = 0; pass < passes; ++pass) {
    const int shift = pass * kRadixBits;
    s_base[t] = 0;
    __syncthreads();
    for (uint32_t i = t; i < m; i += kBlock)
      atomicAdd(&s_base[(__ldcg(ids + i) >> shift) & (kRadix - 1)], 1u);
    __syncthreads();
    const uint32_t all = s_base[t];
    uint32_t upto = all;
#pragma unroll
    for (int k = 1; k < 32; k <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, upto, k);
      if (lane >= k) upto += y;
    }
    if (lane == 31) s_sum[warp] = upto;
    __syncthreads();
    uint32_t first = upto - all;
    for (int w = 0; w < warp; ++w) first += s_sum[w];
    s_base[t] = first;
    for (uint32_t t0 = 0; t0 < m; t0 += kBlock * kOrderItems) {
      for (int k = t; k < kBlock / 32 * (kRadix + 1); k += kBlock) (&s_warp[0][0])[k] = 0;
      __syncthreads();
      uint32_t id[kOrderItems], rank[kOrderItems];
#pragma unroll
      for (int u = 0; u < kOrderItems; ++u) {
        const uint32_t i = t0 + (warp * kOrderItems + u) * 32 + lane;
        id[u] = i < m ? __ldcg(ids + i) : 0u;
        const uint32_t d = i < m ? (id[u] >> shift) & (kRadix - 1) : (uint32_t)kRadix;
        const unsigned same = __match_any_sync(0xffffffffu, d);
        const uint32_t before = s_warp[warp][d];
        __syncwarp();
        rank[u] = before + __popc(same & ((1u << lane) - 1u));
        if (lane == __ffs((int)same) - 1) s_warp[warp][d] = before + __popc(same);
        __syncwarp();
      }
      __syncthreads();
      uint32_t at = s_base[t];
      for (int w = 0; w < kBlock / 32; ++w) {
        const uint32_t c = s_warp[w][t];
        s_warp[w][t] = at;
        at += c;
      }
      s_base[t] = at;
      __syncthreads();
#pragma unroll
      for (int u = 0; u < kOrderItems; ++u) {
        const uint32_t i = t0 + (warp * kOrderItems + u) * 32 + lane;
        if (i >= m) continue;
        const uint32_t to = s_warp[warp][(id[u] >> shift) & (kRadix - 1)] + rank[u];
        ids2[to] = id[u];
        src2[to] = __ldcg(src + i);
      }
      __syncthreads();
    }
    uint32_t* x = ids;
    ids = ids2;
    ids2 = x;
    x = src;
    src = src2;
    src2 = x;
  }
}

// Id and old slot of every particle into its cell's range.  With a crowded cell
// about (`any`), the threads count what they have placed of it in `placed`, a word for
// every kCrowded + 1 slots: no two crowded cells start in the same ones.  The block
// with the last particle of a cell puts it in order.
struct PlaceArgs {
  const uint32_t *keys, *rank, *ids, *any;
  uint32_t *placed;
  uint32_t *cell_ids, *cell_src;  // written by all blocks and read by one
  uint32_t *ids2, *src2;          // scratch
  int passes;                     // digit passes that order ids
};
__global__ void __launch_bounds__(kBlock, 8)
    k_place(int n, const uint32_t* __restrict__ cstart, const PlaceArgs a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool any = __ldg(a.any) != 0;
  uint32_t key = 0, b = 0;
  if (i < n) {
    key = __ldg(a.keys + i);
    b = __ldg(cstart + key);
    const uint32_t j = min(b + __ldg(a.rank + i), (uint32_t)n - 1u);
    a.cell_ids[j] = __ldg(a.ids + i);
    a.cell_src[j] = (uint32_t)i;
  }
  if (!any) return;
  __shared__ uint32_t s_first[kBlock], s_count[kBlock];
  __shared__ int s_cells;
  if (threadIdx.x == 0) s_cells = 0;
  __syncthreads();
  const uint32_t m = i < n ? min(__ldg(cstart + key + 1), (uint32_t)n) - b : 0u;
  const unsigned on = __ballot_sync(0xffffffffu, i < n && m > kCrowded && m <= (uint32_t)n);
  if (on >> (threadIdx.x & 31) & 1u) {
    const unsigned same = __match_any_sync(on, key);
    __threadfence();
    __syncwarp(same);
    if ((int)(threadIdx.x & 31) == __ffs((int)same) - 1) {
      const uint32_t here = (uint32_t)__popc(same);
      if (atomicAdd(a.placed + b / (kCrowded + 1), here) + here == m) {
        const int c = atomicAdd(&s_cells, 1);
        s_first[c] = b;
        s_count[c] = m;
      }
    }
  }
  __syncthreads();
  __threadfence();
  for (int c = 0; c < s_cells; ++c) {
    const uint32_t f = s_first[c];
    order_cell(a.cell_ids + f, a.cell_src + f, a.ids2 + f, a.src2 + f, s_count[c], a.passes);
  }
}

// Keys of the slots from the cell starts.
__global__ void __launch_bounds__(kBlock)
    k_slot_keys(const uint32_t* __restrict__ cstart, uint32_t ncells, uint32_t* __restrict__ keys) {
  const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncells) return;
  for (uint32_t j = cstart[c]; j < cstart[c + 1]; ++j) keys[j] = c;
}

template <bool COUNTED>
__global__ void __launch_bounds__(kBlock)
    k_reorder(const DevParams P, const SlotOrder o, const PD* __restrict__ pd_in,
              const float4* __restrict__ vel_in, PD* __restrict__ pd_out,
              float4* __restrict__ vel_out, float4* __restrict__ xsa, uint4* __restrict__ nr_out,
              uint32_t* __restrict__ cellp, int predict, int move_vel, ReorderExtra ex) {
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= P.n) return;
  const uint32_t id = __ldg(o.ids + j);
  uint32_t src;
  if (COUNTED) {
    src = __ldg(o.src + j);
    const uint32_t key = __ldg(o.keys + src);
    const uint32_t b = __ldg(o.cstart + key), e = __ldg(o.cstart + key + 1);
    if (e - b <= kCrowded) {  // (a crowded cell's are in order)
      uint32_t at = b;
      for (uint32_t k = b; k < e; ++k) at += __ldg(o.ids + k) < id ? 1u : 0u;
      j = (int)min(at, (uint32_t)P.n - 1u);
    }
    o.ids_out[j] = id;
  } else {
    src = __ldg(o.src + id);
  }
  float4 x, dg;
  ld_pd(pd_in, (int)src, x, dg);
  float4 v = (predict || move_vel) ? __ldg(vel_in + src) : make_float4(0.f, 0.f, 0.f, 0.f);
  float4 d;
  double xs, ys, zs;
  canonical_xstar(P, x, v, dg, predict != 0, d, xs, ys, zs);
  int cx, cy, cz;
  grid_cell(P, xs, ys, zs, cx, cy, cz);
  cx = min(cx, P.nx - 1);
  cy = min(cy, P.ny - 1);
  cz = min(cz, P.nz - 1);
  d.w = predict ? 0.0f : dg.w;
  st_pd(pd_out, j, x, d);
  xsa_store(xsa, j, (float)xs, (float)ys, (float)zs);
  nr_out[j] = make_nr(P, xs, ys, zs, d.w);
  cellp[j] = pack_cell(P, cx, cy, cz);
  if (move_vel) {
    if (predict) {
      // the velocity after ApplyGravity, as the reference holds it
      if (P.gaxis == 0) v.x = __fadd_rn(v.x, P.gdt_f);
      else if (P.gaxis == 1) v.y = __fadd_rn(v.y, P.gdt_f);
      else v.z = __fadd_rn(v.z, P.gdt_f);
    }
    vel_out[j] = v;
  }
#pragma unroll
  for (int k = 0; k < 6; ++k)
    if (ex.in4[k]) ex.out4[k][j] = __ldg(ex.in4[k] + src);
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if (ex.in1[k]) ex.out1[k][j] = __ldg(ex.in1[k] + src);
  if (ex.nr_carry) ex.nr_carry[j] = make_nr(P, xs, ys, zs, __ldg(ex.carry_src + src));
}

constexpr int kSmallGap = 32;
constexpr int64_t kGapChunk = 4096;  // worklist entries cover at most this many cells

__device__ __forceinline__ void push_gap(int64_t lo, int64_t hi, uint32_t val, uint4* gaps,
                                         uint32_t* gap_count) {
  const int64_t pieces = (hi - lo + kGapChunk) / kGapChunk;
  const uint32_t g = atomicAdd(gap_count, (uint32_t)pieces);
  for (int64_t k = 0; k < pieces; ++k) {
    const int64_t a = lo + k * kGapChunk;
    const int64_t b = min(hi, a + kGapChunk - 1);
    gaps[g + k] = make_uint4((uint32_t)a, (uint32_t)b, val, 0u);
  }
}

// cstart[lo..hi] = v, inline for a short run of cells, else as worklist
// pieces for k_fill_gaps.
__device__ __forceinline__ void set_cells(int64_t lo, int64_t hi, uint32_t v,
                                          uint32_t* __restrict__ cstart, uint4* gaps,
                                          uint32_t* gap_count) {
  if (hi - lo + 1 <= kSmallGap) {
    for (int64_t c = lo; c <= hi; ++c) cstart[c] = v;
  } else {
    push_gap(lo, hi, v, gaps, gap_count);
  }
}

// start[c] = lower_bound(keys, c): the first slot j of every non-empty key
// writes j into the cells (key[j-1], key[j]]; long runs of empty cells go to
// a worklist filled by k_fill_gaps.  A thread takes four consecutive slots
// (one 128-bit load of keys and the key before them).
constexpr int kStartsPerThread = 4;
__global__ void __launch_bounds__(kBlock)
    k_cell_starts(const uint32_t* __restrict__ keys, int n, uint32_t ncells,
                  uint32_t* __restrict__ cstart, uint4* __restrict__ gaps,
                  uint32_t* __restrict__ gap_count, uint32_t* __restrict__ err) {
  const int j0 = (blockIdx.x * blockDim.x + threadIdx.x) * kStartsPerThread;
  if (j0 >= n) return;
  uint32_t k[kStartsPerThread];
  if (j0 + kStartsPerThread <= n) {
    const uint4 v = __ldg(reinterpret_cast<const uint4*>(keys + j0));
    k[0] = v.x;
    k[1] = v.y;
    k[2] = v.z;
    k[3] = v.w;
  } else {
#pragma unroll
    for (int u = 0; u < kStartsPerThread; ++u) k[u] = j0 + u < n ? __ldg(keys + j0 + u) : 0u;
  }
  int64_t kp = j0 > 0 ? (int64_t)__ldg(keys + j0 - 1) : -1;
#pragma unroll
  for (int u = 0; u < kStartsPerThread; ++u) {
    const int j = j0 + u;
    if (j >= n) break;
    const int64_t kk = (int64_t)k[u];
    if (kk >= (int64_t)ncells) {
      atomicOr(err, kErrCellRange);
      return;
    }
    if (kk != kp) set_cells(kp + 1, kk, (uint32_t)j, cstart, gaps, gap_count);
    kp = kk;
    // after the last key: every cell up to the sentinel cstart[C] starts at n
    if (j == n - 1) set_cells(kk + 1, (int64_t)ncells, (uint32_t)n, cstart, gaps, gap_count);
  }
}

__global__ void __launch_bounds__(kBlock)
    k_fill_gaps(const uint4* __restrict__ gaps, const uint32_t* __restrict__ gap_count,
                uint32_t* __restrict__ cstart) {
  const uint32_t ng = *gap_count;
  for (uint32_t g = blockIdx.x; g < ng; g += gridDim.x) {
    const uint4 e = gaps[g];
    for (uint64_t c = (uint64_t)e.x + threadIdx.x; c <= (uint64_t)e.y; c += blockDim.x)
      cstart[c] = e.z;
  }
}

// FillNeighbors' validity test and HashVal coordinate of one shifted axis
// value (neighbors.c:252-263).
__device__ __forceinline__ bool shifted_coord(double x, double h, int nmax, int& g) {
  const double f = floor(__ddiv_rn(x, h));
  if (f > (double)(nmax - 1) || x < 0.0) return false;
  g = (int)(unsigned)f;
  return true;
}

// Whether the walk visits the cells c-1, c, c+1 of an axis that the grid has, for a
// particle in cell c.  A particle beyond the grid is not regular: its cell is the
// last one, its key another's (key_of), and the rows of a block's tile are found
// from both.
__device__ __forceinline__ bool axis_regular(double x, double h, int c, int nmax) {
  int g;
  if (c == nmax - 1 && !shifted_coord(x, h, nmax, g)) return false;
  const bool vm = shifted_coord(__dadd_rn(x, -h), h, nmax, g);
  const bool okm = vm ? (g == c - 1) : (c == 0);
  const bool vp = shifted_coord(__dadd_rn(x, h), h, nmax, g);
  const bool okp = vp ? (g == c + 1) : (c == nmax - 1);
  return okm && okp;
}

// r^2 < h^2 exactly as neighbors.c:278-285 evaluates it on the canonical
// double positions of slots p and j.  The FP32 absolute positions decide every
// pair whose r^2 lies outside the band [P.bld_h2lo, P.bld_h2hi] about h^2; this
// test decides the rest.  The band is as wide as FP32 rounding of the grid's
// largest coordinate can move r^2 (sphpc_neighbor_pretest_band: 2^-14 h^2 for 128
// cells an axis), and open to every pair beyond about 2^12 h.
__device__ __forceinline__ bool exact_neighbor(const DevParams& P, const PD* __restrict__ pd,
                                               int p, int j) {
  float4 xp, dp, xq, dq;
  ld_pd(pd, p, xp, dp);
  ld_pd(pd, j, xq, dq);
  const double ddx = __dsub_rn(xstar_d(xp.x, dp.x), xstar_d(xq.x, dq.x));
  const double ddy = __dsub_rn(xstar_d(xp.y, dp.y), xstar_d(xq.y, dq.y));
  const double ddz = __dsub_rn(xstar_d(xp.z, dp.z), xstar_d(xq.z, dq.z));
  const double r2 = __dadd_rn(__dadd_rn(__dmul_rn(ddx, ddx), __dmul_rn(ddy, ddy)),
                              __dmul_rn(ddz, ddz));
  return r2 < P.h2d;
}

// FillNeighbors' 27-cell walk (neighbors.c:247-295) verbatim, for a
// particle whose neighbour cells are not cx-1..cx+1 (FP64 rounding at a cell
// face): its bucket goes to list entries 0..count-1 of p in nbr, the last
// block's entries past the count are set to p; returns the count.
__device__ __forceinline__ int walk_27_cells(const DevParams& P, const NbrView& V,
                                             const PD* __restrict__ pd,
                                             const float4* __restrict__ xsa, int p,
                                             uint32_t* __restrict__ nbr) {
  const float4 xf = xsa_load(xsa, p);
  float4 xp, dp;
  ld_pd(pd, p, xp, dp);
  const double xs = xstar_d(xp.x, dp.x), ys = xstar_d(xp.y, dp.y), zs = xstar_d(xp.z, dp.z);
  auto entry = [&](int t) -> uint32_t& { return nbr[(((size_t)(t >> 2) * V.n + p) << 2) + (t & 3)]; };
  int count = 0;
  for (int dz = -1; dz <= 1; ++dz)
    for (int dy = -1; dy <= 1; ++dy)
      for (int dx = -1; dx <= 1; ++dx) {
        int gx, gy, gz;
        if (!shifted_coord(__dadd_rn(xs, (double)dx * P.hd), P.hd, P.nx, gx)) continue;
        if (!shifted_coord(__dadd_rn(ys, (double)dy * P.hd), P.hd, P.ny, gy)) continue;
        if (!shifted_coord(__dadd_rn(zs, (double)dz * P.hd), P.hd, P.nz, gz)) continue;
        const uint32_t key = (uint32_t)P.nx * (uint32_t)P.ny * (uint32_t)gz +
                             ((uint32_t)gy * (uint32_t)P.nx + (uint32_t)gx);
        if (key >= P.ncells) continue;
        const int b = (int)__ldg(V.cstart + key);
        const int e = (int)__ldg(V.cstart + key + 1);
        for (int j = b; j < e && count < kMaxNeighbors; ++j) {
          if (j == p) continue;
          const float4 q = xsa_load(xsa, j);
          const float r2 = norm2(xf.x - q.x, xf.y - q.y, xf.z - q.z);
          if (r2 < P.bld_h2lo || (r2 <= P.bld_h2hi && exact_neighbor(P, pd, p, j)))
            entry(count++) = (uint32_t)j;
        }
      }
  for (int t = count; t & 3; ++t) entry(t) = (uint32_t)p;
  return count;
}

// ---------------------------------------------------------------------------
// Neighbour build (FillNeighbors, neighbors.c:217-298): one thread per
// particle tests its 9 (dz, dy) slot rows in the reference's order (rows of
// cells cx-1..cx+1 are contiguous slot ranges, cells in dx order, particles
// in ascending original index), four candidates at a time without branches,
// each hit one bit shifted into a word of 32 candidates.  The words that hold a
// hit go to the thread's column in shared memory, and the list is written from
// them at the end as 16-byte blocks (for each block index, a warp's 32
// consecutive slots are four whole 128-byte lines), the last block's entries
// past the count set to the particle itself.
//
// The candidates of a block of kTileSlots slots come from its tile of FP32
// positions in shared memory (TileInfo; nine bulk copies), pairs of slots as
// the 64-bit operands of the packed FP32x2 arithmetic of sm_100, and the list's
// entries are byte offsets in the record tile.  A block whose tile does not fit
// loads the pairs from global memory and its list holds slots.
//
// Bound: instruction issue (79% at 41% of the warps), 118 warp instructions a
// particle.  4.2M particles: 1005 us with candidate pairs loaded per lane from
// global memory and every candidate stored and counted on a hit; 854 us so from
// tiles, the shared-memory pipe then as busy as the issue (74%, half of it bank
// conflicts: the lanes of a warp are in four cells whose rows start a cell's
// eight records, one turn of the banks, apart); 739 us with hit words; 663 us
// with the lanes of odd cells half a turn of the banks ahead (conflicts 17M ->
// 4M a launch of 1M particles) and the band as narrow as the grid allows; 618 us
// with the words read back without a test a hit.  Tried for the same work and
// slower: the candidates of a cell held by a warp's lanes, its particles
// broadcast to them and the hits taken from ballots (1462 us).
//
// kWords: rows at rest density take one word; with ten a column seven blocks
// fit an SM.  A particle with more writes whole blocks of its list ahead.
// ---------------------------------------------------------------------------
constexpr int kWords = 10;

// Whether the neighbour cells of a particle with FP32 position x in cell c of
// an axis are c-1, c, c+1 (axis_regular) for certain: x / h lies at least
// (c + 2) 2^-21 inside the cell, more than the FP32 rounding of x and of the
// quotient, (c + 2) 2^-22, plus any FP64 rounding of (x +- h) / h.
__device__ __forceinline__ bool axis_inside(float x, float inv_h, int c) {
  const float f = fmaf(x, inv_h, -(float)c), m = (float)(c + 2) * 0x1p-21f;
  return f > m && f < 1.0f - m;
}

__device__ __forceinline__ float min3_abs(float a, float b, float c) {
  float m;
  asm("min.abs.f32 %0, %1, %2, %3;" : "=f"(m) : "f"(a), "f"(b), "f"(c));
  return m;
}

struct BuildRow {
  const DevParams& P;
  const PD* __restrict__ pd;
  uint64_t pxx, pyy, pzz, mh2;
  int p;
};

// Tests the candidates of `group` = src + j, j even, and the three after it and shifts their hits into `word`, the
// first one highest.  Candidate j is slot j + dslot.
// s = r^2 - h^2 by fused multiply-adds from -h^2: its sign decides, and the
// exact FP64 test where |s| lies in the band (the three roundings of s stay
// within the bound that the band was sized for: near the band every partial
// sum is at most h^2).  Candidates outside [lo, hi) may be any bits: they are
// tested by sign alone, and the caller drops their hits.
template <bool TILE>
__device__ __forceinline__ uint32_t build_four(const BuildRow& c, const float4* __restrict__ src,
                                               const float4* __restrict__ group, int lo, int hi,
                                               int dslot, uint32_t word) {
  uint64_t x0, y0, z0, x1, y1, z1;
  if (TILE) {
    const ulonglong2* t = reinterpret_cast<const ulonglong2*>(group);
    const ulonglong2 a = t[0], b = t[2];
    x0 = a.x;
    y0 = a.y;
    x1 = b.x;
    y1 = b.y;
    z0 = *reinterpret_cast<const uint64_t*>(t + 1);
    z1 = *reinterpret_cast<const uint64_t*>(t + 3);
  } else {
    ld_pair(group, 0, x0, y0, z0);
    ld_pair(group, 2, x1, y1, z1);
  }
  uint64_t d = f2_sub(c.pxx, x0);
  uint64_t s0 = f2_fma(d, d, c.mh2);
  d = f2_sub(c.pyy, y0);
  s0 = f2_fma(d, d, s0);
  d = f2_sub(c.pzz, z0);
  s0 = f2_fma(d, d, s0);
  d = f2_sub(c.pxx, x1);
  uint64_t s1 = f2_fma(d, d, c.mh2);
  d = f2_sub(c.pyy, y1);
  s1 = f2_fma(d, d, s1);
  d = f2_sub(c.pzz, z1);
  s1 = f2_fma(d, d, s1);
  float s[4] = {f2_lo(s0), f2_hi(s0), f2_lo(s1), f2_hi(s1)};
  const float band = c.P.bld_band;
  if (fminf(min3_abs(s[0], s[1], s[2]), fabsf(s[3])) <= band) {
    const int j = (int)(group - src);
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (fabsf(s[u]) <= band && j + u >= lo && j + u < hi)
        s[u] = exact_neighbor(c.P, c.pd, c.p, j + u + dslot) ? -1.0f : 1.0f;
  }
#pragma unroll
  for (int u = 0; u < 4; ++u) word = __funnelshift_l(__float_as_uint(s[u]), word, 1);
  return word;
}

// The hits of one particle between the tests and its list: words of 32
// consecutive candidates that hold a hit, in list order, in the thread's columns
// (stride kTileSlots) of `mask` and `base`; base is the list entry of the word's
// lowest bit, and entries fall by 1 << SHIFT a bit upwards.
template <class B, int SHIFT>
struct Hits {
  uint32_t* mask;
  B* base;
  int words = 0;      // stored
  int found = 0;      // hits so far, at most kMaxNeighbors
  int written = 0;    // entries in the list

  // Writes the list's blocks while more than `keep` hits are not written.
  __device__ __forceinline__ void write(uint4*& out, int n, int keep) {
    constexpr int kPer = sizeof(B) == 2 ? 8 : 4;
    int next = 0;
    uint32_t m = 0, e0 = 0;
    auto take = [&]() -> uint32_t {
      if (m == 0) {
        m = mask[next * kTileSlots];
        e0 = (uint32_t)base[next * kTileSlots];
        next = min(next + 1, words);
      }
      const int f = 31 - __clz((int)m);
      m &= ~(1u << f);
      return e0 - ((uint32_t)f << SHIFT);
    };
#pragma unroll 1
    for (; found - written > keep; out += n, written += kPer) {
      uint32_t w[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        w[u] = take();
        if (kPer == 8) w[u] |= take() << 16;
      }
      *out = make_uint4(w[0], w[1], w[2], w[3]);
    }
    if (keep == 0) return;
    // what is left moves to the front
    int k = 0;
    if (m != 0) {
      mask[0] = m;
      base[0] = (B)e0;
      k = 1;
    }
    for (; next < words; ++next, ++k) {
      mask[k * kTileSlots] = mask[next * kTileSlots];
      base[k * kTileSlots] = base[next * kTileSlots];
    }
    words = k;
  }

  __device__ __forceinline__ void add(uint32_t word, uint32_t entry, uint4*& out, int n) {
    if (word == 0) return;
    // (at most seven hits, in as many words, stay)
    if (words == kWords) write(out, n, 7);
    found += __popc(word);
    for (; found > kMaxNeighbors; --found) word &= word - 1;
    mask[words * kTileSlots] = word;
    base[words * kTileSlots] = (B)entry;
    ++words;
  }

  // The rest of the list, the last block filled up with entry `self`: a word of
  // one hit that is read over and over.
  __device__ __forceinline__ void finish(uint32_t self, uint4*& out, int n) {
    mask[words * kTileSlots] = 1u;
    base[words * kTileSlots] = (B)self;
    write(out, n, 0);
  }
};

// The hits among candidates [lo, hi) of one row except `skip` (< 0: none).
template <bool TILE, class H>
__device__ __forceinline__ void build_range(const BuildRow& c, const float4* __restrict__ src,
                                            int lo, int hi, int skip, int dslot, int odd,
                                            H& hits, uint4*& out, int n) {
  for (int w = lo & ~1; w < hi && hits.found < kMaxNeighbors; w += 32) {
    const int end = min(w + 32, hi), bits = (end - w + 3) & ~3;
    // Lanes of adjacent cells read different halves of the 128 bytes that the
    // banks hold of a tile's pairs: those of the wrong parity start with the
    // second group of four and take the first one last.
    const bool turn = TILE && (((w >> 2) ^ odd) & 1) != 0;
    uint32_t word = 0;
    const float4* g = src + w + (turn ? 4 : 0);
    const float4* const g1 = g + bits - 4;
#pragma unroll 1
    for (; g != g1; g += 4) word = build_four<TILE>(c, src, g, lo, hi, dslot, word);
    word = build_four<TILE>(c, src, turn ? src + w : g, lo, hi, dslot, word);
    word <<= 32 - bits;
    if (turn) {
      const uint32_t first = word & (15u << (32 - bits));
      word = ((word ^ first) >> 4) | (first << (bits - 4));
    }
    if (w < lo) word &= 0x7fffffffu;
    word &= 0xffffffffu << (32 - (end - w));
    if ((unsigned)(skip - w) < 32u) word &= ~(0x80000000u >> (skip - w));
    hits.add(word, (uint32_t)(w + 31) << (TILE ? 4 : 0), out, n);
  }
}

// The nine rows of particle p, tile: src is the tile and off[r] = o[r] - s[r]
// takes slots to tile records; else src is xsa.
template <bool TILE, class H>
__device__ __forceinline__ void build_rows(const BuildRow& c, const NbrView& V, uint32_t cell,
                                           const float4* __restrict__ src, const int* off, H& hits,
                                           uint4*& out) {
  const DevParams& P = c.P;
  int cx, cy, cz;
  unpack_cell(V, cell, cx, cy, cz);
  // rows of the grid among the nine
  const uint32_t ys = (cy > 0 ? 1u : 0u) | 2u | (cy < P.ny - 1 ? 4u : 0u);
  const uint32_t rows = (cz > 0 ? ys : 0u) | ys << 3 | (cz < P.nz - 1 ? ys << 6 : 0u);
  const uint32_t* first = V.cstart + (cx - (cx > 0));
  const int width = (cx > 0) + 1 + (cx < P.nx - 1);
  uint32_t key = (uint32_t)cz * P.nxny + (uint32_t)cy * (uint32_t)P.nx - P.nxny - (uint32_t)P.nx;
  auto bounds = [&](int r, int& b, int& e) {
    b = e = 0;
    if (rows >> r & 1u) {
      b = (int)__ldg(first + key);
      e = (int)__ldg(first + key + width);
    }
    key += (uint32_t)P.nx;
    if (r % 3 == 2) key += P.nxny - 3u * (uint32_t)P.nx;
  };
  int b, e;
  bounds(0, b, e);
#pragma unroll 1
  for (int r = 0; r < 9; ++r) {
    int bn, en;
    bounds(r + 1, bn, en);  // the next row's, ahead of this row's tests
    const int o = TILE ? off[r] : 0;
    build_range<TILE>(c, src, b + o, e + o, r == 4 ? c.p + o : -1, -o, cx, hits, out, V.n);
    b = bn;
    e = en;
  }
}

// The nine ranges of the block's tile (TileInfo): computed by lanes 0..8 of
// warp 0 into t.
__device__ __forceinline__ void tile_ranges(const DevParams& P, const NbrView& V,
                                            const uint32_t* __restrict__ cellp, int first,
                                            int last, TileInfo& t) {
  const int r = threadIdx.x;
  int s = 0, len = 0;
  if (r < 9) {
    int cx, cy, cz;
    unpack_cell(V, __ldg(cellp + first), cx, cy, cz);
    const int64_t k0 = (int64_t)cell_key(P, cx, cy, cz);
    unpack_cell(V, __ldg(cellp + last), cx, cy, cz);
    const int64_t k1 = (int64_t)cell_key(P, cx, cy, cz);
    const int64_t d = (int64_t)(r / 3 - 1) * P.nxny + (int64_t)(r % 3 - 1) * P.nx;
    const int64_t lo = min(max(k0 + d - 1, (int64_t)0), (int64_t)P.ncells);
    const int64_t hi = min(max(k1 + d + 2, (int64_t)0), (int64_t)P.ncells);
    s = (int)__ldg(V.cstart + lo) & ~1;
    len = (((int)__ldg(V.cstart + hi) + 1) & ~1) - s;
    len = max(len, 0);
  }
  int o = len;
#pragma unroll
  for (int k = 1; k < 16; k <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, o, k);
    if (r >= k) o += y;
  }
  if (r < 9) {
    t.s[r] = s;
    t.o[r] = o - len;
  }
  if (r == 8) t.total = o;
}

// Seven blocks of 128 threads per SM with their tiles (32 KB).
__global__ void __launch_bounds__(kTileSlots, 7)
    k_build(const DevParams P, const NbrView V, const PD* __restrict__ pd,
            const float4* __restrict__ xsa, const uint32_t* __restrict__ cellp,
            uint32_t* __restrict__ nbr, uint8_t* __restrict__ ncount, TileInfo* __restrict__ tiles) {
  // the tile (its last group of four may read three records past it), or the
  // bases of the hit words of a block without one
  extern __shared__ __align__(128) float4 s_tile[];
  uint32_t* const s_mask = reinterpret_cast<uint32_t*>(s_tile + V.cap + 4);
  uint16_t* const s_base = reinterpret_cast<uint16_t*>(s_mask + (kWords + 1) * kTileSlots);
  static_assert(sizeof(int) * (kWords + 1) * kTileSlots <= sizeof(float4) * kTileCap,
                "bases fit in the tile");
  __shared__ TileInfo s_info;
  __shared__ int s_off[9];
  __shared__ __align__(8) uint64_t s_mbar;
  const int first = blockIdx.x * kTileSlots;
  const int p = first + threadIdx.x;
  const bool own = p < P.n;
  uint32_t cell = 0;
  bool regular = true;
  float4 xf = make_float4(0.f, 0.f, 0.f, 0.f);
  if (own) {
    xf = xsa_load(xsa, p);
    cell = __ldg(cellp + p);
    int cx, cy, cz;
    unpack_cell(V, cell, cx, cy, cz);
    const float inv_h = 1.0f / P.h;
    if (!(axis_inside(xf.x, inv_h, cx) && axis_inside(xf.y, inv_h, cy) &&
          axis_inside(xf.z, inv_h, cz))) {
      float4 xp, dp;
      ld_pd(pd, p, xp, dp);
      regular = axis_regular(xstar_d(xp.x, dp.x), P.hd, cx, P.nx) &&
                axis_regular(xstar_d(xp.y, dp.y), P.hd, cy, P.ny) &&
                axis_regular(xstar_d(xp.z, dp.z), P.hd, cz, P.nz);
    }
  }
  if (p == 0) V.err[kGridBarrier] = 0;  // (for the solve of this step)
  if (threadIdx.x < 32) tile_ranges(P, V, cellp, first, min(first + kTileSlots, P.n) - 1, s_info);
  const bool all_regular = __syncthreads_and(regular ? 1 : 0) != 0;
  const int total = s_info.total;
  const bool tiled = all_regular && total <= V.cap;
  if (threadIdx.x < 32) {
    const int r = threadIdx.x;
    if (r < 9) {
      s_off[r] = s_info.o[r] - s_info.s[r];
      tiles[blockIdx.x].s[r] = s_info.s[r];
      tiles[blockIdx.x].o[r] = s_info.o[r];
    }
    if (r == 9) tiles[blockIdx.x].total = tiled ? total : -1;
    if (tiled) {
      if (r == 0) {
        mbar_init1(&s_mbar);
        mbar_expect(&s_mbar, (uint32_t)total * 16u);
      }
      __syncwarp();
      if (r < 9) {
        const int o = s_info.o[r], e = r < 8 ? s_info.o[r + 1] : total;
        if (e > o) bulk_load(s_tile + o, xsa + s_info.s[r], (uint32_t)(e - o) * 16u, &s_mbar);
      }
    }
  }
  __syncthreads();
  if (tiled && !mbar_wait0(&s_mbar)) {
    atomicOr(V.err, kErrTileWait);
    mbar_wait0(&s_mbar);
  }
  if (!own) return;
  const BuildRow c{P, pd, f2_dup(xf.x), f2_dup(xf.y), f2_dup(xf.z), f2_dup(-P.h2), p};
  uint4* out = reinterpret_cast<uint4*>(nbr) + p;
  int count;
  if (tiled) {
    Hits<uint16_t, 4> hits{s_mask + threadIdx.x, s_base + threadIdx.x};
    build_rows<true>(c, V, cell, s_tile, s_off, hits, out);
    hits.finish((uint32_t)(p + s_off[4]) << 4, out, P.n);
    count = hits.found;
  } else if (regular) {
    Hits<int, 0> hits{s_mask + threadIdx.x, reinterpret_cast<int*>(s_tile) + threadIdx.x};
    build_rows<false>(c, V, cell, xsa, nullptr, hits, out);
    hits.finish((uint32_t)p, out, P.n);
    count = hits.found;
  } else {
    count = walk_27_cells(P, V, pd, xsa, p, nbr);
  }
  ncount[p] = (uint8_t)count;
}

__global__ void __launch_bounds__(kBlock)
    k_export_buckets(const NbrView V, const uint32_t* __restrict__ ids,
                     uint32_t* __restrict__ nbr, int32_t* __restrict__ count,
                     uint32_t* __restrict__ err) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= V.n) return;
  // the list's last block must hold p past the count (the batched visits
  // read those entries as the pair (p, p))
  const int cnt = (int)__ldg(V.ncount + p), per = has_tile(V, p) ? 8 : 4;
  for (int t = cnt; t & (per - 1); ++t)
    if (nbr_entry(V, p, t) != (uint32_t)p) atomicOr(err, kErrNbrTail);
  const uint32_t idp = __ldg(ids + p);
  uint32_t* out = nbr + (size_t)idp * kMaxNeighbors;
  for (int j = 0; j < kMaxNeighbors; ++j) out[j] = j < cnt ? __ldg(ids + nbr_entry(V, p, j)) : 0u;
  count[idp] = cnt;
}

}  // namespace

void launch_hash(const DevParams& P, const PD* pd, const float4* vel, const uint32_t* ids,
                 uint32_t* keys_by_id, uint32_t* loc_by_id, uint32_t* hist, int passes,
                 bool predict, uint32_t* err, cudaStream_t st) {
  k_hash<<<grid_for(P.n), kBlock, 0, st>>>(P, pd, vel, ids, keys_by_id, loc_by_id, hist,
                                           passes, predict ? 1 : 0, err);
}

size_t cell_table_words(uint32_t ncells, int cap) {
  // cstart[0..C], then the scan's ticket and block states, then whether a cell is
  // crowded and what is placed of the crowded ones
  return (((size_t)ncells + 2) & ~(size_t)1) + 2 * (2 + (size_t)ncells / kScanItems + 1) + 1 +
         (size_t)cap / (kCrowded + 1) + 1;
}

bool counts_cells(int n, uint32_t ncells) {
  return n > 0 && (uint64_t)ncells <= 32ull * (uint64_t)n;
}

int launch_count_cells(const DevParams& P, const PD* pd, const float4* vel, const uint32_t* ids,
                       uint32_t* cstart, const CountScratch& s, bool predict, uint32_t* crowded,
                       uint32_t* err, cudaStream_t st) {
  const uint32_t m = P.ncells + 1;
  uint32_t* after = cstart + (((size_t)P.ncells + 2) & ~(size_t)1);
  unsigned long long* state = reinterpret_cast<unsigned long long*>(after);
  uint32_t* any = after + 2 * (2 + (size_t)P.ncells / kScanItems + 1);
  cudaMemsetAsync(cstart, 0, cell_table_words(P.ncells, P.n) * sizeof(uint32_t), st);
  k_count<<<grid_for(P.n), kBlock, 0, st>>>(P, pd, vel, s.keys, s.rank, cstart, predict ? 1 : 0,
                                            err);
  k_scan_counts<<<(int)(((uint64_t)m + kScanItems - 1) / kScanItems), kScanThreads, 0, st>>>(
      cstart, m, state, crowded, any, err);
  int passes = 2;  // digits of the ids below n, an even number
  while (passes < 4 && (uint64_t)P.n > 1ull << (passes * kRadixBits)) passes += 2;
  const PlaceArgs a{s.keys, s.rank, ids, any, any + 1, s.cell_ids, s.cell_src, s.ids2, s.src2, passes};
  k_place<<<grid_for(P.n), kBlock, 0, st>>>(P.n, cstart, a);
  return 3;
}

void launch_slot_keys(const uint32_t* cstart, uint32_t ncells, uint32_t* keys, cudaStream_t st) {
  k_slot_keys<<<(int)(((uint64_t)ncells + kBlock - 1) / kBlock), kBlock, 0, st>>>(cstart, ncells,
                                                                                 keys);
}

void launch_reorder(const DevParams& P, const SlotOrder& order, const PD* pd_in,
                    const float4* vel_in, PD* pd_out, float4* vel_out, float4* xsa, uint4* nr_out,
                    uint32_t* cellp, bool predict, bool move_vel, const ReorderExtra* extra,
                    cudaStream_t st) {
  ReorderExtra ex = {};
  if (extra) ex = *extra;
  if (order.keys)
    k_reorder<true><<<grid_for(P.n), kBlock, 0, st>>>(P, order, pd_in, vel_in, pd_out, vel_out, xsa,
                                                      nr_out, cellp, predict ? 1 : 0,
                                                      move_vel ? 1 : 0, ex);
  else
    k_reorder<false><<<grid_for(P.n), kBlock, 0, st>>>(P, order, pd_in, vel_in, pd_out, vel_out,
                                                       xsa, nr_out, cellp, predict ? 1 : 0,
                                                       move_vel ? 1 : 0, ex);
}

// Up to kBoundsMaxCells cells the bounds kernel writes the table in one launch
// (256 blocks of 2048 cells, all resident at once); beyond, its two searches per
// block cost more than the worklist's second launch.
constexpr uint32_t kBoundsMaxCells = 1u << 19;

int launch_cell_starts(const uint32_t* keys_sorted, int n, uint32_t ncells, uint32_t* cstart,
                       uint4* gaps, uint32_t* gap_count, uint32_t* err, cudaStream_t st) {
  if (n == 0) {
    cudaMemsetAsync(cstart, 0, sizeof(uint32_t) * ((size_t)ncells + 1), st);
    return 0;
  }
  if (ncells <= kBoundsMaxCells) {
    launch_bounds(keys_sorted, n, (int)ncells + 1, cstart, false, st, err);
    return 1;
  }
  cudaMemsetAsync(gap_count, 0, sizeof(uint32_t), st);
  const int threads = (n + kStartsPerThread - 1) / kStartsPerThread;
  k_cell_starts<<<grid_for(threads), kBlock, 0, st>>>(keys_sorted, n, ncells, cstart, gaps,
                                                       gap_count, err);
  k_fill_gaps<<<148 * 16, kBlock, 0, st>>>(gaps, gap_count, cstart);
  return 2;
}

void launch_build_neighbors(const DevParams& P, const NbrView& V, const PD* pd,
                            const float4* xsa, const uint32_t* cellp, uint32_t* nbr,
                            uint8_t* ncount, TileInfo* tiles, cudaStream_t st) {
  const size_t bytes = (size_t)(V.cap + 4) * sizeof(float4) +
                       (kWords + 1) * kTileSlots * (sizeof(uint32_t) + sizeof(uint16_t));
  allow_shared(k_build, bytes);
  k_build<<<grid_for(P.n, kTileSlots), kTileSlots, bytes, st>>>(P, V, pd, xsa, cellp, nbr, ncount,
                                                                tiles);
}

void launch_export_buckets(const NbrView& V, const uint32_t* ids, uint32_t* nbr, int32_t* count,
                           uint32_t* err, cudaStream_t st) {
  k_export_buckets<<<grid_for(V.n), kBlock, 0, st>>>(V, ids, nbr, count, err);
}

}  // namespace sphpc
