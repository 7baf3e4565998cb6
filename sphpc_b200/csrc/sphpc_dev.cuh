// sphpc_dev.cuh -- device-side layout, parameters and shared primitives of
// the B200 PBF pipeline.
//
// State layout in HBM (slot order = particles sorted by uniform-grid cell
// key, rebuilt every step):
//   pd[n]    PD      32-byte record {x, d}: x the step-start position (.w
//                    unused), d = x* - x the predicted-position displacement
//                    (.w carries lambda after the density/lambda pass and the
//                    density after the position pass).  A neighbour's record
//                    is one 256-bit load.
//   nr[n]    uint4   16-byte neighbour record {X, Y, Z, w}: x* in fixed
//                    point (2^-k units, wrapping mod 2^32, so the difference
//                    of two records is exact for any box) and a payload (w:
//                    lambda after a density/lambda pass, the density after
//                    a position pass).  Neighbour sums gather only these.
//   xsa[n]   float4  x* as absolute FP32 (neighbour-build candidate test),
//                    in pair blocks: slots 2b, 2b+1 share {x0, x1, y0, y1},
//                    {z0, z1, 0, 0} at float4 index 2b
//   vel[n]   float4  v
//   ids[n]   u32     original particle index of each slot
//   cellp[n] u32     packed grid cell (cx | cy<<bx | cz<<(bx+by)) of x* at
//                    neighbour-build time
//   nbr[15][n] uint4 neighbour lists in the reference's bucket order, one
//                    16-byte block of consecutive entries per particle and
//                    block index (column p, so a warp reads four 128-byte
//                    lines per block): eight 16-bit offsets into the record
//                    tile of the particle's block of kTileSlots slots
//                    (TileInfo), or four 32-bit slots where the block has no
//                    tile; the last block's entries past the count are the
//                    particle itself
//   ncount[n] u8     bucket sizes
//   cstart[C+1] u32  start slot of every cell (lower bound), cstart[C] = n
//
// The canonical predicted position is the double fl64(x + d): the hash, the
// neighbour test, the box clamp and the SDF lookup are evaluated on it in
// FP64 exactly as the reference evaluates its double x_star.  Pair
// differences inside the neighbour sums are integer differences of the
// fixed-point records (2^-k units, k = 28 - ceil(log2 h): 7.5e-9 for h = 2)
// converted to FP32, so their precision does not depend on the box size.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace sphpc {

constexpr int kMaxNeighbors = 60;   // MAX_NEIGHBORS, neighbors.h:6

// Position record of one particle: step-start x and displacement d = x* - x.
struct __align__(32) PD {
  float4 x;
  float4 d;
};

// Packed FP32x2 (sm_100): two independent IEEE single-precision operations
// per instruction, each rounded to nearest as its scalar form.
__device__ __forceinline__ uint64_t f2_pack(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ uint64_t f2_dup(float a) { return f2_pack(a, a); }
__device__ __forceinline__ uint64_t f2_add(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t f2_sub(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t f2_mul(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ float f2_lo(uint64_t a) { return __uint_as_float((uint32_t)a); }
__device__ __forceinline__ float f2_hi(uint64_t a) { return __uint_as_float((uint32_t)(a >> 32)); }

// One 256-bit read-only load of a record (ld.global.nc.v8.f32, sm_100).
__device__ __forceinline__ void ld_pd(const PD* __restrict__ base, int i, float4& x, float4& d) {
  asm("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
      : "=f"(x.x), "=f"(x.y), "=f"(x.z), "=f"(x.w), "=f"(d.x), "=f"(d.y), "=f"(d.z), "=f"(d.w)
      : "l"(base + i));
}

__device__ __forceinline__ void st_pd(PD* base, int i, const float4 x, const float4 d) {
  asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(base + i),
               "f"(x.x), "f"(x.y), "f"(x.z), "f"(x.w), "f"(d.x), "f"(d.y), "f"(d.z), "f"(d.w)
               : "memory");
}

// 16-byte neighbour record: fixed-point x* and a payload, one 128-bit load.
__device__ __forceinline__ uint4 ld_nr(const uint4* __restrict__ base, int i) {
  uint4 r;
  asm("ld.global.nc.v4.u32 {%0,%1,%2,%3}, [%4];"
      : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
      : "l"(base + i));
  return r;
}

__device__ __forceinline__ float nr_w(const uint4 r) { return __uint_as_float(r.w); }

// |(x, y, z)|^2 as fma(z, z, fma(y, y, x x)).  The neighbour sums spell out
// every fused multiply-add (fmaf) and every product or sum that must not be
// fused (__fmul_rn, __fadd_rn), so their rounding is the same in every build
// of the library, whatever contractions the compiler would choose.
__device__ __forceinline__ float norm2(float x, float y, float z) {
  return fmaf(z, z, fmaf(y, y, __fmul_rn(x, x)));
}

// Error bits raised by kernels (host reads them back).
enum : uint32_t {
  kErrSortSpin = 1u << 1,          // radix-sort look-back wait gave up
  kErrCellRange = 1u << 2,         // a particle hashed outside the grid
  kErrScanSpin = 1u << 3,
  kErrNbrTail = 1u << 5,           // a list block's entries past the count are not p
  kErrTileWait = 1u << 6,          // the wait for a tile's bulk copies gave up
  kErrGridWait = 1u << 7,          // the solve's wait for the other blocks gave up
};

// Word after the error bits that the blocks of the solve meet at.
constexpr int kGridBarrier = 2;

struct DevParams {
  int n;
  int nx, ny, nz;
  uint32_t nxny;
  uint32_t ncells;      // C = nx*ny*nz
  int bx, by;           // packed-cell bit widths of x and y
  uint32_t mx, my;      // masks for cx and cy
  double hd;            // smoothing radius (double)
  double fx_scale;      // 2^k: fixed-point units per length of the records
  float fx_inv;         // 2^-k
  float fx_inv2;        // 2^-2k
  float h_fx;           // h in fixed-point units (h 2^k)
  float rmin2_fx;       // (1e-4 h)^2 in fixed-point units squared
  double h2d;
  // neighbour-build FP32 pre-test band: pairs with FP32 r^2 in [lo, hi] go
  // to the exact FP64 test (lo = -1, hi = inf: every pair does)
  float bld_h2lo, bld_h2hi;
  float bld_band;       // the band's half width (inf: every pair)
  float h, h2;
  float rmin;           // r floor 1e-4 h (particles.c:636)
  // smoothing-kernel constants; *_m variants carry the particle mass
  float W0m;            // m * W(0)
  float Wn, Wn_m;       // poly6 norm
  float DWn, DWn_m;     // spiky gradient norm
  float DWPn;           // poly6 gradient norm
  float m, rho0, inv_rho0, inv_rho0_sq;
  double rho0_d;
  float lambda_eps;
  float scorr_k;        // s_corr = -k (W/W(dq))^n
  int scorr_n;
  float inv_Wdq;
  float scorr_u;        // 1 / (h^2 - dq^2): W(r)/W(dq) = ((h^2 - r^2) scorr_u)^3
  float scorr_u_fx;     // scorr_u 2^-2k (for r^2 in fixed-point units squared)
  float scorr_uh2;      // scorr_u h^2
  float c_xsph;
  int xsph_exact;       // 0: reference r expression (particles.c:439)
  float gamma, C_norm;  // surface tension
  float vort_eps;
  float dt, inv_dt, v_max;
  double dt_d, gdt_d;   // gravity increment (-g*dt) in double
  int gaxis;
  float gdt_f;
  double bmin[3], bmax[3], bmax_eps[3];  // clamp (particles.c:842-867)
  // obstacle SDF (x fastest), tex3D-style sampling
  int has_sdf;
  int sdim[3];
  const float* sdf;
  double ob_min[3], ob_max[3];
  float ob_len[3];      // world extents as float (obstacle_cuda.cu:74-85)
  float tex_sp[3];      // 1/dim in normalised coordinates
  float model_to_world;
};

// The neighbourhood of kTileSlots consecutive slots as nine contiguous slot
// ranges: with k0 and k1 the cell keys of the first and the last slot, range
// r = 3 (dz + 1) + dy + 1 holds the cells k0 + d - 1 .. k1 + d + 1, d = dz nx ny
// + dy nx, so it covers cells cx-1 .. cx+1 of that row for every slot of the
// block, also where the block runs over the end of a row of cells.  Range r
// starts at slot s[r] and at record o[r] of the tile that holds all nine one
// after the other (total records; -1: more than tile_cap, or a particle whose
// neighbour cells are not the regular ones: the block's lists hold slots).
// Range starts and lengths are even, so that pairs of slots stay together.
//
// tile_cap, the most records of a tile: nine ranges of 128 slots and about four
// cells at the ends hold 1400 records at the rest density, and 1472 records of 16
// bytes leave room for nine blocks per SM.  Where the fluid is pressed or its rows
// are short some blocks need more (34% of 4096 particles 800 steps after a dam
// break, 21% of 290k), and one that has no tile holds the others up when all run
// at once: a set of up to four blocks per SM has the room that its passes over
// two arrays leave a block.
// A step of 4096 particles 115 -> 105 us, of 13,824 125 -> 107, of 32,768 138 ->
// 120, of 68,921 172 -> 167.  In larger sets occupancy is worth more: with 1744
// records 290k take 524 us for 534, 4.2M 5094 for 4982.
// Entries are 16-bit byte offsets, and the build adds up to 32 records to one.
constexpr int kTileSlots = 128;
constexpr int kTileCap = 1472;
constexpr int kTileCapMost = 4056;
inline int tile_cap(int n, int sms) {
  const int blocks = (n + kTileSlots - 1) / kTileSlots;
  const int per_sm = blocks > sms ? (blocks + sms - 1) / sms : 1;
  if (per_sm > 4) return kTileCap;
  const int room = ((226 * 1024 / per_sm - 2048) / 32) & ~7;
  return room < kTileCapMost ? room : kTileCapMost;
}
// Shared memory beyond 48 KB has to be allowed for a kernel: up to two of the
// largest tiles, whatever this launch needs.
template <class K>
inline void allow_shared(K* kernel, size_t bytes) {
  if (bytes > 48 * 1024)
    cudaFuncSetAttribute(reinterpret_cast<const void*>(kernel),
                         cudaFuncAttributeMaxDynamicSharedMemorySize, 2 * kTileCapMost * 16);
}
struct TileInfo {
  int s[9], o[9], total, pad;
};

// View of the per-step neighbour structure.
struct NbrView {
  const uint32_t* __restrict__ nbr;     // [15][n] blocks of 16 bytes
  const uint8_t* __restrict__ ncount;   // [n]
  const uint32_t* __restrict__ cstart;  // [C+1]
  const TileInfo* __restrict__ tiles;   // [ceil(n / kTileSlots)]
  uint32_t* err;
  int n;
  int cap;                              // records of a tile, at most (tile_cap)
  int nx, ny, nz;
  uint32_t nxny;
  int bx, by;
  uint32_t mx, my;
};

__device__ __forceinline__ void unpack_cell(const NbrView& v, uint32_t cp, int& cx,
                                            int& cy, int& cz) {
  cx = (int)(cp & v.mx);
  cy = (int)((cp >> v.bx) & v.my);
  cz = (int)(cp >> (v.bx + v.by));
}

__device__ __forceinline__ uint4 nbr_block(const NbrView& v, int p, int b) {
  return __ldg(reinterpret_cast<const uint4*>(v.nbr) + (size_t)b * v.n + p);
}

__device__ __forceinline__ bool has_tile(const NbrView& v, int p) {
  return __ldg(&v.tiles[p / kTileSlots].total) >= 0;
}

// Slot of list entry j of particle p (entry by entry: for exports and checks).
__device__ __forceinline__ uint32_t nbr_entry(const NbrView& v, int p, int j) {
  if (!has_tile(v, p)) return __ldg(v.nbr + (((size_t)(j >> 2) * v.n + p) << 2) + (j & 3));
  const uint16_t* l = reinterpret_cast<const uint16_t*>(v.nbr);
  const int i = (int)(__ldg(l + (((size_t)(j >> 3) * v.n + p) << 3) + (j & 7)) >> 4);
  const TileInfo* t = v.tiles + p / kTileSlots;
  int r = 8;
  while (r > 0 && __ldg(&t->o[r]) > i) --r;
  return (uint32_t)(__ldg(&t->s[r]) + i - __ldg(&t->o[r]));
}

// ---------------------------------------------------------------------------
// Tiles in shared memory.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

// Bounded wait for a phase (parity) of an mbarrier (~1e6 polls, each of which
// may itself suspend the thread for a while).
__device__ __forceinline__ bool mbar_wait(uint64_t* mbar, uint32_t parity) {
  const uint32_t addr = smem_addr(mbar);
  for (int i = 0; i < (1 << 20); ++i) {
    uint32_t ok;
    asm volatile(
        "{\n.reg .pred P1;\nmbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n"
        "selp.b32 %0, 1, 0, P1;\n}\n"
        : "=r"(ok)
        : "r"(addr), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}
__device__ __forceinline__ bool mbar_wait0(uint64_t* mbar) { return mbar_wait(mbar, 0); }

__device__ __forceinline__ void mbar_init1(uint64_t* mbar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(mbar)));
  asm volatile("fence.mbarrier_init.release.cluster;");
}

__device__ __forceinline__ void mbar_expect(uint64_t* mbar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(mbar)),
               "r"(bytes)
               : "memory");
}

// One bulk copy to this block's shared memory (16-byte aligned, a multiple of
// 16 bytes), counted on mbar.
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes,
                                          uint64_t* mbar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
          "r"(smem_addr(dst)),
      "l"(src), "r"(bytes), "r"(smem_addr(mbar))
      : "memory");
}

// The tile of a block of kTileSlots threads: tile_load starts the copies of
// NARR arrays of 16-byte records (array k at byte k * cap * 16 of `tile`)
// and returns whether the block has a tile; tile_wait waits for them.  Every
// thread of the block calls both.
template <int NARR>
__device__ __forceinline__ bool tile_load(const NbrView& v, const void* a0, const void* a1,
                                          unsigned char* tile, uint64_t* mbar) {
  const TileInfo* t = v.tiles + blockIdx.x;
  const int total = __ldg(&t->total);
  if (total >= 0 && threadIdx.x < 32) {
    const int r = threadIdx.x;
    int s = 0, o = 0, e = 0;
    if (r < 9) {
      s = __ldg(&t->s[r]);
      o = __ldg(&t->o[r]);
      e = r < 8 ? __ldg(&t->o[r + 1]) : total;
    }
    if (r == 0) {
      mbar_init1(mbar);
      mbar_expect(mbar, (uint32_t)total * (16u * NARR));
    }
    __syncwarp();
    if (e > o) {
      const uint32_t bytes = (uint32_t)(e - o) * 16u;
      bulk_load(tile + o * 16, static_cast<const uint4*>(a0) + s, bytes, mbar);
      if (NARR == 2)
        bulk_load(tile + (v.cap + o) * 16, static_cast<const uint4*>(a1) + s, bytes, mbar);
    }
  }
  return total >= 0;
}

__device__ __forceinline__ bool tile_wait(const NbrView& v, bool tiled, uint64_t* mbar) {
  if (!tiled) return true;
  __syncthreads();  // the mbarrier is initialised
  if (mbar_wait0(mbar)) return true;
  atomicOr(v.err, kErrTileWait);
  mbar_wait0(mbar);  // the copies in flight write this block's shared memory
  return false;
}

// A batch of four list entries: the neighbours' records and, with a second
// array, their vectors; entries past the count are the particle itself (the
// pair (p, p): difference 0).
template <int NARR>
struct Batch {
  uint4 r[4];
  float4 e[NARR == 2 ? 4 : 1];
};

// Visits the list of particle p in batches of four: f(batch, nvalid) with
// nvalid = count - (entries before the batch).  tiled: offsets into the tile
// (16-bit entries, eight per block), else slots (gathered from nr and e).  The
// next list block is loaded before this one's bodies run.  (Eight entries a
// round without the test between them measured 5% slower: more registers live
// for no fewer wavefronts.)
// LIVE: the records change while the kernel runs (ordinary loads, after a fence).
template <int NARR, bool LIVE = false, class F>
__device__ __forceinline__ void visit(const NbrView& v, bool tiled, const unsigned char* tile,
                                      const uint4* nr, const float4* __restrict__ e,
                                      int p, int cnt, uint4 blk, F&& f) {
  if (tiled) {
    const unsigned char* tile_e = tile + v.cap * 16;
    auto load = [&](uint32_t w0, uint32_t w1) {
      const uint32_t o[4] = {w0 & 0xffffu, w0 >> 16, w1 & 0xffffu, w1 >> 16};
      Batch<NARR> b;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        b.r[u] = *reinterpret_cast<const uint4*>(tile + o[u]);
        if (NARR == 2) b.e[u] = *reinterpret_cast<const float4*>(tile_e + o[u]);
      }
      return b;
    };
    for (int j0 = 0; j0 < cnt; j0 += 8) {
      const uint4 w = blk;
      if (j0 + 8 < cnt) blk = nbr_block(v, p, (j0 >> 3) + 1);
      f(load(w.x, w.y), cnt - j0);
      if (j0 + 4 < cnt) f(load(w.z, w.w), cnt - j0 - 4);
    }
  } else {
    for (int j0 = 0; j0 < cnt; j0 += 4) {
      const int q[4] = {(int)blk.x, (int)blk.y, (int)blk.z, (int)blk.w};
      if (j0 + 4 < cnt) blk = nbr_block(v, p, (j0 >> 2) + 1);
      Batch<NARR> b;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        b.r[u] = LIVE ? *(nr + q[u]) : ld_nr(nr, q[u]);
        if (NARR == 2) b.e[u] = __ldg(e + q[u]);
      }
      f(b, cnt - j0);
    }
  }
}

// ---------------------------------------------------------------------------
// Canonical double predicted position and the reference's box clamp.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double xstar_d(float x, float d) {
  return __dadd_rn((double)x, (double)d);
}

// ApplyBoundaryConditions, particles.c:842-867, on one axis.
__device__ __forceinline__ double clamp_axis(double x, double lo, double hi,
                                             double hi_eps) {
  if (x < lo) return lo;
  if (x >= hi) return hi_eps;
  return x;
}

// Fixed-point coordinate of a double position (round to nearest, mod 2^32).
__device__ __forceinline__ uint32_t fx_of(const DevParams& P, double x) {
  return (uint32_t)(unsigned long long)__double2ll_rn(__dmul_rn(x, P.fx_scale));
}

__device__ __forceinline__ uint4 make_nr(const DevParams& P, double x, double y, double z,
                                         float w) {
  return make_uint4(fx_of(P, x), fx_of(P, y), fx_of(P, z), __float_as_uint(w));
}

// HashVal, neighbors.c:79-98, per axis: floor(x / spacing) in FP64.
__device__ __forceinline__ int grid_coord(double x, double h) {
  return (int)(unsigned)floor(__ddiv_rn(x, h));
}

// ---------------------------------------------------------------------------
// SDF obstacle: tex3D<float> (linear filter, clamp addressing, normalised
// coordinates; obstacle_cuda.cu:166-181) with exact FP32 weights.
// ---------------------------------------------------------------------------
__device__ __forceinline__ float sdf_texel(const DevParams& P, int i, int j, int k) {
  i = min(max(i, 0), P.sdim[0] - 1);
  j = min(max(j, 0), P.sdim[1] - 1);
  k = min(max(k, 0), P.sdim[2] - 1);
  return __ldg(P.sdf + ((size_t)k * P.sdim[1] + j) * P.sdim[0] + i);
}

__device__ __forceinline__ float lerp_rn(float a, float b, float t) {
  return __fmaf_rn(t, __fsub_rn(b, a), a);
}

__device__ __forceinline__ float sdf_sample(const DevParams& P, float u, float v, float w) {
  const float xb = __fsub_rn(__fmul_rn(u, (float)P.sdim[0]), 0.5f);
  const float yb = __fsub_rn(__fmul_rn(v, (float)P.sdim[1]), 0.5f);
  const float zb = __fsub_rn(__fmul_rn(w, (float)P.sdim[2]), 0.5f);
  const float fx = floorf(xb), fy = floorf(yb), fz = floorf(zb);
  const float ax = __fsub_rn(xb, fx), ay = __fsub_rn(yb, fy), az = __fsub_rn(zb, fz);
  const int i = (int)fx, j = (int)fy, k = (int)fz;
  const float c00 = lerp_rn(sdf_texel(P, i, j, k), sdf_texel(P, i + 1, j, k), ax);
  const float c10 = lerp_rn(sdf_texel(P, i, j + 1, k), sdf_texel(P, i + 1, j + 1, k), ax);
  const float c01 = lerp_rn(sdf_texel(P, i, j, k + 1), sdf_texel(P, i + 1, j, k + 1), ax);
  const float c11 = lerp_rn(sdf_texel(P, i, j + 1, k + 1), sdf_texel(P, i + 1, j + 1, k + 1), ax);
  const float c0 = lerp_rn(c00, c10, ay);
  const float c1 = lerp_rn(c01, c11, ay);
  return lerp_rn(c0, c1, az);
}

// CalculateParticleCollisions_kernel body (obstacle_cuda.cu:62-115) on one
// double position.  Returns true and updates xyz when the particle is pushed.
__device__ __forceinline__ bool sdf_collide(const DevParams& P, double& x, double& y,
                                            double& z) {
  if (!(x > P.ob_min[0] && x < P.ob_max[0] && y > P.ob_min[1] && y < P.ob_max[1] &&
        z > P.ob_min[2] && z < P.ob_max[2]))
    return false;
  const float xt = (float)__ddiv_rn(__dsub_rn(x, P.ob_min[0]), (double)P.ob_len[0]);
  const float yt = (float)__ddiv_rn(__dsub_rn(y, P.ob_min[1]), (double)P.ob_len[1]);
  const float zt = (float)__ddiv_rn(__dsub_rn(z, P.ob_min[2]), (double)P.ob_len[2]);
  const float dist = sdf_sample(P, xt, yt, zt);
  if (!(dist < 0.0f)) return false;
  const float gx = __fsub_rn(sdf_sample(P, __fadd_rn(xt, P.tex_sp[0]), yt, zt),
                             sdf_sample(P, __fsub_rn(xt, P.tex_sp[0]), yt, zt));
  const float gy = __fsub_rn(sdf_sample(P, xt, __fadd_rn(yt, P.tex_sp[1]), zt),
                             sdf_sample(P, xt, __fsub_rn(yt, P.tex_sp[1]), zt));
  const float gz = __fsub_rn(sdf_sample(P, xt, yt, __fadd_rn(zt, P.tex_sp[2])),
                             sdf_sample(P, xt, yt, __fsub_rn(zt, P.tex_sp[2])));
  const float dot = __fadd_rn(__fadd_rn(__fmul_rn(gx, gx), __fmul_rn(gy, gy)),
                              __fmul_rn(gz, gz));
  const float inv = __fdiv_rn(1.0f, __fsqrt_rn(dot));
  const float dw = __fmul_rn(fabsf(dist), P.model_to_world);
  y = __dadd_rn(y, (double)__fmul_rn(dw, __fmul_rn(gy, inv)));
  x = __dadd_rn(x, (double)__fmul_rn(dw, __fmul_rn(gx, inv)));
  z = __dadd_rn(z, (double)__fmul_rn(dw, __fmul_rn(gz, inv)));
  return true;
}

}  // namespace sphpc
