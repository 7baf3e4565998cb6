// pbf.cu -- the neighbour passes and pointwise steps of one PBF time step.
//
// Every pass is one thread per particle in slot (cell-sorted) order; the
// neighbour loop visits the bucket of the particle in the reference's order.
// Sums are FP32 (density with Kahan compensation); the box clamp, the SDF
// lookup and the position update are FP64 on the canonical double x* = x + d
// of the particle's own record.  Neighbours are read from the 16-byte records
// (fixed-point x* and a payload), and a vector beside them in the passes that
// need one; the pair difference is their exact integer difference.
//
// A block of kTileSlots threads first brings the records of its neighbourhood
// into shared memory (its tile, sphpc_dev.cuh: nine bulk copies, about 1400
// records) and its lists index them; a block without a tile gathers from
// global memory.
//
// Bounds: the shared-memory pipe (70-80% of its wavefronts).  A warp's gather
// of 32 16-byte records costs about nine wavefronts (eight lanes at a time, a
// conflict where two of them read different records of one 16-byte bank
// group), where the same gather through the L1 touched thirteen 128-byte
// lines, and a list entry takes two bytes instead of four.  At 16.7M
// particles, per launch: density 917 -> 724 us, position 1048 -> 904, colour
// and tension 2582 -> 2255, XSPH 1647 -> 1622, vorticity and confinement
// 2585 -> 2442.
#include "kernels.cuh"

#include <algorithm>

namespace sphpc {

namespace {

struct Pair {
  float dx, dy, dz, r2;
};

// Resident blocks of kTileSlots threads asked of the compiler: one tile of
// records (23.5 KB) fits nine times into an SM's shared memory, two four times.
constexpr int kMinBlocks1 = 9;
constexpr int kMinBlocks2 = 4;
constexpr int kMinBlocksFeatures = 8;

// Head of a neighbour pass: the particle, its list's size and first block, and
// the start of the tile's copies (NARR arrays of records).
#define SPHPC_PASS_HEAD(NARR, arr0, arr1)                                          \
  extern __shared__ __align__(128) unsigned char tile[];                           \
  __shared__ __align__(8) uint64_t s_mbar;                                         \
  const bool tiled = tile_load<NARR>(V, arr0, arr1, tile, &s_mbar);                \
  const int p = blockIdx.x * blockDim.x + threadIdx.x;                             \
  const bool own = p < P.n;                                                        \
  int cnt = own ? (int)__ldg(V.ncount + p) : 0;                                    \
  const uint4 blk = cnt > 0 ? nbr_block(V, p, 0) : make_uint4(0u, 0u, 0u, 0u)
// Before the list is visited: the tile has arrived (a wait that gave up raises
// its error bit and visits nothing).
#define SPHPC_PASS_READY() \
  if (!tile_wait(V, tiled, &s_mbar)) cnt = 0

__device__ __forceinline__ void ld_rw(const PD* base, int i, float4& x, float4& d) {
  x = base[i].x;
  d = base[i].d;
}

// x*_p - x*_q as (x_p - x_q) + (d_p - d_q): exact in the first term for any
// box size, so the FP32 pair geometry keeps its relative precision.
__device__ __forceinline__ Pair pair_geom(const float4 xp, const float4 dp, const float4 xq,
                                          const float4 dq) {
  Pair g;
  g.dx = (xp.x - xq.x) + (dp.x - dq.x);
  g.dy = (xp.y - xq.y) + (dp.y - dq.y);
  g.dz = (xp.z - xq.z) + (dp.z - dq.z);
  g.r2 = norm2(g.dx, g.dy, g.dz);
  return g;
}

// x*_p - x*_q from two 16-byte records: the wrapping integer difference is
// exact, its conversion to FP32 rounds like any FP32 difference.
__device__ __forceinline__ Pair pair_nr(const DevParams& P, const uint4 a, const uint4 b) {
  Pair g;
  g.dx = __fmul_rn((float)(int)(a.x - b.x), P.fx_inv);
  g.dy = __fmul_rn((float)(int)(a.y - b.y), P.fx_inv);
  g.dz = __fmul_rn((float)(int)(a.z - b.z), P.fx_inv);
  g.r2 = norm2(g.dx, g.dy, g.dz);
  return g;
}

// Two neighbours' pair geometry at a time as packed FP32x2 values (low half:
// the first neighbour): a packed operation is issued once for two neighbours
// and rounds each as its scalar form; what a list's order fixes -- the running
// sums -- stays scalar.  Kept where issue comes next after the shared-memory
// pipe (4.2M particles, scalar -> packed: density 204 -> 190 us, position 241
// -> 234); the passes that gather a vector too are no faster with it (tension
// 581 -> 598, XSPH 409 -> 411, vorticity 620 -> 626) and stay scalar.
//
// Differences x*_p - x*_q of two 16-byte records in fixed-point units: the
// wrapping integer difference is exact, its conversion to FP32 rounds like any
// FP32 difference.
struct Pair2 {
  uint64_t x, y, z;
};
__device__ __forceinline__ Pair2 diff2(const uint4 p, const uint4 a, const uint4 b) {
  return {f2_pack((float)(int)(p.x - a.x), (float)(int)(p.x - b.x)),
          f2_pack((float)(int)(p.y - a.y), (float)(int)(p.y - b.y)),
          f2_pack((float)(int)(p.z - a.z), (float)(int)(p.z - b.z))};
}
// |d|^2 of both, as norm2.
__device__ __forceinline__ uint64_t norm2_2(const Pair2& d) {
  return f2_fma(d.z, d.z, f2_fma(d.y, d.y, f2_mul(d.x, d.x)));
}
__device__ __forceinline__ uint64_t max2(uint64_t a, float b) {
  return f2_pack(fmaxf(f2_lo(a), b), fmaxf(f2_hi(a), b));
}

// 1/sqrt(x) of a normal x (PTX rsqrt.approx.ftz.f32): the value rsqrtf gives,
// without the range test and the two scalings that rsqrtf spends on subnormal
// arguments, which the floors below rule out.
__device__ __forceinline__ float rsqrt_normal(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

__device__ __forceinline__ uint64_t rsqrt2(uint64_t a) {
  return f2_pack(rsqrt_normal(f2_lo(a)), rsqrt_normal(f2_hi(a)));
}

// r_mag floored at 1e-4 h (particles.c:635-637): returns r and 1/r.
__device__ __forceinline__ void floored_r(const DevParams& P, float r2, float& r, float& rinv) {
  const float r2c = fmaxf(r2, P.rmin * P.rmin);
  rinv = rsqrt_normal(r2c);
  r = __fmul_rn(r2c, rinv);
}

// max(h - r, 0) of two neighbours in fixed-point units, from r^2 floored at
// r_min^2 and its reciprocal root, one fused multiply-add each: r - h
// (rounded as h - r), then the sign turned with the floor.
__device__ __forceinline__ uint64_t h_minus_r(const DevParams& P, uint64_t r2c, uint64_t rinv) {
  const uint64_t m = f2_fma(r2c, rinv, f2_dup(-P.h_fx));
  return f2_pack(fmaxf(-f2_lo(m), 0.0f), fmaxf(-f2_hi(m), 0.0f));
}

// The same in fixed-point units (r2f = |d|^2 of the record difference):
// r2c = max(r2f, r_min^2) and rinv_f = 2^-k / r, so the loops need no
// rescaling of r^2; r_f = r 2^k is r2c rinv, and h_f - r_f, floored at
// 0, one fused multiply-add (fx_hm).
__device__ __forceinline__ void floored_r_fx(const DevParams& P, float r2f, float& r2c,
                                             float& rinv) {
  r2c = fmaxf(r2f, P.rmin2_fx);
  rinv = rsqrt_normal(r2c);
}
__device__ __forceinline__ float fx_hm(const DevParams& P, float r2c, float rinv) {
  return fmaxf(fmaf(-r2c, rinv, P.h_fx), 0.0f);
}

// 1/x by the hardware's approximate reciprocal (PTX rcp.approx.ftz.f32, at
// most 1 ulp from the rounded quotient): one instruction where the correctly
// rounded reciprocal takes a refinement sequence.  Used for the neighbour
// densities of the post passes (x near rho0, never subnormal).
__device__ __forceinline__ float rcp_fast(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// max and sum of the per-particle density error over the block (FP64).
__device__ __forceinline__ void block_resid(double e, double* resid) {
  double m = e, s = e;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    s += __shfl_xor_sync(0xffffffffu, s, o);
  }
  __shared__ double sm[kBlock / 32], ss[kBlock / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) {
    sm[warp] = m;
    ss[warp] = s;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double bm = 0.0, bs = 0.0;
    for (int w = 0; w < (int)blockDim.x / 32; ++w) {
      bm = fmax(bm, sm[w]);
      bs += ss[w];
    }
    atomicMax(reinterpret_cast<unsigned long long*>(resid),
              (unsigned long long)__double_as_longlong(bm));
    atomicAdd(resid + 1, bs);
  }
}

// Density (MODE 0, 1) and multiplier (MODE 0, 2, from rho) of particle p with
// record rp over its list.
template <int MODE, bool LIVE>
__device__ __forceinline__ void density_lambda_of(const DevParams& P, const NbrView& V, bool tiled,
                                                  const unsigned char* tile, const uint4* nr, int p,
                                                  const uint4 rp, int cnt, const uint4 blk,
                                                  float& rho, float& lam) {
  // The loop keeps only what varies per pair: the density sums t^3 with
  // t = h^2 - r^2 and the gradient sums c d with c = (h - r)^2 / r and d
  // the pair difference, both in fixed-point units; the kernel norms, the
  // mass and 2^-2k multiply the sums once afterwards.  The density sum is
  // Kahan-compensated per batch: a batch's four terms are added pairwise
  // (relative error at most 2 ulp of the batch sum, all terms >= 0) and the
  // batch sum enters the compensated running sum.  Padding slots past the
  // count are the pair (p, p): their density term is masked, their gradient
  // terms carry d = 0.
  float st = 0.0f, comp = 0.0f;
  float sgx = 0.f, sgy = 0.f, sgz = 0.f, sC = 0.f;
  visit<1, LIVE>(V, tiled, tile, nr, nullptr, p, cnt, blk,
                  [&](const Batch<1>& q, int nvalid) {
    float t[4], t2[4];
#pragma unroll
    for (int u = 0; u < 4; u += 2) {
      const Pair2 d = diff2(rp, q.r[u], q.r[u + 1]);
      const uint64_t r2f = norm2_2(d);
      if (MODE != 2) {
        uint64_t tt = max2(f2_fma(f2_dup(-P.fx_inv2), r2f, f2_dup(P.h2)), 0.0f);
        tt = f2_pack(u < nvalid ? f2_lo(tt) : 0.0f, u + 1 < nvalid ? f2_hi(tt) : 0.0f);
        t[u] = f2_lo(tt);
        t[u + 1] = f2_hi(tt);
        tt = f2_mul(tt, tt);
        t2[u] = f2_lo(tt);
        t2[u + 1] = f2_hi(tt);
      }
      if (MODE != 1) {
        // in fixed-point units: c_f = (h_f - r_f)^2 / r_f = 2^k c
        const uint64_t r2c = max2(r2f, P.rmin2_fx);
        const uint64_t rinv = rsqrt2(r2c);
        const uint64_t hm = h_minus_r(P, r2c, rinv);
        const uint64_t c = f2_mul(f2_mul(hm, hm), rinv);
        const uint64_t cc = f2_mul(c, c);
        // |c d|^2 = c^2 |d|^2: three fused accumulations and one for the norm
        sgx = fmaf(f2_lo(c), f2_lo(d.x), sgx);
        sgy = fmaf(f2_lo(c), f2_lo(d.y), sgy);
        sgz = fmaf(f2_lo(c), f2_lo(d.z), sgz);
        sC = fmaf(f2_lo(cc), f2_lo(r2f), sC);
        sgx = fmaf(f2_hi(c), f2_hi(d.x), sgx);
        sgy = fmaf(f2_hi(c), f2_hi(d.y), sgy);
        sgz = fmaf(f2_hi(c), f2_hi(d.z), sgz);
        sC = fmaf(f2_hi(cc), f2_hi(r2f), sC);
      }
    }
    if (MODE != 2) {
      // t0^3 + t1^3 + t2^3 + t3^3 as a chain of fused multiply-adds
      const float yb = fmaf(t2[0], t[0], fmaf(t2[1], t[1],
                            fmaf(t2[2], t[2], __fmul_rn(t2[3], t[3]))));
      const float y = yb - comp;
      const float s = st + y;
      comp = (s - st) - y;
      st = s;
    }
  });
  if (MODE != 2) rho = fmaf(P.Wn_m, st - comp, P.W0m);
  if (MODE != 1) {
    // ComputeLambda's constraint (particles.c:616-617) in FP64
    const float C = (float)fmax(__ddiv_rn((double)rho, P.rho0_d) - 1.0, 0.0);
    const float g = P.DWn_m * P.fx_inv2;  // gradient scale (2^-2k is exact)
    sC = __fadd_rn(sC, norm2(sgx, sgy, sgz));
    sC *= (g * g) * P.inv_rho0_sq;
    lam = -C / (sC + P.lambda_eps);
  }
}

template <int MODE, bool RESID>
__global__ void __launch_bounds__(kTileSlots, kMinBlocks1)
    k_density_lambda(const DevParams P, const NbrView V, const PassArgs a) {
  SPHPC_PASS_HEAD(1, a.nr, nullptr);
  double err = 0.0;
  const uint4 rp = own ? ld_nr(a.nr, p) : make_uint4(0u, 0u, 0u, 0u);
  SPHPC_PASS_READY();
  if (own) {
    float rho = 0.0f, lam = 0.0f;
    if (MODE == 2) rho = a.rho[p];
    density_lambda_of<MODE, false>(P, V, tiled, tile, a.nr, p, rp, cnt, blk, rho, lam);
    if (MODE != 2) a.rho[p] = rho;
    if (MODE != 1) {
      if (a.nr_out) a.nr_out[p] = make_uint4(rp.x, rp.y, rp.z, __float_as_uint(lam));
      if (a.lam) a.lam[p] = lam;
    }
    if (RESID) err = fmax((double)rho / (double)P.rho0 - 1.0, 0.0);
  }
  if (RESID) block_resid(err, a.resid);
}

// The first density/lambda pass of a step (mode 0, with residual) that also
// forms the 16 warm-start features of each particle p < limit:
//   0 rho/rho0 - 1       1 C = max(rho/rho0 - 1, 0)     2 lambda
//   3 sum_q |grad_q C|^2 4 |grad_p C|^2 (both with the 1/rho0^2 of lambda)
//   5 neighbour count    6-8 mean neighbour offset (x*_q - x*_p) / h
//   9-11 mean relative predicted displacement (d_q - d_p) / h, d = x* - x
//        (= the mean relative velocity * dt / h away from the box walls)
//   12 SDF distance at x* / h, clamped to [-4, 4] (4 without an obstacle)
//   13 nearest-neighbour distance / h (1 without neighbours)
//   14 distance to the nearest box wall / h, clamped to [0, 4]
//   15 own predicted displacement along the gravity axis / h
// RAW: FP32 features to feat[p][16]; otherwise the network's input row
// bf16((f - mean) * inv_std) (norm = mean[16], inv_std[16]) to xbf[p][16].
// It gathers the 32-byte particle records; in a block with a tile the slots of
// the tile's records are laid out in shared memory for that.
template <bool RAW>
__global__ void __launch_bounds__(kTileSlots, kMinBlocksFeatures)
    k_features(const DevParams P, const NbrView V, const PassArgs a, float* __restrict__ feat,
               __nv_bfloat16* __restrict__ xbf, const float* __restrict__ norm, int limit) {
  __shared__ int s_slot[kTileCapMost];
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  const TileInfo* info = V.tiles + blockIdx.x;
  const int total = __ldg(&info->total);
  if (total >= 0) {
    for (int r = 0; r < 9; ++r) {
      const int s = __ldg(&info->s[r]), o = __ldg(&info->o[r]),
                len = (r < 8 ? __ldg(&info->o[r + 1]) : total) - o;
      for (int t = threadIdx.x; t < len; t += kTileSlots) s_slot[o + t] = s + t;
    }
    __syncthreads();
  }
  double err = 0.0;
  if (p < P.n) {
    float4 xp, dp;
    ld_pd(a.pd, p, xp, dp);
    // Only what varies per pair stays in the loop: the sum of t^3
    // (t = h^2 - r^2), the sums of c d with c = (h - r)^2 / r and of c^2 r^2,
    // the neighbour offsets and displacements; the kernel norms and the mass
    // multiply the sums once afterwards, as in the density pass.  The t^3
    // sum is Kahan-compensated per batch of four neighbours, as there.
    float st = 0.0f, comp = 0.0f;
    float sgx = 0.f, sgy = 0.f, sgz = 0.f, sC = 0.f;
    float ox = 0.f, oy = 0.f, oz = 0.f, ux = 0.f, uy = 0.f, uz = 0.f, rmin2 = P.h2;
    const int cnt = (int)__ldg(V.ncount + p);
    uint4 blk = cnt > 0 ? nbr_block(V, p, 0) : make_uint4(0u, 0u, 0u, 0u);
    for (int j0 = 0; j0 < cnt; j0 += 4) {
      const int nvalid = cnt - j0;
      int q[4];
      if (total >= 0) {
        // the low half of a block, then the high half, eight entries in all
        const uint32_t w0 = (j0 & 4) ? blk.z : blk.x, w1 = (j0 & 4) ? blk.w : blk.y;
        const uint32_t o[4] = {w0 & 0xffffu, w0 >> 16, w1 & 0xffffu, w1 >> 16};
#pragma unroll
        for (int u = 0; u < 4; ++u) q[u] = s_slot[o[u] >> 4];
        if ((j0 & 4) && j0 + 4 < cnt) blk = nbr_block(V, p, (j0 >> 3) + 1);
      } else {
        q[0] = (int)blk.x;
        q[1] = (int)blk.y;
        q[2] = (int)blk.z;
        q[3] = (int)blk.w;
        if (j0 + 4 < cnt) blk = nbr_block(V, p, (j0 >> 2) + 1);
      }
      float4 xq[4], dq[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) ld_pd(a.pd, q[u], xq[u], dq[u]);
      float yb = 0.0f;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (u < nvalid) {
          const Pair g = pair_geom(xp, dp, xq[u], dq[u]);
          const float t = fmaxf(P.h2 - g.r2, 0.0f);
          yb = fmaf(__fmul_rn(t, t), t, yb);
          float r, rinv;
          floored_r(P, g.r2, r, rinv);
          const float hm = fmaxf(P.h - r, 0.0f);
          const float c = __fmul_rn(__fmul_rn(hm, hm), rinv);
          sgx = fmaf(c, g.dx, sgx);
          sgy = fmaf(c, g.dy, sgy);
          sgz = fmaf(c, g.dz, sgz);
          sC = fmaf(__fmul_rn(c, c), g.r2, sC);
          ox -= g.dx;
          oy -= g.dy;
          oz -= g.dz;
          ux += dq[u].x;
          uy += dq[u].y;
          uz += dq[u].z;
          rmin2 = fminf(rmin2, g.r2);
        }
      }
      const float y = yb - comp;
      const float s = st + y;
      comp = (s - st) - y;
      st = s;
    }
    // sum_q (d_q - d_p) from sum_q d_q
    ux = fmaf(-(float)cnt, dp.x, ux);
    uy = fmaf(-(float)cnt, dp.y, uy);
    uz = fmaf(-(float)cnt, dp.z, uz);
    sgx *= P.DWn_m;
    sgy *= P.DWn_m;
    sgz *= P.DWn_m;
    sC *= P.DWn_m * P.DWn_m;
    const float rho = fmaf(P.Wn_m, st - comp, P.W0m);
    a.rho[p] = rho;
    const float C = (float)fmax(__ddiv_rn((double)rho, P.rho0_d) - 1.0, 0.0);
    const float s_pairs = sC * P.inv_rho0_sq;
    sC = __fadd_rn(sC, norm2(sgx, sgy, sgz));
    sC *= P.inv_rho0_sq;
    const float lam = -C / (sC + P.lambda_eps);
    const double xs = xstar_d(xp.x, dp.x), ys = xstar_d(xp.y, dp.y), zs = xstar_d(xp.z, dp.z);
    a.nr_out[p] = make_nr(P, xs, ys, zs, lam);
    err = fmax((double)rho / (double)P.rho0 - 1.0, 0.0);
    if (p < limit) {
      const float inv_h = 1.0f / P.h;
      const float s_self = __fmul_rn(norm2(sgx, sgy, sgz), P.inv_rho0_sq);
      const float inv_cnt = cnt > 0 ? 1.0f / (float)cnt : 0.0f;
      const float sc = inv_h * inv_cnt;
      float sdf = 4.0f;
      if (P.has_sdf && xs > P.ob_min[0] && xs < P.ob_max[0] && ys > P.ob_min[1] &&
          ys < P.ob_max[1] && zs > P.ob_min[2] && zs < P.ob_max[2]) {
        const float xt = (float)((xs - P.ob_min[0]) / (double)P.ob_len[0]);
        const float yt = (float)((ys - P.ob_min[1]) / (double)P.ob_len[1]);
        const float zt = (float)((zs - P.ob_min[2]) / (double)P.ob_len[2]);
        sdf = fminf(fmaxf(sdf_sample(P, xt, yt, zt) * P.model_to_world * inv_h, -4.0f), 4.0f);
      }
      const double wall =
          fmin(fmin(xs - P.bmin[0], P.bmax[0] - xs),
               fmin(fmin(ys - P.bmin[1], P.bmax[1] - ys), fmin(zs - P.bmin[2], P.bmax[2] - zs)));
      const float fw = fminf(fmaxf((float)(wall / P.hd), 0.0f), 4.0f);
      const float vg = (P.gaxis == 0 ? dp.x : (P.gaxis == 1 ? dp.y : dp.z)) * inv_h;
      const float f[16] = {fmaf(rho, P.inv_rho0, -1.0f), C, lam, s_pairs, s_self, (float)cnt,
                           ox * sc, oy * sc, oz * sc, ux * sc, uy * sc, uz * sc,
                           sdf, sqrtf(rmin2) * inv_h, fw, vg};
      if (RAW) {
        float4* out = reinterpret_cast<float4*>(feat + (size_t)p * 16);
#pragma unroll
        for (int k = 0; k < 4; ++k)
          out[k] = make_float4(f[4 * k], f[4 * k + 1], f[4 * k + 2], f[4 * k + 3]);
      } else {
        uint32_t w[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const float lo = (f[2 * k] - __ldg(norm + 2 * k)) * __ldg(norm + 16 + 2 * k);
          const float hi = (f[2 * k + 1] - __ldg(norm + 2 * k + 1)) * __ldg(norm + 17 + 2 * k);
          const __nv_bfloat162 b2 = __floats2bfloat162_rn(lo, hi);
          w[k] = *reinterpret_cast<const uint32_t*>(&b2);
        }
        uint4* out = reinterpret_cast<uint4*>(xbf + (size_t)p * 16);
        out[0] = make_uint4(w[0], w[1], w[2], w[3]);
        out[1] = make_uint4(w[4], w[5], w[6], w[7]);
      }
    }
  }
  block_resid(err, a.resid);
}

// target[p] += s * lambda_p (lambda in d.w of the records) for p < limit:
// the stiffness-weighted multiplier sum of a plain solve, the warm-start
// network's training target.
__global__ void k_accum_lambda(const uint4* __restrict__ rec, float s, float* __restrict__ target,
                               int limit) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p < limit) target[p] = fmaf(s, __uint_as_float(rec[p].w), target[p]);
}

// Displacement of particle p with record rp (payload lambda) over its list
// (UpdateDPs), for the stiffness of the substep.
template <int SCORR_N, bool LIVE>
__device__ __forceinline__ float3 displacement_of(const DevParams& P, const NbrView& V, bool tiled,
                                                  const unsigned char* tile, const uint4* nr, int p,
                                                  const uint4 rp, int cnt, const uint4 blk,
                                                  float stiffness) {
  const float lp = nr_w(rp);
  // sums of c d with c = (lambda_p + lambda_q + s_corr) (h - r)^2 / r and d
  // the pair difference, both in fixed-point units; the spiky norm, the mass
  // and 2^-2k multiply them once afterwards.  Every term carries d, so the batch's
  // padding slots (q = p, d = 0) add nothing and are not masked.
  float ax = 0.f, ay = 0.f, az = 0.f;
  visit<1, LIVE>(V, tiled, tile, nr, nullptr, p, cnt, blk, [&](const Batch<1>& q, int) {
#pragma unroll
    for (int u = 0; u < 4; u += 2) {
      const Pair2 d = diff2(rp, q.r[u], q.r[u + 1]);
      // in fixed-point units: c_f = s (h_f - r_f)^2 / r_f = 2^k c
      const uint64_t r2c = max2(norm2_2(d), P.rmin2_fx);
      const uint64_t rinv = rsqrt2(r2c);
      const uint64_t hm = h_minus_r(P, r2c, rinv);
      uint64_t s = f2_pack(lp + nr_w(q.r[u]), lp + nr_w(q.r[u + 1]));
      if (SCORR_N != 0) {
        // W(r) / W(dq) = w^3 with w = (h^2 - r^2) / (h^2 - dq^2), w <= 1.05
        const uint64_t w =
            max2(f2_fma(f2_dup(-P.scorr_u_fx), r2c, f2_dup(P.scorr_uh2)), 0.0f);
        if (SCORR_N == 4) {
          const uint64_t w2 = f2_mul(w, w);
          const uint64_t w4 = f2_mul(w2, w2);
          s = f2_fma(f2_dup(-P.scorr_k), f2_mul(f2_mul(w4, w4), w4), s);
        } else {
          const uint64_t ratio = f2_mul(f2_mul(w, w), w);
          uint64_t sc = f2_dup(-P.scorr_k);
          for (int e = 0; e < P.scorr_n; ++e) sc = f2_mul(sc, ratio);
          s = f2_add(s, sc);
        }
      }
      const uint64_t c = f2_mul(f2_mul(f2_mul(s, hm), hm), rinv);
      ax = fmaf(f2_lo(c), f2_lo(d.x), ax);
      ay = fmaf(f2_lo(c), f2_lo(d.y), ay);
      az = fmaf(f2_lo(c), f2_lo(d.z), az);
      ax = fmaf(f2_hi(c), f2_hi(d.x), ax);
      ay = fmaf(f2_hi(c), f2_hi(d.y), ay);
      az = fmaf(f2_hi(c), f2_hi(d.z), az);
    }
  });
  const float s = stiffness * P.inv_rho0 * (P.DWn_m * P.fx_inv2);
  return make_float3(ax * s, ay * s, az * s);
}

// x* of the record {xp, d} moved by dp (UpdatePositionStars): the new d, with
// rho as its payload, and the exact x* - x.
template <bool SDF>
__device__ __forceinline__ float4 move_star(const DevParams& P, const float4 xp, const float4 d,
                                            const float3 dp, float rho, double& ex, double& ey,
                                            double& ez) {
  double xs = __dadd_rn(xstar_d(xp.x, d.x), (double)dp.x);
  double ys = __dadd_rn(xstar_d(xp.y, d.y), (double)dp.y);
  double zs = __dadd_rn(xstar_d(xp.z, d.z), (double)dp.z);
  xs = clamp_axis(xs, P.bmin[0], P.bmax[0], P.bmax_eps[0]);
  ys = clamp_axis(ys, P.bmin[1], P.bmax[1], P.bmax_eps[1]);
  zs = clamp_axis(zs, P.bmin[2], P.bmax[2], P.bmax_eps[2]);
  if (SDF) sdf_collide(P, xs, ys, zs);
  ex = __dsub_rn(xs, (double)xp.x);
  ey = __dsub_rn(ys, (double)xp.y);
  ez = __dsub_rn(zs, (double)xp.z);
  return make_float4(__double2float_rn(ex), __double2float_rn(ey), __double2float_rn(ez), rho);
}

// UpdateVelocities, particles.c:814-837
__device__ __forceinline__ float4 velocity_of(const DevParams& P, double ex, double ey, double ez) {
  float vx = __double2float_rn(__ddiv_rn(ex, P.dt_d));
  float vy = __double2float_rn(__ddiv_rn(ey, P.dt_d));
  float vz = __double2float_rn(__ddiv_rn(ez, P.dt_d));
  vx = fminf(fmaxf(vx, -P.v_max), P.v_max);
  vy = fminf(fmaxf(vy, -P.v_max), P.v_max);
  vz = fminf(fmaxf(vz, -P.v_max), P.v_max);
  return make_float4(vx, vy, vz, 0.0f);
}

// The record of the canonical x* = x + d.
__device__ __forceinline__ uint4 record_of(const DevParams& P, const float4 xp, const float4 d) {
  return make_nr(P, xstar_d(xp.x, d.x), xstar_d(xp.y, d.y), xstar_d(xp.z, d.z), d.w);
}

template <int MODE, int SCORR_N, bool SDF>
__global__ void __launch_bounds__(kTileSlots, kMinBlocks1)
    k_position(const DevParams P, const NbrView V, const PassArgs a) {
  SPHPC_PASS_HEAD(1, a.nr, nullptr);
  const uint4 rp = own ? ld_nr(a.nr, p) : make_uint4(0u, 0u, 0u, 0u);
  SPHPC_PASS_READY();
  if (!own) return;
  float4 xp, d;  // own particle record, loaded ahead of the neighbour loop
  if (MODE == 0) ld_pd(a.pd, p, xp, d);
  const float3 dp = displacement_of<SCORR_N, false>(P, V, tiled, tile, a.nr, p, rp, cnt, blk,
                                                    a.stiffness);
  if (MODE == 1) {
    a.dp[p] = make_float4(dp.x, dp.y, dp.z, 0.0f);
    return;
  }
  double ex, ey, ez;
  const float4 dn = move_star<SDF>(P, xp, d, dp, a.rho[p], ex, ey, ez);
  st_pd(a.pd_out, p, xp, dn);
  // the record carries the canonical x* of what was just stored
  a.nr_out[p] = record_of(P, xp, dn);
  if (a.lam_acc) a.lam_acc[p] = fmaf(a.stiffness, nr_w(rp), a.acc_add ? a.lam_acc[p] : 0.0f);
  if (a.last) a.vel_out[p] = velocity_of(P, ex, ey, ez);
}

// ---------------------------------------------------------------------------
// The whole solve of a small set in one launch: every iteration's density and
// position pass, with the blocks meeting between them.  A block keeps its slots:
// records, multipliers, densities and positions of its particles stay in
// registers, and a pass reads only its tile and its lists.
//
// Bound: latency.  A pass of a set that is resident at once is a chain of a
// launch, the tile's ranges, the copies, the lists and the sums; the meeting takes
// the place of the launch and the first loads.
// Step of 4096 particles (200 steps after the dam broke, four iterations) 123 ->
// 115 us, of 32,768 152 -> 138, of 68,921 178 -> 172; at the start of a scene 4096
// 140 -> 121 us a step.  Larger sets fill the device with one pass and have their
// own kernels (nine blocks an SM instead of four).
// A cooperative launch, so every block is resident; the wait is bounded all
// the same.  The records are written by other blocks while the kernel runs:
// ordinary loads and fences on both sides of the meeting, also between the
// ordinary stores and the bulk copies (fence.proxy.async).
// ---------------------------------------------------------------------------
__device__ __forceinline__ bool grid_meet(uint32_t* count, uint32_t target, bool wait) {
  __shared__ int s_met;
  asm volatile("fence.proxy.async;" ::: "memory");
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(count, 1u);
    bool met = false;
    for (int i = 0; wait && i < (1 << 20); ++i) {
      uint32_t c;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(c) : "l"(count) : "memory");
      if ((met = c >= target)) break;
    }
    __threadfence();
    s_met = met ? 1 : 0;
  }
  __syncthreads();
  asm volatile("fence.proxy.async;" ::: "memory");
  return s_met != 0;
}

template <int SCORR_N, bool SDF>
__global__ void __launch_bounds__(kTileSlots, 4)
    k_solve(const DevParams P, const NbrView V, const SolveArgs a) {
  extern __shared__ __align__(128) unsigned char tile[];
  __shared__ __align__(8) uint64_t s_mbar;
  __shared__ TileInfo s_info;
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  const bool own = p < P.n;
  const int cnt = own ? (int)__ldg(V.ncount + p) : 0;
  const uint4 blk = cnt > 0 ? nbr_block(V, p, 0) : make_uint4(0u, 0u, 0u, 0u);
  if (threadIdx.x < sizeof(TileInfo) / sizeof(int))
    reinterpret_cast<int*>(&s_info)[threadIdx.x] =
        __ldg(reinterpret_cast<const int*>(V.tiles + blockIdx.x) + threadIdx.x);
  if (threadIdx.x == 0) mbar_init1(&s_mbar);
  uint4 rp = make_uint4(0u, 0u, 0u, 0u);
  float4 xp = make_float4(0.f, 0.f, 0.f, 0.f), d = xp;
  if (own) {
    rp = a.nr[p];
    ld_pd(a.pd, p, xp, d);
  }
  __syncthreads();
  const bool tiled = s_info.total >= 0;
  uint32_t* const count = V.err + kGridBarrier;
  uint32_t target = 0, phase = 0;
  bool good = true;  // the same in every thread of the block
  // a pass's tile of `nr`; false: it did not arrive
  auto fetch = [&](const uint4* nr) {
    if (!tiled) return;
    if (threadIdx.x == 0) mbar_expect(&s_mbar, (uint32_t)s_info.total * 16u);
    __syncwarp();
    if (threadIdx.x < 9) {
      const int r = threadIdx.x, s = s_info.s[r], o = s_info.o[r],
                e = r < 8 ? s_info.o[r + 1] : s_info.total;
      if (e > o) bulk_load(tile + o * 16, nr + s, (uint32_t)(e - o) * 16u, &s_mbar);
    }
  };
  auto arrived = [&]() {
    if (!tiled) return true;
    if (mbar_wait(&s_mbar, phase)) return true;
    atomicOr(V.err, kErrTileWait);
    mbar_wait(&s_mbar, phase);
    return false;
  };
  auto meet = [&]() {
    target += gridDim.x;
    if (!grid_meet(count, target, good)) {
      if (good && threadIdx.x == 0) atomicOr(V.err, kErrGridWait);
      good = false;
    }
  };
  double ex = 0.0, ey = 0.0, ez = 0.0;
  float rho = 0.0f;
  for (int it = 0; it < a.iterations; ++it) {
    if (it > 0) meet();
    fetch(a.nr);
    bool here = arrived();
    phase ^= 1u;
    float lam = 0.0f;
    if (own) {
      density_lambda_of<0, true>(P, V, tiled, tile, a.nr, p, rp, here ? cnt : 0, blk, rho, lam);
      rp.w = __float_as_uint(lam);
      a.nr_lam[p] = rp;
    }
    meet();
    fetch(a.nr_lam);
    here = arrived();
    phase ^= 1u;
    if (own) {
      const float3 dp = displacement_of<SCORR_N, true>(P, V, tiled, tile, a.nr_lam, p, rp,
                                                       here ? cnt : 0, blk, a.stiffness[it]);
      d = move_star<SDF>(P, xp, d, dp, rho, ex, ey, ez);
      rp = record_of(P, xp, d);
      a.nr[p] = rp;
    }
  }
  if (!own) return;
  a.rho[p] = rho;
  st_pd(a.pd_out, p, xp, d);
  a.vel_out[p] = velocity_of(P, ex, ey, ez);
}

template <bool SDF>
__global__ void __launch_bounds__(kBlock) k_apply_dp(const DevParams P, const PassArgs a) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= P.n) return;
  float4 xp, dp;
  ld_rw(a.pd_out, p, xp, dp);
  const float4 dd = __ldg(a.dp + p);
  double xs = __dadd_rn(xstar_d(xp.x, dp.x), (double)dd.x);
  double ys = __dadd_rn(xstar_d(xp.y, dp.y), (double)dd.y);
  double zs = __dadd_rn(xstar_d(xp.z, dp.z), (double)dd.z);
  xs = clamp_axis(xs, P.bmin[0], P.bmax[0], P.bmax_eps[0]);
  ys = clamp_axis(ys, P.bmin[1], P.bmax[1], P.bmax_eps[1]);
  zs = clamp_axis(zs, P.bmin[2], P.bmax[2], P.bmax_eps[2]);
  if (SDF) sdf_collide(P, xs, ys, zs);
  const float4 d = make_float4(__double2float_rn(__dsub_rn(xs, (double)xp.x)),
                               __double2float_rn(__dsub_rn(ys, (double)xp.y)),
                               __double2float_rn(__dsub_rn(zs, (double)xp.z)), dp.w);
  a.pd_out[p].d = d;
  a.nr_out[p] = make_nr(P, xstar_d(xp.x, d.x), xstar_d(xp.y, d.y), xstar_d(xp.z, d.z), 0.0f);
}

__global__ void __launch_bounds__(kTileSlots, kMinBlocks1)
    k_color(const DevParams P, const NbrView V, const PassArgs a) {
  SPHPC_PASS_HEAD(1, a.nr, nullptr);
  const uint4 rp = own ? ld_nr(a.nr, p) : make_uint4(0u, 0u, 0u, 0u);
  SPHPC_PASS_READY();
  if (!own) return;
  // sums of (h^2 - r^2)^2 r / (r rho_q) d, d in fixed-point units; the
  // poly6-gradient norm, m, h and 2^-k multiply them once (every term carries
  // d, so the padding slots add nothing)
  float cx = 0.f, cy = 0.f, cz = 0.f;
  visit<1>(V, tiled, tile, a.nr, nullptr, p, cnt, blk, [&](const Batch<1>& q, int) {
#pragma unroll
    for (int u = 0; u < 4; u += 2) {
      const Pair2 d = diff2(rp, q.r[u], q.r[u + 1]);
      // r and 1/r in fixed-point units (their product is unit-free)
      const uint64_t r2c = max2(norm2_2(d), P.rmin2_fx);
      const uint64_t rinv = rsqrt2(r2c);
      const uint64_t t = max2(f2_fma(f2_dup(-P.fx_inv2), r2c, f2_dup(P.h2)), 0.0f);
      const uint64_t irho = f2_pack(rcp_fast(nr_w(q.r[u])), rcp_fast(nr_w(q.r[u + 1])));
      const uint64_t c =
          f2_mul(f2_mul(f2_mul(t, t), f2_mul(r2c, rinv)), f2_mul(rinv, irho));
      cx = fmaf(f2_lo(c), f2_lo(d.x), cx);
      cy = fmaf(f2_lo(c), f2_lo(d.y), cy);
      cz = fmaf(f2_lo(c), f2_lo(d.z), cz);
      cx = fmaf(f2_hi(c), f2_hi(d.x), cx);
      cy = fmaf(f2_hi(c), f2_hi(d.y), cy);
      cz = fmaf(f2_hi(c), f2_hi(d.z), cz);
    }
  });
  const float s = P.h * (P.DWPn * P.m * P.fx_inv);
  a.color[p] = make_float4(s * cx, s * cy, s * cz, 0.0f);
}

// Akinci cohesion spline (particles.c:54-65) without its norm: with
// y = ((h - r) r)^3, 2y - h^6/64 for r <= h/2, y up to h, 0 beyond (h6_64 =
// h^6/64); selects, no branches.
__device__ __forceinline__ float cohesion_unnormed(const DevParams& P, float r, float h6_64) {
  const float hr = (P.h - r) * r;
  const float y = hr * hr * hr;
  float c = r <= 0.5f * P.h ? fmaf(2.0f, y, -h6_64) : y;
  return r > P.h ? 0.0f : c;
}

__global__ void __launch_bounds__(kTileSlots, kMinBlocks2)
    k_tension(const DevParams P, const NbrView V, const PassArgs a) {
  SPHPC_PASS_HEAD(2, a.nr, a.color);
  const uint4 recp = own ? ld_nr(a.nr, p) : make_uint4(0u, 0u, 0u, 0u);
  const float4 cp = own ? __ldg(a.color + p) : make_float4(0.f, 0.f, 0.f, 0.f);
  SPHPC_PASS_READY();
  if (!own) return;
  const float rp = nr_w(recp);
  const float kcoh = -20.0f * P.gamma * P.m * P.m;
  const float kcur = -P.gamma * P.m;
  // colour of each neighbour fetched with its record; the self terms of the
  // padding slots vanish (d = 0, c_p - c_q = 0)
  // the spline's norm and 2^-k for d in fixed-point units (exact)
  const float kcoh_fx = kcoh * P.C_norm * P.fx_inv;
  const float h3 = P.h * P.h * P.h;
  const float h6_64 = h3 * h3 * (1.0f / 64.0f);
  const float two_rho0 = 2.0f * P.rho0;
  // kcur (c_p - c_q) = kcur c_p - kcur c_q
  const float kpx = kcur * cp.x, kpy = kcur * cp.y, kpz = kcur * cp.z;
  float fx = 0.f, fy = 0.f, fz = 0.f;
  visit<2>(V, tiled, tile, a.nr, a.color, p, cnt, blk, [&](const Batch<2>& q, int) {
#pragma unroll
   for (int u = 0; u < 4; ++u) {
    const uint4 rq = q.r[u];
    const float4 cq = q.e[u];
    const float dx = (float)(int)(recp.x - rq.x);
    const float dy = (float)(int)(recp.y - rq.y);
    const float dz = (float)(int)(recp.z - rq.z);
    const float r2 = __fmul_rn(norm2(dx, dy, dz), P.fx_inv2);
    float r, rinv;
    floored_r(P, r2, r, rinv);
    const float coh = kcoh_fx * cohesion_unnormed(P, r, h6_64) * rinv;
    const float K = two_rho0 * rcp_fast(rp + nr_w(rq));
    fx = fmaf(K, fmaf(coh, dx, fmaf(-kcur, cq.x, kpx)), fx);
    fy = fmaf(K, fmaf(coh, dy, fmaf(-kcur, cq.y, kpy)), fy);
    fz = fmaf(K, fmaf(coh, dz, fmaf(-kcur, cq.z, kpz)), fz);
   }
  });
  float4 v = a.vel[p];
  const float s = P.dt / rp;
  v.x = fmaf(s, fx, v.x);
  v.y = fmaf(s, fy, v.y);
  v.z = fmaf(s, fz, v.z);
  a.vel[p] = v;
}

__global__ void __launch_bounds__(kTileSlots, kMinBlocks2)
    k_xsph(const DevParams P, const NbrView V, const PassArgs a) {
  SPHPC_PASS_HEAD(2, a.nr, a.vel);
  const uint4 rp = own ? ld_nr(a.nr, p) : make_uint4(0u, 0u, 0u, 0u);
  const float4 vp = own ? __ldg(a.vel + p) : make_float4(0.f, 0.f, 0.f, 0.f);
  SPHPC_PASS_READY();
  if (!own) return;
  // sums of (v_q - v_p) t^3 / rho_q; the poly6 norm, m and c multiply them
  // once (the padding slots' v_q - v_p is 0)
  float sx = 0.f, sy = 0.f, sz = 0.f;
  visit<2>(V, tiled, tile, a.nr, a.vel, p, cnt, blk, [&](const Batch<2>& q, int) {
#pragma unroll
   for (int u = 0; u < 4; ++u) {
    const uint4 rq = q.r[u];
    const float4 vq = q.e[u];
    const Pair g = pair_nr(P, rp, rq);
    // particles.c:439 evaluates x^2 + y^2 * z^2 (kept unless xsph_exact)
    const float rr =
        P.xsph_exact ? g.r2
                     : fmaf(g.dx, g.dx, __fmul_rn(__fmul_rn(__fmul_rn(g.dy, g.dy), g.dz), g.dz));
    const float t = fmaxf(P.h2 - rr, 0.0f);
    const float w = __fmul_rn(__fmul_rn(__fmul_rn(t, t), t), rcp_fast(nr_w(rq)));
    sx = fmaf(vq.x - vp.x, w, sx);
    sy = fmaf(vq.y - vp.y, w, sy);
    sz = fmaf(vq.z - vp.z, w, sz);
   }
  });
  const float cw = P.c_xsph * P.Wn_m;
  const float4 vn = make_float4(fmaf(cw, sx, vp.x), fmaf(cw, sy, vp.y), fmaf(cw, sz, vp.z), 0.0f);
  a.vel_out[p] = vn;
  if (a.write_pos) {
    float4 xp, dp;
    ld_pd(a.pd, p, xp, dp);
    st_pd(a.pd_out, p,
          make_float4(__double2float_rn(xstar_d(xp.x, dp.x)),
                      __double2float_rn(xstar_d(xp.y, dp.y)),
                      __double2float_rn(xstar_d(xp.z, dp.z)), 0.0f),
          make_float4(0.f, 0.f, 0.f, nr_w(rp)));
  }
}

// With nr_out, also the records {X, |omega|} the confinement pass gathers
// (one 16-byte load per neighbour instead of a record and omega[q]).
__global__ void __launch_bounds__(kTileSlots, kMinBlocks2)
    k_vorticity(const DevParams P, const NbrView V, const PassArgs a) {
  SPHPC_PASS_HEAD(2, a.nr, a.vel);
  const uint4 rp = own ? ld_nr(a.nr, p) : make_uint4(0u, 0u, 0u, 0u);
  const float4 vp = own ? __ldg(a.vel + p) : make_float4(0.f, 0.f, 0.f, 0.f);
  SPHPC_PASS_READY();
  if (!own) return;
  // sums of (v_q - v_p) x c d with c = (h - r)^2 / r and d in fixed-point
  // units (r too); the spiky norm and 2^-2k multiply them once (the padding slots'
  // v_q - v_p and d are 0)
  float wx = 0.f, wy = 0.f, wz = 0.f;
  visit<2>(V, tiled, tile, a.nr, a.vel, p, cnt, blk, [&](const Batch<2>& q, int) {
#pragma unroll
   for (int u = 0; u < 4; ++u) {
    const uint4 rq = q.r[u];
    const float4 vq = q.e[u];
    const float dx = (float)(int)(rp.x - rq.x);
    const float dy = (float)(int)(rp.y - rq.y);
    const float dz = (float)(int)(rp.z - rq.z);
    float r2c, rinv;
    floored_r_fx(P, norm2(dx, dy, dz), r2c, rinv);
    const float hm = fx_hm(P, r2c, rinv);
    const float c = __fmul_rn(__fmul_rn(hm, hm), rinv);
    const float gx = __fmul_rn(c, dx), gy = __fmul_rn(c, dy), gz = __fmul_rn(c, dz);
    const float ux = vq.x - vp.x, uy = vq.y - vp.y, uz = vq.z - vp.z;
    wx = __fadd_rn(wx, fmaf(uy, gz, -__fmul_rn(uz, gy)));
    wy = __fadd_rn(wy, fmaf(uz, gx, -__fmul_rn(ux, gz)));
    wz = __fadd_rn(wz, fmaf(ux, gy, -__fmul_rn(uy, gx)));
   }
  });
  const float sw = P.DWn * P.fx_inv2;
  wx *= sw;
  wy *= sw;
  wz *= sw;
  const float wm = sqrtf(norm2(wx, wy, wz));
  a.omega[p] = make_float4(wx, wy, wz, wm);
  if (a.nr_out) a.nr_out[p] = make_uint4(rp.x, rp.y, rp.z, __float_as_uint(wm));
}

// a.nr carries |omega| as its payload (the vorticity pass's records).
__global__ void __launch_bounds__(kTileSlots, kMinBlocks1)
    k_confinement(const DevParams P, const NbrView V, const PassArgs a) {
  SPHPC_PASS_HEAD(1, a.nr, nullptr);
  const uint4 rp = own ? ld_nr(a.nr, p) : make_uint4(0u, 0u, 0u, 0u);
  SPHPC_PASS_READY();
  if (!own) return;
  // sums of |omega_q| (h - r)^2 / r d, d and r in fixed-point units; the
  // spiky norm and 2^-2k multiply them once (the padding slots' d is 0)
  float ex = 0.f, ey = 0.f, ez = 0.f;
  visit<1>(V, tiled, tile, a.nr, nullptr, p, cnt, blk, [&](const Batch<1>& q, int) {
#pragma unroll
    for (int u = 0; u < 4; u += 2) {
      const Pair2 d = diff2(rp, q.r[u], q.r[u + 1]);
      const uint64_t r2c = max2(norm2_2(d), P.rmin2_fx);
      const uint64_t rinv = rsqrt2(r2c);
      const uint64_t hm = h_minus_r(P, r2c, rinv);
      const uint64_t g = f2_mul(f2_mul(hm, hm), rinv);
      const float ca = __fmul_rn(f2_lo(g), nr_w(q.r[u])), cb = __fmul_rn(f2_hi(g), nr_w(q.r[u + 1]));
      ex = fmaf(ca, f2_lo(d.x), ex);
      ey = fmaf(ca, f2_lo(d.y), ey);
      ez = fmaf(ca, f2_lo(d.z), ez);
      ex = fmaf(cb, f2_hi(d.x), ex);
      ey = fmaf(cb, f2_hi(d.y), ey);
      ez = fmaf(cb, f2_hi(d.z), ez);
    }
  });
  const float se = P.DWn * P.fx_inv2;
  ex *= se;
  ey *= se;
  ez *= se;
  const float em = fmaxf(sqrtf(norm2(ex, ey, ez)), P.rmin);
  const float nx = ex / em, ny = ey / em, nz = ez / em;
  const float4 w = __ldg(a.omega + p);
  const float s = P.dt * P.vort_eps / P.m;
  float4 v = a.vel[p];
  v.x = fmaf(s, fmaf(ny, w.z, -__fmul_rn(nz, w.y)), v.x);
  v.y = fmaf(s, fmaf(nz, w.x, -__fmul_rn(nx, w.z)), v.y);
  v.z = fmaf(s, fmaf(nx, w.y, -__fmul_rn(ny, w.x)), v.z);
  a.vel[p] = v;
  if (a.write_pos) {
    float4 xp, dp;
    ld_pd(a.pd, p, xp, dp);
    st_pd(a.pd_out, p,
          make_float4(__double2float_rn(xstar_d(xp.x, dp.x)),
                      __double2float_rn(xstar_d(xp.y, dp.y)),
                      __double2float_rn(xstar_d(xp.z, dp.z)), 0.0f),
          make_float4(0.f, 0.f, 0.f, 0.0f));
  }
}

__global__ void __launch_bounds__(kBlock) k_gravity(const DevParams P, float4* vel) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= P.n) return;
  float4 v = vel[p];
  if (P.gaxis == 0) v.x = __fadd_rn(v.x, P.gdt_f);
  else if (P.gaxis == 1) v.y = __fadd_rn(v.y, P.gdt_f);
  else v.z = __fadd_rn(v.z, P.gdt_f);
  vel[p] = v;
}

__global__ void __launch_bounds__(kBlock)
    k_predict(const DevParams P, PD* pd, const float4* __restrict__ vel) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= P.n) return;
  const float4 x = pd[p].x, v = vel[p];
  double xs = __dadd_rn((double)x.x, __dmul_rn((double)v.x, P.dt_d));
  double ys = __dadd_rn((double)x.y, __dmul_rn((double)v.y, P.dt_d));
  double zs = __dadd_rn((double)x.z, __dmul_rn((double)v.z, P.dt_d));
  xs = clamp_axis(xs, P.bmin[0], P.bmax[0], P.bmax_eps[0]);
  ys = clamp_axis(ys, P.bmin[1], P.bmax[1], P.bmax_eps[1]);
  zs = clamp_axis(zs, P.bmin[2], P.bmax[2], P.bmax_eps[2]);
  const float w = pd[p].d.w;
  pd[p].d = make_float4(__double2float_rn(__dsub_rn(xs, (double)x.x)),
                        __double2float_rn(__dsub_rn(ys, (double)x.y)),
                        __double2float_rn(__dsub_rn(zs, (double)x.z)), w);
}

__global__ void __launch_bounds__(kBlock)
    k_update_velocities(const DevParams P, const PD* __restrict__ pd,
                        float4* __restrict__ vel, const float* __restrict__ w_src,
                        uint4* __restrict__ nr) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= P.n) return;
  if (nr) nr[p].w = __float_as_uint(w_src[p]);
  const float4 d = pd[p].d;
  float vx = __double2float_rn(__ddiv_rn((double)d.x, P.dt_d));
  float vy = __double2float_rn(__ddiv_rn((double)d.y, P.dt_d));
  float vz = __double2float_rn(__ddiv_rn((double)d.z, P.dt_d));
  vx = fminf(fmaxf(vx, -P.v_max), P.v_max);
  vy = fminf(fmaxf(vy, -P.v_max), P.v_max);
  vz = fminf(fmaxf(vz, -P.v_max), P.v_max);
  vel[p] = make_float4(vx, vy, vz, 0.0f);
}

__global__ void __launch_bounds__(kBlock)
    k_update_positions(const DevParams P, PD* pd) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= P.n) return;
  const float4 x = pd[p].x;
  const float4 d = pd[p].d;
  const float nx = __double2float_rn(xstar_d(x.x, d.x));
  const float ny = __double2float_rn(xstar_d(x.y, d.y));
  const float nz = __double2float_rn(xstar_d(x.z, d.z));
  pd[p].x = make_float4(nx, ny, nz, 0.0f);
  // keep x* unchanged: d' = x* - x_new (exactly representable residue)
  pd[p].d = make_float4(__double2float_rn(__dsub_rn(xstar_d(x.x, d.x), (double)nx)),
                        __double2float_rn(__dsub_rn(xstar_d(x.y, d.y), (double)ny)),
                        __double2float_rn(__dsub_rn(xstar_d(x.z, d.z), (double)nz)), d.w);
}

// 16-byte records from the particle records: canonical x* = x + d and the
// payload src[p * stride] (0 without src).
__global__ void __launch_bounds__(kBlock)
    k_make_nr(const DevParams P, const PD* __restrict__ pd, const float* __restrict__ src,
              int stride, uint4* __restrict__ nr) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= P.n) return;
  const float4 x = pd[p].x, d = pd[p].d;
  nr[p] = make_nr(P, xstar_d(x.x, d.x), xstar_d(x.y, d.y), xstar_d(x.z, d.z),
                  src ? src[(size_t)p * stride] : 0.0f);
}

__global__ void __launch_bounds__(kBlock)
    k_collisions_double(const DevParams P, double* x, double* y, double* z, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double a = x[i], b = y[i], c = z[i];
  if (sdf_collide(P, a, b, c)) {
    x[i] = a;
    y[i] = b;
    z[i] = c;
  }
}

}  // namespace

// Launch of a neighbour pass with the tiles of NARR arrays.
#define SPHPC_PASS(NARR, ...)                                                       \
  do {                                                                              \
    const size_t bytes = (size_t)NARR * V.cap * 16;                                 \
    allow_shared(__VA_ARGS__, bytes);                                               \
    __VA_ARGS__<<<grid_for(P.n, kTileSlots), kTileSlots, bytes, st>>>(P, V, a);     \
  } while (0)

void launch_density_lambda(const DevParams& P, const NbrView& V, const PassArgs& a, int mode,
                           bool residual, cudaStream_t st) {
  if (mode == 0) {
    if (residual) SPHPC_PASS(1, k_density_lambda<0, true>);
    else SPHPC_PASS(1, k_density_lambda<0, false>);
  } else if (mode == 1) {
    if (residual) SPHPC_PASS(1, k_density_lambda<1, true>);
    else SPHPC_PASS(1, k_density_lambda<1, false>);
  } else {
    SPHPC_PASS(1, k_density_lambda<2, false>);
  }
}

void launch_features(const DevParams& P, const NbrView& V, const PassArgs& a, float* feat,
                     int limit, cudaStream_t st) {
  k_features<true><<<grid_for(P.n, kTileSlots), kTileSlots, 0, st>>>(P, V, a, feat, nullptr, nullptr, limit);
}

void launch_features_bf16(const DevParams& P, const NbrView& V, const PassArgs& a,
                          __nv_bfloat16* xbf, const float* norm, cudaStream_t st) {
  k_features<false><<<grid_for(P.n, kTileSlots), kTileSlots, 0, st>>>(P, V, a, nullptr, xbf, norm, P.n);
}

void launch_accum_lambda(const uint4* rec, float s, float* target, int limit, cudaStream_t st) {
  if (limit > 0) k_accum_lambda<<<(limit + kBlock - 1) / kBlock, kBlock, 0, st>>>(rec, s, target, limit);
}

void launch_position(const DevParams& P, const NbrView& V, const PassArgs& a, int mode,
                     cudaStream_t st) {
  const int sn = P.scorr_k != 0.0f ? (P.scorr_n == 4 ? 4 : -1) : 0;
  const bool sdf = P.has_sdf != 0;
#define SPHPC_POS(M, N, S) \
  SPHPC_PASS(1, k_position<M, N, S>)
  if (mode == 0) {
    if (sn == 0) { if (sdf) SPHPC_POS(0, 0, true); else SPHPC_POS(0, 0, false); }
    else if (sn == 4) { if (sdf) SPHPC_POS(0, 4, true); else SPHPC_POS(0, 4, false); }
    else { if (sdf) SPHPC_POS(0, -1, true); else SPHPC_POS(0, -1, false); }
  } else {
    if (sn == 0) SPHPC_POS(1, 0, false);
    else if (sn == 4) SPHPC_POS(1, 4, false);
    else SPHPC_POS(1, -1, false);
  }
#undef SPHPC_POS
}

namespace {
using SolveKernel = void (*)(DevParams, NbrView, SolveArgs);
SolveKernel solve_kernel(const DevParams& P) {
  const int sn = P.scorr_k != 0.0f ? (P.scorr_n == 4 ? 4 : -1) : 0;
  if (P.has_sdf) return sn == 0 ? k_solve<0, true> : sn == 4 ? k_solve<4, true> : k_solve<-1, true>;
  return sn == 0 ? k_solve<0, false> : sn == 4 ? k_solve<4, false> : k_solve<-1, false>;
}
}  // namespace

bool solve_fits(const DevParams& P, const NbrView& V, int device, int sms) {
  const int per_sm = (grid_for(P.n, kTileSlots) + sms - 1) / sms;
  if (P.n <= 0 || per_sm > kSolveBlocksPerSm) return false;
  const size_t bytes = (size_t)V.cap * 16;
  int blocks = 0, coop = 0;
  allow_shared(solve_kernel(P), bytes);
  if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device) == cudaSuccess && coop &&
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, solve_kernel(P), kTileSlots, bytes) ==
          cudaSuccess)
    return per_sm <= blocks;
  cudaGetLastError();
  return false;
}

cudaError_t launch_solve(const DevParams& P, const NbrView& V, const SolveArgs& a,
                         cudaStream_t st) {
  DevParams p = P;
  NbrView v = V;
  SolveArgs s = a;
  void* args[] = {&p, &v, &s};
  return cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(solve_kernel(P)),
                                     dim3(grid_for(P.n, kTileSlots)), dim3(kTileSlots), args,
                                     (size_t)V.cap * 16, st);
}

void launch_apply_dp(const DevParams& P, const PassArgs& a, cudaStream_t st) {
  if (P.has_sdf) k_apply_dp<true><<<grid_for(P.n), kBlock, 0, st>>>(P, a);
  else k_apply_dp<false><<<grid_for(P.n), kBlock, 0, st>>>(P, a);
}

void launch_color(const DevParams& P, const NbrView& V, const PassArgs& a, cudaStream_t st) {
  SPHPC_PASS(1, k_color);
}
void launch_tension(const DevParams& P, const NbrView& V, const PassArgs& a, cudaStream_t st) {
  SPHPC_PASS(2, k_tension);
}
void launch_xsph(const DevParams& P, const NbrView& V, const PassArgs& a, cudaStream_t st) {
  SPHPC_PASS(2, k_xsph);
}
void launch_vorticity(const DevParams& P, const NbrView& V, const PassArgs& a, cudaStream_t st) {
  SPHPC_PASS(2, k_vorticity);
}
void launch_confinement(const DevParams& P, const NbrView& V, const PassArgs& a,
                        cudaStream_t st) {
  SPHPC_PASS(1, k_confinement);
}
void launch_gravity(const DevParams& P, float4* vel, cudaStream_t st) {
  k_gravity<<<grid_for(P.n), kBlock, 0, st>>>(P, vel);
}
void launch_predict(const DevParams& P, PD* pd, const float4* vel, cudaStream_t st) {
  k_predict<<<grid_for(P.n), kBlock, 0, st>>>(P, pd, vel);
}
void launch_update_velocities(const DevParams& P, const PD* pd, float4* vel, cudaStream_t st,
                              const float* w_src, uint4* nr) {
  k_update_velocities<<<grid_for(P.n), kBlock, 0, st>>>(P, pd, vel, w_src, nr);
}
void launch_update_positions(const DevParams& P, PD* pd, cudaStream_t st) {
  k_update_positions<<<grid_for(P.n), kBlock, 0, st>>>(P, pd);
}
void launch_make_nr(const DevParams& P, const PD* pd, const float* src, uint4* nr,
                    cudaStream_t st, int stride) {
  k_make_nr<<<grid_for(P.n), kBlock, 0, st>>>(P, pd, src, stride, nr);
}
void launch_collisions_double(const DevParams& P, double* x, double* y, double* z, int n,
                              cudaStream_t st) {
  k_collisions_double<<<grid_for(n), kBlock, 0, st>>>(P, x, y, z, n);
}

}  // namespace sphpc
