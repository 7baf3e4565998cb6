// surface.cu -- particle-to-level-set surface reconstruction on a dense
// grid, the operations of the reference's post-processing tool
// (PostProcessing/OpenVDB/src/ConstructSurface.cc:39-72): voxel size = r/2,
// spheres of radius r rasterised as phi = min_p (|x - p| - r), then "dilate"
// by r, smooth, "erode" by r (the tool's offset(-r), gaussian(),
// offset(+r)).  The reference does this with OpenVDB's sparse narrow-band
// grids on the CPU; here the grid is dense on the device:
//   * distances: per voxel the nearest particle, found over bins of particles;
//     values are fixed-point (2^-20 length units), clamped to +-band (band =
//     (halfWidth voxels + r), wide enough that the offsets by r stay inside it);
//   * dilate: phi - r; smooth: three passes of a 3-tap mean along x, y, z
//     (a box-filter approximation of a Gaussian); erode: phi + r.
#include <algorithm>
#include <climits>
#include <cmath>
#include <utility>
#include <cuda_runtime.h>

#include "host_internal.h"
#include "scratch.cuh"

namespace sphpc {
namespace {

constexpr float kFixScale = 1048576.0f;  // 2^20 units per length

// Cubic bins of particles over the grid and `pad` bins around it.
struct Bins {
  int n[3], pad;
  float edge, inv_edge;
  float slack;  // bins that FP32 rounding can move a particle by, at most
  int rings;    // bins more than this many away are out of reach
};

__device__ __forceinline__ bool bin_of(const Bins& b, float x, float y, float z, int& c) {
  const float fx = floorf(x * b.inv_edge) + b.pad, fy = floorf(y * b.inv_edge) + b.pad,
              fz = floorf(z * b.inv_edge) + b.pad;
  if (!(fx >= 0.f && fy >= 0.f && fz >= 0.f && fx < b.n[0] && fy < b.n[1] && fz < b.n[2]))
    return false;
  c = ((int)fz * b.n[1] + (int)fy) * b.n[0] + (int)fx;
  return true;
}

__device__ __forceinline__ float3 local_pos(const double* __restrict__ xyz, int p, double ox,
                                            double oy, double oz) {
  return make_float3((float)(xyz[3 * (size_t)p] - ox), (float)(xyz[3 * (size_t)p + 1] - oy),
                     (float)(xyz[3 * (size_t)p + 2] - oz));
}

__global__ void k_bin_count(const double* __restrict__ xyz, int np, double ox, double oy, double oz,
                            const Bins b, int* __restrict__ count, int2* __restrict__ place) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= np) return;
  const float3 x = local_pos(xyz, p, ox, oy, oz);
  int c = -1, rank = 0;
  if (bin_of(b, x.x, x.y, x.z, c)) rank = atomicAdd(count + c, 1);
  place[p] = make_int2(c, rank);
}

// A range of the binned particles for each bin, in no particular order.
__global__ void k_bin_ranges(const int* __restrict__ count, int bins, int* __restrict__ used,
                             int2* __restrict__ range) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31;
  const int n = c < bins ? count[c] : 0;
  int end = n;
#pragma unroll
  for (int k = 1; k < 32; k <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, end, k);
    if (lane >= k) end += y;
  }
  int base = 0;
  if (lane == 31 && end > 0) base = atomicAdd(used, end);
  base = __shfl_sync(0xffffffffu, base, 31) + end - n;
  if (c < bins) range[c] = make_int2(base, n);
}

__global__ void k_bin_place(const double* __restrict__ xyz, int np, double ox, double oy, double oz,
                            const int2* __restrict__ place, const int2* __restrict__ range,
                            float4* __restrict__ pos) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= np) return;
  const int2 at = place[p];
  if (at.x < 0) return;
  const float3 x = local_pos(xyz, p, ox, oy, oz);
  pos[range[at.x].x + at.y] = make_float4(x.x, x.y, x.z, 0.0f);
}

// phi - r of the particles on the grid: a warp takes 4 x 4 x 4 voxels, two a
// lane, the bins about them and one ring, and then the rings that can still hold a
// nearer particle for any of them.  Inside the fluid there are none: some 64
// particles a block, where a particle that writes its distance to every voxel
// within r + band visits 2197 voxels.  The nearest squared
// distance gives the bits of the least rounded distance, since the root, the
// clamp and the rounding are monotone.
// 97,336 particles, 1.1M voxels: 441 us by atomic minima from the particles,
// 94 us so with the bins' launches.
constexpr int kFewInBin = 16;
__global__ void __launch_bounds__(128)
    k_nearest(const int2* __restrict__ range, const float4* __restrict__ pos, const Bins b, int nx,
              int ny, int nz, int bx, int by, long long blocks, float voxel, float radius,
              float band, float* __restrict__ out) {
  __shared__ float4 s_pos[4][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long blk = (long long)blockIdx.x * 4 + warp;
  if (blk >= blocks) return;
  const int i0 = (int)(blk % bx) * 4, j0 = (int)(blk / bx % by) * 4,
            k0 = (int)(blk / bx / by) * 4;
  const int i = i0 + (lane & 3), j = j0 + (lane >> 2 & 3), k = k0 + (lane >> 4);
  const float x = i * voxel, y = j * voxel, za = k * voxel, zb = (k + 2) * voxel;
  const bool in = i < nx && j < ny, ina = in && k < nz, inb = in && k + 2 < nz;
  const float reach = radius + band, far2 = 1.001f * reach * reach;
  // squared distances; a voxel outside the grid needs none
  float ma = ina ? far2 : 0.0f, mb = inb ? far2 : 0.0f;
  // the block's corners and bins
  const float lo[3] = {i0 * voxel, j0 * voxel, k0 * voxel};
  const float hi[3] = {min(i0 + 3, nx - 1) * voxel, min(j0 + 3, ny - 1) * voxel,
                       min(k0 + 3, nz - 1) * voxel};
  int c0[3], c1[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    c0[d] = (int)floorf(lo[d] * b.inv_edge) + b.pad;
    c1[d] = (int)floorf(hi[d] * b.inv_edge) + b.pad;
  }
  auto nearer = [&](const float4 q) {
    const float dx = x - q.x, dy = y - q.y, da = za - q.z, db = zb - q.z;
    const float d2 = fmaf(dy, dy, dx * dx);
    ma = fminf(ma, fmaf(da, da, d2));
    mb = fminf(mb, fmaf(db, db, d2));
  };
  float worst = far2;
  for (int ring = 1, done = -1;;) {
    int a0[3], m[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      a0[d] = max(c0[d] - ring, 0);
      m[d] = min(c1[d] + ring, b.n[d] - 1) - a0[d] + 1;
    }
    const int cells = m[0] * m[1] * m[2];
    for (int t0 = 0; t0 < cells; t0 += 32) {
      const int t = t0 + lane;
      int2 rg = make_int2(0, 0);
      if (t < cells) {
        const int q = t / m[0], cx = a0[0] + t - q * m[0], r = q / m[1],
                  cy = a0[1] + q - r * m[1], cz = a0[2] + r;
        const int away = max(max(max(c0[0] - cx, cx - c1[0]), max(c0[1] - cy, cy - c1[1])),
                             max(c0[2] - cz, cz - c1[2]));
        if (away > done) {
          float d2 = 0.0f;
          const int cc[3] = {cx, cy, cz};
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            const float e0 = ((float)(cc[d] - b.pad) - b.slack) * b.edge,
                        e1 = ((float)(cc[d] - b.pad + 1) + b.slack) * b.edge;
            const float g = fmaxf(fmaxf(e0 - hi[d], lo[d] - e1), 0.0f);
            d2 = fmaf(g, g, d2);
          }
          if (d2 <= worst) rg = range[(cz * b.n[1] + cy) * b.n[0] + cx];
        }
      }
      // bins of few particles together, a particle of each at a time
      const bool few = rg.y <= kFewInBin;
      for (int u = 0;; ++u) {
        const unsigned on = __ballot_sync(0xffffffffu, few && u < rg.y);
        if (on == 0) break;
        if (few && u < rg.y) s_pos[warp][__popc(on & ((1u << lane) - 1u))] = pos[rg.x + u];
        __syncwarp();
        const int n = __popc(on);
        for (int v = 0; v < n; ++v) nearer(s_pos[warp][v]);
        __syncwarp();
      }
      // bins of many one after the other
      for (unsigned on = __ballot_sync(0xffffffffu, !few); on != 0; on &= on - 1) {
        const int src = __ffs((int)on) - 1;
        const int base = __shfl_sync(0xffffffffu, rg.x, src), n = __shfl_sync(0xffffffffu, rg.y, src);
        for (int v = 0; v < n; ++v) nearer(__ldg(pos + base + v));
      }
    }
    worst = fmaxf(ma, mb);
#pragma unroll
    for (int d = 16; d; d >>= 1) worst = fmaxf(worst, __shfl_xor_sync(0xffffffffu, worst, d));
    // rings that can still hold a nearer one
    const int more = min(b.rings, (int)floorf(sqrtf(worst) * 1.0001f * b.inv_edge + b.slack) + 1);
    if (more <= ring) break;
    done = ring;
    ring = more;
  }
  auto value = [&](float m2) {
    const float d = fminf(fmaxf(sqrtf(m2) - radius, -band), band);
    return (float)__float2int_rn(d * kFixScale) * (1.0f / kFixScale) - radius;
  };
  if (ina) out[((size_t)k * ny + j) * nx + i] = value(ma);
  if (inb) out[((size_t)(k + 2) * ny + j) * nx + i] = value(mb);
}

// One round of smoothing: 3-tap means along x, then y, then z, edges replicated,
// plus `shift`.  A block takes 32 x 8 x 8 voxels and their halo of one through
// shared memory, so a round reads and writes the grid once instead of three times.
// 1.1M voxels: nine passes of one axis 68 us, three rounds 36 us.
constexpr int kMx = 32, kMy = 8, kMz = 8;
__global__ void __launch_bounds__(256)
    k_smooth(const float* __restrict__ in, float* __restrict__ out, int nx, int ny, int nz, int bx,
             int by, float shift) {
  __shared__ float s_in[(kMz + 2) * (kMy + 2) * (kMx + 2)];
  __shared__ float s_x[(kMz + 2) * (kMy + 2) * kMx];
  float* s_y = s_in;  // [kMz + 2][kMy][kMx]
  const int i0 = (int)(blockIdx.x % bx) * kMx, j0 = (int)(blockIdx.x / bx % by) * kMy,
            k0 = (int)(blockIdx.x / bx / by) * kMz;
  auto mean = [](float a, float b, float c) { return (a + b + c) * (1.0f / 3.0f); };
  for (int t = threadIdx.x; t < (kMz + 2) * (kMy + 2) * (kMx + 2); t += 256) {
    const int i = i0 - 1 + t % (kMx + 2), j = j0 - 1 + t / (kMx + 2) % (kMy + 2),
              k = k0 - 1 + t / ((kMx + 2) * (kMy + 2));
    if ((unsigned)i < (unsigned)nx && (unsigned)j < (unsigned)ny && (unsigned)k < (unsigned)nz)
      s_in[t] = in[((size_t)k * ny + j) * nx + i];
  }
  __syncthreads();
  const int x = threadIdx.x % kMx, i = i0 + x;
  for (int r = threadIdx.x / kMx; r < (kMz + 2) * (kMy + 2); r += 256 / kMx) {
    const float* c = s_in + r * (kMx + 2) + x + 1;
    const float v = c[0];
    s_x[r * kMx + x] = mean(i > 0 ? c[-1] : v, v, i < nx - 1 ? c[1] : v);
  }
  __syncthreads();
  for (int r = threadIdx.x / kMx; r < (kMz + 2) * kMy; r += 256 / kMx) {
    const int y = r % kMy, z = r / kMy, j = j0 + y;
    const float* c = s_x + (z * (kMy + 2) + y + 1) * kMx + x;
    const float v = c[0];
    s_y[r * kMx + x] = mean(j > 0 ? c[-kMx] : v, v, j < ny - 1 ? c[kMx] : v);
  }
  __syncthreads();
  for (int r = threadIdx.x / kMx; r < kMz * kMy; r += 256 / kMx) {
    const int y = r % kMy, z = r / kMy, j = j0 + y, k = k0 + z;
    if (i >= nx || j >= ny || k >= nz) continue;
    const float* c = s_y + ((z + 1) * kMy + y) * kMx + x;
    const float v = c[0];
    out[((size_t)k * ny + j) * nx + i] =
        mean(k > 0 ? c[-kMy * kMx] : v, v, k < nz - 1 ? c[kMy * kMx] : v) + shift;
  }
}

}  // namespace
}  // namespace sphpc

using namespace sphpc;

// Level set of particles xyz[3 * np] (interleaved doubles, host memory, as
// WriteParticles writes them) on the dense grid dims at origin with voxel
// size radius / 2: phi[i + dims[0] * (j + dims[1] * k)] (host), negative
// inside.  half_width is the narrow band in voxels (the tool uses 2).
extern "C" int sphpc_particle_surface(const double* xyz, int np, double radius, int half_width,
                                      const int* dims, const double* origin, float* phi) {
  if (!xyz || np <= 0 || !(radius > 0.0) || half_width < 1 || !dims || !origin || !phi)
    return set_error(SPHPC_EINVAL, "sphpc_particle_surface: bad arguments");
  for (int d = 0; d < 3; ++d)
    if (dims[d] <= 0) return set_error(SPHPC_EINVAL, "sphpc_particle_surface: empty grid");
  const long long n = (long long)dims[0] * dims[1] * dims[2];
  const float voxel = (float)(radius / 2.0);
  const float r = (float)radius;
  const float band = half_width * voxel + r;
  if ((double)band * kFixScale > 2.0e9)
    return set_error(SPHPC_EINVAL, "sphpc_particle_surface: radius too large for the grid units");
  // Bins of two voxels (about a particle each), of more where the reach is long:
  // at most five rings.
  const float reach = r + band;
  Bins bins;
  bins.edge = 2.0f * voxel * fmaxf(1.0f, floorf(reach / (8.0f * voxel)));
  long long nbins;
  for (;; bins.edge *= 2.0f) {
    bins.inv_edge = 1.0f / bins.edge;
    bins.rings = (int)floorf(reach / bins.edge) + 1;
    bins.pad = bins.rings + 1;
    nbins = 1;
    for (int d = 0; d < 3; ++d) {
      bins.n[d] = (int)floorf((dims[d] - 1) * voxel * bins.inv_edge) + 2 + 2 * bins.pad;
      nbins *= bins.n[d];
    }
    // (of a long thin grid most bins are padding: wider ones)
    if (nbins <= std::min(std::max(n, 1ll << 22), 1ll << 30)) break;
  }
  const int longest = std::max(bins.n[0], std::max(bins.n[1], bins.n[2]));
  bins.slack = std::max(1.0e-3f, (float)longest * 0x1p-21f);
  auto tiles = [&](int d, int m) { return (dims[d] + m - 1) / m; };
  const long long blocks = (long long)tiles(0, 4) * tiles(1, 4) * tiles(2, 4);
  const long long smooth = (long long)tiles(0, kMx) * tiles(1, kMy) * tiles(2, kMz);
  if (blocks / 4 >= INT_MAX || smooth > INT_MAX)
    return set_error(SPHPC_EINVAL, "sphpc_particle_surface: grid too large");
  // the bins' places and the binned positions lie where the distances and their
  // smoothed copy follow
  ScratchLayout lay;
  const size_t grid_bytes = sizeof(float) * (size_t)n;
  const size_t o_xyz = lay.part(sizeof(double) * 3 * (size_t)np),
               o_count = lay.part(sizeof(int) * (size_t)(nbins + 1)),
               o_range = lay.part(sizeof(int2) * (size_t)nbins),
               o_a = lay.part(std::max(grid_bytes, sizeof(int2) * (size_t)np)),
               o_b = lay.part(std::max(grid_bytes, sizeof(float4) * (size_t)np));
  CallScratch mem;
  cudaError_t e = mem.take(lay.bytes(), 0);
  double* d_xyz = mem.at<double>(o_xyz);
  int2 *d_place = mem.at<int2>(o_a), *d_range = mem.at<int2>(o_range);
  float4* d_pos = mem.at<float4>(o_b);
  int* d_count = mem.at<int>(o_count);
  float *d_a = mem.at<float>(o_a), *d_b = mem.at<float>(o_b);
  if (e == cudaSuccess)
    e = cudaMemcpy(d_xyz, xyz, sizeof(double) * 3 * (size_t)np, cudaMemcpyHostToDevice);
  if (e == cudaSuccess)
    e = cudaMemsetAsync(d_count, 0, sizeof(int) * (size_t)(nbins + 1), 0);
  if (e == cudaSuccess) {
    const double ox = origin[0], oy = origin[1], oz = origin[2];
    const int gp = (int)(((long long)np + 255) / 256), gb = (int)((nbins + 255) / 256);
    k_bin_count<<<gp, 256>>>(d_xyz, np, ox, oy, oz, bins, d_count, d_place);
    k_bin_ranges<<<gb, 256>>>(d_count, (int)nbins, d_count + nbins, d_range);
    k_bin_place<<<gp, 256>>>(d_xyz, np, ox, oy, oz, d_place, d_range, d_pos);
    // distances, dilated by r; smoothed; eroded by r (ConstructSurface.cc:54-63)
    k_nearest<<<(int)((blocks + 3) / 4), 128>>>(d_range, d_pos, bins, dims[0], dims[1], dims[2],
                                                tiles(0, 4), tiles(1, 4), blocks, voxel, r, band,
                                                d_a);
    for (int it = 0; it < 3; ++it) {
      k_smooth<<<(int)smooth, 256>>>(d_a, d_b, dims[0], dims[1], dims[2], tiles(0, kMx),
                                     tiles(1, kMy), it == 2 ? r : 0.0f);
      std::swap(d_a, d_b);
    }
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(phi, d_a, sizeof(float) * (size_t)n, cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return set_error(SPHPC_ECUDA, "sphpc_particle_surface: %s", cudaGetErrorString(e));
  }
  return SPHPC_OK;
}
