// meshsdf.cu -- signed distance field of a closed triangle mesh on the
// device, in the sample layout of the SDFGen files the reference's obstacle
// loader reads (obstacle.c:13-79): samples at origin + (i, j, k) * dx, i
// fastest, negative inside.  The reference runtime names such a file
// (Runtime/sim-config.ini: bunny_watertight.sdf) but ships only the mesh.
//
// |phi| is the exact distance to the nearest triangle (closest point on a
// triangle by Voronoi regions: Ericson, "Real-Time Collision Detection",
// 2005, section 5.1.5).  The sign comes from the generalized winding number
// (Jacobson, Kavan, Sorkine-Hornung, SIGGRAPH 2013): the sum of the
// triangles' solid angles (Van Oosterom and Strackee, IEEE TBME 1983) is
// 4 pi inside a closed mesh and 0 outside, and a sample is inside when it
// exceeds 2 pi.
//
// Neither is computed over all pairs of samples and triangles:
//   * distances: the triangles, in Morton order of their centres, form clusters
//     of 8 with a bounding box each; a warp takes a box of 4 x 4 x 2 samples and
//     visits only the clusters that can hold the nearest triangle of one of them;
//   * signs of a closed mesh: its winding number is a whole number that changes
//     only where a row of samples crosses a triangle, so the crossings of each
//     triangle with the rows it spans are added up along the rows;
//   * signs of any other mesh (a boundary edge left, so the winding number is a
//     fraction): the sum of all solid angles per sample.
// 4,224 triangles, 104,544 samples: 3511 us for all pairs, 173 us for the
// distances and about 15 for the signs so; 72,000 triangles: 1.4 ms.
#include <cmath>
#include <cuda_runtime.h>

#include "host_internal.h"
#include "radix_sort.cuh"
#include "scratch.cuh"

namespace sphpc {
namespace {

constexpr int kSdfBlock = 256;
constexpr int kTriTile = 256;
constexpr int kCluster = 8;  // triangles per cluster

__device__ __forceinline__ float3 sub3(float3 a, float3 b) { return make_float3(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ float dot3(float3 a, float3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ float3 cross3(float3 a, float3 b) {
  return make_float3(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}

// Squared distance from p to triangle abc (Ericson 5.1.5).  The closest point is
// a + v (b - a) + w (c - a); the regions (corner, edge or face nearest) choose
// numerators and one denominator of v and w by selects, from the last region to
// the first, so the lanes of a warp stay together.
__device__ __forceinline__ float tri_dist2(float3 p, float3 a, float3 b, float3 c) {
  const float3 ab = sub3(b, a), ac = sub3(c, a), ap = sub3(p, a), bp = sub3(p, b), cp = sub3(p, c);
  const float d1 = dot3(ab, ap), d2 = dot3(ac, ap);
  const float d3 = dot3(ab, bp), d4 = dot3(ac, bp);
  const float d5 = dot3(ab, cp), d6 = dot3(ac, cp);
  const float vc = d1 * d4 - d3 * d2, vb = d5 * d2 - d1 * d6, va = d3 * d6 - d5 * d4;
  const float e = d4 - d3, f = d5 - d6;
  float nv = vb, nw = vc, den = va + vb + vc;  // face
  if (va <= 0.f && e >= 0.f && f >= 0.f) { nv = f; nw = e; den = e + f; }                // bc
  if (vb <= 0.f && d2 >= 0.f && d6 <= 0.f) { nv = 0.f; nw = d2; den = d2 - d6; }         // ac
  if (d6 >= 0.f && d5 <= d6) { nv = 0.f; nw = 1.f; den = 1.f; }                          // c
  if (vc <= 0.f && d1 >= 0.f && d3 <= 0.f) { nv = d1; nw = 0.f; den = d1 - d3; }         // ab
  if (d3 >= 0.f && d4 <= d3) { nv = 1.f; nw = 0.f; den = 1.f; }                          // b
  if (d1 <= 0.f && d2 <= 0.f) { nv = 0.f; nw = 0.f; den = 1.f; }                         // a
  const float s = 1.f / den, v = nv * s, w = nw * s;
  const float3 d = make_float3(ap.x - (ab.x * v + ac.x * w), ap.y - (ab.y * v + ac.y * w),
                               ap.z - (ab.z * v + ac.z * w));
  return dot3(d, d);
}

// Signed solid angle of triangle abc seen from the origin (a, b, c relative
// to the sample), Van Oosterom and Strackee.
__device__ __forceinline__ float solid_angle(float3 a, float3 b, float3 c) {
  const float la = sqrtf(dot3(a, a)), lb = sqrtf(dot3(b, b)), lc = sqrtf(dot3(c, c));
  const float num = dot3(a, cross3(b, c));
  const float den = la * lb * lc + dot3(a, b) * lc + dot3(a, c) * lb + dot3(b, c) * la;
  return 2.0f * atan2f(num, den);
}

struct SdfGrid {
  int ni, nj, nk;
  double ox, oy, oz, dx;
};
__device__ __forceinline__ float3 sample_pos(const SdfGrid& g, int i, int j, int k) {
  return make_float3((float)(g.ox + i * g.dx), (float)(g.oy + j * g.dx), (float)(g.oz + k * g.dx));
}

__device__ __forceinline__ uint64_t mix64(uint64_t z) {
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
__device__ __forceinline__ uint64_t point_hash(float3 p, uint64_t seed) {
  // + 0.0f: -0 and 0 are one point
  const uint64_t a = __float_as_uint(p.x + 0.0f), b = __float_as_uint(p.y + 0.0f),
                 c = __float_as_uint(p.z + 0.0f);
  return mix64(seed + mix64(a + (b << 32)) * 3 + mix64(c + 0x9E3779B97F4A7C15ull));
}
__device__ __forceinline__ uint32_t spread10(uint32_t v) {  // bit k of v to bit 3k
  v = (v | (v << 16)) & 0x030000FFu;
  v = (v | (v << 8)) & 0x0300F00Fu;
  v = (v | (v << 4)) & 0x030C30C3u;
  return (v | (v << 2)) & 0x09249249u;
}

// Corners of each triangle, its Morton key (30 bits of the centre in the
// mesh's box lo + [0, 1024) / scale), and the mesh's boundary: `open` receives
// two independent sums, over all triangles' edges u -> v, of +-h(u, v) with the
// sign of the direction in which the edge is walked (h a 64-bit hash of the two
// end points' coordinates).  An edge that its triangles walk as often one way as
// the other cancels, so the sums vanish for a closed mesh, and for no other but
// by an accident of 2^-128.  (open[2] is the host's: a vertex is not finite.)
__global__ void __launch_bounds__(kSdfBlock)
    k_triangles(const float3* __restrict__ verts, const int* __restrict__ tris, int nt, float3 lo,
                float3 scale, float3* __restrict__ corners, uint32_t* __restrict__ keys,
                unsigned long long* __restrict__ open) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  uint64_t sum[2] = {0, 0};
  if (t < nt) {
    float3 v[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      v[k] = verts[tris[3 * (size_t)t + k]];
      corners[3 * (size_t)t + k] = v[k];
    }
    auto cell = [](float x, float l, float s) {
      return (uint32_t)fminf(fmaxf((x - l) * s, 0.0f), 1023.0f);
    };
    const float third = 1.0f / 3.0f;
    keys[t] = spread10(cell((v[0].x + v[1].x + v[2].x) * third, lo.x, scale.x)) |
              (spread10(cell((v[0].y + v[1].y + v[2].y) * third, lo.y, scale.y)) << 1) |
              (spread10(cell((v[0].z + v[1].z + v[2].z) * third, lo.z, scale.z)) << 2);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      uint64_t h[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) h[k] = point_hash(v[k], 0x632BE59BD9B4E019ull * (q + 1));
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const uint64_t a = h[k], b = h[(k + 1) % 3];
        const uint64_t e = mix64(min(a, b) * 3 + mix64(max(a, b)));
        sum[q] += a < b ? e : a > b ? (uint64_t)0 - e : (uint64_t)0;
      }
    }
  }
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    for (int o = 16; o > 0; o >>= 1) sum[q] += __shfl_xor_sync(0xffffffffu, sum[q], o);
    if ((threadIdx.x & 31) == 0 && sum[q]) atomicAdd(open + q, (unsigned long long)sum[q]);
  }
}

// Clusters of kCluster triangles in the sorted order: the corners, 9 floats in
// three float4 per triangle (the last cluster is filled up with its last
// triangle), the box of the cluster and one of its corners.
__global__ void __launch_bounds__(kSdfBlock)
    k_clusters(const float3* __restrict__ corners, const uint32_t* __restrict__ order, int nt,
               int nc, float4* __restrict__ tri, float4* __restrict__ box,
               float4* __restrict__ rep) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nc * kCluster) return;  // whole clusters: eight lanes stay or leave together
  const size_t src = 3 * (size_t)order[min(t, nt - 1)];
  const float3 a = corners[src], b = corners[src + 1], c = corners[src + 2];
  tri[3 * (size_t)t] = make_float4(a.x, a.y, a.z, b.x);
  tri[3 * (size_t)t + 1] = make_float4(b.y, b.z, c.x, c.y);
  tri[3 * (size_t)t + 2] = make_float4(c.z, 0.f, 0.f, 0.f);
  float lo[3] = {fminf(a.x, fminf(b.x, c.x)), fminf(a.y, fminf(b.y, c.y)), fminf(a.z, fminf(b.z, c.z))};
  float hi[3] = {fmaxf(a.x, fmaxf(b.x, c.x)), fmaxf(a.y, fmaxf(b.y, c.y)), fmaxf(a.z, fmaxf(b.z, c.z))};
  const unsigned mask = 0xffu << (threadIdx.x & 24);
#pragma unroll
  for (int o = kCluster / 2; o > 0; o >>= 1)
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      lo[k] = fminf(lo[k], __shfl_xor_sync(mask, lo[k], o));
      hi[k] = fmaxf(hi[k], __shfl_xor_sync(mask, hi[k], o));
    }
  if (t % kCluster == 0) {
    box[2 * (t / kCluster)] = make_float4(lo[0], lo[1], lo[2], 0.f);
    box[2 * (t / kCluster) + 1] = make_float4(hi[0], hi[1], hi[2], 0.f);
    rep[t / kCluster] = make_float4(a.x, a.y, a.z, 0.f);
  }
}

// Squared distance between the boxes [alo, ahi] and [blo, bhi].
__device__ __forceinline__ float box_dist2(float3 alo, float3 ahi, float4 blo, float4 bhi) {
  const float x = fmaxf(fmaxf(blo.x - ahi.x, alo.x - bhi.x), 0.0f);
  const float y = fmaxf(fmaxf(blo.y - ahi.y, alo.y - bhi.y), 0.0f);
  const float z = fmaxf(fmaxf(blo.z - ahi.z, alo.z - bhi.z), 0.0f);
  return x * x + y * y + z * z;
}

// |phi|: a block per box of 4 x 4 x 2 samples, one per lane in each of its
// warps, which share the clusters (a sample at the middle of a hollow has many
// near-nearest ones, and one warp alone would hold up the launch).  Pass 1: the
// cluster whose corner is the nearest to each sample; those clusters (a few per
// box) are visited first and leave bounds near the distances themselves.  Pass 2,
// 32 clusters a round: the clusters whose box is near enough to the box of
// samples, then to some sample, are visited, each against the lanes' best so
// far.  The bounds carry a relative margin of 2^-18, more than their FP32
// rounding (about 2^-21), so a triangle that is left out is not the nearest by
// more than the rounding of its distance.
// Bounds: issue, in pass 1 and in tri_dist2 of the clusters visited.  Measured
// on the way (us, 4,224 triangles): one warp per box with clusters of 16 and a
// bound from the nearest cluster's farthest point 297, clusters of 8 236, four
// warps and pass 1 as above 173.  tri_dist2 without branches is no faster there
// but halves small meshes (192 triangles: 50 -> 31), and its error against 64
// bits is smaller (7.4e-8 of the field's norm against 1.0e-7).
constexpr int kDistWarps = 4;
__global__ void __launch_bounds__(kDistWarps * 32)
    k_mesh_dist(const float4* __restrict__ tri, const float4* __restrict__ box,
                const float4* __restrict__ rep, int nc, SdfGrid g, float* __restrict__ phi) {
  constexpr unsigned kAll = 0xffffffffu;
  constexpr float kMargin = 1.0f + 0x1p-18f;
  __shared__ float s_d[kDistWarps][32];
  __shared__ int s_c[kDistWarps][32];
  __shared__ float4 s_tri[kDistWarps][3 * kCluster];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int bi = (g.ni + 3) / 4, bj = (g.nj + 3) / 4;
  const long long w = blockIdx.x;
  const int i = (int)(w % bi) * 4 + (lane & 3), j = (int)(w / bi % bj) * 4 + (lane >> 2 & 3),
            k = (int)(w / ((long long)bi * bj)) * 2 + (lane >> 4);
  const bool live = i < g.ni && j < g.nj && k < g.nk;
  const float3 p = sample_pos(g, min(i, g.ni - 1), min(j, g.nj - 1), min(k, g.nk - 1));
  float3 lo = p, hi = p;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lo.x = fminf(lo.x, __shfl_xor_sync(kAll, lo.x, o));
    lo.y = fminf(lo.y, __shfl_xor_sync(kAll, lo.y, o));
    lo.z = fminf(lo.z, __shfl_xor_sync(kAll, lo.z, o));
    hi.x = fmaxf(hi.x, __shfl_xor_sync(kAll, hi.x, o));
    hi.y = fmaxf(hi.y, __shfl_xor_sync(kAll, hi.y, o));
    hi.z = fmaxf(hi.z, __shfl_xor_sync(kAll, hi.z, o));
  }
  float bound = 3.0e38f;  // of the lane's sample
  int nearest = 0;
#pragma unroll 8
  for (int c = warp; c < nc; c += kDistWarps) {
    const float4 r = __ldg(rep + c);
    const float x = p.x - r.x, y = p.y - r.y, z = p.z - r.z;
    const float d = x * x + y * y + z * z;
    if (d < bound) {
      bound = d;
      nearest = c;
    }
  }
  s_d[warp][lane] = bound;
  s_c[warp][lane] = nearest;
  __syncthreads();
#pragma unroll
  for (int q = 0; q < kDistWarps; ++q)
    if (s_d[q][lane] < bound) {
      bound = s_d[q][lane];
      nearest = s_c[q][lane];
    }
  float best = 3.0e38f;
  // a cluster's triangles, fetched by the lanes together (one load's latency)
  static_assert(3 * kCluster <= 32, "one float4 of the cluster per lane");
  auto visit = [&](int c) {
    __syncwarp();
    if (lane < 3 * kCluster) s_tri[warp][lane] = __ldg(tri + (size_t)c * (3 * kCluster) + lane);
    __syncwarp();
    const float4* t = s_tri[warp];
#pragma unroll 2
    for (int n = 0; n < kCluster; ++n, t += 3) {
      const float4 u = t[0], v = t[1];
      const float cz = t[2].x;
      best = fminf(best, tri_dist2(p, make_float3(u.x, u.y, u.z), make_float3(u.w, v.x, v.y),
                                   make_float3(v.z, v.w, cz)));
    }
  };
  int turn = 0;
  for (unsigned left = kAll; left; ++turn) {
    const int c = __shfl_sync(kAll, nearest, __ffs(left) - 1);
    if (turn % kDistWarps == warp) visit(c);
    left &= ~__ballot_sync(kAll, nearest == c);
  }
  // the warps hold the same samples, so the minimum over them is each lane's
  auto share = [&]() {
    __syncthreads();
    s_d[warp][lane] = best;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kDistWarps; ++q) best = fminf(best, s_d[q][lane]);
  };
  share();
  bound = fminf(bound, best) * kMargin;
  for (int c0 = warp * 32; c0 < nc; c0 += 32 * kDistWarps) {
    float worst = bound;  // of the box
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) worst = fmaxf(worst, __shfl_xor_sync(kAll, worst, o));
    const int c = c0 + lane;
    bool near = false;
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
    if (c < nc) {
      a = __ldg(box + 2 * (size_t)c);
      b = __ldg(box + 2 * (size_t)c + 1);
      near = box_dist2(lo, hi, a, b) <= worst;
    }
    for (unsigned m = __ballot_sync(kAll, near); m; m &= m - 1) {
      const int q = __ffs(m) - 1;
      const float4 qa = make_float4(__shfl_sync(kAll, a.x, q), __shfl_sync(kAll, a.y, q),
                                    __shfl_sync(kAll, a.z, q), 0.f),
                   qb = make_float4(__shfl_sync(kAll, b.x, q), __shfl_sync(kAll, b.y, q),
                                    __shfl_sync(kAll, b.z, q), 0.f);
      if (__any_sync(kAll, box_dist2(p, p, qa, qb) <= bound)) {
        visit(c0 + q);
        bound = fminf(bound, best * kMargin);
      }
    }
  }
  share();
  if (live && warp == 0) phi[((long long)k * g.nj + j) * g.ni + i] = sqrtf(best);
}

// The part of edge a -> b in the winding number, in the (y, z) plane, of a triangle
// about the row (y, z): +-1 where the ray from the row towards +y crosses the
// edge, by the direction in which the triangle walks it.  The edge holds its lower
// end and not its upper one, so a row through a corner crosses one of the edges
// that pass it; the side is computed from the lower end whichever way the edge is
// walked, by spelled-out operations.  So the two triangles of an edge always add
// opposite parts, whatever rounds, and the crossings of a closed mesh with a row
// add up to zero.
__device__ __forceinline__ int edge_part(const float3& a, const float3& b, double y, double z) {
  const bool below_a = a.z <= z, below_b = b.z <= z;
  if (below_a == below_b) return 0;
  const float3 u = below_a ? a : b, v = below_a ? b : a;
  const double ey = __dsub_rn(v.y, u.y), ez = __dsub_rn(v.z, u.z);
  const double side = __dsub_rn(__dmul_rn(ey, __dsub_rn(z, u.z)), __dmul_rn(ez, __dsub_rn(y, u.y)));
  return side > 0.0 ? (below_a ? 1 : -1) : 0;
}

// Crossings of a closed mesh with the rows of samples along x: each triangle
// walks the rows that its (y, z) box spans; a crossing before sample i of row
// (j, k) adds its orientation to step[(k nj + j) ni + i] (a row's running sum
// is then the winding number behind the crossings passed).  One warp per
// triangle.
__global__ void __launch_bounds__(kSdfBlock)
    k_crossings(const float3* __restrict__ corners, int nt, SdfGrid g,
                const unsigned long long* __restrict__ open, int* __restrict__ step) {
  if (open[0] | open[1] | open[2]) return;
  const int lane = threadIdx.x & 31;
  const int t = blockIdx.x * (kSdfBlock / 32) + (threadIdx.x >> 5);
  if (t >= nt) return;
  const float3 a = corners[3 * (size_t)t], b = corners[3 * (size_t)t + 1],
               c = corners[3 * (size_t)t + 2];
  const double xlo = fmin(fmin((double)a.x, b.x), c.x), xhi = fmax(fmax((double)a.x, b.x), c.x);
  const double ylo = fmin(fmin((double)a.y, b.y), c.y), yhi = fmax(fmax((double)a.y, b.y), c.y);
  const double zlo = fmin(fmin((double)a.z, b.z), c.z), zhi = fmax(fmax((double)a.z, b.z), c.z);
  // one row more on each side, and what rounding to FP32 moves a sample's coordinate
  auto clip = [](double v, int n) { return (int)fmin(fmax(v, 0.0), (double)n); };
  const double ym = 0x1p-23 * fmax(fabs(ylo), fabs(yhi)), zm = 0x1p-23 * fmax(fabs(zlo), fabs(zhi));
  const int j0 = clip(floor((ylo - ym - g.oy) / g.dx) - 1, g.nj),
            j1 = clip(ceil((yhi + ym - g.oy) / g.dx) + 2, g.nj),
            k0 = clip(floor((zlo - zm - g.oz) / g.dx) - 1, g.nk),
            k1 = clip(ceil((zhi + zm - g.oz) / g.dx) + 2, g.nk);
  const int nj = j1 - j0;
  if (nj <= 0 || k1 <= k0) return;
  for (long long r = lane; r < (long long)nj * (k1 - k0); r += 32) {
    const int j = j0 + (int)(r % nj), k = k0 + (int)(r / nj);
    const float3 s = sample_pos(g, 0, j, k);
    const int wind = edge_part(a, b, s.y, s.z) + edge_part(b, c, s.y, s.z) + edge_part(c, a, s.y, s.z);
    if (wind == 0) continue;
    // the plane through the triangle at (y, z), within the triangle's range (also
    // where rounding leaves no normal along x)
    const double ux = (double)b.x - a.x, uy = (double)b.y - a.y, uz = (double)b.z - a.z;
    const double vx = (double)c.x - a.x, vy = (double)c.y - a.y, vz = (double)c.z - a.z;
    const double nx = uy * vz - uz * vy, ny = uz * vx - ux * vz, nz = ux * vy - uy * vx;
    const double plane = a.x - (ny * ((double)s.y - a.y) + nz * ((double)s.z - a.z)) / nx;
    const double x = fmin(fmax(plane, xlo), xhi);
    int i = (int)fmin(fmax(ceil((x - g.ox) / g.dx), 0.0), (double)g.ni);
    while (i > 0 && (double)sample_pos(g, i - 1, j, k).x > x) --i;
    while (i < g.ni && (double)sample_pos(g, i, j, k).x <= x) ++i;
    // walking +x, the winding number drops by one where the normal points to +x
    if (i < g.ni) atomicAdd(step + ((long long)k * g.nj + j) * g.ni + i, -wind);
  }
}

// Signs of a closed mesh: a warp per row sums the steps along x.
__global__ void __launch_bounds__(kSdfBlock)
    k_row_signs(const int* __restrict__ step, SdfGrid g,
                const unsigned long long* __restrict__ open, float* __restrict__ phi) {
  if (open[0] | open[1] | open[2]) return;
  const int lane = threadIdx.x & 31;
  const long long row = (long long)blockIdx.x * (kSdfBlock / 32) + (threadIdx.x >> 5);
  if (row >= (long long)g.nj * g.nk) return;
  int base = 0;
  for (int i0 = 0; i0 < g.ni; i0 += 32) {
    const int i = i0 + lane;
    int x = i < g.ni ? step[row * g.ni + i] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    x += base;
    if (i < g.ni && x != 0) phi[row * g.ni + i] = -phi[row * g.ni + i];
    base = __shfl_sync(0xffffffffu, x, 31);
  }
}

// Signs of a mesh with a boundary: the solid angles of all triangles, staged
// through shared memory in tiles, one thread per sample.
__global__ void __launch_bounds__(kSdfBlock)
    k_solid_signs(const float3* __restrict__ tv, int nt, SdfGrid g,
                  const unsigned long long* __restrict__ open, float* __restrict__ phi) {
  if (!(open[0] | open[1] | open[2])) return;
  __shared__ float3 s[3 * kTriTile];
  const long long total = (long long)g.ni * g.nj * g.nk;
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const bool live = idx < total;
  const int i = live ? (int)(idx % g.ni) : 0;
  const int j = live ? (int)((idx / g.ni) % g.nj) : 0;
  const int k = live ? (int)(idx / ((long long)g.ni * g.nj)) : 0;
  const float3 p = sample_pos(g, i, j, k);
  float wind = 0.0f;
  for (int t0 = 0; t0 < nt; t0 += kTriTile) {
    const int cnt = min(kTriTile, nt - t0);
    __syncthreads();
    for (int e = threadIdx.x; e < 3 * cnt; e += blockDim.x) s[e] = tv[3 * (size_t)t0 + e];
    __syncthreads();
    if (live)
      for (int t = 0; t < cnt; ++t)
        wind += solid_angle(sub3(s[3 * t], p), sub3(s[3 * t + 1], p), sub3(s[3 * t + 2], p));
  }
  if (live && fabsf(wind) > 6.283185307f) phi[idx] = -phi[idx];
}

}  // namespace
}  // namespace sphpc

using namespace sphpc;

// Signed distance of the mesh (vertices[3 * nv], triangles[3 * nt]
// vertex indices, host memory) at the samples origin + (i, j, k) * dx of a
// dims[0] x dims[1] x dims[2] grid, into phi (host, i fastest).
extern "C" int sphpc_mesh_sdf(const float* vertices, int n_vertices, const int* triangles,
                              int n_triangles, const int* dims, const double* origin, double dx,
                              float* phi) {
  if (!vertices || !triangles || !dims || !origin || !phi || n_vertices <= 0 ||
      n_triangles <= 0 || !(dx > 0.0))
    return set_error(SPHPC_EINVAL, "sphpc_mesh_sdf: bad arguments");
  for (int d = 0; d < 3; ++d)
    if (dims[d] <= 0) return set_error(SPHPC_EINVAL, "sphpc_mesh_sdf: empty grid");
  const long long total = (long long)dims[0] * dims[1] * dims[2];
  for (long long k = 0; k < 3ll * n_triangles; ++k)
    if (triangles[k] < 0 || triangles[k] >= n_vertices)
      return set_error(SPHPC_EINVAL, "sphpc_mesh_sdf: triangle %d has vertex index %d",
                       (int)(k / 3), triangles[k]);
  // the mesh's box, for the Morton keys
  bool finite = true;
  float lo[3] = {0.f, 0.f, 0.f}, scale[3] = {0.f, 0.f, 0.f};
  for (int c = 0; c < 3; ++c) {
    float a = INFINITY, b = -INFINITY;
    for (int v = 0; v < n_vertices; ++v) {
      const float x = vertices[3 * (size_t)v + c];
      finite = finite && std::isfinite(x);
      a = fminf(a, x);
      b = fmaxf(b, x);
    }
    lo[c] = a;
    scale[c] = b > a ? 1024.0f / (b - a) : 0.0f;
  }
  const size_t nt = (size_t)n_triangles, nc = (nt + kCluster - 1) / kCluster;
  ScratchLayout lay;
  auto part = [&](size_t bytes) { return lay.part(bytes); };
  const size_t o_vert = part(12 * (size_t)n_vertices), o_tri = part(12 * nt),
               o_corner = part(36 * nt), o_key = part(4 * nt), o_order = part(4 * nt),
               o_keys2 = part(4 * nt), o_order2 = part(4 * nt), o_aux = part(4 * sort_aux_words(n_triangles)),
               o_sorted = part(48 * nc * kCluster), o_box = part(32 * nc), o_rep = part(16 * nc), o_open = part(24),
               o_step = part(4 * (size_t)total), o_phi = part(4 * (size_t)total);
  CallScratch mem;
  cudaError_t e = mem.take(lay.bytes(), 0);
  char* buf = mem.at<char>(0);
  const SdfGrid g{dims[0], dims[1], dims[2], origin[0], origin[1], origin[2], dx};
  auto blocks = [](long long n, int per) { return (unsigned)((n + per - 1) / per); };
  if (e == cudaSuccess) {
    float* d_phi = (float*)(buf + o_phi);
    float3* corners = (float3*)(buf + o_corner);
    auto* open = (unsigned long long*)(buf + o_open);
    SortScratch sc;
    sc.keys_alt = (uint32_t*)(buf + o_keys2);
    sc.vals_alt = (uint32_t*)(buf + o_order2);
    sort_layout(sc, (uint32_t*)(buf + o_aux));
    e = cudaMemcpyAsync(buf + o_vert, vertices, 12 * (size_t)n_vertices, cudaMemcpyHostToDevice, 0);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(buf + o_tri, triangles, 12 * nt, cudaMemcpyHostToDevice, 0);
    if (e == cudaSuccess) e = cudaMemsetAsync(open, 0, 16, 0);
    if (e == cudaSuccess) e = cudaMemsetAsync(open + 2, finite ? 0 : 1, 8, 0);
    if (e == cudaSuccess) e = cudaMemsetAsync(buf + o_step, 0, 4 * (size_t)total, 0);
    if (e == cudaSuccess) {
      k_triangles<<<blocks(nt, kSdfBlock), kSdfBlock>>>(
          (const float3*)(buf + o_vert), (const int*)(buf + o_tri), n_triangles,
          make_float3(lo[0], lo[1], lo[2]), make_float3(scale[0], scale[1], scale[2]), corners,
          (uint32_t*)(buf + o_key), open);
      e = radix_sort_pairs((uint32_t*)(buf + o_key), (uint32_t*)(buf + o_order), n_triangles,
                           kMaxPasses, sc, 0, false, true, true, nullptr, nullptr);
    }
    if (e == cudaSuccess) {
      const float4* tri = (const float4*)(buf + o_sorted);
      const float4* box = (const float4*)(buf + o_box);
      k_clusters<<<blocks(nc * kCluster, kSdfBlock), kSdfBlock>>>(
          corners, (const uint32_t*)(buf + o_order), n_triangles, (int)nc, (float4*)tri, (float4*)box,
          (float4*)(buf + o_rep));
      const long long boxes =
          (long long)((g.ni + 3) / 4) * ((g.nj + 3) / 4) * ((g.nk + 1) / 2);
      k_mesh_dist<<<(unsigned)boxes, kDistWarps * 32>>>(
          tri, box, (const float4*)(buf + o_rep), (int)nc, g, d_phi);
      k_crossings<<<blocks(nt, kSdfBlock / 32), kSdfBlock>>>(corners, n_triangles, g, open,
                                                             (int*)(buf + o_step));
      k_row_signs<<<blocks((long long)g.nj * g.nk, kSdfBlock / 32), kSdfBlock>>>(
          (const int*)(buf + o_step), g, open, d_phi);
      k_solid_signs<<<blocks(total, kSdfBlock), kSdfBlock>>>(corners, n_triangles, g, open, d_phi);
      e = cudaGetLastError();
    }
    if (e == cudaSuccess)
      e = cudaMemcpy(phi, d_phi, sizeof(float) * (size_t)total, cudaMemcpyDeviceToHost);
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    return set_error(SPHPC_ECUDA, "sphpc_mesh_sdf: %s", cudaGetErrorString(e));
  }
  return SPHPC_OK;
}
