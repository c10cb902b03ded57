// Mesh -> particle setup on the GPU: the voxeliser (src/softbody/voxelize.ts)
// and the signed-distance baker (src/sdf/bake.ts).
//
// Both are brute force in the reference (every grid point against every
// triangle, in JavaScript doubles). Here one thread takes one grid point, in
// double precision: the voxeliser walks all triangles, tiled through shared
// memory; the baker walks the chunks of triangles its warp's brick of voxels
// can reach. This file is compiled with -fmad=false, so every double
// multiply and add is rounded on its own as the reference's arithmetic is,
// and the occupancy, hit counts and distances equal the reference's. The
// integer bookkeeping that follows the inside test (largest piece, surface
// classification, ordering, edges) runs on the host, in O(cells).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <limits>
#include <string>
#include <vector>

#include "common.cuh"
#include "devmem.cuh"
#include "pfsim.h"

namespace pf {
namespace {

constexpr uint32_t kTileTris = 128;

// One triangle as the kernels read it: the three corners (f32, as the
// mesh's Float32Array holds them), 48 bytes.
struct alignas(16) MeshTri {
  float a[3], b[3], c[3], pad[3];
};
constexpr uint32_t kTriWords = sizeof(MeshTri) / 4;

// Shared-memory staging of triangles [t0, t0 + kTileTris).
__device__ __forceinline__ uint32_t stage_tris(MeshTri* st, const MeshTri* __restrict__ tris, uint32_t t0,
                                               uint32_t n_tris) {
  const uint32_t cnt = min(kTileTris, n_tris - t0);
  const float* src = reinterpret_cast<const float*>(tris + t0);
  float* dst = reinterpret_cast<float*>(st);
  for (uint32_t i = threadIdx.x; i < cnt * kTriWords; i += blockDim.x) dst[i] = src[i];
  __syncthreads();
  return cnt;
}

// voxelize.ts:178-228: Moller-Trumbore, the ray parameter of the hit or -1.
__device__ __forceinline__ double ray_tri_t(double ox, double oy, double oz, double dx, double dy, double dz,
                                            const MeshTri& T) {
  const double ax = T.a[0], ay = T.a[1], az = T.a[2];
  const double e1x = (double)T.b[0] - ax, e1y = (double)T.b[1] - ay, e1z = (double)T.b[2] - az;
  const double e2x = (double)T.c[0] - ax, e2y = (double)T.c[1] - ay, e2z = (double)T.c[2] - az;
  const double hx = dy * e2z - dz * e2y;
  const double hy = dz * e2x - dx * e2z;
  const double hz = dx * e2y - dy * e2x;
  const double a = e1x * hx + e1y * hy + e1z * hz;
  if (a > -1e-9 && a < 1e-9) return -1.0;
  const double f = 1.0 / a;
  const double sx = ox - ax, sy = oy - ay, sz = oz - az;
  const double u = f * (sx * hx + sy * hy + sz * hz);
  if (u < 0.0 || u > 1.0) return -1.0;
  const double qx = sy * e1z - sz * e1y;
  const double qy = sz * e1x - sx * e1z;
  const double qz = sx * e1y - sy * e1x;
  const double v = f * (dx * qx + dy * qy + dz * qz);
  if (v < 0.0 || u + v > 1.0) return -1.0;
  const double t = f * (e2x * qx + e2y * qy + e2z * qz);
  if (t < 1e-9) return -1.0;
  return t;
}

// voxelize.ts:86-90, 234-259: grid point `cell` of an nx x ny x nz lattice
// at min + r + 2r i, inside the mesh when a slightly off-axis ray crosses it
// an odd number of times.
__global__ void __launch_bounds__(256) k_vox_mesh(const MeshTri* __restrict__ tris, uint32_t n_tris, double mnx,
                                                  double mny, double mnz, double r, double spacing, uint32_t nx,
                                                  uint32_t ny, uint64_t cells, uint8_t* __restrict__ occ) {
  __shared__ MeshTri st[kTileTris];
  const uint64_t cell = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool live = cell < cells;
  double px = 0, py = 0, pz = 0;
  if (live) {
    px = mnx + r + spacing * (double)(cell % nx);
    py = mny + r + spacing * (double)((cell / nx) % ny);
    pz = mnz + r + spacing * (double)(cell / ((uint64_t)nx * ny));
  }
  uint32_t crossings = 0;
  for (uint32_t t0 = 0; t0 < n_tris; t0 += kTileTris) {
    const uint32_t cnt = stage_tris(st, tris, t0, n_tris);
    if (live)
      for (uint32_t t = 0; t < cnt; ++t)
        if (ray_tri_t(px, py, pz, 1.0, 0.00137, 0.00241, st[t]) > 0.0) ++crossings;
    __syncthreads();
  }
  if (live) occ[cell] = (crossings & 1u) ? 1 : 0;
}

// sample.ts:12-47 in doubles over the f32 field.
__device__ __forceinline__ double sample_field(const float* __restrict__ data, uint32_t rx, uint32_t ry,
                                               uint32_t rz, double ox, double oy, double oz, double vx,
                                               double vy, double vz, double x, double y, double z) {
  const double gx = (x - ox) / vx - 0.5, gy = (y - oy) / vy - 0.5, gz = (z - oz) / vz - 0.5;
  auto clampi = [](double v, double hi) { return v < 0.0 ? 0.0 : (v > hi ? hi : v); };
  const double i0 = clampi(floor(gx), (double)(rx - 2)), j0 = clampi(floor(gy), (double)(ry - 2)),
               k0 = clampi(floor(gz), (double)(rz - 2));
  auto c01 = [](double t) { return t < 0.0 ? 0.0 : (t > 1.0 ? 1.0 : t); };
  const double tx = c01(gx - i0), ty = c01(gy - j0), tz = c01(gz - k0);
  const uint64_t stride = rx, slice = (uint64_t)rx * ry;
  const uint64_t base = (uint64_t)i0 + (uint64_t)j0 * stride + (uint64_t)k0 * slice;
  auto lerp = [](double a, double b, double t) { return a + (b - a) * t; };
  const double c00 = lerp(data[base], data[base + 1], tx);
  const double c10 = lerp(data[base + stride], data[base + stride + 1], tx);
  const double c01v = lerp(data[base + slice], data[base + slice + 1], tx);
  const double c11 = lerp(data[base + slice + stride], data[base + slice + stride + 1], tx);
  const double c0 = lerp(c00, c10, ty), c1 = lerp(c01v, c11, ty);
  return lerp(c0, c1, tz);
}

// voxelize.ts:173-177: inside where the sampled field is below `dilation`.
__global__ void __launch_bounds__(256) k_vox_sdf(const float* __restrict__ data, uint32_t rx, uint32_t ry,
                                                 uint32_t rz, double ox, double oy, double oz, double vx, double vy,
                                                 double vz, double dilation, double r, double spacing, uint32_t nx,
                                                 uint32_t ny, uint64_t cells, uint8_t* __restrict__ occ) {
  const uint64_t cell = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (cell >= cells) return;
  const double px = ox + r + spacing * (double)(cell % nx);
  const double py = oy + r + spacing * (double)((cell / nx) % ny);
  const double pz = oz + r + spacing * (double)(cell / ((uint64_t)nx * ny));
  occ[cell] = sample_field(data, rx, ry, rz, ox, oy, oz, vx, vy, vz, px, py, pz) < dilation ? 1 : 0;
}

// bake.ts:297-368: squared distance from P to a triangle (Ericson RTCD
// 5.1.5, the seven Voronoi regions).
__device__ __forceinline__ double point_tri_d2(double px, double py, double pz, const MeshTri& T) {
  const double ax = T.a[0], ay = T.a[1], az = T.a[2];
  const double bx = T.b[0], by = T.b[1], bz = T.b[2];
  const double cx = T.c[0], cy = T.c[1], cz = T.c[2];
  const double abx = bx - ax, aby = by - ay, abz = bz - az;
  const double acx = cx - ax, acy = cy - ay, acz = cz - az;
  const double apx = px - ax, apy = py - ay, apz = pz - az;
  const double d1 = abx * apx + aby * apy + abz * apz;
  const double d2 = acx * apx + acy * apy + acz * apz;
  if (d1 <= 0.0 && d2 <= 0.0) return apx * apx + apy * apy + apz * apz;
  const double bpx = px - bx, bpy = py - by, bpz = pz - bz;
  const double d3 = abx * bpx + aby * bpy + abz * bpz;
  const double d4 = acx * bpx + acy * bpy + acz * bpz;
  if (d3 >= 0.0 && d4 <= d3) return bpx * bpx + bpy * bpy + bpz * bpz;
  const double vc = d1 * d4 - d3 * d2;
  if (vc <= 0.0 && d1 >= 0.0 && d3 <= 0.0) {
    const double v = d1 / (d1 - d3);
    const double qx = apx - v * abx, qy = apy - v * aby, qz = apz - v * abz;
    return qx * qx + qy * qy + qz * qz;
  }
  const double cpx = px - cx, cpy = py - cy, cpz = pz - cz;
  const double d5 = abx * cpx + aby * cpy + abz * cpz;
  const double d6 = acx * cpx + acy * cpy + acz * cpz;
  if (d6 >= 0.0 && d5 <= d6) return cpx * cpx + cpy * cpy + cpz * cpz;
  const double vb = d5 * d2 - d1 * d6;
  if (vb <= 0.0 && d2 >= 0.0 && d6 <= 0.0) {
    const double w = d2 / (d2 - d6);
    const double qx = apx - w * acx, qy = apy - w * acy, qz = apz - w * acz;
    return qx * qx + qy * qy + qz * qz;
  }
  const double va = d3 * d6 - d5 * d4;
  if (va <= 0.0 && d4 - d3 >= 0.0 && d5 - d6 >= 0.0) {
    const double w = (d4 - d3) / (d4 - d3 + (d5 - d6));
    const double qx = bpx - w * (cx - bx), qy = bpy - w * (cy - by), qz = bpz - w * (cz - bz);
    return qx * qx + qy * qy + qz * qz;
  }
  const double denom = 1.0 / (va + vb + vc);
  const double v = vb * denom, w = vc * denom;
  const double qx = apx - v * abx - w * acx, qy = apy - v * aby - w * acy, qz = apz - v * abz - w * acz;
  return qx * qx + qy * qy + qz * qz;
}

// bake.ts:460-486: the axis ray along +x, +y or +z against one triangle.
__device__ __forceinline__ bool axis_hit(double px, double py, double pz, int axis, const MeshTri& T) {
  const double ax = T.a[0], ay = T.a[1], az = T.a[2];
  const double e1x = (double)T.b[0] - ax, e1y = (double)T.b[1] - ay, e1z = (double)T.b[2] - az;
  const double e2x = (double)T.c[0] - ax, e2y = (double)T.c[1] - ay, e2z = (double)T.c[2] - az;
  double hx, hy, hz;
  if (axis == 0) {
    hx = 0.0;
    hy = -e2z;
    hz = e2y;
  } else if (axis == 1) {
    hx = e2z;
    hy = 0.0;
    hz = -e2x;
  } else {
    hx = -e2y;
    hy = e2x;
    hz = 0.0;
  }
  const double a = e1x * hx + e1y * hy + e1z * hz;
  if (fabs(a) < 1e-7) return false;
  const double inv = 1.0 / a;
  const double sx = px - ax, sy = py - ay, sz = pz - az;
  const double u = inv * (sx * hx + sy * hy + sz * hz);
  if (u < 0.0 || u > 1.0) return false;
  const double qx = sy * e1z - sz * e1y;
  const double qy = sz * e1x - sx * e1z;
  const double qz = sx * e1y - sy * e1x;
  const double v = inv * (axis == 0 ? qx : (axis == 1 ? qy : qz));
  if (v < 0.0 || u + v > 1.0) return false;
  return inv * (e2x * qx + e2y * qy + e2z * qz) > 1e-7;
}

// A double between two floats: the nearest float at or below it and at or
// above it. Against a float bound L, v < L exactly when lo < L, and v > L
// exactly when hi > L, so the box culls below compare in FP32 (full rate, no
// conversions of the boxes) and decide as the doubles would.
struct Span {
  float lo, hi;
};
__device__ __forceinline__ Span span_of(double v) { return {__double2float_rd(v), __double2float_ru(v)}; }

// What the baker rejects a triangle by: its bounding box, and its plane
// n . x = d (n unit, zero where the triangle has none); slack is what FP32
// makes of the plane's distance at the triangle's corners at most.
struct alignas(16) TriCull {
  float lo[3], hi[3], n[3], d, slack, pad;
};
// What bounds kBakeChunk consecutive triangles (in the baker's order): a box,
// and the slab d0 <= n . x <= d1 of their mean normal n (unit; zero where the
// triangles have none, a slab that bounds nothing).
struct alignas(16) ChunkBox {
  float lo[3], hi[3], n[3], d0, d1, pad;
};
constexpr uint32_t kBakeChunk = 32;  // a lane tests one triangle of a chunk
constexpr uint32_t kBakeWarps = 4;
// A warp takes a brick of 4 x 4 x 2 voxels.
constexpr uint32_t kBrickX = 4, kBrickY = 4, kBrickZ = 2;

// bake.ts:106-127: per voxel centre, the closest triangle (each skipped when
// its box is no closer than the best so far), the three jittered axis-ray
// parities and their majority.
//
// The reference tests every triangle at every voxel; in FP64 that was bound
// by instruction issue. A warp's 32 voxels form a brick, the triangles come in
// chunks of 32 neighbours (sorted along a Morton curve on the host), and a
// warp leaves out what none of its voxels can need, in three steps. The lanes
// test 32 chunks at a time against the brick: for the distance, by the
// chunk's box and slab against the worst of the lanes' best distances (the
// closest chunk is taken first, so that bound is tight at once); for a ray
// axis, by the box culls of bake.ts:422-448 over the brick's rays. Then the
// lanes test a chunk's 32 triangles in the same way. Each lane then tests
// its own voxel against the box and the plane of a triangle that is left
// (of 8,064 triangles about 140 per warp), and the exact test in doubles runs
// where some lane needs it (about 30). All of the rejecting runs in FP32,
// rounded so that it drops only what the doubles drop, so the hit counts are
// the brute force's and the distance is the minimum over every triangle that
// can be the closest.
// 8,064 triangles, 128^3 voxels: 75.4 ms before (every pair), 2.2 ms now;
// boxes alone, with every lane testing every triangle of a chunk, took 4.4 ms.
// It waits on FP64 and L1 latency, so eight blocks per SM (64 registers) are
// better than what the registers alone would take: 2.8 ms at 126, 2.5 at 80.
__global__ void __launch_bounds__(32 * kBakeWarps, 8) k_bake(const MeshTri* __restrict__ tris,
                                                          const TriCull* __restrict__ culls, uint32_t n_tris,
                                                          const ChunkBox* __restrict__ boxes, uint32_t n_chunks,
                                                          uint32_t res, double ox, double oy, double oz, double voxel,
                                                          double jitter, float* __restrict__ data,
                                                          unsigned long long* __restrict__ inconsistent) {
  constexpr uint32_t kAll = 0xffffffffu;
  const uint32_t lane = threadIdx.x & 31u;
  const uint64_t brick = (uint64_t)blockIdx.x * kBakeWarps + (threadIdx.x >> 5);
  const uint32_t nbx = div_up(res, kBrickX), nby = div_up(res, kBrickY), nbz = div_up(res, kBrickZ);
  if (brick >= (uint64_t)nbx * nby * nbz) return;  // whole warps
  const uint32_t x0 = (uint32_t)(brick % nbx) * kBrickX, y0 = (uint32_t)((brick / nbx) % nby) * kBrickY,
                 z0 = (uint32_t)(brick / ((uint64_t)nbx * nby)) * kBrickZ;
  const uint32_t xi = x0 + lane % kBrickX, yi = y0 + (lane / kBrickX) % kBrickY, zi = z0 + lane / (kBrickX * kBrickY);
  const bool live = xi < res && yi < res && zi < res;
  const uint32_t top = res - 1;
  auto at = [&](double o, uint32_t i) { return o + ((double)min(i, top) + 0.5) * voxel; };
  // voxels past the grid's end stand on its last voxel and write nothing
  const double px = at(ox, xi), py = at(oy, yi), pz = at(oz, zi);
  const double ja = jitter * 1.4142135623730951, jb = jitter * 3.141592653589793;
  const Span sx = span_of(px), sy = span_of(py), sz = span_of(pz);
  // the three rays' fixed coordinates: axis x at (ya, zb), y at (xb, za), z at (xa, yb)
  const Span ya = span_of(py + ja), zb = span_of(pz + jb), xb = span_of(px + jb), za = span_of(pz + ja),
             xa = span_of(px + ja), yb = span_of(py + jb);
  double best = INFINITY;
  float best_up = INFINITY;  // best, rounded up
  uint32_t hx = 0, hy = 0, hz = 0;
  // squared distance from a span of points to a box, every operation rounded
  // down: at most the per-triangle box distance of the doubles
  auto gap = [](float p0, float p1, float lo, float hi) {
    return fmaxf(fmaxf(__fsub_rd(lo, p1), __fsub_rd(p0, hi)), 0.0f);
  };
  auto square = [](float dx, float dy, float dz) {
    return __fmul_rd(__fadd_rd(__fadd_rd(__fmul_rd(dx, dx), __fmul_rd(dy, dy)), __fmul_rd(dz, dz)), 1.0f - 0x1p-20f);
  };
  // the brick's box, and its rays' (by shuffles: lane 0 has the lowest voxel
  // on every axis, lane 31 the highest)
  auto hull = [&](Span s) { return Span{__shfl_sync(kAll, s.lo, 0), __shfl_sync(kAll, s.hi, 31)}; };
  const Span wx = hull(sx), wy = hull(sy), wz = hull(sz), wya = hull(ya), wzb = hull(zb), wxb = hull(xb),
             wza = hull(za), wxa = hull(xa), wyb = hull(yb);
  // the brick's centre and half extents (rounded outwards)
  const float hxl = __fmul_ru(0.5f, __fsub_ru(wx.hi, wx.lo)), hyl = __fmul_ru(0.5f, __fsub_ru(wy.hi, wy.lo)),
              hzl = __fmul_ru(0.5f, __fsub_ru(wz.hi, wz.lo));
  const double cx = 0.5 * ((double)wx.lo + wx.hi), cy = 0.5 * ((double)wy.lo + wy.hi),
               cz = 0.5 * ((double)wz.lo + wz.hi);
  // squared distance from the brick to a chunk, rounded down: to its box, or
  // to its slab where that is further (a smooth patch is a thin slab, but a
  // thick box when it lies askew)
  auto apart = [&](const ChunkBox& B) {
    const float box = square(gap(wx.lo, wx.hi, B.lo[0], B.hi[0]), gap(wy.lo, wy.hi, B.lo[1], B.hi[1]),
                             gap(wz.lo, wz.hi, B.lo[2], B.hi[2]));
    const double h = B.n[0] * cx + B.n[1] * cy + B.n[2] * cz;
    const float reach = fabsf(B.n[0]) * hxl + fabsf(B.n[1]) * hyl + fabsf(B.n[2]) * hzl;
    const float off = (__double2float_rd(fmax((double)B.d0 - h, h - (double)B.d1)) - reach * 1.000001f) * 0.999999f;
    return off > 0.0f ? fmaxf(box, __fmul_rd(off, off)) : box;
  };
  // the worst of the lanes' best distances (non-negative floats order as
  // their bits)
  auto worst = [&]() { return __uint_as_float(__reduce_max_sync(kAll, __float_as_uint(best_up))); };
  // the rounding of a plane distance in FP32 (a few parts in 2^24 of its terms)
  const float fx = (float)px, fy = (float)py, fz = (float)pz;
  const float fuzz = 1e-6f * (fabsf(fx) + fabsf(fy) + fabsf(fz));
  float limit = INFINITY;
  auto take = [&](uint32_t c) {
    const uint32_t t0 = c * kBakeChunk;
    bool near = false;
    if (t0 + lane < n_tris) {
      const TriCull& C = culls[t0 + lane];
      near = !(square(gap(wx.lo, wx.hi, C.lo[0], C.hi[0]), gap(wy.lo, wy.hi, C.lo[1], C.hi[1]),
                      gap(wz.lo, wz.hi, C.lo[2], C.hi[2])) > limit);
    }
    for (uint32_t m = __ballot_sync(kAll, near); m; m &= m - 1) {
      const uint32_t t = t0 + __ffs(m) - 1;
      const TriCull& C = culls[t];
      const float far = square(gap(sx.lo, sx.hi, C.lo[0], C.hi[0]), gap(sy.lo, sy.hi, C.lo[1], C.hi[1]),
                               gap(sz.lo, sz.hi, C.lo[2], C.hi[2]));
      const float off =
          fmaxf(fabsf(C.n[0] * fx + C.n[1] * fy + C.n[2] * fz - C.d) - (fuzz + C.slack), 0.0f) * 0.999999f;
      if (far > best_up || off * off > best_up) continue;  // no closer than the best so far
      const double d = point_tri_d2(px, py, pz, tris[t]);
      if (d < best) {
        best = d;
        best_up = __double2float_ru(d);
      }
    }
  };
  // the closest chunk first
  uint32_t first = 0;
  {
    float lb = INFINITY;
    for (uint32_t c = lane; c < n_chunks; c += 32) {
      const float v = apart(boxes[c]);
      if (v < lb) {
        lb = v;
        first = c;
      }
    }
    const uint32_t low = __reduce_min_sync(kAll, __float_as_uint(lb));
    const uint32_t who = __ballot_sync(kAll, __float_as_uint(lb) == low);
    first = __shfl_sync(kAll, first, __ffs(who) - 1);
  }
  take(first);
  limit = worst();
  // whether no ray of a brick can meet a box
  auto misses = [](Span u, Span v, float w, const float* lo, const float* hi, int a, int b, int c) {
    return u.hi < lo[a] || u.lo > hi[a] || v.hi < lo[b] || v.lo > hi[b] || w > hi[c];
  };
  for (uint32_t c0 = 0; c0 < n_chunks; c0 += 32) {
    const uint32_t c = c0 + lane;
    float lb = INFINITY;
    bool near = false, rx = false, ry = false, rz = false;
    if (c < n_chunks) {
      const ChunkBox B = boxes[c];
      lb = apart(B);
      near = c != first && !(lb > limit);
      rx = !misses(wya, wzb, wx.lo, B.lo, B.hi, 1, 2, 0);
      ry = !misses(wxb, wza, wy.lo, B.lo, B.hi, 0, 2, 1);
      rz = !misses(wxa, wyb, wz.lo, B.lo, B.hi, 0, 1, 2);
    }
    for (uint32_t m = __ballot_sync(kAll, near); m; m &= m - 1) {
      const uint32_t b = __ffs(m) - 1;
      if (__shfl_sync(kAll, lb, b) > limit) continue;  // the limit has come down
      take(c0 + b);
      limit = worst();
    }
    // an axis's chunks, their triangles against the brick's rays (a lane
    // each), then each lane's ray against what is left: bake.ts:422-448
    auto clear = [](Span u, Span v, Span w, const TriCull& C, int a, int b, int c) {
      return u.lo < C.lo[a] || u.hi > C.hi[a] || v.lo < C.lo[b] || v.hi > C.hi[b] || w.hi > C.hi[c];
    };
    auto rays = [&](bool mine, Span wu, Span wv, Span ww, Span u, Span v, Span w, int a, int b, int c, double rx,
                    double ry, double rz) {
      uint32_t hits = 0;
      for (uint32_t m = __ballot_sync(kAll, mine); m; m &= m - 1) {
        const uint32_t t0 = (c0 + __ffs(m) - 1) * kBakeChunk;
        bool some = false;
        if (t0 + lane < n_tris) some = !misses(wu, wv, ww.lo, culls[t0 + lane].lo, culls[t0 + lane].hi, a, b, c);
        for (uint32_t q = __ballot_sync(kAll, some); q; q &= q - 1) {
          const uint32_t t = t0 + __ffs(q) - 1;
          if (!clear(u, v, w, culls[t], a, b, c)) hits += axis_hit(rx, ry, rz, c, tris[t]) ? 1u : 0u;
        }
      }
      return hits;
    };
    hx += rays(rx, wya, wzb, wx, ya, zb, sx, 1, 2, 0, px, py + ja, pz + jb);
    hy += rays(ry, wxb, wza, wy, xb, za, sy, 0, 2, 1, px + jb, py, pz + ja);
    hz += rays(rz, wxa, wyb, wz, xa, yb, sz, 0, 1, 2, px + ja, py + jb, pz);
  }
  if (!live) return;
  const uint32_t votes = (hx & 1u) + (hy & 1u) + (hz & 1u);
  if (votes == 1 || votes == 2) atomicAdd(inconsistent, 1ull);
  const double dist = sqrt(best);
  data[xi + (uint64_t)res * (yi + (uint64_t)res * zi)] = (float)(votes >= 2 ? -dist : dist);
}

// A triangle's box and plane.
TriCull cull_of(const MeshTri& T) {
  TriCull C{};
  double e[3], f[3], n[3];
  for (int a = 0; a < 3; ++a) {
    C.lo[a] = std::min(std::min(T.a[a], T.b[a]), T.c[a]);
    C.hi[a] = std::max(std::max(T.a[a], T.b[a]), T.c[a]);
    e[a] = (double)T.b[a] - T.a[a];
    f[a] = (double)T.c[a] - T.a[a];
  }
  for (int a = 0; a < 3; ++a) n[a] = e[(a + 1) % 3] * f[(a + 2) % 3] - e[(a + 2) % 3] * f[(a + 1) % 3];
  const double len = std::sqrt(n[0] * n[0] + n[1] * n[1] + n[2] * n[2]);
  // a sliver's normal is not to be trusted: it has no plane
  double longest = 0;
  for (int a = 0; a < 3; ++a) longest = std::max(longest, std::max(std::fabs(e[a]), std::fabs(f[a])));
  if (std::isfinite(len) && len > 1e-6 * longest * longest) {
    double d = 0, most = 0;
    for (int a = 0; a < 3; ++a) {
      C.n[a] = (float)(n[a] / len);
      d += (double)C.n[a] * T.a[a];
      most += std::max(std::fabs(C.lo[a]), std::fabs(C.hi[a]));
    }
    C.d = (float)d;
    C.slack = (float)(1e-6 * most);
  }
  return C;
}

// The baker's order: triangles along a Morton curve through their boxes'
// centres (10 bits an axis over the mesh's box), so that kBakeChunk
// consecutive ones lie close together; their culling records and their
// chunks' bounds. Coordinates that are not finite take code 0 and leave the
// boxes alone: such a triangle is neither closer than another nor hit.
void order_for_bake(std::vector<MeshTri>& tris, const double mn[3], const double mx[3], std::vector<TriCull>* culls,
                    std::vector<ChunkBox>* chunks) {
  auto spread = [](uint32_t v) {
    v = (v | (v << 16)) & 0x030000ffu;
    v = (v | (v << 8)) & 0x0300f00fu;
    v = (v | (v << 4)) & 0x030c30c3u;
    return (v | (v << 2)) & 0x09249249u;
  };
  std::vector<TriCull> raw(tris.size());
  std::vector<std::pair<uint32_t, uint32_t>> key(tris.size());
  for (size_t t = 0; t < tris.size(); ++t) {
    raw[t] = cull_of(tris[t]);
    uint32_t code = 0;
    for (int a = 0; a < 3; ++a) {
      const double u = (0.5 * ((double)raw[t].lo[a] + raw[t].hi[a]) - mn[a]) / (mx[a] - mn[a]) * 1024.0;
      code |= spread(u >= 0 ? (uint32_t)std::min(u, 1023.0) : 0u) << a;
    }
    key[t] = {code, (uint32_t)t};
  }
  std::sort(key.begin(), key.end());
  std::vector<MeshTri> sorted(tris.size());
  culls->resize(tris.size());
  chunks->resize((tris.size() + kBakeChunk - 1) / kBakeChunk);
  for (size_t c = 0; c < chunks->size(); ++c) {
    ChunkBox& B = (*chunks)[c];
    const size_t t0 = c * kBakeChunk, t1 = std::min(tris.size(), t0 + kBakeChunk);
    double n[3] = {0, 0, 0};
    for (int a = 0; a < 3; ++a) {
      B.lo[a] = INFINITY;
      B.hi[a] = -INFINITY;
    }
    for (size_t t = t0; t < t1; ++t) {
      const MeshTri& T = sorted[t] = tris[key[t].second];
      const TriCull& C = (*culls)[t] = raw[key[t].second];
      for (int a = 0; a < 3; ++a) {
        if (C.lo[a] < B.lo[a]) B.lo[a] = C.lo[a];
        if (C.hi[a] > B.hi[a]) B.hi[a] = C.hi[a];
        const int p = (a + 1) % 3, q = (a + 2) % 3;
        n[a] += ((double)T.b[p] - T.a[p]) * ((double)T.c[q] - T.a[q]) -
                ((double)T.b[q] - T.a[q]) * ((double)T.c[p] - T.a[p]);
      }
    }
    const double len = std::sqrt(n[0] * n[0] + n[1] * n[1] + n[2] * n[2]);
    const bool flat = std::isfinite(len) && len > 0;  // not so with a corner that is no number
    for (int a = 0; a < 3; ++a) B.n[a] = flat ? (float)(n[a] / len) : 0.0f;
    double d0 = INFINITY, d1 = -INFINITY, most = 0;
    for (size_t t = t0; t < t1; ++t) {
      const float* corner[3] = {sorted[t].a, sorted[t].b, sorted[t].c};
      for (const float* v : corner) {
        const double d = (double)B.n[0] * v[0] + (double)B.n[1] * v[1] + (double)B.n[2] * v[2];
        d0 = std::min(d0, d);
        d1 = std::max(d1, d);
        most = std::max(most, std::fabs((double)v[0]) + std::fabs((double)v[1]) + std::fabs((double)v[2]));
      }
    }
    // rounded outwards
    B.d0 = flat ? std::nextafterf((float)(d0 - 1e-12 * most), -INFINITY) : -INFINITY;
    B.d1 = flat ? std::nextafterf((float)(d1 + 1e-12 * most), INFINITY) : INFINITY;
  }
  tris.swap(sorted);
}

// toTriangleMesh + validated (src/core/mesh.ts:16-56).
pf_status read_mesh(const pf_mesh* m, std::vector<MeshTri>* out) {
  if (!m) return fail(PF_ERR_INVALID, "toTriangleMesh: expected a mesh");
  if (m->n_vertices && !m->vertices) return fail(PF_ERR_INVALID, "TriangleMesh: vertices are NULL");
  if (m->n_indices && !m->indices) return fail(PF_ERR_INVALID, "TriangleMesh: indices are NULL");
  if (m->n_indices % 3 != 0)
    return fail(PF_ERR_INVALID, "TriangleMesh: indices length " + std::to_string(m->n_indices) +
                                    " is not a multiple of 3");
  for (uint32_t i = 0; i < m->n_indices; ++i)
    if (m->indices[i] >= m->n_vertices)
      return fail(PF_ERR_INVALID, "TriangleMesh: index " + std::to_string(m->indices[i]) + " is out of range");
  out->resize(m->n_indices / 3);
  for (size_t t = 0; t < out->size(); ++t) {
    MeshTri& T = (*out)[t];
    const float* v[3] = {m->vertices + 3ull * m->indices[3 * t], m->vertices + 3ull * m->indices[3 * t + 1],
                         m->vertices + 3ull * m->indices[3 * t + 2]};
    for (int a = 0; a < 3; ++a) {
      T.a[a] = v[0][a];
      T.b[a] = v[1][a];
      T.c[a] = v[2][a];
      T.pad[a] = 0.0f;
    }
  }
  return PF_OK;
}

// A scratch buffer of one call. Up to kPooled bytes come from the library's
// device pool, in the order of the default stream, which the kernels here run
// on: mapping and unmapping pages on every call cost a bake about a millisecond.
// Larger ones are given back to the device at once.
struct DevBuf {
  static constexpr size_t kPooled = 32ull << 20;
  void* p = nullptr;
  bool pooled = false;
  ~DevBuf() {
    if (pooled) dev_free(p, nullptr);
    else if (p) cudaFree(p);
  }
  cudaError_t alloc(size_t bytes) {
    pooled = bytes <= kPooled;
    return pooled ? dev_alloc(&p, bytes, nullptr) : cudaMalloc(&p, bytes);
  }
};

template <typename T>
pf_status to_device(const std::vector<T>& v, DevBuf* d) {
  const size_t bytes = std::max<size_t>(1, v.size()) * sizeof(T);
  PF_CUDA(d->alloc(bytes));
  if (!v.empty()) PF_CUDA(cudaMemcpy(d->p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice));
  return PF_OK;
}

// voxelize.ts:92-161 from the occupancy: the largest face-connected piece
// (when asked), surface cells (a face neighbour missing) first, positions
// at the grid points, face-adjacent pairs.
pf_status finish_voxels(std::vector<uint8_t>& occ, const double mn[3], double r, double spacing, uint32_t nx,
                        uint32_t ny, uint32_t nz, bool largest, pf_voxels* out) {
  const uint64_t cells = (uint64_t)nx * ny * nz;
  auto nbrs = [&](uint64_t cell, uint64_t* o) {
    const uint64_t x = cell % nx, y = (cell / nx) % ny, z = cell / ((uint64_t)nx * ny);
    int n = 0;
    if (x > 0 && occ[cell - 1]) o[n++] = cell - 1;
    if (x + 1 < nx && occ[cell + 1]) o[n++] = cell + 1;
    if (y > 0 && occ[cell - nx]) o[n++] = cell - nx;
    if (y + 1 < ny && occ[cell + nx]) o[n++] = cell + nx;
    if (z > 0 && occ[cell - (uint64_t)nx * ny]) o[n++] = cell - (uint64_t)nx * ny;
    if (z + 1 < nz && occ[cell + (uint64_t)nx * ny]) o[n++] = cell + (uint64_t)nx * ny;
    return n;
  };
  if (largest) {
    std::vector<int64_t> piece(cells, -1);
    std::vector<uint64_t> best, members;
    uint64_t nb[6];
    for (uint64_t seed = 0; seed < cells; ++seed) {
      if (!occ[seed] || piece[seed] != -1) continue;
      members.assign(1, seed);
      piece[seed] = (int64_t)seed;
      for (size_t k = 0; k < members.size(); ++k) {
        const int c = nbrs(members[k], nb);
        for (int q = 0; q < c; ++q)
          if (piece[nb[q]] == -1) {
            piece[nb[q]] = (int64_t)seed;
            members.push_back(nb[q]);
          }
      }
      if (members.size() > best.size()) best.swap(members);
    }
    std::fill(occ.begin(), occ.end(), 0);
    for (uint64_t c : best) occ[c] = 1;
  }
  std::vector<uint64_t> surf, inner;
  uint64_t nb[6];
  for (uint64_t cell = 0; cell < cells; ++cell) {
    if (!occ[cell]) continue;
    (nbrs(cell, nb) < 6 ? surf : inner).push_back(cell);
  }
  const uint64_t count = surf.size() + inner.size();
  if (count > 0xffffffffull) return fail(PF_ERR_INVALID, "voxelize: too many particles");
  out->count = (uint32_t)count;
  out->surface_count = (uint32_t)surf.size();
  std::vector<uint32_t> particle_of;
  std::vector<uint64_t> ordered(surf);
  ordered.insert(ordered.end(), inner.begin(), inner.end());
  // cell -> particle through a sorted lookup (cells can be many)
  std::vector<std::pair<uint64_t, uint32_t>> lut(count);
  for (uint32_t i = 0; i < count; ++i) lut[i] = {ordered[i], i};
  std::sort(lut.begin(), lut.end());
  auto pid = [&](uint64_t cell) {
    return std::lower_bound(lut.begin(), lut.end(), std::make_pair(cell, 0u))->second;
  };
  if (out->positions && out->capacity >= count)
    for (uint32_t i = 0; i < count; ++i) {
      const uint64_t cell = ordered[i];
      const uint64_t ix[3] = {cell % nx, (cell / nx) % ny, cell / ((uint64_t)nx * ny)};
      for (int a = 0; a < 3; ++a) out->positions[3ull * i + a] = (float)(mn[a] + r + spacing * (double)ix[a]);
    }
  uint64_t ne = 0;
  for (uint32_t i = 0; i < count; ++i) {
    const int c = nbrs(ordered[i], nb);
    for (int q = 0; q < c; ++q) {
      const uint32_t j = pid(nb[q]);
      if (i < j) {
        if (out->edges && ne < out->edge_capacity) {
          out->edges[2 * ne] = i;
          out->edges[2 * ne + 1] = j;
        }
        ++ne;
      }
    }
  }
  out->edge_count = (uint32_t)ne;
  return PF_OK;
}

pf_status occupancy_launch_check() {
  PF_CUDA(cudaGetLastError());
  PF_CUDA(cudaDeviceSynchronize());
  return PF_OK;
}

}  // namespace
}  // namespace pf

using namespace pf;

extern "C" {

pf_status pf_voxelize_mesh(const pf_mesh* mesh, double particle_radius, uint32_t largest_piece, pf_voxels* out) {
  if (!out) return fail(PF_ERR_INVALID, "voxelize: output is NULL");
  if (!(particle_radius > 0) || !std::isfinite(particle_radius))
    return fail(PF_ERR_INVALID, "voxelize: particleRadius must be positive, got " + std::to_string(particle_radius));
  if (mesh && mesh->n_vertices == 0) return fail(PF_ERR_INVALID, "voxelize: mesh has no vertices");
  std::vector<MeshTri> tris;
  PF_TRY(read_mesh(mesh, &tris));
  // voxelize.ts:164-172: bounds of the vertices
  double mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
  for (uint32_t v = 0; v < mesh->n_vertices; ++v)
    for (int a = 0; a < 3; ++a) {
      mn[a] = std::min(mn[a], (double)mesh->vertices[3ull * v + a]);
      mx[a] = std::max(mx[a], (double)mesh->vertices[3ull * v + a]);
    }
  const double spacing = 2 * particle_radius;
  uint32_t dims[3];
  for (int a = 0; a < 3; ++a) {
    const double d = std::ceil((mx[a] - mn[a]) / spacing);
    if (!(d < 4294967295.0)) return fail(PF_ERR_INVALID, "voxelize: grid too large");
    dims[a] = (uint32_t)std::max(1.0, d);
  }
  const uint64_t cells = (uint64_t)dims[0] * dims[1] * dims[2];
  if (cells > (1ull << 31)) return fail(PF_ERR_INVALID, "voxelize: grid too large");
  DevBuf dt, docc;
  PF_TRY(to_device(tris, &dt));
  PF_CUDA(docc.alloc(std::max<uint64_t>(cells, 1)));
  k_vox_mesh<<<(unsigned)((cells + 255) / 256), 256>>>(static_cast<const MeshTri*>(dt.p), (uint32_t)tris.size(),
                                                        mn[0], mn[1], mn[2], particle_radius, spacing, dims[0],
                                                        dims[1], cells, static_cast<uint8_t*>(docc.p));
  PF_TRY(occupancy_launch_check());
  std::vector<uint8_t> occ(cells);
  PF_CUDA(cudaMemcpy(occ.data(), docc.p, cells, cudaMemcpyDeviceToHost));
  return finish_voxels(occ, mn, particle_radius, spacing, dims[0], dims[1], dims[2], largest_piece != 0, out);
}

pf_status pf_voxelize_sdf(const float* data, const uint32_t res[3], const double origin[3], const double voxel[3],
                          double particle_radius, double dilation, uint32_t largest_piece, pf_voxels* out) {
  if (!out || !data || !res || !origin || !voxel) return fail(PF_ERR_INVALID, "voxelize: NULL argument");
  if (!(particle_radius > 0) || !std::isfinite(particle_radius))
    return fail(PF_ERR_INVALID, "voxelize: particleRadius must be positive, got " + std::to_string(particle_radius));
  if (!std::isfinite(dilation))
    return fail(PF_ERR_INVALID, "voxelize: dilation must be a finite number, got " + std::to_string(dilation));
  for (int a = 0; a < 3; ++a) {
    if (res[a] < 2)
      return fail(PF_ERR_INVALID, "sampleSdf: resolution must be integers >= 2, got [" + std::to_string(res[0]) +
                                      ", " + std::to_string(res[1]) + ", " + std::to_string(res[2]) + "]");
    if (!(voxel[a] > 0) || !std::isfinite(voxel[a]) || !std::isfinite(origin[a]))
      return fail(PF_ERR_INVALID, "voxelize: voxelSize must be positive and origin finite");
  }
  // voxelize.ts:173-177: the field's box
  double mn[3], mx[3];
  for (int a = 0; a < 3; ++a) {
    mn[a] = origin[a];
    mx[a] = origin[a] + (double)res[a] * voxel[a];
  }
  const double spacing = 2 * particle_radius;
  uint32_t dims[3];
  for (int a = 0; a < 3; ++a) {
    const double d = std::ceil((mx[a] - mn[a]) / spacing);
    if (!(d < 4294967295.0)) return fail(PF_ERR_INVALID, "voxelize: grid too large");
    dims[a] = (uint32_t)std::max(1.0, d);
  }
  const uint64_t cells = (uint64_t)dims[0] * dims[1] * dims[2];
  const uint64_t nv = (uint64_t)res[0] * res[1] * res[2];
  if (cells > (1ull << 31) || nv > (1ull << 31)) return fail(PF_ERR_INVALID, "voxelize: grid too large");
  DevBuf dd, docc;
  PF_CUDA(dd.alloc(4 * nv));
  PF_CUDA(cudaMemcpy(dd.p, data, 4 * nv, cudaMemcpyHostToDevice));
  PF_CUDA(docc.alloc(std::max<uint64_t>(cells, 1)));
  k_vox_sdf<<<(unsigned)((cells + 255) / 256), 256>>>(static_cast<const float*>(dd.p), res[0], res[1], res[2],
                                                       origin[0], origin[1], origin[2], voxel[0], voxel[1], voxel[2],
                                                       dilation, particle_radius, spacing, dims[0], dims[1], cells,
                                                       static_cast<uint8_t*>(docc.p));
  PF_TRY(occupancy_launch_check());
  std::vector<uint8_t> occ(cells);
  PF_CUDA(cudaMemcpy(occ.data(), docc.p, cells, cudaMemcpyDeviceToHost));
  return finish_voxels(occ, mn, particle_radius, spacing, dims[0], dims[1], dims[2], largest_piece != 0, out);
}

pf_status pf_bake_sdf(const pf_mesh* mesh, uint32_t resolution, double padding, float* data, double origin[3],
                      double* voxel_size, uint64_t* inconsistent) {
  if (!data || !origin || !voxel_size) return fail(PF_ERR_INVALID, "bakeMeshToSdf: NULL argument");
  std::vector<MeshTri> tris;
  PF_TRY(read_mesh(mesh, &tris));
  // bake.ts:142-172
  if (resolution < 4)
    return fail(PF_ERR_INVALID, "bakeMeshToSdf: resolution must be an integer >= 4, got " + std::to_string(resolution));
  const bool default_pad = padding < 0;
  if (!default_pad && !std::isfinite(padding))
    return fail(PF_ERR_INVALID, "bakeMeshToSdf: padding must be a non-negative finite number, got " +
                                    std::to_string(padding));
  if (tris.empty()) return fail(PF_ERR_INVALID, "bakeMeshToSdf: mesh has zero triangles");
  if ((uint64_t)resolution * resolution * resolution > (1ull << 31))
    return fail(PF_ERR_INVALID, "bakeMeshToSdf: resolution too large");
  // bake.ts:216-255: a cubic grid around the triangles' box
  double mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
  for (const MeshTri& T : tris)
    for (int a = 0; a < 3; ++a) {
      const float lo = std::min(std::min(T.a[a], T.b[a]), T.c[a]), hi = std::max(std::max(T.a[a], T.b[a]), T.c[a]);
      if (lo < mn[a]) mn[a] = lo;
      if (hi > mx[a]) mx[a] = hi;
    }
  std::vector<TriCull> culls;
  std::vector<ChunkBox> boxes;
  order_for_bake(tris, mn, mx, &culls, &boxes);
  if (default_pad) {
    const double extent = std::max(std::max(mx[0] - mn[0], mx[1] - mn[1]), mx[2] - mn[2]);
    const double k = resolution >= 8 ? 2 : 1;
    padding = (k * extent) / ((double)resolution - 2 * k);
  }
  for (int a = 0; a < 3; ++a) {
    mn[a] -= padding;
    mx[a] += padding;
  }
  const double side = std::max(std::max(mx[0] - mn[0], mx[1] - mn[1]), mx[2] - mn[2]);
  const double vs = side / (double)resolution;
  for (int a = 0; a < 3; ++a) origin[a] = 0.5 * (mn[a] + mx[a]) - 0.5 * side;
  *voxel_size = vs;
  const uint64_t n = (uint64_t)resolution * resolution * resolution;
  DevBuf dt, dk, db, dd, dc;
  PF_TRY(to_device(tris, &dt));
  PF_TRY(to_device(culls, &dk));
  PF_TRY(to_device(boxes, &db));
  PF_CUDA(dd.alloc(4 * n));
  PF_CUDA(dc.alloc(8));
  PF_CUDA(cudaMemset(dc.p, 0, 8));
  const uint64_t bricks =
      (uint64_t)div_up(resolution, kBrickX) * div_up(resolution, kBrickY) * div_up(resolution, kBrickZ);
  k_bake<<<(unsigned)((bricks + kBakeWarps - 1) / kBakeWarps), 32 * kBakeWarps>>>(
      static_cast<const MeshTri*>(dt.p), static_cast<const TriCull*>(dk.p), (uint32_t)tris.size(),
      static_cast<const ChunkBox*>(db.p), (uint32_t)boxes.size(), resolution, origin[0], origin[1], origin[2], vs,
      vs * 1e-4, static_cast<float*>(dd.p), static_cast<unsigned long long*>(dc.p));
  PF_TRY(occupancy_launch_check());
  PF_CUDA(cudaMemcpy(data, dd.p, 4 * n, cudaMemcpyDeviceToHost));
  unsigned long long bad = 0;
  PF_CUDA(cudaMemcpy(&bad, dc.p, 8, cudaMemcpyDeviceToHost));
  if (inconsistent) *inconsistent = bad;
  // bake.ts:129-138
  const double frac = (double)bad / (double)n;
  if (frac > 0.01) {
    char pct[32];
    std::snprintf(pct, sizeof pct, "%.2f", frac * 100);
    return fail(PF_ERR_INVALID, "bakeMeshToSdf: mesh appears non-watertight - " + std::to_string(bad) + " of " +
                                    std::to_string(n) + " voxels (" + pct +
                                    "%) had disagreeing axis sign votes. Threshold is 1.00%. Check the input mesh "
                                    "for holes, T-junctions, or non-manifold edges.");
  }
  return PF_OK;
}

}  // extern "C"
