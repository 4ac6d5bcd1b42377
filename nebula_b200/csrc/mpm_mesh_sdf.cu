// mpm_mesh_sdf.cu -- mesh -> Morton-ordered SDF on the GPU (buildMeshSDF,
// src/core/MeshSDF.h:98-132, with transformTriangles, MeshSDF.h:134-141,
// applied on the device).
//
// Same definition as the reference: for every cell centre (ix+0.5, iy+0.5,
// iz+0.5) * cellSize inside gridRes, the distance to the closest triangle,
// signed by that triangle's normal (outside when dot(p - cp, n) >= 0); the
// first triangle wins ties (strict <); cells of the Morton cube beyond gridRes
// hold 1e9.  The closest point is Ericson's complete region test: the
// reference's closestPtOnTriangle (MeshSDF.h:48-78) leaves out the edge-BC
// region and then returns a point outside the triangle (too short, wrongly
// signed distances); that case is added here.
//
// The reference loops over all cells x all triangles on the host.  Here a CTA
// owns 256 consecutive Morton codes (an 8 x 8 x 4 box of cells), one per
// thread, and culls the triangle list for the whole box before any thread
// computes a closest point:
//   1. U = min over triangles and their vertices of the distance from the
//      vertex to the farthest cell centre of the box.  Every cell of the box
//      has a triangle within U, so its closest distance is <= U.  A triangle
//      that may never be closest (a vertex that is not finite, hardly any area)
//      bounds nothing.
//   2. The triangles are staged through shared memory in tiles of 256, in
//      list order.  A triangle whose bounding sphere is farther than U from
//      the box cannot be any cell's closest and is dropped from the tile; the
//      survivors are compacted in list order.
//   3. Each thread walks the survivors, skipping a triangle whose bounding
//      sphere is no closer than min(its best so far, U).
// Every skipped triangle is strictly farther than the cell's closest one (the
// bounds carry a margin above float rounding), so the distances and the
// winning triangle are those of the brute-force loop.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <future>
#include <memory>
#include <system_error>
#include <vector>

#include "mpm_device.cuh"
#include "mpm_engine.h"

namespace nebula {
namespace {

constexpr int kThreads = 256;  // = the Morton codes of one 8 x 8 x 4 box

// Bounding disc of a set of points: a thickness on both sides of a plane
// through the centre, and a radius.  A surface patch much smaller than its
// distance is skipped for every point whose foot lies beside it, where its
// bounding sphere, which is as thick as it is wide, keeps every patch within
// sqrt(2 distance radius) of the foot.  gx..gz is a unit vector or zero (then
// the disc is the sphere).
struct Disc {
  float sx, sy, sz, sr;  // centre, radius
  float gx, gy, gz, gt;  // plane normal, half thickness
};

struct Tri {  // a, b - a, c - a, normal
  float ax, ay, az, bx, by, bz, cx, cy, cz, nx, ny, nz;
};
struct TriS : Tri {  // with a bounding sphere (centre, radius)
  float sx, sy, sz, sr;
};
struct TriD : Tri {  // with a bounding disc
  Disc d;
};

__device__ __forceinline__ float dot3f(float ax, float ay, float az, float bx, float by, float bz) { return ax * bx + ay * by + az * bz; }

// glm::quat * vec3 for a unit quaternion (w, u): v + 2 (w (u x v) + u x (u x v)).
__device__ __forceinline__ void rotate(const MeshPose& q, float& vx, float& vy, float& vz) {
  const float cx = q.q[2] * vz - q.q[3] * vy, cy = q.q[3] * vx - q.q[1] * vz, cz = q.q[1] * vy - q.q[2] * vx;
  const float dx = q.q[2] * cz - q.q[3] * cy, dy = q.q[3] * cx - q.q[1] * cz, dz = q.q[1] * cy - q.q[2] * cx;
  vx += (cx * q.q[0] + dx) * 2.0f;
  vy += (cy * q.q[0] + dy) * 2.0f;
  vz += (cz * q.q[0] + dz) * 2.0f;
}

// Triangle k as (normal, v0, v1, v2), the binary STL order, after the pose.
__device__ __forceinline__ void loadTri(const float4* __restrict__ t4, uint32_t k, const MeshPose& p, float (&v)[12]) {
  const float4 r0 = __ldg(t4 + 3 * size_t(k)), r1 = __ldg(t4 + 3 * size_t(k) + 1), r2 = __ldg(t4 + 3 * size_t(k) + 2);
  v[0] = r0.x; v[1] = r0.y; v[2] = r0.z; v[3] = r0.w;
  v[4] = r1.x; v[5] = r1.y; v[6] = r1.z; v[7] = r1.w;
  v[8] = r2.x; v[9] = r2.y; v[10] = r2.z; v[11] = r2.w;
  if (p.posed) {
#pragma unroll
    for (int j = 0; j < 4; ++j) rotate(p, v[3 * j], v[3 * j + 1], v[3 * j + 2]);
#pragma unroll
    for (int j = 1; j < 4; ++j) {
      v[3 * j] += p.t[0];
      v[3 * j + 1] += p.t[1];
      v[3 * j + 2] += p.t[2];
    }
  }
}

// True when every point of the disc's set is at least `best` away from p, by a
// margin: `pad` widens the disc, and the factors cover the float rounding of
// the plane distance and, under the root, of the lateral one.  False when the
// disc holds a NaN.
__device__ __forceinline__ bool discBeyond(const Disc& d, float px, float py, float pz, float pad, float best) {
  const float ex = px - d.sx, ey = py - d.sy, ez = pz - d.sz;
  const float q = dot3f(ex, ey, ez, ex, ey, ez);
  const float h = dot3f(ex, ey, ez, d.gx, d.gy, d.gz);
  const float lat = sqrtf(fmaxf(q * (1.0f - 4e-6f) - h * h, 0.f)) - d.sr - pad;
  const float out = fabsf(h) * (1.0f - 2e-6f) - d.gt - pad;
  const float l = fmaxf(lat, 0.f), o = fmaxf(out, 0.f);
  // fmaxf drops a NaN: q, h, sr and gt are tested through the plain difference
  return (l * l + o * o) * (1.0f - 1e-6f) >= best * best && lat == lat && out == out && q == q;
}

// Disc of the triangle (a, a + b, a + c).
__device__ __forceinline__ Disc triDisc(const Tri& t, float eps) {
  Disc d;
  d.sx = t.ax + (t.bx + t.cx) * (1.0f / 3.0f);
  d.sy = t.ay + (t.by + t.cy) * (1.0f / 3.0f);
  d.sz = t.az + (t.bz + t.cz) * (1.0f / 3.0f);
  float gx = t.by * t.cz - t.bz * t.cy, gy = t.bz * t.cx - t.bx * t.cz, gz = t.bx * t.cy - t.by * t.cx;
  const float g2 = dot3f(gx, gy, gz, gx, gy, gz);
  const float inv = g2 > 1e-30f && g2 < 1e30f ? rsqrtf(g2) : 0.f;
  d.gx = gx * inv;
  d.gy = gy * inv;
  d.gz = gz * inv;
  float rr = 0.f, th = 0.f;
  auto vertex = [&](float x, float y, float z) {
    const float dx = x - d.sx, dy = y - d.sy, dz = z - d.sz;
    const float r2 = dot3f(dx, dy, dz, dx, dy, dz);
    rr = r2 > rr || r2 != r2 ? r2 : rr;
    th = fmaxf(th, fabsf(dot3f(dx, dy, dz, d.gx, d.gy, d.gz)));
  };
  vertex(t.ax, t.ay, t.az);
  vertex(t.ax + t.bx, t.ay + t.by, t.az + t.bz);
  vertex(t.ax + t.cx, t.ay + t.cy, t.az + t.cz);
  d.sr = sqrtf(rr) * 1.0001f + eps;  // covers the triangle despite rounding
  d.gt = th * 1.0001f + eps;
  return d;
}

// a b - c d with every operation rounded: zero where the products are equal.  A
// fused multiply-add leaves the rounding of one product, and a triangle with two
// equal vertices then falls through its edge tests.
__device__ __forceinline__ float cross2(float a, float b, float c, float d) { return __fsub_rn(__fmul_rn(a, b), __fmul_rn(c, d)); }

// Closest point of triangle (a, a + ab, a + ac) to p (MeshSDF.h:48-78).
__device__ __forceinline__ void closestOnTriangle(const Tri& t, float px, float py, float pz, float& qx, float& qy, float& qz) {
  const float apx = px - t.ax, apy = py - t.ay, apz = pz - t.az;
  const float d1 = dot3f(t.bx, t.by, t.bz, apx, apy, apz), d2 = dot3f(t.cx, t.cy, t.cz, apx, apy, apz);
  if (d1 <= 0.f && d2 <= 0.f) {
    qx = t.ax; qy = t.ay; qz = t.az;
    return;
  }
  const float bpx = apx - t.bx, bpy = apy - t.by, bpz = apz - t.bz;  // p - b
  const float d3 = dot3f(t.bx, t.by, t.bz, bpx, bpy, bpz), d4 = dot3f(t.cx, t.cy, t.cz, bpx, bpy, bpz);
  if (d3 >= 0.f && d4 <= d3) {
    qx = t.ax + t.bx; qy = t.ay + t.by; qz = t.az + t.bz;
    return;
  }
  const float vc = cross2(d1, d4, d3, d2);
  if (vc <= 0.f && d1 >= 0.f && d3 <= 0.f) {
    const float v = d1 / (d1 - d3);
    qx = t.ax + v * t.bx; qy = t.ay + v * t.by; qz = t.az + v * t.bz;
    return;
  }
  const float cpx = apx - t.cx, cpy = apy - t.cy, cpz = apz - t.cz;  // p - c
  const float d5 = dot3f(t.bx, t.by, t.bz, cpx, cpy, cpz), d6 = dot3f(t.cx, t.cy, t.cz, cpx, cpy, cpz);
  if (d6 >= 0.f && d5 <= d6) {
    qx = t.ax + t.cx; qy = t.ay + t.cy; qz = t.az + t.cz;
    return;
  }
  const float vb = cross2(d5, d2, d1, d6);
  if (vb <= 0.f && d2 >= 0.f && d6 <= 0.f) {
    const float w = d2 / (d2 - d6);
    qx = t.ax + w * t.cx; qy = t.ay + w * t.cy; qz = t.az + w * t.cz;
    return;
  }
  const float va = cross2(d3, d6, d5, d4);
  if (va <= 0.f && (d4 - d3) >= 0.f && (d5 - d6) >= 0.f) {  // edge BC (Ericson 5.1.5; left out by MeshSDF.h:76-78)
    const float w = (d4 - d3) / ((d4 - d3) + (d5 - d6));
    qx = t.ax + t.bx + w * (t.cx - t.bx); qy = t.ay + t.by + w * (t.cy - t.by); qz = t.az + t.bz + w * (t.cz - t.bz);
    return;
  }
  const float sum = va + vb + vc;
  const float v = vb / sum, w = vc / sum;
  qx = t.ax + v * t.bx + w * t.cx;
  qy = t.ay + v * t.by + w * t.cy;
  qz = t.az + v * t.bz + w * t.cz;
}

// Lower bound of the distance from p to the disc's set (NaN when the disc
// holds one).
__device__ __forceinline__ float discBound(const Disc& d, float px, float py, float pz, float pad) {
  const float ex = px - d.sx, ey = py - d.sy, ez = pz - d.sz;
  const float q = dot3f(ex, ey, ez, ex, ey, ez);
  const float h = dot3f(ex, ey, ez, d.gx, d.gy, d.gz);
  const float lat = sqrtf(fmaxf(q * (1.0f - 4e-6f) - h * h, 0.f)) - d.sr - pad;
  const float out = fabsf(h) * (1.0f - 2e-6f) - d.gt - pad;
  const float l = fmaxf(lat, 0.f), o = fmaxf(out, 0.f);
  const float nan = (lat + out + q) * 0.f;  // keeps a NaN that fmaxf dropped
  return sqrtf(l * l + o * o) * (1.0f - 1e-6f) + (nan == nan ? 0.f : nan);
}

// Whether a (posed) triangle is sure to be as close as its vertices: nine finite
// coordinates and some area.  (A NaN or an overflow fails the comparison.  With a
// NaN the closest point is NaN; with hardly any area rounding decides the region
// test, and the point may lie far off: of 4,000,000 points around triangles 100,000
// times as long as wide 30 got one farther than the nearest vertex, by up to 9
// times the distance, at 10,000 times 5, at 1,000 times 1; at 500 times, where the
// line is, 1 of 40,000,000, by 0.8 of it.)  A list of slivers alone bounds nothing
// and is walked whole: 1,000 of them 100,000 times as long as wide on 128^3 0.40 ->
// 2.15 ms.
__device__ __forceinline__ bool canBeClosest(const float (&v)[12]) {
  const float ax = v[6] - v[3], ay = v[7] - v[4], az = v[8] - v[5], cx = v[9] - v[3], cy = v[10] - v[4], cz = v[11] - v[5];
  const float gx = ay * cz - az * cy, gy = az * cx - ax * cz, gz = ax * cy - ay * cx;
  const float e2 = dot3f(ax, ay, az, ax, ay, az) + dot3f(cx, cy, cz, cx, cy, cz);
  return dot3f(gx, gy, gz, gx, gy, gz) > 1e-6f * e2 * e2;
}

// Squared distance from the triangle's nearest vertex to the farthest point of a box.
__device__ __forceinline__ float farthestCell2(const float (&v)[12], float lox, float loy, float loz, float hix, float hiy, float hiz) {
  float m2 = INFINITY;
#pragma unroll
  for (int j = 1; j < 4; ++j) {
    const float ex = fmaxf(v[3 * j] - lox, hix - v[3 * j]);
    const float ey = fmaxf(v[3 * j + 1] - loy, hiy - v[3 * j + 1]);
    const float ez = fmaxf(v[3 * j + 2] - loz, hiz - v[3 * j + 2]);
    m2 = fminf(m2, ex * ex + ey * ey + ez * ez);
  }
  return m2;
}

__global__ void __launch_bounds__(kThreads) k_mesh_sdf(const float4* __restrict__ tris, uint32_t n, MeshPose pose, int rx, int ry, int rz,
                                                       uint32_t totalCells, float cs, float eps, float* __restrict__ sdf) {
  __shared__ TriS tile[kThreads];
  __shared__ uint32_t warpCount[kThreads / 32];
  __shared__ uint32_t boundBits;
  const uint32_t base = blockIdx.x * kThreads;
  const uint32_t code = base + threadIdx.x;
  int bx0, by0, bz0;
  mortonDecode(base, bx0, by0, bz0);
  if (bx0 >= rx || by0 >= ry || bz0 >= rz) {  // the whole box lies in the padding of the Morton cube
    if (code < totalCells) sdf[code] = 1e9f;
    return;
  }
  int bx1, by1, bz1;
  mortonDecode(base | uint32_t(kThreads - 1), bx1, by1, bz1);
  const float lox = (float(bx0) + 0.5f) * cs, loy = (float(by0) + 0.5f) * cs, loz = (float(bz0) + 0.5f) * cs;
  const float hix = (float(min(bx1, rx - 1)) + 0.5f) * cs, hiy = (float(min(by1, ry - 1)) + 0.5f) * cs, hiz = (float(min(bz1, rz - 1)) + 0.5f) * cs;

  // 1. U^2 over the box
  if (threadIdx.x == 0) boundBits = __float_as_uint(INFINITY);
  __syncthreads();
  // A triangle that may never be closest bounds nothing.  A thread with one
  // triangle looks at it first; one with several looks at the nearest alone, and
  // leaves the bound to the other threads if it is such a triangle.
  float u2 = INFINITY;
  if (n <= kThreads) {
    if (threadIdx.x < n) {
      float v[12];
      loadTri(tris, threadIdx.x, pose, v);
      if (canBeClosest(v)) u2 = farthestCell2(v, lox, loy, loz, hix, hiy, hiz);
    }
  } else {
    uint32_t nearest = n;
#pragma unroll 4
    for (uint32_t k = threadIdx.x; k < n; k += kThreads) {
      float v[12];
      loadTri(tris, k, pose, v);
      const float m2 = farthestCell2(v, lox, loy, loz, hix, hiy, hiz);
      nearest = m2 < u2 ? k : nearest;
      u2 = fminf(u2, m2);
    }
    if (nearest < n) {
      float v[12];
      loadTri(tris, nearest, pose, v);
      if (!canBeClosest(v)) u2 = INFINITY;
    }
  }
  u2 = __uint_as_float(__reduce_min_sync(0xffffffffu, __float_as_uint(u2)));  // non-negative floats order as their bits
  if ((threadIdx.x & 31) == 0) atomicMin(&boundBits, __float_as_uint(u2));
  __syncthreads();
  const float U = sqrtf(__uint_as_float(boundBits)) * (1.0f + 1e-5f) + eps;

  int ix = 0, iy = 0, iz = 0;
  if (code < totalCells) mortonDecode(code, ix, iy, iz);
  const bool inside = code < totalCells && ix < rx && iy < ry && iz < rz;
  const float px = (float(ix) + 0.5f) * cs, py = (float(iy) + 0.5f) * cs, pz = (float(iz) + 0.5f) * cs;
  float best = 1e9f;
  bool outer = true;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (uint32_t t0 = 0; t0 < n; t0 += kThreads) {
    // 2. stage the tile's triangles that can be closest to some cell of the box
    const uint32_t k = t0 + threadIdx.x;
    TriS t;
    bool keep = false;
    if (k < n) {
      float v[12];
      loadTri(tris, k, pose, v);
      t.nx = v[0]; t.ny = v[1]; t.nz = v[2];
      t.ax = v[3]; t.ay = v[4]; t.az = v[5];
      t.bx = v[6] - v[3]; t.by = v[7] - v[4]; t.bz = v[8] - v[5];
      t.cx = v[9] - v[3]; t.cy = v[10] - v[4]; t.cz = v[11] - v[5];
      t.sx = (v[3] + v[6] + v[9]) * (1.0f / 3.0f);
      t.sy = (v[4] + v[7] + v[10]) * (1.0f / 3.0f);
      t.sz = (v[5] + v[8] + v[11]) * (1.0f / 3.0f);
      float rr = 0.f;
#pragma unroll
      for (int j = 1; j < 4; ++j) {
        const float dx = v[3 * j] - t.sx, dy = v[3 * j + 1] - t.sy, dz = v[3 * j + 2] - t.sz;
        rr = fmaxf(rr, dx * dx + dy * dy + dz * dz);
      }
      t.sr = sqrtf(rr) * 1.0001f + eps;  // covers the triangle despite rounding
      const float gx = fmaxf(fmaxf(lox - t.sx, t.sx - hix), 0.f), gy = fmaxf(fmaxf(loy - t.sy, t.sy - hiy), 0.f),
                  gz = fmaxf(fmaxf(loz - t.sz, t.sz - hiz), 0.f);
      keep = sqrtf(gx * gx + gy * gy + gz * gz) - t.sr <= U;
    }
    const uint32_t mask = __ballot_sync(0xffffffffu, keep);
    __syncthreads();  // the previous tile has been consumed
    if (lane == 0) warpCount[warp] = __popc(mask);
    __syncthreads();
    uint32_t off = 0, m = 0;
#pragma unroll
    for (int w = 0; w < kThreads / 32; ++w) {
      const uint32_t c = warpCount[w];
      off += uint32_t(w) < warp ? c : 0u;
      m += c;
    }
    if (keep) tile[off + __popc(mask & ((1u << lane) - 1u))] = t;
    __syncthreads();
    if (!inside) continue;
    // 3. closest points against the survivors, in list order
    for (uint32_t j = 0; j < m; ++j) {
      const TriS& s = tile[j];
      const float ex = px - s.sx, ey = py - s.sy, ez = pz - s.sz;
      const float dc = sqrtf(ex * ex + ey * ey + ez * ez);
      if (dc - s.sr >= fminf(best, U)) continue;  // every point of the triangle is at least this far
      float qx, qy, qz;
      closestOnTriangle(s, px, py, pz, qx, qy, qz);
      const float dx = px - qx, dy = py - qy, dz = pz - qz;
      const float d = sqrtf(dx * dx + dy * dy + dz * dz);
      if (d < best) {
        best = d;
        outer = dot3f(dx, dy, dz, s.nx, s.ny, s.nz) >= 0.f;
      }
    }
  }
  if (code < totalCells) sdf[code] = inside ? (outer ? best : -best) : 1e9f;
}

// ---------------------------------------------------------------- prepared meshes
// The same SDF from a prepared mesh: triangles in an order of median splits
// (orderTriangles), in leaves of 8, 64 leaves to a group and 64 groups to a
// block, with a bounding disc (mesh frame) at each level.  A warp takes 32
// consecutive Morton codes (a 4 x 4 x 2 box of cells) and works alone:
//   1. A greedy descent to the leaf nearest the box's centre: the distance to a
//      vertex of it bounds every lane's distance from above.
//   2. Blocks, groups and leaves are tested 32 at a time, one per lane,
//      against the whole box (the centre's bound less the box's radius) and
//      the lanes' largest bound.  Every lane takes the distance to one vertex
//      of each surviving leaf: the nearest of these is within a leaf's width
//      of the foot, so it is its distance to second order.
//   3. The leaves that gave the bounds are taken first, then the tree is walked
//      again with the distances they leave: a surviving leaf is tested by every
//      lane for its own cell and taken if some lane needs it.  Leaves are posed
//      into shared memory four at a time, one triangle per lane, and every lane
//      walks the 32 triangles, computing closest points for those whose disc
//      comes nearer than its bound.
// What bounds it is arithmetic (a bumpy sphere of 20,480 triangles moved to a new
// pose, 128^3: 1.50 ms, where clusters of 32 with bounding spheres took 4.3).
// Without step 2 a warp inside a closed mesh, where many leaves are almost equally
// far, walked 518 triangles on average.
// The discs are not posed: the cell goes to the mesh frame by the inverse
// pose, and `pad` covers the rounding of that (and a quaternion off unit
// length).  Triangles are visited out of list order, so a tie in distance
// goes to the smaller list index: the first triangle of the list reaching the
// minimum, as in the brute-force loop.

__device__ __forceinline__ Disc loadDisc(const float4* __restrict__ discs, uint32_t i) {
  const float4 a = __ldg(discs + 2 * size_t(i)), b = __ldg(discs + 2 * size_t(i) + 1);
  return Disc{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
}

// Index in [0, count) of the disc of discs[base ...] with the smallest bound at p (whole warp).
__device__ __forceinline__ uint32_t nearestDisc(const float4* __restrict__ discs, uint32_t base, uint32_t count, float px, float py, float pz) {
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t key = 0xffffffffu, at = 0;
  for (uint32_t i = lane; i < count; i += 32u) {
    const uint32_t k = __float_as_uint(discBound(loadDisc(discs, base + i), px, py, pz, 0.f));  // non-negative floats order as their bits
    if (k < key) {
      key = k;
      at = i;
    }
  }
  const uint32_t m = __reduce_min_sync(0xffffffffu, key);
  return __shfl_sync(0xffffffffu, at, __ffs(__ballot_sync(0xffffffffu, key == m)) - 1);
}

__global__ void __launch_bounds__(kThreads) k_mesh_sdf_discs(const float4* __restrict__ tris, const uint32_t* __restrict__ index,
                                                             const float4* __restrict__ discs, const float4* __restrict__ points, uint32_t n, uint32_t nLeaves, uint32_t nGroups,
                                                             uint32_t nBlocks, MeshPose pose, int rx, int ry, int rz, uint32_t totalCells, float cs,
                                                             float eps, float pad, float* __restrict__ sdf) {
  constexpr uint32_t kFull = 0xffffffffu, kTileLeaves = 32u / kMeshLeaf;
  __shared__ __align__(16) TriD tiles[kThreads];
  __shared__ uint32_t tileIdx[kThreads];
  const uint32_t code = blockIdx.x * kThreads + threadIdx.x;
  const uint32_t lane = threadIdx.x & 31u;
  TriD* tile = tiles + (threadIdx.x & ~31u);
  uint32_t* ids = tileIdx + (threadIdx.x & ~31u);
  int ix = 0, iy = 0, iz = 0;
  if (code < totalCells) mortonDecode(code, ix, iy, iz);
  const bool inside = code < totalCells && ix < rx && iy < ry && iz < rz;
  if (!__any_sync(kFull, inside)) {  // the whole box lies in the padding of the Morton cube
    if (code < totalCells) sdf[code] = 1e9f;
    return;
  }
  const float px = (float(ix) + 0.5f) * cs, py = (float(iy) + 0.5f) * cs, pz = (float(iz) + 0.5f) * cs;
  // cell centre and box centre in the mesh frame
  const float bx = (float(__shfl_sync(kFull, ix, 0)) + 2.0f) * cs, by = (float(__shfl_sync(kFull, iy, 0)) + 2.0f) * cs,
              bz = (float(__shfl_sync(kFull, iz, 0)) + 1.0f) * cs;
  float mx = px, my = py, mz = pz, cx = bx, cy = by, cz = bz;
  if (pose.posed) {
    MeshPose inv = pose;
    inv.q[1] = -pose.q[1];
    inv.q[2] = -pose.q[2];
    inv.q[3] = -pose.q[3];
    mx -= pose.t[0]; my -= pose.t[1]; mz -= pose.t[2];
    cx -= pose.t[0]; cy -= pose.t[1]; cz -= pose.t[2];
    rotate(inv, mx, my, mz);
    rotate(inv, cx, cy, cz);
  }
  const float boxR = 2.1795f * cs * 1.0001f + pad;  // half diagonal of 3 x 3 x 1 cells
  float best = inside ? 1e9f : 0.f;  // a lane without a cell needs nothing
  float bound = best;                // every lane's distance is at most this
  uint32_t bestIdx = 0xffffffffu;
  bool outer = true;
  float most = 1e9f;           // the lanes' largest bound
  uint32_t hot = 0, nHot = 0;  // collected leaves, one in each of the lanes 0..nHot-1
  uint32_t near = 0;           // the leaf that gave the bound

  auto tighten = [&]() { most = __uint_as_float(__reduce_max_sync(kFull, __float_as_uint(bound))); };
  // the distance to a vertex of leaf l
  auto vertexBound = [&](uint32_t l) {
    const float4 v = __ldg(points + l);
    const float ex = mx - v.x, ey = my - v.y, ez = mz - v.z;
    const float d = sqrtf(dot3f(ex, ey, ez, ex, ey, ez)) * (1.0f + 1e-5f) + pad;
    if (d < bound) {  // (not with a NaN)
      bound = d;
      near = l;
    }
  };
  auto flush = [&]() {
    const uint32_t leaf = __shfl_sync(kFull, hot, lane >> 3);
    const uint32_t t = leaf * kMeshLeaf + (lane & 7u);
    const bool valid = (lane >> 3) < nHot && t < n;
    if (valid) {
      float v[12];
      loadTri(tris, t, pose, v);
      TriD s;
      s.nx = v[0]; s.ny = v[1]; s.nz = v[2];
      s.ax = v[3]; s.ay = v[4]; s.az = v[5];
      s.bx = v[6] - v[3]; s.by = v[7] - v[4]; s.bz = v[8] - v[5];
      s.cx = v[9] - v[3]; s.cy = v[10] - v[4]; s.cz = v[11] - v[5];
      s.d = triDisc(s, eps);
      tile[lane] = s;
      ids[lane] = index[t];
    }
    uint32_t mask = __ballot_sync(kFull, valid);
    __syncwarp();
    while (mask) {
      const int j = __ffs(mask) - 1;
      mask &= mask - 1u;
      const TriD& s = tile[j];
      if (discBeyond(s.d, px, py, pz, 0.f, bound)) continue;  // every point of the triangle is at least this far
      float qx, qy, qz;
      closestOnTriangle(s, px, py, pz, qx, qy, qz);
      const float dx = px - qx, dy = py - qy, dz = pz - qz;
      const float d = sqrtf(dx * dx + dy * dy + dz * dz);
      const uint32_t id = ids[j];
      if (inside && (d < best || (d == best && id < bestIdx))) {
        best = d;
        bestIdx = id;
        outer = dot3f(dx, dy, dz, s.nx, s.ny, s.nz) >= 0.f;
        bound = fminf(bound, d);
      }
    }
    __syncwarp();  // the tile is consumed
    nHot = 0;
    tighten();
  };
  // discs [from, from + 32) of a level, up to `end`, that the box may need (one bit each)
  auto needed = [&](uint32_t base, uint32_t from, uint32_t end) {
    const uint32_t i = from + lane;
    return __ballot_sync(kFull, i < end && !(discBound(loadDisc(discs, base + i), cx, cy, cz, pad) - boxR >= most));
  };
  // walk(leaf, group): every leaf the box may need, `group` after each group
  auto walk = [&](auto&& leaf, auto&& group) {
    for (uint32_t b0 = 0; b0 < nBlocks; b0 += 32u) {
      uint32_t bm = needed(nLeaves + nGroups, b0, nBlocks);
      while (bm) {
        const uint32_t b = b0 + uint32_t(__ffs(bm) - 1);
        bm &= bm - 1u;
        const uint32_t gEnd = min((b + 1u) * kMeshFan, nGroups);
        for (uint32_t g0 = b * kMeshFan; g0 < gEnd; g0 += 32u) {
          uint32_t gm = needed(nLeaves, g0, gEnd);
          while (gm) {
            const uint32_t g = g0 + uint32_t(__ffs(gm) - 1);
            gm &= gm - 1u;
            const uint32_t lEnd = min((g + 1u) * kMeshFan, nLeaves);
            for (uint32_t l0 = g * kMeshFan; l0 < lEnd; l0 += 32u) {
              uint32_t lm = needed(0u, l0, lEnd);
              while (lm) {
                const uint32_t l = l0 + uint32_t(__ffs(lm) - 1);
                lm &= lm - 1u;
                leaf(l);
              }
            }
            group();
          }
        }
      }
    }
  };

  // Small meshes leave steps out, whose fixed cost per warp is most of their
  // time.  Up to 32 triangles are one tile: no search (a soup of 4 on 128^3 108 ->
  // 54 us, of 32 183 -> 145; the clusters with bounding spheres that the tree
  // replaced took 95 and 201).  Up to a group of leaves, every leaf gives its
  // bound, without the descent and the first walk (40 triangles 197 -> 157 us, the
  // clusters 161; 300: 322 -> 294, the clusters 304); from there on the walk pays
  // (450: 327 -> 322, 512: 345 -> 347).
  if (nLeaves <= kTileLeaves) {
    for (uint32_t l = 0; l < nLeaves; ++l) vertexBound(l);
    hot = lane;
    nHot = nLeaves;
  } else {
    if (nLeaves <= kMeshFan) {
      // 1., 2. a bound per lane
      for (uint32_t l = 0; l < nLeaves; ++l) vertexBound(l);
      tighten();
    } else {
      // 1. the leaf nearest the box's centre
      const uint32_t b = nearestDisc(discs, nLeaves + nGroups, nBlocks, cx, cy, cz);
      const uint32_t g = b * kMeshFan + nearestDisc(discs, nLeaves + b * kMeshFan, min(kMeshFan, nGroups - b * kMeshFan), cx, cy, cz);
      near = g * kMeshFan + nearestDisc(discs, g * kMeshFan, min(kMeshFan, nLeaves - g * kMeshFan), cx, cy, cz);
      vertexBound(near);
      tighten();
      // 2. a bound per lane
      walk(vertexBound, tighten);
    }
    // 3. the closest triangles: first the leaves that gave the bounds (the
    // nearest leaf where no vertex may bound: a mesh of slivers)
    auto collect = [&](uint32_t l) {
      if (lane == nHot) hot = l;
      if (++nHot == kTileLeaves) flush();
    };
    uint32_t todo = __ballot_sync(kFull, inside);
    while (todo) {
      const uint32_t l = __shfl_sync(kFull, near, __ffs(todo) - 1);
      todo &= ~__ballot_sync(kFull, near == l);
      collect(l);
    }
    if (nHot) flush();
    walk(
        [&](uint32_t l) {
          if (__any_sync(kFull, inside && near == l)) return;  // done above
          if (__any_sync(kFull, !discBeyond(loadDisc(discs, l), mx, my, mz, pad, bound))) collect(l);
        },
        [] {});
  }
  if (nHot) flush();
  if (code < totalCells) sdf[code] = inside ? (outer ? best : -best) : 1e9f;
}

// ------------------------------------------------------------------ the reference's closest point
// closestPtOnTriangle (MeshSDF.h:48-78) step for step, including its gap: a
// point whose closest feature is edge BC falls through to the barycentric
// face case and gets the projection onto the triangle's plane, outside the
// triangle.  That point can be nearer than any point of the triangle, so no
// distance bound culls triangles here: every cell visits every triangle, as
// buildMeshSDF's loop does (MeshSDF.h:113-126).
struct TriRef {  // posed vertices and normal
  float ax, ay, az, bx, by, bz, cx, cy, cz, nx, ny, nz;
};

// Float operations rounded one at a time, in the reference's order (no fused
// multiply-add): the missing region makes the result jump where a region test
// flips, so its arithmetic is kept operation for operation.
__device__ __forceinline__ float mulr(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float addr(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float subr(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float dotr(float ax, float ay, float az, float bx, float by, float bz) {
  return addr(addr(mulr(ax, bx), mulr(ay, by)), mulr(az, bz));
}

__device__ __forceinline__ void closestRef(const TriRef& t, float px, float py, float pz, float& qx, float& qy, float& qz) {
  const float abx = subr(t.bx, t.ax), aby = subr(t.by, t.ay), abz = subr(t.bz, t.az);
  const float acx = subr(t.cx, t.ax), acy = subr(t.cy, t.ay), acz = subr(t.cz, t.az);
  const float apx = subr(px, t.ax), apy = subr(py, t.ay), apz = subr(pz, t.az);
  const float d1 = dotr(abx, aby, abz, apx, apy, apz), d2 = dotr(acx, acy, acz, apx, apy, apz);
  if (d1 <= 0.f && d2 <= 0.f) {
    qx = t.ax; qy = t.ay; qz = t.az;
    return;
  }
  const float bpx = subr(px, t.bx), bpy = subr(py, t.by), bpz = subr(pz, t.bz);
  const float d3 = dotr(abx, aby, abz, bpx, bpy, bpz), d4 = dotr(acx, acy, acz, bpx, bpy, bpz);
  if (d3 >= 0.f && d4 <= d3) {
    qx = t.bx; qy = t.by; qz = t.bz;
    return;
  }
  const float vc = subr(mulr(d1, d4), mulr(d3, d2));
  if (vc <= 0.f && d1 >= 0.f && d3 <= 0.f) {
    const float v = __fdiv_rn(d1, subr(d1, d3));
    qx = addr(t.ax, mulr(v, abx)); qy = addr(t.ay, mulr(v, aby)); qz = addr(t.az, mulr(v, abz));
    return;
  }
  const float cpx = subr(px, t.cx), cpy = subr(py, t.cy), cpz = subr(pz, t.cz);
  const float d5 = dotr(abx, aby, abz, cpx, cpy, cpz), d6 = dotr(acx, acy, acz, cpx, cpy, cpz);
  if (d6 >= 0.f && d5 <= d6) {
    qx = t.cx; qy = t.cy; qz = t.cz;
    return;
  }
  const float vb = subr(mulr(d5, d2), mulr(d1, d6));
  if (vb <= 0.f && d2 >= 0.f && d6 <= 0.f) {
    const float w = __fdiv_rn(d2, subr(d2, d6));
    qx = addr(t.ax, mulr(w, acx)); qy = addr(t.ay, mulr(w, acy)); qz = addr(t.az, mulr(w, acz));
    return;
  }
  const float va = subr(mulr(d3, d6), mulr(d5, d4));
  const float sum = addr(addr(va, vb), vc);
  const float v = __fdiv_rn(vb, sum), w = __fdiv_rn(vc, sum);
  qx = addr(addr(t.ax, mulr(v, abx)), mulr(w, acx));
  qy = addr(addr(t.ay, mulr(v, aby)), mulr(w, acy));
  qz = addr(addr(t.az, mulr(v, abz)), mulr(w, acz));
}

// One thread per Morton code; the (posed) triangles pass through shared
// memory in tiles of kThreads.  `index` (may be null: list order) gives each
// triangle's place in the caller's list, so a list in another order still
// resolves equal distances to the first triangle of the caller's list, as
// the strict < of the reference's loop does.
__global__ void __launch_bounds__(kThreads) k_mesh_sdf_ref(const float4* __restrict__ tris, const uint32_t* __restrict__ index, uint32_t n,
                                                           MeshPose pose, int rx, int ry, int rz, uint32_t totalCells, float cs,
                                                           float* __restrict__ sdf) {
  __shared__ TriRef tile[kThreads];
  __shared__ uint32_t tileIdx[kThreads];
  const uint32_t code = blockIdx.x * kThreads + threadIdx.x;
  int ix, iy, iz;
  mortonDecode(code, ix, iy, iz);
  const bool inside = code < totalCells && ix < rx && iy < ry && iz < rz;
  const float px = mulr(addr(float(ix), 0.5f), cs), py = mulr(addr(float(iy), 0.5f), cs), pz = mulr(addr(float(iz), 0.5f), cs);
  float best = 1e9f;
  uint32_t bestIdx = 0xffffffffu;
  bool outer = true;
  for (uint32_t t0 = 0; t0 < n; t0 += kThreads) {
    __syncthreads();  // the previous tile is consumed
    const uint32_t t = t0 + threadIdx.x;
    if (t < n) {
      float v[12];
      loadTri(tris, t, pose, v);
      tile[threadIdx.x] = TriRef{v[3], v[4], v[5], v[6], v[7], v[8], v[9], v[10], v[11], v[0], v[1], v[2]};
      tileIdx[threadIdx.x] = index ? __ldg(index + t) : t;
    }
    __syncthreads();
    if (!inside) continue;
    const uint32_t m = min(uint32_t(kThreads), n - t0);
    for (uint32_t j = 0; j < m; ++j) {
      const TriRef& tr = tile[j];
      float qx, qy, qz;
      closestRef(tr, px, py, pz, qx, qy, qz);
      const float dx = subr(px, qx), dy = subr(py, qy), dz = subr(pz, qz);
      const float d = __fsqrt_rn(dotr(dx, dy, dz, dx, dy, dz));
      const uint32_t id = tileIdx[j];
      if (d < best || (d == best && id < bestIdx)) {
        best = d;
        bestIdx = id;
        outer = dotr(dx, dy, dz, tr.nx, tr.ny, tr.nz) >= 0.f;
      }
    }
  }
  if (code < totalCells) sdf[code] = inside ? (outer ? best : -best) : 1e9f;
}

}  // namespace

cudaError_t launchMeshSdfReference(const float* dTris, const uint32_t* dIndex, uint32_t n, const MeshPose& pose, const uint32_t res[3],
                                   uint32_t totalCells, float cellSize, float* dSdf, cudaStream_t s, uint64_t* launches) {
  if (totalCells == 0) return cudaSuccess;
  k_mesh_sdf_ref<<<(totalCells + kThreads - 1) / kThreads, kThreads, 0, s>>>(reinterpret_cast<const float4*>(dTris), dIndex, n, pose, int(res[0]),
                                                                             int(res[1]), int(res[2]), totalCells, cellSize, dSdf);
  ++*launches;
  return cudaGetLastError();
}

cudaError_t launchMeshSdf(const float* dTris, uint32_t n, const MeshPose& pose, const uint32_t res[3], uint32_t totalCells, float cellSize,
                          float* dSdf, cudaStream_t s, uint64_t* launches) {
  if (totalCells == 0) return cudaSuccess;
  // Margin of the culling bounds over float rounding: distances within the
  // domain are O(cellSize * cubeRes).
  const float extent = cellSize * float(domainCubeRes(res));
  const float eps = 1e-5f * fmaxf(extent, 1.0f);
  k_mesh_sdf<<<(totalCells + kThreads - 1) / kThreads, kThreads, 0, s>>>(reinterpret_cast<const float4*>(dTris), n, pose, int(res[0]),
                                                                         int(res[1]), int(res[2]), totalCells, cellSize, eps, dSdf);
  ++*launches;
  return cudaGetLastError();
}

cudaError_t launchMeshSdfPrepared(const PreparedMesh& m, const MeshPose& pose, const uint32_t res[3], uint32_t totalCells, float cellSize,
                                  float* dSdf, cudaStream_t s, uint64_t* launches) {
  if (totalCells == 0) return cudaSuccess;
  const float extent = cellSize * float(domainCubeRes(res));
  const float eps = 1e-5f * fmaxf(extent, 1.0f);
  // rounding of a cell taken to the mesh frame, and a quaternion off unit length
  float pad = eps;
  if (pose.posed) {
    const float q2 = pose.q[0] * pose.q[0] + pose.q[1] * pose.q[1] + pose.q[2] * pose.q[2] + pose.q[3] * pose.q[3];
    const float reach = m.reach + extent + fabsf(pose.t[0]) + fabsf(pose.t[1]) + fabsf(pose.t[2]);
    pad += (2e-6f + 8.0f * fabsf(q2 - 1.0f)) * reach;
  }
  k_mesh_sdf_discs<<<(totalCells + kThreads - 1) / kThreads, kThreads, 0, s>>>(
      static_cast<const float4*>(m.tris.ptr), static_cast<const uint32_t*>(m.index.ptr), static_cast<const float4*>(m.discs.ptr),
      static_cast<const float4*>(m.discs.ptr) + 2 * (size_t(m.leaves) + m.groups + m.blocks), m.n, m.leaves,
      m.groups, m.blocks, pose, int(res[0]), int(res[1]), int(res[2]), totalCells, cellSize, eps, pad, dSdf);
  ++*launches;
  return cudaGetLastError();
}

namespace {

// Bounding box, area-weighted normal and finiteness of a run of triangles.
struct Extent {
  float l[3] = {INFINITY, INFINITY, INFINITY}, u[3] = {-INFINITY, -INFINITY, -INFINITY};
  double g[3] = {0.0, 0.0, 0.0};
  float bad = 0.f;  // NaN when a coordinate is not finite
  void add(const float* v) {
    for (int k = 0; k < 9; k += 3)
      for (int a = 0; a < 3; ++a) {
        bad += v[k + a] * 0.f;
        l[a] = std::min(l[a], v[k + a]);
        u[a] = std::max(u[a], v[k + a]);
      }
    const double x1 = double(v[3]) - v[0], y1 = double(v[4]) - v[1], z1 = double(v[5]) - v[2];
    const double x2 = double(v[6]) - v[0], y2 = double(v[7]) - v[1], z2 = double(v[8]) - v[2];
    g[0] += y1 * z2 - z1 * y2;
    g[1] += z1 * x2 - x1 * z2;
    g[2] += x1 * y2 - y1 * x2;
  }
  void add(const Extent& e) {
    bad += e.bad;
    for (int a = 0; a < 3; ++a) {
      l[a] = std::min(l[a], e.l[a]);
      u[a] = std::max(u[a], e.u[a]);
      g[a] += e.g[a];
    }
  }
};

// Bounding disc of the vertices of sorted triangles [t0, t1): the plane of
// their area-weighted normal through the middle of their bounding box.
void hostDisc(const float* tris, uint32_t t0, uint32_t t1, const Extent& e, float4* out) {
  if (e.bad != 0.f) {  // never skipped
    out[0] = make_float4(NAN, NAN, NAN, NAN);
    out[1] = make_float4(0.f, 0.f, 0.f, NAN);
    return;
  }
  const double len = std::sqrt(e.g[0] * e.g[0] + e.g[1] * e.g[1] + e.g[2] * e.g[2]);
  float n[3], c[3];
  for (int a = 0; a < 3; ++a) {
    c[a] = 0.5f * e.l[a] + 0.5f * e.u[a];
    n[a] = len > 1e-30 && std::isfinite(len) ? float(e.g[a] / len) : 0.f;
  }
  double r2 = 0.0, th = 0.0;
  for (uint32_t t = t0; t < t1; ++t)
    for (int k = 0; k < 3; ++k) {
      const float* v = tris + 12 * size_t(t) + 3 + 3 * k;
      const double d[3] = {double(v[0]) - c[0], double(v[1]) - c[1], double(v[2]) - c[2]};
      const double h = d[0] * n[0] + d[1] * n[1] + d[2] * n[2];
      th = std::max(th, std::fabs(h));
      r2 = std::max(r2, d[0] * d[0] + d[1] * d[1] + d[2] * d[2] - h * h);
    }
  const float slack = 1e-6f * std::max(1.0f, std::fabs(c[0]) + std::fabs(c[1]) + std::fabs(c[2]));
  out[0] = make_float4(c[0], c[1], c[2], float(std::sqrt(r2)) * 1.0001f + slack);
  out[1] = make_float4(n[0], n[1], n[2], float(th) * 1.0001f + slack);
}

constexpr size_t kForkTriangles = 8192;  // a split below this takes less than starting a thread is worth

struct Centroid {
  float c[3];
  uint32_t index;  // in the caller's list
  // position along an axis, ties by list index: unsigned integers order as the pairs
  uint64_t key(int axis) const {
    const float f = c[axis] + 0.0f;  // (-0 and 0 are one place)
    uint32_t u;
    std::memcpy(&u, &f, sizeof(u));
    u ^= (u >> 31) ? 0xffffffffu : 0x80000000u;
    return (uint64_t(u) << 32) | index;
  }
};

// The mid - lo smallest of t[lo, hi) along an axis to the front, as
// std::nth_element, by partitions without a branch per element: the comparisons
// are unpredictable and were most of the preparation.
void selectFront(std::vector<Centroid>& t, size_t lo, size_t mid, size_t hi, int axis) {
  for (int rounds = 0; hi - lo > 16 && rounds < 64; ++rounds) {
    uint64_t s[9];  // the pivot is the median of nine
    for (size_t k = 0; k < 9; ++k) s[k] = t[lo + (hi - 1 - lo) * k / 8].key(axis);
    std::sort(s, s + 9);
    size_t m = lo;
    for (size_t i = lo; i < hi; ++i) {
      const Centroid c = t[i];
      t[i] = t[m];
      t[m] = c;
      m += c.key(axis) < s[4] ? 1u : 0u;
    }
    if (m == mid) return;
    if (mid < m) hi = m;
    else lo = m;
  }
  std::nth_element(t.begin() + lo, t.begin() + mid, t.begin() + hi, [axis](const Centroid& p, const Centroid& q) { return p.key(axis) < q.key(axis); });
}

// Order of the triangles: median splits of the centroids along their longest
// extent, cut at multiples of a block, then a group, then a leaf, so that the
// runs of every level are compact.  (Runs of a Morton order jump between
// distant patches of a surface and make wide leaves: 2.41 ms where median splits
// give 1.50.)
// t[t0, t1); ties by list index, so the runs depend on the mesh alone.  The
// halves are independent: those of the first `forks` splits of a large mesh go to
// threads of their own.
void orderTriangles(std::vector<Centroid>& t, size_t t0, size_t t1, int forks) {
  std::vector<std::future<void>> others;  // (joined on the way out)
  while (t1 - t0 > kMeshLeaf) {
    const size_t len = t1 - t0;
    size_t unit = kMeshLeaf;
    while (unit * kMeshFan < len) unit *= kMeshFan;
    const size_t mid = t0 + unit * (((len + unit - 1) / unit) / 2);
    float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (size_t k = t0; k < t1; ++k)
      for (int a = 0; a < 3; ++a) {
        lo[a] = std::min(lo[a], t[k].c[a]);
        hi[a] = std::max(hi[a], t[k].c[a]);
      }
    int axis = 0;
    for (int a = 1; a < 3; ++a)
      if (hi[a] - lo[a] > hi[axis] - lo[axis]) axis = a;
    selectFront(t, t0, mid, t1, axis);
    // the larger half here, the smaller one below (the depth stays logarithmic)
    const bool lower = mid - t0 < t1 - mid;
    const size_t s0 = lower ? t0 : mid, s1 = lower ? mid : t1;
    (lower ? t0 : t1) = mid;
    if (forks > 0 && len >= kForkTriangles) {
      --forks;
      try {
        others.push_back(std::async(std::launch::async, [&t, s0, s1, forks] { orderTriangles(t, s0, s1, forks); }));
        continue;
      } catch (const std::system_error&) {  // no thread to be had
      }
    }
    orderTriangles(t, s0, s1, forks);
  }
}
}  // namespace

void PreparedMesh::build(const float* h, uint32_t count) {
  checkMeshArgs(h, count);
  n = count;
  leaves = (count + kMeshLeaf - 1) / kMeshLeaf;
  groups = (leaves + kMeshFan - 1) / kMeshFan;
  blocks = (groups + kMeshFan - 1) / kMeshFan;
  std::vector<Centroid> cen(count);
  for (uint32_t k = 0; k < count; ++k) {
    cen[k].index = k;
    for (int a = 0; a < 3; ++a) {
      const float c = (h[12 * size_t(k) + 3 + a] + h[12 * size_t(k) + 6 + a] + h[12 * size_t(k) + 9 + a]) / 3.0f;
      cen[k].c[a] = std::isfinite(c) ? c : 0.f;  // (any place: a triangle that is never closest)
    }
  }
  orderTriangles(cen, 0, count, 3);
  std::vector<float> sorted(size_t(count) * 12);
  std::vector<uint32_t> idx(count);
  for (uint32_t i = 0; i < count; ++i) {
    idx[i] = cen[i].index;
    std::memcpy(&sorted[12 * size_t(i)], h + 12 * size_t(idx[i]), 12 * sizeof(float));
  }
  reach = 0.f;
  for (size_t t = 0; t < count; ++t)
    for (int k = 3; k < 12; ++k)
      if (std::isfinite(sorted[12 * t + k])) reach = std::max(reach, std::fabs(sorted[12 * t + k]));
  reach *= 1.7320509f;
  const size_t total = size_t(leaves) + groups + blocks;
  std::vector<float4> disc(std::max<size_t>(2 * total + leaves, 1));  // the discs, then a vertex of each leaf
  const uint32_t per[3] = {kMeshLeaf, kMeshLeaf * kMeshFan, kMeshLeaf * kMeshFan * kMeshFan}, runs[3] = {leaves, groups, blocks};
  std::vector<Extent> ext(total);  // of the leaves, then of what they make up
  for (uint32_t t = 0; t < count; ++t) ext[t / kMeshLeaf].add(&sorted[12 * size_t(t) + 3]);
  for (uint32_t l = 0; l < leaves; ++l) ext[leaves + l / kMeshFan].add(ext[l]);
  for (uint32_t g = 0; g < groups; ++g) ext[leaves + groups + g / kMeshFan].add(ext[leaves + g]);
  size_t at = 0;
  for (int lv = 0; lv < 3; ++lv)
    for (uint32_t r = 0; r < runs[lv]; ++r, at += 2)
      hostDisc(sorted.data(), r * per[lv], std::min(count, (r + 1) * per[lv]), ext[at / 2], &disc[at]);
  for (uint32_t l = 0; l < leaves; ++l, ++at) {
    // of a triangle that can be closest: finite and of some area (none: NaN, no bound)
    disc[at] = make_float4(NAN, NAN, NAN, 0.f);
    for (uint32_t t = l * kMeshLeaf; t < std::min(count, (l + 1) * kMeshLeaf); ++t) {
      const float* v = &sorted[12 * size_t(t) + 3];
      double e[3][3], e2 = 0.0, g2 = 0.0;  // two edges, their cross product
      for (int a = 0; a < 3; ++a) {
        e[0][a] = double(v[3 + a]) - v[a];
        e[1][a] = double(v[6 + a]) - v[a];
        e2 += e[0][a] * e[0][a] + e[1][a] * e[1][a];
      }
      for (int a = 0; a < 3; ++a) {
        e[2][a] = e[0][(a + 1) % 3] * e[1][(a + 2) % 3] - e[0][(a + 2) % 3] * e[1][(a + 1) % 3];
        g2 += e[2][a] * e[2][a];
      }
      if (std::isfinite(e2) && g2 > 1e-6 * e2 * e2) {
        disc[at] = make_float4(v[0], v[1], v[2], 0.f);
        break;
      }
    }
  }
  tris.ensure(std::max<size_t>(sorted.size() * sizeof(float), 16));
  index.ensure(std::max<size_t>(idx.size() * sizeof(uint32_t), 16));
  discs.ensure(disc.size() * sizeof(float4));
  if (count) {
    check(cudaMemcpy(tris.ptr, sorted.data(), sorted.size() * sizeof(float), cudaMemcpyHostToDevice), "upload mesh");
    check(cudaMemcpy(index.ptr, idx.data(), idx.size() * sizeof(uint32_t), cudaMemcpyHostToDevice), "upload mesh");
    check(cudaMemcpy(discs.ptr, disc.data(), disc.size() * sizeof(float4), cudaMemcpyHostToDevice), "upload mesh");
  }
}

MeshPose meshPose(const float* translation, const float* rotationWxyz) {
  MeshPose p{};
  p.q[0] = 1.0f;
  if (translation)
    for (int i = 0; i < 3; ++i) p.t[i] = translation[i];
  if (rotationWxyz)
    for (int i = 0; i < 4; ++i) p.q[i] = rotationWxyz[i];
  p.posed = translation != nullptr || rotationWxyz != nullptr;
  return p;
}

void checkMeshArgs(const float* tris, uint32_t nTris) {
  if (nTris && !tris) throw Error(NEBULA_MPM_ERR_INVALID, "null triangles");
  if (nTris > (1u << 26)) throw Error(NEBULA_MPM_ERR_INVALID, "at most 2^26 triangles");
}

}  // namespace nebula

using namespace nebula;

struct nebula_mpm_mesh {
  nebula::PreparedMesh mesh;
};

namespace {
template <class F> int guardedMesh(F&& f) {
  try {
    f();
    return NEBULA_MPM_OK;
  } catch (const Error& e) {
    g_last_error = e.what();
    return e.code;
  } catch (const std::bad_alloc&) {
    g_last_error = "host allocation failed";
    return NEBULA_MPM_ERR_OOM;
  } catch (const std::exception& e) {
    g_last_error = e.what();
    return NEBULA_MPM_ERR_INVALID;
  }
}
void checkGrid(const uint32_t realRes[3], uint32_t totalCells, float cellSize, const float* dSdf) {
  if (!realRes || !dSdf) throw Error(NEBULA_MPM_ERR_INVALID, "null argument");
  if (!(cellSize > 0.f)) throw Error(NEBULA_MPM_ERR_INVALID, "cellSize must be > 0");
  if (!realRes[0] || !realRes[1] || !realRes[2]) throw Error(NEBULA_MPM_ERR_INVALID, "realRes must be >= 1");
  const uint32_t cube = domainCubeRes(realRes);
  if (cube > 1024u || uint64_t(totalCells) < uint64_t(cube) * cube * cube)
    throw Error(NEBULA_MPM_ERR_INVALID, "totalCells must hold the Morton cube of realRes (cubeRes <= 1024)");
}
}  // namespace

extern "C" {

int nebula_mpm_mesh_create(const float* tris, uint32_t n, nebula_mpm_mesh** out) {
  return guardedMesh([&] {
    if (!out) throw Error(NEBULA_MPM_ERR_INVALID, "null output");
    auto m = std::make_unique<nebula_mpm_mesh>();
    m->mesh.build(tris, n);
    *out = m.release();
  });
}

int nebula_mpm_mesh_destroy(nebula_mpm_mesh* m) {
  delete m;
  return NEBULA_MPM_OK;
}

int nebula_mpm_mesh_build_sdf(const nebula_mpm_mesh* m, const float translation[3], const float rotation_wxyz[4], const uint32_t realRes[3],
                              uint32_t totalCells, float cellSize, float* dSdf, void* stream) {
  return guardedMesh([&] {
    if (!m) throw Error(NEBULA_MPM_ERR_INVALID, "null mesh");
    checkGrid(realRes, totalCells, cellSize, dSdf);
    uint64_t l = 0;
    check(launchMeshSdfPrepared(m->mesh, meshPose(translation, rotation_wxyz), realRes, totalCells, cellSize, dSdf, static_cast<cudaStream_t>(stream),
                                &l),
          "mesh sdf");
  });
}

int nebula_mpm_mesh_build_sdf_reference(const nebula_mpm_mesh* m, const float translation[3], const float rotation_wxyz[4],
                                        const uint32_t realRes[3], uint32_t totalCells, float cellSize, float* dSdf, void* stream) {
  return guardedMesh([&] {
    if (!m) throw Error(NEBULA_MPM_ERR_INVALID, "null mesh");
    checkGrid(realRes, totalCells, cellSize, dSdf);
    uint64_t l = 0;
    check(launchMeshSdfReference(static_cast<const float*>(m->mesh.tris.ptr), static_cast<const uint32_t*>(m->mesh.index.ptr), m->mesh.n,
                                 meshPose(translation, rotation_wxyz), realRes, totalCells, cellSize, dSdf, static_cast<cudaStream_t>(stream), &l),
          "mesh sdf (reference closest point)");
  });
}

int nebula_mpm_mesh_sdf_reference(const float* dTris, uint32_t nTris, const float translation[3], const float rotation_wxyz[4],
                                  const uint32_t realRes[3], uint32_t totalCells, float cellSize, float* dSdf, void* stream) {
  return guardedMesh([&] {
    checkGrid(realRes, totalCells, cellSize, dSdf);
    checkMeshArgs(dTris, nTris);
    if (reinterpret_cast<uintptr_t>(dTris) % 16u) throw Error(NEBULA_MPM_ERR_INVALID, "triangles must be 16-byte aligned");
    uint64_t l = 0;
    check(launchMeshSdfReference(dTris, nullptr, nTris, meshPose(translation, rotation_wxyz), realRes, totalCells, cellSize, dSdf,
                                 static_cast<cudaStream_t>(stream), &l),
          "mesh sdf (reference closest point)");
  });
}

int nebula_mpm_mesh_sdf(const float* dTris, uint32_t nTris, const uint32_t realRes[3], uint32_t totalCells, float cellSize, float* dSdf,
                        void* stream) {
  return nebula_mpm_mesh_sdf_posed(dTris, nTris, nullptr, nullptr, realRes, totalCells, cellSize, dSdf, stream);
}

int nebula_mpm_mesh_sdf_posed(const float* dTris, uint32_t nTris, const float translation[3], const float rotationWxyz[4],
                              const uint32_t realRes[3], uint32_t totalCells, float cellSize, float* dSdf, void* stream) {
  return guardedMesh([&] {
    checkGrid(realRes, totalCells, cellSize, dSdf);
    checkMeshArgs(dTris, nTris);
    if (reinterpret_cast<uintptr_t>(dTris) % 16u) throw Error(NEBULA_MPM_ERR_INVALID, "triangles must be 16-byte aligned");
    uint64_t l = 0;
    check(launchMeshSdf(dTris, nTris, meshPose(translation, rotationWxyz), realRes, totalCells, cellSize, dSdf,
                        static_cast<cudaStream_t>(stream), &l),
          "mesh sdf");
  });
}

}  // extern "C"
