// mpm_p2g.cuh -- P2G of a warp's particles (sm_100a device code): the terms the
// per-node gather of mpm_p2g.comp:40-82 sums, taken for the particles of a warp
// that share a cell before anything goes to the grid.
//
// Each particle's P2G inputs go to its lane's row in shared memory in
// separable form (p2gRow); the lanes of a warp are grouped by the cell their
// stencils are centred on, and for each group lanes 0..26 take the cell's 27
// nodes, sum the group's rows and hand each node's sums over (p2gGroup).
#pragma once
#include "mpm_particle.cuh"

namespace nebula {

constexpr int kRow = 9;                   // float4 per input row: 3 axes x 3 offsets (see p2gRow)
constexpr uint32_t kNoKey = 0xFFFFFFFFu;  // a lane with no row for the warp's P2G

struct WarpRows {
  float4 rows[32 * kRow];  // row of lane l at l * kRow
  float mass[32];          // the particle mass of an exact-form row
};

// P2G inputs of one particle in separable form.  The quadratic B-spline weight
// of node (dx,dy,dz) is W_x[dx] W_y[dy] W_z[dz], so the particle's momentum
// term  w (m v + m (4/h^2) B r) - dt Vp tau grad w  equals
//   W_y W_z A_x[dx] + W_x W_z A_y[dy] + W_x W_y A_z[dz]
// with, per axis c and offset d (r_c = x_i,c - x_p,c, G = N'/h):
//   A_c[d] = [c == x] m v W_c + (m 4/h^2 B)[:, c] W_c r_c - (dt Vp tau)[:, c] G_c
// and the mass term is m W_x W_y W_z.  The usual form folds the mass into the
// x factors:
//   row[d]     = (A_x[d],     m W_x[d])
//   row[3 + d] = (A_y[d] / m, W_y[d])
//   row[6 + d] = (A_z[d] / m, W_z[d])
// so a node term is  wyz X.xyz + (X.w Z.w) Y.xyz + (X.w Y.w) Z.xyz  and its
// mass X.w wyz: three vector loads, no per-particle scalar, and no weight
// test.  The shader skips a node whose weight is below 1e-12
// (mpm_p2g.comp:47); the smallest of the 27 weights is the product of the
// three axis minima, so when that product is below 1e-12 (0.15% of the slope
// scene's particles: near a cell face in all three axes, or very near one),
// or the mass is not positive (or so small that 1/m may overflow: far below what
// the grid update counts as mass), the row is written in the exact form instead,
// (A_c[d], W_c[d]) for every axis with the mass in `mass`, whose terms carry
// the shader's test (p2gNodeTermExact).  Returns true for the exact form.
__device__ __forceinline__ bool p2gRow(const SubstepParams& P, const PState& s, float dtStress, int cx, int cy, int cz, float4* row, float& m) {
  const float invH = 1.0f / P.cellSize;
  m = fetchRho0(P, __float_as_uint(s.v.w)) * s.P.w;
  const float av[3] = {m * s.v.x, m * s.v.y, m * s.v.z};
  float Q[3][3];  // GLSL [col][row]
  if (P.flip_ratio < -0.5f) {
    const float k = m * (4.0f / (P.cellSize * P.cellSize));
    Q[0][0] = k * s.B0.x; Q[0][1] = k * s.B0.y; Q[0][2] = k * s.B0.z;
    Q[1][0] = k * s.B1.x; Q[1][1] = k * s.B1.y; Q[1][2] = k * s.B1.z;
    Q[2][0] = k * s.B2.x; Q[2][1] = k * s.B2.y; Q[2][2] = k * s.B2.z;
  } else {
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int q = 0; q < 3; ++q) Q[c][q] = 0.f;
  }
  const float sdt = dtStress * s.P.w;
  const float T[3][3] = {{sdt * s.F0.w, sdt * s.B0.w, sdt * s.B1.w},
                         {sdt * s.B0.w, sdt * s.F1.w, sdt * s.B2.w},
                         {sdt * s.B1.w, sdt * s.B2.w, sdt * s.F2.w}};
  const float xp[3] = {s.P.x, s.P.y, s.P.z};
  const int cc[3] = {cx, cy, cz};
  float xs[3][3], W[3][3], G[3][3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    float ds[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      xs[c][d] = nodeCentre(P, c, cc[c] - 1 + d);
      ds[d] = (xp[c] - xs[c][d]) * invH;
    }
    bsplineStencil(ds[0], ds[1], ds[2], W[c], G[c]);
  }
  const float wmin = (fminf(W[0][0], fminf(W[0][1], W[0][2])) * fminf(W[1][0], fminf(W[1][1], W[1][2]))) * fminf(W[2][0], fminf(W[2][1], W[2][2]));
  const bool exact = !(m > 1e-30f && wmin >= 1e-12f);
  const float sx = exact ? 1.0f : m, sa = exact ? 1.0f : 1.0f / m;
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const float Wc = W[c][d], Gc = G[c][d] * invH;
      const float Rw = Wc * (xs[c][d] - xp[c]);
      float A[3];
#pragma unroll
      for (int q = 0; q < 3; ++q) A[q] = (c == 0 ? av[q] * Wc : 0.f) + Q[c][q] * Rw - T[c][q] * Gc;
      if (c == 0) row[d] = make_float4(A[0], A[1], A[2], sx * Wc);
      else row[3 * c + d] = make_float4(A[0] * sa, A[1] * sa, A[2] * sa, Wc);
    }
  return exact;
}

// Contribution of a usual-form row's three factors to its stencil node.
__device__ __forceinline__ void p2gNodeTermXYZ(const float4 X, const float4 Y, const float4 Z, float acc[4]) {
  const float wyz = Y.w * Z.w;
  const float wxz = X.w * Z.w, wxy = X.w * Y.w;
  acc[0] += wyz * X.x + wxz * Y.x + wxy * Z.x;
  acc[1] += wyz * X.y + wxz * Y.y + wxy * Z.y;
  acc[2] += wyz * X.z + wxz * Y.z + wxy * Z.z;
  acc[3] += X.w * wyz;
}

// Contribution of a usual-form row to its stencil node (dx, dy, dz).
__device__ __forceinline__ void p2gNodeTerm(const float4* __restrict__ row, int dx, int dy, int dz, float acc[4]) {
  p2gNodeTermXYZ(row[dx], row[3 + dy], row[6 + dz], acc);
}

// Contribution of an exact-form row (mass m) to its stencil node, skipped
// below w = 1e-12.
__device__ __forceinline__ void p2gNodeTermExact(const float4* __restrict__ row, float m, int dx, int dy, int dz, float acc[4]) {
  const float4 X = row[dx], Y = row[3 + dy], Z = row[6 + dz];
  const float wyz = Y.w * Z.w;
  const float w = X.w * wyz;
  if (w < 1e-12f) return;
  const float wxz = X.w * Z.w, wxy = X.w * Y.w;
  acc[0] += wyz * X.x + wxz * Y.x + wxy * Z.x;
  acc[1] += wyz * X.y + wxz * Y.y + wxy * Z.y;
  acc[2] += wyz * X.z + wxz * Y.z + wxy * Z.z;
  acc[3] += w * m;
}

// The cell a lane's stencil is centred on, as the key its group shares.
__device__ __forceinline__ uint32_t packCell(int cx, int cy, int cz) { return uint32_t(cx) | (uint32_t(cy) << 10) | (uint32_t(cz) << 20); }

// One group of the warp's rows: the lanes of `peers`, all centred on cell k.
// Lanes 0..26 take the cell's 27 stencil nodes, sum the group's rows (each read
// at a known address) and call add(Morton code, sums): momentum and mass.
template <class Add>
__device__ __forceinline__ void p2gGroup(const SubstepParams& P, const WarpRows& W, uint32_t k, uint32_t peers, uint32_t exactMask, Add&& add) {
  const int lane = threadIdx.x & 31;
  const int dx = lane % 3, dy = (lane / 3) % 3, dz = lane / 9;
  const uint32_t cr = P.cubeRes;
  const uint32_t nx = (k & 1023u) + uint32_t(dx) - 1u, ny = ((k >> 10) & 1023u) + uint32_t(dy) - 1u, nz = (k >> 20) + uint32_t(dz) - 1u;
  if (lane >= 27 || nx >= cr || ny >= cr || nz >= cr) return;
  float a[4] = {0.f, 0.f, 0.f, 0.f};
  if (!(peers & exactMask)) {
    // usual-form rows: two per step, loads of both issued before their sums
    uint32_t m = peers;
    while (m & (m - 1u)) {
      const int j0 = __ffs(m) - 1;
      m &= m - 1u;
      const int j1 = __ffs(m) - 1;
      m &= m - 1u;
      const float4 *r0 = W.rows + j0 * kRow, *r1 = W.rows + j1 * kRow;
      const float4 X0 = r0[dx], Y0 = r0[3 + dy], Z0 = r0[6 + dz];
      const float4 X1 = r1[dx], Y1 = r1[3 + dy], Z1 = r1[6 + dz];
      p2gNodeTermXYZ(X0, Y0, Z0, a);
      p2gNodeTermXYZ(X1, Y1, Z1, a);
    }
    if (m) p2gNodeTerm(W.rows + (__ffs(m) - 1) * kRow, dx, dy, dz, a);
  } else {
    uint32_t m = peers;
    while (m) {
      const int j = __ffs(m) - 1;
      m &= m - 1u;
      if ((exactMask >> j) & 1u) p2gNodeTermExact(W.rows + j * kRow, W.mass[j], dx, dy, dz, a);
      else p2gNodeTerm(W.rows + j * kRow, dx, dy, dz, a);
    }
  }
  add(mortonEncode(int(nx), int(ny), int(nz)), a);
}

}  // namespace nebula
