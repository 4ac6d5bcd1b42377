// mpm_passes.cu -- single-pass kernels on the reference's dense grid layout.
//
// These run one reference dispatch each (binning, P2G, grid update + SDF
// boundary, G2P) on gridMom (float4 x 2 hashCells: [0,NC) momentum/velocity,
// [NC,2NC) pre-force velocity) and gridMass (float x NC), as the shaders do.
// They back the single-pass C ABI and the dense engine path.
#include "mpm_internal.h"
#include "mpm_p2g.cuh"
#include "mpm_scan_kernel.cuh"

#include <algorithm>

namespace nebula {

namespace {

constexpr int kThreads = 256;

inline uint32_t blocksFor(uint64_t n, int t = kThreads) { return uint32_t((n + t - 1) / t); }

constexpr uint32_t kKeyExcluded = 0xffffffffu;

// mpm_hash_count.comp:7-14 / hash_count.comp:7-20 (+ the slot the sort would take).
// Runs of equal keys in neighbouring lanes (particles stored in cell order, or
// lattice order along x) take their slots with one atomic per run; the whole
// warp stays converged for the shuffles, lanes without a particle carrying
// the excluded key.  A thread takes kCountItems particles, all of whose
// positions are loaded before the first atomic.  The kernel also zeroes the
// scan's status words, its ticket and the large-cell flag behind them (`words`
// of 64 bits from `status`) and, when given, the error word: two memset
// launches less.  What bounds it is the atomics' round trips: 8,388,608
// particles on 128^3 60 -> 51 us.
constexpr int kCountItems = 4;
__global__ void __launch_bounds__(kThreads) k_bin_count(SubstepParams P, const float4* __restrict__ pos, const uint32_t* __restrict__ typeFlag,
                                                        uint32_t n, uint32_t* cellCount, uint32_t* key, uint32_t* rank, unsigned long long* status,
                                                        uint32_t words, uint32_t* err) {
  for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < words; q += gridDim.x * blockDim.x) status[q] = 0ull;
  if (err && blockIdx.x == 0 && threadIdx.x == 0) *err = 0u;
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t i0 = blockIdx.x * (kThreads * kCountItems) + threadIdx.x;
  uint32_t c[kCountItems];
#pragma unroll
  for (int r = 0; r < kCountItems; ++r) {
    const uint32_t i = i0 + uint32_t(r) * kThreads;
    c[r] = kKeyExcluded;
    if (i < n && !(typeFlag && typeFlag[i] == kTypeFlagUnused)) {
      const float4 p = pos[i];
      int cx, cy, cz;
      cellCoords(P, p.x, p.y, p.z, cx, cy, cz);
      c[r] = mortonEncode(cx, cy, cz);
    }
  }
  uint32_t base[kCountItems], head[kCountItems];
#pragma unroll
  for (int r = 0; r < kCountItems; ++r) {
    const uint32_t up = __shfl_up_sync(0xffffffffu, c[r], 1);
    const uint32_t heads = __ballot_sync(0xffffffffu, lane == 0 || up != c[r]);
    const uint32_t le = 0xffffffffu >> (31u - lane);  // lanes 0..lane
    head[r] = 31u - __clz(heads & le);                 // first lane of this lane's run
    const uint32_t after = heads & ~le;
    const uint32_t runEnd = after ? uint32_t(__ffs(after) - 1) : 32u;
    base[r] = 0;
    if (lane == head[r] && c[r] != kKeyExcluded) base[r] = atomicAdd(cellCount + c[r], runEnd - lane);
  }
#pragma unroll
  for (int r = 0; r < kCountItems; ++r) {
    const uint32_t i = i0 + uint32_t(r) * kThreads;
    base[r] = __shfl_sync(0xffffffffu, base[r], head[r]);
    if (i < n) {
      key[i] = c[r];
      rank[i] = base[r] + (lane - head[r]);
    }
  }
}

// mpm_hash_sort.comp:7-15 with the slot taken at count time.  A thread takes
// kScatterItems particles, the loads of all of them before the first store:
// the kernel is two dependent memory round trips (key, then the cell's start).
// 8,388,608 particles (with the count kernel's four items): 156 -> 146 us for the whole sort.
constexpr int kScatterItems = 4;
__global__ void __launch_bounds__(kThreads) k_bin_scatter(uint32_t n, const uint32_t* __restrict__ key, const uint32_t* __restrict__ rank,
                                                          const uint32_t* __restrict__ cellStart, uint32_t* sortedTmp, uint32_t* err) {
  const uint32_t i0 = blockIdx.x * (kThreads * kScatterItems) + threadIdx.x;
  uint32_t c[kScatterItems], slot[kScatterItems];
#pragma unroll
  for (int r = 0; r < kScatterItems; ++r) {
    const uint32_t i = i0 + uint32_t(r) * kThreads;
    c[r] = i < n ? key[i] : kKeyExcluded;
    slot[r] = i < n ? rank[i] : 0u;
  }
#pragma unroll
  for (int r = 0; r < kScatterItems; ++r)
    if (c[r] != kKeyExcluded) slot[r] += cellStart[c[r]];
#pragma unroll
  for (int r = 0; r < kScatterItems; ++r) {
    if (c[r] == kKeyExcluded) continue;
    if (slot[r] < n) sortedTmp[slot[r]] = i0 + uint32_t(r) * kThreads;
    else atomicOr(err, kErrBinRange);  // only after an expired scan wait
  }
}

// In-cell canonical order (ascending particle index).  Cells of at most
// kCanonCellMax particles: one thread per cell loads the cell's slots (the
// warp reads one contiguous span) and ranks them in registers, up to the
// warp's largest such cell (1,900,000 occupied cells of 128^3:
// 39 -> 33 us).  Larger cells: one thread per particle counts the
// smaller indices of its cell, in a launch that ends at once unless a cell
// raised the flag.
constexpr uint32_t kCanonCellMax = 16;

__global__ void __launch_bounds__(kThreads) k_bin_canon_cells(uint32_t nc, uint32_t n, const uint32_t* __restrict__ cellStart,
                                                              const uint32_t* __restrict__ cellCount, const uint32_t* __restrict__ sortedTmp,
                                                              uint32_t* sorted, uint32_t* large, uint32_t* err) {
  const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t cnt = c < nc ? cellCount[c] : 0u, st = 0;
  if (cnt > kCanonCellMax) {
    *large = 1u;
    cnt = 0;
  }
  if (cnt) {
    st = cellStart[c];
    if (st > n || cnt > n - st) {
      atomicOr(err, kErrBinRange);
      cnt = 0;
    }
  }
  const uint32_t most = __reduce_max_sync(0xffffffffu, cnt);
  uint32_t v[kCanonCellMax];
#pragma unroll
  for (uint32_t k = 0; k < kCanonCellMax; ++k) {
    if (k >= most) break;
    v[k] = k < cnt ? sortedTmp[st + k] : 0xffffffffu;  // padding never ranks below
  }
#pragma unroll
  for (uint32_t k = 0; k < kCanonCellMax; ++k) {
    if (k >= most) break;
    uint32_t r = 0;
#pragma unroll
    for (uint32_t j = 0; j < kCanonCellMax; ++j) {
      if (j >= most) break;
      r += v[j] < v[k] ? 1u : 0u;
    }
    if (k < cnt) sorted[st + r] = v[k];
  }
}

__global__ void __launch_bounds__(kThreads) k_bin_canon_particles(uint32_t n, const uint32_t* __restrict__ key,
                                                                  const uint32_t* __restrict__ cellStart, const uint32_t* __restrict__ cellCount,
                                                                  const uint32_t* __restrict__ sortedTmp, uint32_t* sorted,
                                                                  const uint32_t* __restrict__ large, uint32_t* err) {
  if (*large == 0u) return;
  for (uint64_t t = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; t < n; t += uint64_t(gridDim.x) * blockDim.x) {
    const uint32_t i = uint32_t(t);
    const uint32_t c = key[i];
    if (c == kKeyExcluded) continue;
    const uint32_t st = cellStart[c], cnt = cellCount[c];
    if (cnt <= kCanonCellMax) continue;  // ranked by k_bin_canon_cells
    if (st > n || cnt > n - st) {
      atomicOr(err, kErrBinRange);
      continue;
    }
    uint32_t r = 0;
    for (uint32_t j = st; j < st + cnt; ++j) r += sortedTmp[j] < i ? 1u : 0u;
    sorted[st + r] = i;
  }
}
constexpr uint32_t kCanonParticleBlocks = 1184;  // as many as 148 SMs hold (the blocks stride, so any number is right); a launch whose cells are all small pays only their start

// P2G: a warp takes `slots` (a power of two up to 32) sorted slots, sums the
// particles that share a cell (mpm_p2g.cuh) and adds each group's 27 nodes to the
// dense grid.  What bounds it is the reductions to L2: 27 of 16 bytes and 27 of 4
// per group, where one thread per particle issued as many per particle.  300,000
// particles in cell order: 31 us (bin to grid update of 128^3: 225 -> 102 us a
// pass, most of the rest the zeroing of the 75 MB grid).
//
// A warp's groups come one after another, up to one per slot: with few warps
// that chain is the pass, and scattered particles in 32 slots a warp were slower
// than one thread each (4,000 at random: 15.7 -> 16.7 us with the zeroing of a
// 64^3 grid).  So up to kP2GSmall particles a warp takes 8 slots: 9.7 us there, 8.3
// instead of 10.4 in cell order; 10,000: 11.1 for 17.1, 9.4 for 10.9.  At 30,000
// the warps are enough and the groups count: 11.3 for 10.5 in cell order.
constexpr uint32_t kP2GSmall = 16384;
__global__ void __launch_bounds__(kThreads) k_p2g_dense(SubstepParams P, StatePtrs st, const uint32_t* __restrict__ sorted, uint32_t n, uint32_t slots,
                                                        float4* gridMom, float* gridMass) {
  __shared__ __align__(16) WarpRows rows[kThreads / 32];
  const uint32_t lane = threadIdx.x & 31u, warp = (blockIdx.x * kThreads + threadIdx.x) >> 5;
  const uint32_t t = lane < slots ? warp * slots + lane : n;
  WarpRows& W = rows[threadIdx.x >> 5];
  uint32_t key = kNoKey;
  bool exact = false;
  if (t < n) {
    const uint32_t p = sorted[t];
    if (p < n) {  // (a caller-supplied order may hold an out-of-range index)
      const PState s = loadState(st.f, p);
      int cx, cy, cz;
      cellCoords(P, s.P.x, s.P.y, s.P.z, cx, cy, cz);
      float m;
      exact = p2gRow(P, s, P.dt, cx, cy, cz, W.rows + lane * kRow, m);
      W.mass[lane] = m;
      key = packCell(cx, cy, cz);
    }
  }
  const uint32_t exactMask = __ballot_sync(0xffffffffu, exact);
  __syncwarp();  // the rows are visible to every lane
  uint32_t pending = __ballot_sync(0xffffffffu, key != kNoKey);
  while (pending) {
    const uint32_t k = __shfl_sync(0xffffffffu, key, __ffs(pending) - 1);
    const uint32_t peers = __ballot_sync(0xffffffffu, key == k);
    pending &= ~peers;
    p2gGroup(P, W, k, peers, exactMask, [&](uint32_t c, const float* a) {
      redAddV4(gridMom + c, a[0], a[1], a[2], 0.f);
      atomicAdd(gridMass + c, a[3]);
    });
  }
}

// mpm_grid_update.comp + mpm_nanovdb_bc.comp, one thread per node.
__global__ void __launch_bounds__(kThreads) k_grid_dense(SubstepParams P, float4* gridMom, const float* __restrict__ gridMass) {
  uint32_t gid = blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= P.hashCells) return;
  float mass = gridMass[gid];
  if (mass < 1e-10f) return;
  float4 mom = gridMom[gid];
  int ix, iy, iz;
  mortonDecode(gid, ix, iy, iz);
  float3 v, vo;
  gridNode(P, ix, iy, iz, mass, mom.x, mom.y, mom.z, v, vo);
  gridMom[P.hashCells + gid] = make_float4(vo.x, vo.y, vo.z, 0.f);
  gridMom[gid] = make_float4(v.x, v.y, v.z, 0.f);
}

struct DenseGrid {
  const float4* mom;
  const float* mass;
  uint32_t nc;
  __device__ __forceinline__ bool node(int x, int y, int z, float& m, float3& v, float3& vo) const {
    uint32_t nid = mortonEncode(x, y, z);
    m = __ldg(mass + nid);
    if (m < 1e-10f) return false;
    float4 a = __ldg(mom + nid);
    float4 b = __ldg(mom + nc + nid);
    v = make_float3(a.x, a.y, a.z);
    vo = make_float3(b.x, b.y, b.z);
    return true;
  }
};

__global__ void __launch_bounds__(kThreads) k_g2p_dense(SubstepParams P, StatePtrs st, uint32_t n, const float4* __restrict__ gridMom,
                                                        const float* __restrict__ gridMass, uint32_t* err) {
  uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  PState s;
  s.P = st.f[0][p]; s.v = st.f[1][p];
  s.F0 = st.f[2][p]; s.F1 = st.f[3][p]; s.F2 = st.f[4][p];
  s.B0 = st.f[5][p]; s.B1 = st.f[6][p]; s.B2 = st.f[7][p];
  DenseGrid g{gridMom, gridMass, P.hashCells};
  g2pParticle(P, s, g, P.dt);
  if (err && !(isfinite(s.P.x) && isfinite(s.P.y) && isfinite(s.P.z))) atomicOr(err, kErrNonFinite);
  st.f[0][p] = s.P; st.f[1][p] = s.v;
  st.f[2][p] = s.F0; st.f[3][p] = s.F1; st.f[4][p] = s.F2;
  st.f[5][p] = s.B0; st.f[6][p] = s.B1; st.f[7][p] = s.B2;
}

}  // namespace

size_t scanWorkspaceBytes(uint64_t n) { return (size_t(scanTiles(n)) + 2) * sizeof(unsigned long long); }

cudaError_t launchBin(const SubstepParams& P, const float4* pos, uint32_t n, const BinBuffers& b, cudaStream_t s, uint64_t* launches) {
  const uint64_t nc = P.hashCells;
  cudaError_t e = cudaMemsetAsync(b.cellCount, 0, nc * sizeof(uint32_t), s);
  if (e != cudaSuccess) return e;
  const uint32_t tiles = scanTiles(nc);
  uint32_t* large = b.tileCounter + 1;
  if (n > 0) {
    k_bin_count<<<blocksFor(n, kThreads * kCountItems), kThreads, 0, s>>>(P, pos, b.typeFlag, n, b.cellCount, b.key, b.rank, b.tileState, tiles + 1,
                                                                           b.clearErr ? b.err : nullptr);
    ++*launches;
  } else {
    e = cudaMemsetAsync(b.tileState, 0, (size_t(tiles) + 1) * sizeof(unsigned long long), s);
    if (e == cudaSuccess && b.clearErr) e = cudaMemsetAsync(b.err, 0, sizeof(uint32_t), s);
    if (e != cudaSuccess) return e;
  }
  launchScanExclusive(b.cellCount, b.cellStart, b.cellEnd, nc, b.tileState, b.tileCounter, b.err, s);
  ++*launches;
  if (n > 0) {
    k_bin_scatter<<<blocksFor(n, kThreads * kScatterItems), kThreads, 0, s>>>(n, b.key, b.rank, b.cellStart, b.sortedTmp, b.err);
    k_bin_canon_cells<<<blocksFor(nc), kThreads, 0, s>>>(uint32_t(nc), n, b.cellStart, b.cellCount, b.sortedTmp, b.sorted, large, b.err);
    k_bin_canon_particles<<<std::min(blocksFor(n), kCanonParticleBlocks), kThreads, 0, s>>>(n, b.key, b.cellStart, b.cellCount, b.sortedTmp, b.sorted,
                                                                                            large, b.err);
    *launches += 3;
  }
  return cudaGetLastError();
}

cudaError_t launchBinScanExpiryProbe(const SubstepParams& P, const BinBuffers& b, cudaStream_t s, uint64_t* launches) {
  const uint64_t nc = P.hashCells;
  const uint32_t tiles = scanTiles(nc);
  if (tiles < 2) return cudaErrorInvalidValue;
  // every status word unpublished and the tile ticket at 1: the single CTA
  // below becomes tile 1 and waits on a tile 0 that never runs
  cudaError_t e = cudaMemsetAsync(b.tileState, 0, (size_t(tiles) + 1) * sizeof(unsigned long long), s);
  if (e == cudaSuccess) e = cudaMemsetAsync(b.err, 0, sizeof(uint32_t), s);
  if (e == cudaSuccess) e = cudaMemsetAsync(b.tileCounter, 1, 1, s);  // little-endian u32 = 1
  if (e != cudaSuccess) return e;
  k_scan_exclusive<false><<<1, kScanThreads, 0, s>>>(b.cellCount, b.cellStart, nullptr, nc, b.tileState, b.tileCounter, b.err);
  ++*launches;
  return cudaGetLastError();
}

cudaError_t launchP2GDense(const SubstepParams& P, StatePtrs st, const uint32_t* sorted, uint32_t n, float4* gridMom, float* gridMass,
                           cudaStream_t s, uint64_t* launches) {
  if (n == 0) return cudaSuccess;
  const uint32_t slots = n <= kP2GSmall ? 8u : 32u;
  k_p2g_dense<<<blocksFor(uint64_t(n) * (32u / slots)), kThreads, 0, s>>>(P, st, sorted, n, slots, gridMom, gridMass);
  ++*launches;
  return cudaGetLastError();
}

cudaError_t launchGridDense(const SubstepParams& P, float4* gridMom, const float* gridMass, cudaStream_t s, uint64_t* launches) {
  k_grid_dense<<<blocksFor(P.hashCells), kThreads, 0, s>>>(P, gridMom, gridMass);
  ++*launches;
  return cudaGetLastError();
}

cudaError_t launchG2PDense(const SubstepParams& P, StatePtrs st, uint32_t n, const float4* gridMom, const float* gridMass, uint32_t* err,
                           cudaStream_t s, uint64_t* launches) {
  if (n == 0) return cudaSuccess;
  k_g2p_dense<<<blocksFor(n), kThreads, 0, s>>>(P, st, n, gridMom, gridMass, err);
  ++*launches;
  return cudaGetLastError();
}

}  // namespace nebula
