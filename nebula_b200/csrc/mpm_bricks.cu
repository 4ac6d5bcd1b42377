// mpm_bricks.cu -- brick-sparse fused substep kernels (sm_100a).
//
// Same per-particle and per-node math as the single-pass kernels
// (mpm_particle.cuh, restating mpm_p2g.comp, mpm_grid_update.comp,
// mpm_nanovdb_bc.comp and mpm_g2p.comp), organised for HBM:
//   * particles live in cell order, read once and written once per substep, 32
//     consecutive ones per warp;
//   * P2G sums the particles of a warp that share a cell before one vector
//     reduction per node to global memory;
//   * only bricks some particle stencil touched are updated or cleared.
#include "mpm_bricks.cuh"
#include "mpm_p2g.cuh"
#include "mpm_scan.cuh"

#include <algorithm>
#include <atomic>
#include <mutex>

namespace nebula {
namespace {

constexpr int kThreads = 256;
constexpr uint32_t kBrickScanSpinLimit = 1u << 22;
constexpr unsigned long long kStFlagAgg = 1ull << 48;
constexpr unsigned long long kStFlagPre = 2ull << 48;
constexpr unsigned long long kStValue = (1ull << 48) - 1;

inline uint32_t blocksFor(uint64_t n, int t = kThreads) { return uint32_t((n + t - 1) / t); }

__device__ __forceinline__ uint32_t laneId() { return threadIdx.x & 31u; }

// Programmatic dependent launch: the per-substep kernels are launched with
// programmatic stream serialization, so a kernel's CTAs may be scheduled as
// soon as the previous kernel's CTAs have all exited (no kernel triggers
// earlier), hiding the launch latency between them.  Every such kernel waits
// here, before its first memory access, until the previous grid has
// completed and its writes are visible; without the launch attribute the
// wait returns at once.
__device__ __forceinline__ void waitForPredecessorGrid() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <class... KArgs, class... Args>
cudaError_t launchSerialized(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args&&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

// Lanes in `mask` holding the same key take consecutive slots of counter[key].
__device__ __forceinline__ uint32_t warpAggInc(uint32_t mask, uint32_t* counter, uint32_t key) {
  const uint32_t peers = __match_any_sync(mask, key);
  const int leader = __ffs(peers) - 1;
  const uint32_t lane = laneId();
  uint32_t base = 0;
  if (int(lane) == leader) base = atomicAdd(counter + key, uint32_t(__popc(peers)));
  base = __shfl_sync(peers, base, leader);
  return base + __popc(peers & ((1u << lane) - 1u));
}

// Mark every brick holding a node of the 3x3x3 stencil around cell (cx,cy,cz).
__device__ __forceinline__ void markStencilBricks(const SubstepParams& P, int cx, int cy, int cz, uint32_t* flag) {
  const int cr = int(P.cubeRes) - 1;
  const int x0 = max(cx - 1, 0) >> 2, x1 = min(cx + 1, cr) >> 2;
  const int y0 = max(cy - 1, 0) >> 2, y1 = min(cy + 1, cr) >> 2;
  const int z0 = max(cz - 1, 0) >> 2, z1 = min(cz + 1, cr) >> 2;
  for (int bz = z0; bz <= z1; ++bz)
    for (int by = y0; by <= y1; ++by)
      for (int bx = x0; bx <= x1; ++bx) flag[mortonEncode(bx, by, bz)] = 1u;
}

// ------------------------------------------------------------------ batch scenes
// The scene s with base[s] <= x < base[s+1] (base non-decreasing, x < base[count]).
__device__ __forceinline__ uint32_t findScene(const uint32_t* __restrict__ base, uint32_t count, uint32_t x) {
  uint32_t lo = 0, hi = count;
  while (hi - lo > 1u) {
    const uint32_t mid = (lo + hi) >> 1;
    if (base[mid] <= x) lo = mid;
    else hi = mid;
  }
  return lo;
}

static_assert(sizeof(SubstepParams) % 4 == 0, "SubstepParams is copied as 32-bit words");
constexpr int kParamWords = int(sizeof(SubstepParams) / 4);

// Word copy of one scene's parameters by threads t = 0..nthreads-1.
__device__ __forceinline__ void copyParams(SubstepParams* dst, const SubstepParams* src, int t, int nthreads) {
  const uint32_t* a = reinterpret_cast<const uint32_t*>(src);
  uint32_t* d = reinterpret_cast<uint32_t*>(dst);
  for (int q = t; q < kParamWords; q += nthreads) d[q] = a[q];
}

__device__ __forceinline__ GridBuffers offsetGrid(const GridBuffers& G, uint32_t brickBase) {
  const size_t c = size_t(brickBase) << 6;
  return GridBuffers{G.acc + c, G.vel + c, G.vold ? G.vold + c : nullptr};
}

// ------------------------------------------------------------------ binning count (standalone)
template <bool BATCH>
__global__ void __launch_bounds__(kThreads) k_brick_count(SubstepParams P0, SceneTable T, const float4* __restrict__ pos, uint32_t n,
                                                          BrickBuffers B) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool act = i < n;
  const uint32_t mask = __ballot_sync(0xffffffffu, act);
  if (!act) return;
  const float4 p = pos[i];
  auto body = [&](const SubstepParams& P, uint32_t base) {
    int cx, cy, cz;
    cellCoords(P, p.x, p.y, p.z, cx, cy, cz);
    const uint32_t c = (base << 6) + mortonEncode(cx, cy, cz);
    B.binKey[i] = c;
    B.binRank[i] = warpAggInc(mask, B.cellCount, c);
    (void)warpAggInc(mask, B.brickCount, c >> 6);
    markStencilBricks(P, cx, cy, cz, B.brickFlag + base);
  };
  if constexpr (BATCH) {
    const uint32_t sc = findScene(T.partBase, T.count, i);
    body(T.params[sc], T.brickBase[sc]);
  } else {
    body(P0, 0u);
  }
}

// ------------------------------------------------------------------ compaction scan
__device__ __forceinline__ unsigned long long ldv64(const unsigned long long* p) { return *reinterpret_cast<const volatile unsigned long long*>(p); }

// One chain of the decoupled look-back, run by a whole warp: returns the
// exclusive prefix of `tile` (in every lane).  The warp reads 32 predecessor
// status words at once; it may add them up to the nearest published prefix
// once every tile in between has published its aggregate, and otherwise
// takes all 32 aggregates and moves 32 tiles back.  Waits are bounded.
__device__ uint32_t lookBackWarp(unsigned long long* st, uint32_t tile, uint32_t aggregate, unsigned long long tag, uint32_t* err) {
  const int lane = threadIdx.x & 31;
  if (tile == 0) {
    if (lane == 0) atomicExch(st, tag | kStFlagPre | aggregate);
    return 0;
  }
  if (lane == 0) atomicExch(st + tile, tag | kStFlagAgg | aggregate);
  uint32_t prefix = 0;
  int64_t j = int64_t(tile) - 1;  // nearest predecessor not yet added
  uint32_t spins = 0;
  for (;;) {
    const int64_t idx = j - lane;
    bool ready = true, isPre = true;  // before tile 0: an empty prefix
    uint32_t val = 0;
    if (idx >= 0) {
      const unsigned long long s = ldv64(st + idx);
      const bool mine = (s & ~((1ull << 50) - 1)) == tag;
      const unsigned long long flag = s & (3ull << 48);
      ready = mine && flag != 0;
      isPre = ready && flag == kStFlagPre;
      val = uint32_t(s & kStValue);
    }
    const uint32_t preMask = __ballot_sync(0xffffffffu, isPre);
    const uint32_t notReady = __ballot_sync(0xffffffffu, !ready);
    const int last = preMask ? __ffs(preMask) - 1 : 31;  // lanes 0..last are consumed
    const uint32_t need = last == 31 ? 0xffffffffu : ((2u << last) - 1u);
    if ((notReady & need) == 0u) {
      uint32_t v = lane <= last ? val : 0u;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      prefix += v;
      if (preMask) break;
      j -= 32;
      continue;
    }
    if (++spins > kBrickScanSpinLimit) {
      if (lane == 0) atomicOr(err, kErrScanTimeout);
      break;
    }
    __nanosleep(32);
  }
  if (lane == 0) atomicExch(st + tile, tag | kStFlagPre | uint32_t(prefix + aggregate));
  return prefix;
}

// One warp waits as tile 1 on a tile 0 that never publishes: the bounded
// look-back must give up after kBrickScanSpinLimit polls (a second or two),
// set kErrScanTimeout and return.
__global__ void k_wait_expiry_probe(unsigned long long* st, uint32_t* err) { (void)lookBackWarp(st, 1u, 0u, 0ull, err); }

// Tickets from the monotone counter number every tile of every launch: tile =
// ticket % tiles, launch = ticket / tiles.  Launches are stream-ordered, so one
// launch's tickets are contiguous, and no host-side value changes between
// launches (the kernel can be replayed from a CUDA graph).
__global__ void __launch_bounds__(kBrickScanThreads) k_brick_scan(BrickBuffers B, uint32_t* err) {
  __shared__ unsigned long long s_ticket;
  __shared__ uint32_t s_warp[3][kBrickScanThreads / 32];
  __shared__ uint32_t s_prefix[3];
  waitForPredecessorGrid();
  if (threadIdx.x == 0) s_ticket = atomicAdd(B.scanTile, 1ull);
  __syncthreads();
  const uint32_t tile = uint32_t(s_ticket % B.tiles);
  const uint32_t epoch = uint32_t(s_ticket / B.tiles);
  const unsigned long long tag = (unsigned long long)(epoch & 0x3fffu) << 50;
  const uint32_t b0 = tile * kBrickScanTile + threadIdx.x * kBrickScanItems;
  static_assert(kBrickScanItems == 8, "the vector path moves 8 bricks as two uint4");
  uint32_t cnt[kBrickScanItems];
  uint32_t flg = 0;  // bit k: grid-active
  uint32_t sc = 0, sp = 0, sg = 0;
  const bool full = b0 + kBrickScanItems <= B.nb;  // b0 is a multiple of 8: 32-byte aligned
  if (full) {
    uint4* pc = reinterpret_cast<uint4*>(B.brickCount + b0);
    uint4* pf = reinterpret_cast<uint4*>(B.brickFlag + b0);
    const uint4 c0 = pc[0], c1 = pc[1], f0 = pf[0], f1 = pf[1];
    const uint4 z = make_uint4(0u, 0u, 0u, 0u);
    pc[0] = z; pc[1] = z; pf[0] = z; pf[1] = z;
    cnt[0] = c0.x; cnt[1] = c0.y; cnt[2] = c0.z; cnt[3] = c0.w;
    cnt[4] = c1.x; cnt[5] = c1.y; cnt[6] = c1.z; cnt[7] = c1.w;
    const uint32_t fv[8] = {f0.x, f0.y, f0.z, f0.w, f1.x, f1.y, f1.z, f1.w};
#pragma unroll
    for (int k = 0; k < kBrickScanItems; ++k)
      if (fv[k]) flg |= 1u << k;
  } else {
#pragma unroll
    for (int k = 0; k < kBrickScanItems; ++k) {
      const uint32_t b = b0 + k;
      cnt[k] = 0;
      if (b < B.nb) {
        cnt[k] = B.brickCount[b];
        const uint32_t f = B.brickFlag[b];
        B.brickCount[b] = 0;
        B.brickFlag[b] = 0;
        if (f) flg |= 1u << k;
      }
    }
  }
#pragma unroll
  for (int k = 0; k < kBrickScanItems; ++k) {
    sc += cnt[k];
    sp += cnt[k] ? 1u : 0u;
  }
  sg = __popc(flg);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t ic = sc, ip = sp, ig = sg;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t yc = __shfl_up_sync(0xffffffffu, ic, o), yp = __shfl_up_sync(0xffffffffu, ip, o), yg = __shfl_up_sync(0xffffffffu, ig, o);
    if (lane >= o) {
      ic += yc;
      ip += yp;
      ig += yg;
    }
  }
  if (lane == 31) {
    s_warp[0][warp] = ic;
    s_warp[1][warp] = ip;
    s_warp[2][warp] = ig;
  }
  __syncthreads();
  if (warp == 0) {
    constexpr int W = kBrickScanThreads / 32;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      uint32_t w = lane < W ? s_warp[c][lane] : 0u;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += y;
      }
      if (lane < W) s_warp[c][lane] = w;
    }
  }
  __syncthreads();
  constexpr int WL = kBrickScanThreads / 32 - 1;
  // chains run in three different warps
  if (warp < 3) {
    const int c = warp;
    const uint32_t agg = s_warp[c][WL];
    const uint32_t pre = lookBackWarp(B.scanState + size_t(c) * B.tiles, tile, agg, tag, err);
    if (lane == 0) s_prefix[c] = pre;
    if (lane == 0 && tile == B.tiles - 1) {
      const uint32_t total = pre + agg;
      if (c == 0) {
        B.counters[kCntTotal] = total;
      } else if (c == 1) {
        B.counters[kCntNumPB] = total;
      } else {
        B.counters[kCntNumGB] = total;
      }
    }
  }
  __syncthreads();
  uint32_t rc = s_prefix[0] + (warp > 0 ? s_warp[0][warp - 1] : 0u) + ic - sc;
  uint32_t rp = s_prefix[1] + (warp > 0 ? s_warp[1][warp - 1] : 0u) + ip - sp;
  uint32_t rg = s_prefix[2] + (warp > 0 ? s_warp[2][warp - 1] : 0u) + ig - sg;
  uint32_t starts[kBrickScanItems];
#pragma unroll
  for (int k = 0; k < kBrickScanItems; ++k) {
    const uint32_t b = b0 + k;
    starts[k] = rc;
    if (b < B.nb) {
      if (!full) B.brickStart[b] = rc;
      if (cnt[k]) {
        B.pbBrick[rp] = b;
        B.pbStart[rp] = rc;
        ++rp;
      }
      if (flg & (1u << k)) {
        B.gbBrick[rg] = b;
        ++rg;
      }
    }
    rc += cnt[k];
  }
  if (full) {
    uint4* ps = reinterpret_cast<uint4*>(B.brickStart + b0);
    ps[0] = make_uint4(starts[0], starts[1], starts[2], starts[3]);
    ps[1] = make_uint4(starts[4], starts[5], starts[6], starts[7]);
  }
  if (tile == B.tiles - 1 && threadIdx.x == 0) {
    // the last tile's look-back finished, so all three totals are final
    const uint32_t npb = s_prefix[1] + s_warp[1][WL];
    B.pbStart[npb] = s_prefix[0] + s_warp[0][WL];
  }
}

// Sorted slots of the buffer indices t of one warp (every lane calls it; `valid`
// per lane): the start of the particle's brick, plus the counts of the cells
// of the brick below its cell, plus its rank in its cell.  The lanes' keys
// come in a few bricks (the buffer holds particles in cell order), and for
// each distinct brick the warp reads its 64 counts once (two per lane) and
// scans them.
__device__ __forceinline__ void permScatterWarp(const BrickBuffers& B, uint32_t n, uint32_t* err, uint32_t t, bool valid) {
  const uint32_t lane = laneId();
  const uint32_t key = valid ? B.binKey[t] : 0u;
  const uint32_t rank = valid ? B.binRank[t] : 0u;
  const uint32_t brick = key >> 6, cell = key & 63u;
  const uint32_t start = valid ? B.brickStart[brick] : 0u;
  uint32_t below = 0;
  uint32_t pending = __ballot_sync(0xffffffffu, valid);
  while (pending) {
    const uint32_t b = __shfl_sync(0xffffffffu, brick, __ffs(pending) - 1);
    const uint2 c = reinterpret_cast<const uint2*>(B.cellCount + (size_t(b) << 6))[lane];
    uint32_t incl = c.x + c.y;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= uint32_t(o)) incl += y;
    }
    const uint32_t pairBelow = __shfl_sync(0xffffffffu, incl - c.x - c.y, cell >> 1);
    const uint32_t evenCount = __shfl_sync(0xffffffffu, c.x, cell >> 1);
    const bool mine = valid && brick == b;
    if (mine) below = pairBelow + ((cell & 1u) ? evenCount : 0u);
    pending &= ~__ballot_sync(0xffffffffu, mine);
  }
  if (valid) {
    const uint32_t slot = start + below + rank;
    if (slot < n) B.perm[slot] = t;
    else atomicOr(err, kErrBinRange);
  }
}

// The same over buffer indices t0, t0 + stride, ... < n (t0 - lane and stride
// multiples of 32, so the warp's lanes stay together).
__device__ __forceinline__ void permScatterStrided(const BrickBuffers& B, uint32_t n, uint32_t* err, uint64_t t0, uint64_t stride) {
  for (uint64_t w = t0 - laneId(); w < n; w += stride) {
    const uint64_t t = w + laneId();
    permScatterWarp(B, n, err, uint32_t(t < n ? t : 0u), t < n);
  }
}

// The separate permutation launch: each warp takes kPermRounds groups of 32
// buffer indices and issues the loads of all groups before their sums (the
// key -> brick start / counts -> slot chain is the kernel's latency); a group
// whose lanes hold more than one brick finishes the other bricks one by one.
constexpr int kPermRounds = 4;
__global__ void __launch_bounds__(kThreads) k_perm_scatter(BrickBuffers B, uint32_t n, uint32_t* err) {
  waitForPredecessorGrid();
  const uint32_t lane = laneId();
  const uint32_t base = (blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5)) * (32u * kPermRounds);
  uint32_t t[kPermRounds], key[kPermRounds], rank[kPermRounds], start[kPermRounds], lead[kPermRounds];
  uint2 c[kPermRounds];
#pragma unroll
  for (int r = 0; r < kPermRounds; ++r) {
    t[r] = base + uint32_t(r) * 32u + lane;
    const bool v = t[r] < n;
    key[r] = v ? B.binKey[t[r]] : 0u;
    rank[r] = v ? B.binRank[t[r]] : 0u;
  }
#pragma unroll
  for (int r = 0; r < kPermRounds; ++r) {
    const bool v = t[r] < n;
    start[r] = v ? B.brickStart[key[r] >> 6] : 0u;
    lead[r] = __shfl_sync(0xffffffffu, key[r] >> 6, 0);  // the brick of the group's first lane (lane 0 is valid whenever any lane is)
    c[r] = reinterpret_cast<const uint2*>(B.cellCount + (size_t(lead[r]) << 6))[lane];
  }
#pragma unroll
  for (int r = 0; r < kPermRounds; ++r) {
    const bool v = t[r] < n;
    const uint32_t brick = key[r] >> 6, cell = key[r] & 63u;
    uint32_t incl = c[r].x + c[r].y;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= uint32_t(o)) incl += y;
    }
    const uint32_t pairBelow = __shfl_sync(0xffffffffu, incl - c[r].x - c[r].y, cell >> 1);
    const uint32_t evenCount = __shfl_sync(0xffffffffu, c[r].x, cell >> 1);
    const bool first = v && brick == lead[r];
    uint32_t below = first ? pairBelow + ((cell & 1u) ? evenCount : 0u) : 0u;
    if (__ballot_sync(0xffffffffu, v && !first)) {
      // lanes of other bricks: the general per-brick walk
      uint32_t pending = __ballot_sync(0xffffffffu, v && !first);
      while (pending) {
        const uint32_t b = __shfl_sync(0xffffffffu, brick, __ffs(pending) - 1);
        const uint2 cb = reinterpret_cast<const uint2*>(B.cellCount + (size_t(b) << 6))[lane];
        uint32_t in2 = cb.x + cb.y;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t y = __shfl_up_sync(0xffffffffu, in2, o);
          if (lane >= uint32_t(o)) in2 += y;
        }
        const uint32_t pb = __shfl_sync(0xffffffffu, in2 - cb.x - cb.y, cell >> 1);
        const uint32_t ec = __shfl_sync(0xffffffffu, cb.x, cell >> 1);
        const bool mine = v && !first && brick == b;
        if (mine) below = pb + ((cell & 1u) ? ec : 0u);
        pending &= ~__ballot_sync(0xffffffffu, mine);
      }
    }
    if (v) {
      const uint32_t slot = start[r] + below + rank[r];
      if (slot < n) B.perm[slot] = t[r];
      else atomicOr(err, kErrBinRange);
    }
  }
}

// ------------------------------------------------------------------ P2G of sorted particles (standalone)
// Slots [0, n) in rounds of 32, one per warp; a round of a batch that spans
// scenes is taken scene by scene.
template <bool BATCH>
__global__ void __launch_bounds__(kThreads) k_p2g_sorted(SubstepParams P0, SceneTable T, StatePtrs cur, uint32_t n, BrickBuffers B, GridBuffers G,
                                                         float dtStress) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int warp = threadIdx.x >> 5;
  const uint32_t lane = laneId();
  WarpRows& W = reinterpret_cast<WarpRows*>(smem_raw)[warp];
  const uint32_t warps = blockDim.x >> 5;
  auto part = [&](const SubstepParams& P, const GridBuffers& g, float dts, uint32_t t, bool act) {
    uint32_t key = kNoKey;
    bool exact = false;
    if (act) {
      const uint32_t s = B.perm[t];
      if (s < n) {
        const PState st = loadState(cur.f, s);
        int cx, cy, cz;
        cellCoords(P, st.P.x, st.P.y, st.P.z, cx, cy, cz);
        float m;
        exact = p2gRow(P, st, dts, cx, cy, cz, W.rows + lane * kRow, m);
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
      p2gGroup(P, W, k, peers, exactMask, [&](uint32_t c, const float* a) { redAddV4(g.acc + c, a[0], a[1], a[2], a[3]); });
    }
    __syncwarp();  // every lane has read the rows before they are written again
  };
  for (uint64_t t0 = (uint64_t(blockIdx.x) * warps + warp) * 32u; t0 < n; t0 += uint64_t(gridDim.x) * warps * 32u) {
    const uint32_t t = uint32_t(t0) + lane;
    if constexpr (BATCH) {
      __shared__ SubstepParams sP[kThreads / 32];
      const uint32_t end = min(uint32_t(t0) + 32u, n);
      for (uint32_t lo = uint32_t(t0); lo < end;) {
        const uint32_t sc = findScene(T.partBase, T.count, lo), hi = min(T.partBase[sc + 1u], end);
        __syncwarp();
        copyParams(&sP[warp], T.params + sc, int(lane), 32);
        __syncwarp();
        part(sP[warp], offsetGrid(G, T.brickBase[sc]), sP[warp].dt, t, t >= lo && t < hi);
        lo = hi;
      }
    } else {
      part(P0, G, dtStress, t, t < n);
    }
  }
}

// ------------------------------------------------------------------ sparse grid update
// Per thread, kGridBatch nodes per round (2 or 4, picked by the launch
// configuration): their brick ids, then their accumulators (and an L1
// prefetch of their SDF samples) are loaded before any node is updated, so
// one round costs about the memory round trips of one node.
// The kernel also scatters the permutation of the binning that precedes it
// (the scan's brick starts, the fused kernel's keys and ranks) when n > 0:
// the grid update does not read it and the next fused kernel does, so the
// scatter needs no launch of its own.  Scattering the same binning twice
// writes the same values.
template <int kGridBatch>
__global__ void __launch_bounds__(kThreads) k_grid_bricks(SubstepParams P, BrickBuffers B, GridBuffers G, uint32_t n, uint32_t* err) {
  waitForPredecessorGrid();
  const uint64_t total = uint64_t(B.counters[kCntNumGB]) * 64u;
  const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
  permScatterStrided(B, n, err, uint64_t(blockIdx.x) * blockDim.x + threadIdx.x, stride);
  for (uint64_t g0 = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; g0 < total; g0 += stride * kGridBatch) {
    uint32_t code[kGridBatch];
    bool live[kGridBatch];
#pragma unroll
    for (int k = 0; k < kGridBatch; ++k) {
      const uint64_t g = g0 + uint64_t(k) * stride;
      live[k] = g < total;
      code[k] = live[k] ? ((B.gbBrick[g >> 6] << 6) | uint32_t(g & 63u)) : 0u;
      live[k] = live[k] && code[k] < P.hashCells;
    }
    float4 a[kGridBatch];
#pragma unroll
    for (int k = 0; k < kGridBatch; ++k) {
      a[k] = live[k] ? G.acc[code[k]] : make_float4(0.f, 0.f, 0.f, 0.f);
      if (live[k] && P.sdf) {
        // the node's SDF sample and its six neighbours (read when the node is
        // within 1.5 h of the surface): the second read hits L1 (-7% per launch)
        int ix, iy, iz;
        mortonDecode(code[k], ix, iy, iz);
        const int cm = int(P.cubeRes) - 1;
        const float* f = P.sdf;
        asm volatile("prefetch.global.L1 [%0];" ::"l"(f + code[k]));
        asm volatile("prefetch.global.L1 [%0];" ::"l"(f + mortonEncode(min(ix + 1, cm), iy, iz)));
        asm volatile("prefetch.global.L1 [%0];" ::"l"(f + mortonEncode(max(ix - 1, 0), iy, iz)));
        asm volatile("prefetch.global.L1 [%0];" ::"l"(f + mortonEncode(ix, min(iy + 1, cm), iz)));
        asm volatile("prefetch.global.L1 [%0];" ::"l"(f + mortonEncode(ix, max(iy - 1, 0), iz)));
        asm volatile("prefetch.global.L1 [%0];" ::"l"(f + mortonEncode(ix, iy, min(iz + 1, cm))));
        asm volatile("prefetch.global.L1 [%0];" ::"l"(f + mortonEncode(ix, iy, max(iz - 1, 0))));
      }
    }
#pragma unroll
    for (int k = 0; k < kGridBatch; ++k) {
      if (!live[k]) continue;
      const uint32_t c = code[k];
      G.acc[c] = make_float4(0.f, 0.f, 0.f, 0.f);
      int ix, iy, iz;
      mortonDecode(c, ix, iy, iz);
      float3 v, vo;
      const bool ok = gridNode(P, ix, iy, iz, a[k].w, a[k].x, a[k].y, a[k].z, v, vo);
      G.vel[c] = ok ? make_float4(v.x, v.y, v.z, a[k].w) : make_float4(0.f, 0.f, 0.f, a[k].w);
      if (G.vold) G.vold[c] = ok ? make_float4(vo.x, vo.y, vo.z, 0.f) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
}

// Batched grid update: one warp per listed grid brick, two nodes per lane, the
// brick's scene parameters in a warp-private shared copy.
// Also scatters the permutation of the preceding binning (as k_grid_bricks).
__global__ void __launch_bounds__(kThreads) k_grid_bricks_batch(SceneTable T, uint32_t substep, BrickBuffers B, GridBuffers G, uint32_t n,
                                                                uint32_t* err) {
  __shared__ SubstepParams sP[kThreads / 32];
  waitForPredecessorGrid();
  permScatterStrided(B, n, err, uint64_t(blockIdx.x) * blockDim.x + threadIdx.x, uint64_t(gridDim.x) * blockDim.x);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t numGB = B.counters[kCntNumGB];
  // Each warp takes a contiguous run of the (ascending) grid-brick list, so
  // consecutive bricks mostly share a scene: the scene is searched once and
  // then advanced, and its parameters are copied only when it changes.
  const uint32_t warps = gridDim.x * (kThreads / 32), gw = blockIdx.x * (kThreads / 32) + warp;
  const uint32_t per = (numGB + warps - 1) / warps;
  const uint32_t g0 = min(gw * per, numGB), g1 = min(g0 + per, numGB);
  uint32_t sc = g0 < g1 ? findScene(T.brickBase, T.count, B.gbBrick[g0]) : 0u;
  uint32_t loaded = 0xFFFFFFFFu;
  for (uint32_t gb = g0; gb < g1; ++gb) {
    const uint32_t bg = B.gbBrick[gb];
    // k_brick_scan lists grid bricks in ascending order, so the scene only
    // moves forward; a brick below the current scene's base (a list built
    // otherwise) is searched for again instead of taking the wrong scene
    if (bg < T.brickBase[sc]) sc = findScene(T.brickBase, T.count, bg);
    while (sc + 1u < T.count && T.brickBase[sc + 1u] <= bg) ++sc;
    const uint32_t base = T.brickBase[sc];
    if (sc != loaded) {
      __syncwarp();
      copyParams(&sP[warp], T.params + sc, lane, 32);
      __syncwarp();
      if (lane == 0) sP[warp].colliders += size_t(substep) * sP[warp].colliderCount;
      __syncwarp();
      loaded = sc;
    }
    const SubstepParams& P = sP[warp];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint32_t sub = uint32_t(lane + 32 * h);
      const uint32_t local = ((bg - base) << 6) | sub;
      if (local >= P.hashCells) continue;
      const size_t code = (size_t(bg) << 6) | sub;
      const float4 a = G.acc[code];
      G.acc[code] = make_float4(0.f, 0.f, 0.f, 0.f);
      int ix, iy, iz;
      mortonDecode(local, ix, iy, iz);
      float3 v, vo;
      const bool ok = gridNode(P, ix, iy, iz, a.w, a.x, a.y, a.z, v, vo);
      G.vel[code] = ok ? make_float4(v.x, v.y, v.z, a.w) : make_float4(0.f, 0.f, 0.f, a.w);
      if (G.vold) G.vold[code] = ok ? make_float4(vo.x, vo.y, vo.z, 0.f) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
}

__global__ void __launch_bounds__(kThreads) k_clear_bricks(BrickBuffers B, GridBuffers G) {
  const uint64_t total = uint64_t(B.counters[kCntNumGB]) * 64u;
  for (uint64_t g = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; g < total; g += uint64_t(gridDim.x) * blockDim.x) {
    const uint32_t code = (B.gbBrick[g >> 6] << 6) | uint32_t(g & 63u);
    G.acc[code] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
}

// ------------------------------------------------------------------ fused G2P -> update -> P2G
// G2P node source: the grid in global memory (velocities are zero where a
// node is lighter than 1e-10).
template <bool FLIP>
struct GlobalGrid {
  const float4* gvel;
  const float4* gvold;
  __device__ __forceinline__ bool node(int x, int y, int z, float& m, float3& v, float3& vo) const {
    const uint32_t c = mortonEncode(x, y, z);
    const float4 a = gvel[c];
    m = a.w;
    if (m < 1e-10f) return false;
    v = make_float3(a.x, a.y, a.z);
    if (FLIP) {
      const float4 b = gvold[c];
      vo = make_float3(b.x, b.y, b.z);
    }
    return true;
  }
};

// The gather of a particle whose stencil leaves [0, gridRes), out of line: it
// takes a caller's state outside the domain to get here, and inline it was half
// of a kernel whose warps run apart and whose largest stall is the instruction
// cache (8,000 elastic particles 19 -> 17 us, 1,000,000 Drucker-Prager 302 ->
// 286).  The parameters are a __grid_constant__, so that passing them by
// reference copies nothing.
struct Gathered {
  float v[3], vo[3], G[3][3], B[3][3];
};
template <bool FLIP>
__device__ __noinline__ Gathered gatherOutside(const SubstepParams& P, float x, float y, float z, const float4* vel, const float4* vold) {
  Gathered g;
  PState s;
  s.P = make_float4(x, y, z, 0.f);
  g2pGather(P, s, GlobalGrid<FLIP>{vel, vold}, g.v, g.vo, g.G, g.B);
  return g;
}

// One round: the sorted slots t of a warp's lanes (`act`).  The binning orders
// particles by cell (bricks in Morton order, the 64 cells of a brick in Morton
// order), so the 32 slots hold the particles of a few neighbouring cells: the
// gather's loads are mostly the same few cache lines, and the lanes' new cells
// fall into a few groups.  Per particle: G2P from the grid, particle update,
// write to its slot in the next buffer and its P2G row.  Per group of lanes
// with the same new cell: binning counts under the global cell key 64
// brickBase + Morton code (the rank is read after the P2G, so the atomic's
// round trip overlaps it), P2G into the grid, and the marks of its stencil's
// bricks.
template <bool FLIP, int MS>
__device__ __forceinline__ void g2p2gRound(const SubstepParams& P, WarpRows& W, uint32_t t, bool act, uint32_t brickBase, StatePtrs cur,
                                           const uint32_t* __restrict__ pidCur, StatePtrs nxt, uint32_t* __restrict__ pidNxt, uint32_t n,
                                           const BrickBuffers& B, const GridBuffers& G, float dtStress, uint32_t* err) {
  const uint32_t lane = laneId();
  uint32_t key = kNoKey, nc = 0;
  bool exact = false, placed = false;
  if (act) {
    const uint32_t s = B.perm[t];
    if (s < n) {
      PState st = loadState(cur.f, s);
      const uint32_t pid = pidCur[s];
      float vpic[3], vpo[3], Gv[3][3], Bn[3][3];
      int ox, oy, oz;
      if (!g2pGatherGrid<FLIP>(P, st, G.vel, G.vold, vpic, vpo, Gv, Bn, ox, oy, oz)) {
        const Gathered g = gatherOutside<FLIP>(P, st.P.x, st.P.y, st.P.z, G.vel, G.vold);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          vpic[i] = g.v[i];
          vpo[i] = g.vo[i];
#pragma unroll
          for (int j = 0; j < 3; ++j) {
            Gv[i][j] = g.G[i][j];
            Bn[i][j] = g.B[i][j];
          }
        }
      }
      g2pUpdate<MS>(P, st, P.dt, vpic, vpo, Gv, Bn);
      storeState(nxt.f, t, st);
      pidNxt[t] = pid;
      if (!(isfinite(st.P.x) && isfinite(st.P.y) && isfinite(st.P.z))) atomicOr(err, kErrNonFinite);
      int cx, cy, cz;
      cellCoords(P, st.P.x, st.P.y, st.P.z, cx, cy, cz);
      // particles that left the cells around their brick in one substep are counted
      if (((unsigned(cx + 1 - (ox & ~3)) > 5u) | (unsigned(cy + 1 - (oy & ~3)) > 5u) | (unsigned(cz + 1 - (oz & ~3)) > 5u)))
        atomicAdd(B.counters + kCntOverflow, 1u);
      nc = (brickBase << 6) + mortonEncode(cx, cy, cz);
      float m;
      exact = p2gRow(P, st, dtStress, cx, cy, cz, W.rows + lane * kRow, m);
      W.mass[lane] = m;
      key = packCell(cx, cy, cz);
      placed = true;
    } else {
      atomicOr(err, kErrBinRange);  // a slot that maps nowhere: only after an expired scan wait
      nc = brickBase << 6;
      key = 0u;  // counted in the scene's first cell, without P2G
    }
    B.binKey[t] = nc;
  }
  const uint32_t exactMask = __ballot_sync(0xffffffffu, exact), placedMask = __ballot_sync(0xffffffffu, placed);
  __syncwarp();  // the rows are visible to every lane
  uint32_t pending = __ballot_sync(0xffffffffu, act), mine = 0, base = 0;
  while (pending) {
    const int leader = __ffs(pending) - 1;
    const uint32_t k = __shfl_sync(0xffffffffu, key, leader);
    const uint32_t peers = __ballot_sync(0xffffffffu, key == k);
    pending &= ~peers;
    if (key == k) mine = peers;
    if (int(lane) == leader) {
      base = atomicAdd(B.cellCount + nc, uint32_t(__popc(peers)));
      atomicAdd(B.brickCount + (nc >> 6), uint32_t(__popc(peers)));
    }
    if (peers & placedMask)
      p2gGroup(P, W, k, peers & placedMask, exactMask, [&](uint32_t c, const float* a) {
        redAddV4(G.acc + c, a[0], a[1], a[2], a[3]);
        B.brickFlag[brickBase + (c >> 6)] = 1u;  // grid-active mark
      });
  }
  __syncwarp();  // every lane has read the rows before they are written again
  base = __shfl_sync(0xffffffffu, base, mine ? __ffs(mine) - 1 : int(lane));
  if (act) B.binRank[t] = base + uint32_t(__popc(mine & ((1u << lane) - 1u)));
}

// Warps take rounds of 32 sorted slots, `gridDim x warps` apart, and use nothing
// of one another's work (the CTAs of large scenes start their rounds together,
// below): no brick owns a CTA, so a scene of few or unevenly filled bricks spreads
// over the SMs as evenly as its rounds do, and a CTA has no staging or tile
// flush.  (The kernel used to hand particle bricks to CTAs: staged 6^3 velocities,
// an 8^3 shared accumulation tile, two barriers per brick.  A warp then waited for
// the slowest of its CTA -- the largest stall -- and a scene of 160 bricks left
// most warps idle.)  What bounds it is
// instruction issue and its latencies (60% of cycles issue on 1,000,000
// Drucker-Prager particles; L1 loads are the largest stall).  Per launch, bricks ->
// rounds, before the changes whose figures stand at gatherOutside and inStep:
// 8,000 elastic particles 26 -> 19 us, 85,184 Von Mises under FLIP 78 -> 38,
// 80,000 of the two-material scene 75 -> 33, 250,007 of all models 128 -> 92,
// 1,000,000 Drucker-Prager 363 -> 302.  With particles thinly spread, a warp's
// cells are many and its reductions with them, but the bricks are emptier still:
// a substep of 250,000 Drucker-Prager particles on 256^3 takes 91 us at 8 to a
// cell (bricks: 189), 120 at 2 (210), 127 at 1 (326), and 458 strewn at random over
// the domain (4,185).  256 threads, 3 CTAs per SM: 80 registers with some spills
// to L1-cached local memory.  MS: the material-model set compiled in.
template <bool FLIP, bool BATCH, int MS>
__global__ void __launch_bounds__(kThreads, 3) k_g2p2g(const __grid_constant__ SubstepParams P0, SceneTable T, StatePtrs cur, const uint32_t* __restrict__ pidCur, StatePtrs nxt,
                                                       uint32_t* __restrict__ pidNxt, uint32_t n, BrickBuffers B, GridBuffers G, float dtStress,
                                                       uint32_t* err) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  waitForPredecessorGrid();
  const int warp = threadIdx.x >> 5;
  const uint32_t lane = laneId();
  WarpRows& W = reinterpret_cast<WarpRows*>(smem_raw)[warp];
  const uint32_t gw = blockIdx.x * (blockDim.x >> 5) + uint32_t(warp), tw = gridDim.x * (blockDim.x >> 5);
  uint32_t loaded = 0xffffffffu;
  // The warps of a large scene's CTAs start their rounds together: what one
  // fetches of the 4,000 instructions of a round the others then find in the
  // instruction cache (1,000,000 particles 7.27 -> 6.84 ms a step of 25
  // substeps, 250,007 1.59 -> 1.52, a batch of 1,090,000 50.2 -> 45.4).  Scenes
  // in smaller CTAs run one or two rounds per warp and only lost the wait.
  const bool inStep = blockDim.x == kThreads;
#pragma unroll 1
  for (uint64_t c0 = uint64_t(gw - uint32_t(warp)) * 32u; c0 < n; c0 += uint64_t(tw) * 32u) {  // (the CTA's first slot: the same for all its warps)
    const uint64_t t0 = c0 + uint64_t(warp) * 32u;
    const uint32_t t = uint32_t(t0) + lane;
    if (inStep) __syncthreads();
    if (t0 >= n) continue;
    if constexpr (BATCH) {
      // a round that spans scenes is taken scene by scene
      __shared__ SubstepParams sP[kThreads / 32];
      const uint32_t end = min(uint32_t(t0) + 32u, n);
      for (uint32_t lo = uint32_t(t0); lo < end;) {
        const uint32_t sc = findScene(T.partBase, T.count, lo), hi = min(T.partBase[sc + 1u], end), bb = T.brickBase[sc];
        if (sc != loaded) {
          __syncwarp();
          copyParams(&sP[warp], T.params + sc, int(lane), 32);
          __syncwarp();
          loaded = sc;
        }
        g2p2gRound<FLIP, MS>(sP[warp], W, t, t >= lo && t < hi, bb, cur, pidCur, nxt, pidNxt, n, B, offsetGrid(G, bb), sP[warp].dt, err);
        lo = hi;
      }
    } else {
      g2p2gRound<FLIP, MS>(P0, W, t, t < n, 0u, cur, pidCur, nxt, pidNxt, n, B, G, dtStress, err);
    }
  }
  // the permutation has read the previous binning's counts: clear them for the binning after this one
  const uint32_t numPB = B.counters[kCntNumPB];
  for (uint32_t i = gw; i < numPB; i += tw)
    reinterpret_cast<uint2*>(B.cellPrev + (size_t(B.pbBrick[i]) << 6))[lane] = make_uint2(0u, 0u);
}

__global__ void __launch_bounds__(kThreads) k_unpermute(StatePtrs in, const uint32_t* __restrict__ pid, StatePtrs out, uint32_t n) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t d = pid[i];
  if (d >= n) return;
#pragma unroll
  for (int k = 0; k < 8; ++k) out.f[k][d] = in.f[k][i];
}

__global__ void __launch_bounds__(kThreads) k_sorted_pid(const uint32_t* __restrict__ perm, const uint32_t* __restrict__ pid, uint32_t* out,
                                                         uint32_t n) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const uint32_t s = perm[t];
  out[t] = s < n ? pid[s] : 0xffffffffu;
}

__global__ void __launch_bounds__(kThreads) k_iota(uint32_t* pid, uint32_t n) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) pid[i] = i;
}

template <class K> int ctasPerSm(K kernel, int threads, size_t smem = 0) {
  int perSM = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, kernel, threads, smem) != cudaSuccess || perSM < 1) perSM = 1;
  return perSM;
}

// Warps of a fused CTA that the launches use: 1, 2, 4 and 8 by scene size, 6 and 8 on request.
constexpr int kFusedWarps[] = {1, 2, 4, 6, 8};
constexpr int fusedSlot(int warps) { return warps <= 1 ? 0 : warps <= 2 ? 1 : warps <= 4 ? 2 : warps <= 6 ? 3 : 4; }

// Most CTAs per SM of every kernel variant, resolved once per device (kernel
// attributes are per device; the queries stay outside stream capture).
struct LaunchShapes {
  std::atomic<bool> ready{false};
  int p2g[2] = {0, 0};      // [BATCH]
  int grid[2] = {0, 0};     // [gridBatch == 4]
  int gridBatch = 0;        // batched grid kernel
  int fused[2][2][5] = {};  // [FLIP][BATCH][fusedSlot(warps)]
};
constexpr int kShapeSlots = 64;  // device ordinals beyond this share slots modulo 64
LaunchShapes g_shapes[kShapeSlots];
std::mutex g_shapesMutex;

template <bool FLIP, bool BATCH, int MS> void setupFused(LaunchShapes& L) {
  // every model set has the same shared memory and register bound
  for (int w : kFusedWarps) L.fused[FLIP][BATCH][fusedSlot(w)] = ctasPerSm(k_g2p2g<FLIP, BATCH, MS>, 32 * w, size_t(w) * sizeof(WarpRows));
}

const LaunchShapes& shapes() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0) dev = 0;
  LaunchShapes& L = g_shapes[dev % kShapeSlots];
  if (L.ready.load(std::memory_order_acquire)) return L;
  std::lock_guard<std::mutex> lock(g_shapesMutex);
  if (L.ready.load(std::memory_order_relaxed)) return L;
  L.p2g[0] = ctasPerSm(k_p2g_sorted<false>, kThreads, kThreads / 32 * sizeof(WarpRows));
  L.p2g[1] = ctasPerSm(k_p2g_sorted<true>, kThreads, kThreads / 32 * sizeof(WarpRows));
  L.grid[0] = ctasPerSm(k_grid_bricks<2>, kThreads);
  L.grid[1] = ctasPerSm(k_grid_bricks<4>, kThreads);
  L.gridBatch = ctasPerSm(k_grid_bricks_batch, kThreads);
  setupFused<false, false, kModelsElastic>(L);
  setupFused<false, false, kModelsDruckerPrager>(L);
  setupFused<false, false, kModelsElasticVonMises>(L);
  setupFused<false, false, kModelsElasticDruckerPrager>(L);
  setupFused<false, false, kModelsAny>(L);
  setupFused<false, true, kModelsElasticVonMises>(L);
  setupFused<false, true, kModelsAny>(L);
  setupFused<true, false, kModelsElasticVonMises>(L);
  setupFused<true, false, kModelsElasticDruckerPrager>(L);
  setupFused<true, false, kModelsAny>(L);
  setupFused<true, true, kModelsAny>(L);
  L.ready.store(true, std::memory_order_release);
  return L;
}

// Blocks of a persistent launch: the requested CTAs per SM (0 = most that fit), capped by occupancy.
int persistentGrid(uint32_t requested, int most, int numSMs) {
  const int per = requested == 0 ? most : std::min(int(requested), most);
  return std::max(per, 1) * numSMs;
}

}  // namespace

LaunchLimits launchLimits(bool flip, bool batch) {
  const LaunchShapes& L = shapes();
  LaunchLimits out;
  out.fusedCtasPerSm[0] = uint32_t(L.fused[flip][batch][fusedSlot(6)]);
  out.fusedCtasPerSm[1] = uint32_t(L.fused[flip][batch][fusedSlot(8)]);
  out.gridCtasPerSm[0] = uint32_t(L.grid[0]);
  out.gridCtasPerSm[1] = uint32_t(L.grid[1]);
  return out;
}

cudaError_t probeWaitExpiry(uint32_t* errorBits) {
  unsigned long long* st = nullptr;
  uint32_t* err = nullptr;
  cudaError_t e = cudaMalloc(&st, 2 * sizeof(unsigned long long));
  if (e == cudaSuccess) e = cudaMalloc(&err, sizeof(uint32_t));
  if (e == cudaSuccess) e = cudaMemset(st, 0, 2 * sizeof(unsigned long long));
  if (e == cudaSuccess) e = cudaMemset(err, 0, sizeof(uint32_t));
  if (e == cudaSuccess) {
    k_wait_expiry_probe<<<1, 32>>>(st, err);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(errorBits, err, sizeof(uint32_t), cudaMemcpyDeviceToHost);
  cudaFree(st);
  cudaFree(err);
  return e;
}

void prepareBrickKernels(int numSMs) {
  (void)numSMs;
  (void)shapes();
}

cudaError_t launchBrickCount(const SubstepParams& P, const float4* pos, uint32_t n, const BrickBuffers& b, uint32_t* err, cudaStream_t s,
                             uint64_t* launches) {
  (void)err;
  if (n == 0) return cudaSuccess;
  k_brick_count<false><<<blocksFor(n), kThreads, 0, s>>>(P, SceneTable{}, pos, n, b);
  ++*launches;
  return cudaGetLastError();
}

cudaError_t launchBrickCountBatch(const SceneTable& T, const float4* pos, uint32_t n, const BrickBuffers& b, cudaStream_t s, uint64_t* launches) {
  if (n == 0) return cudaSuccess;
  k_brick_count<true><<<blocksFor(n), kThreads, 0, s>>>(SubstepParams{}, T, pos, n, b);
  ++*launches;
  return cudaGetLastError();
}

cudaError_t launchBrickScan(const BrickBuffers& b, uint32_t* err, cudaStream_t s, uint64_t* launches) {
  const cudaError_t e = launchSerialized(k_brick_scan, dim3(b.tiles), dim3(kBrickScanThreads), 0, s, b, err);
  ++*launches;
  return e;
}

cudaError_t launchPermScatter(const BrickBuffers& b, uint32_t n, uint32_t* err, cudaStream_t s, uint64_t* launches) {
  if (n == 0) return cudaSuccess;
  const cudaError_t e = launchSerialized(k_perm_scatter, dim3(blocksFor(n, kThreads * kPermRounds)), dim3(kThreads), 0, s, b, n, err);
  ++*launches;
  return e;
}

cudaError_t launchP2GBricks(const SubstepParams& P, StatePtrs cur, uint32_t n, const BrickBuffers& b, GridBuffers g, float dtStress,
                            int numSMs, cudaStream_t s, uint64_t* launches) {
  if (n == 0) return cudaSuccess;
  const int blocks = std::min(shapes().p2g[0] * numSMs, int(blocksFor(n)));
  k_p2g_sorted<false><<<blocks, kThreads, kThreads / 32 * sizeof(WarpRows), s>>>(P, SceneTable{}, cur, n, b, g, dtStress);
  ++*launches;
  return cudaGetLastError();
}

cudaError_t launchP2GBricksBatch(const SceneTable& T, StatePtrs cur, uint32_t n, const BrickBuffers& b, GridBuffers g, int numSMs,
                                 cudaStream_t s, uint64_t* launches) {
  if (n == 0) return cudaSuccess;
  const int blocks = std::min(shapes().p2g[1] * numSMs, int(blocksFor(n)));
  k_p2g_sorted<true><<<blocks, kThreads, kThreads / 32 * sizeof(WarpRows), s>>>(SubstepParams{}, T, cur, n, b, g, 0.f);
  ++*launches;
  return cudaGetLastError();
}

cudaError_t launchGridBricks(const SubstepParams& P, const BrickBuffers& b, GridBuffers g, uint32_t n, uint32_t* err, const LaunchConfig& lc,
                             int numSMs, cudaStream_t s, uint64_t* launches) {
  const LaunchShapes& L = shapes();
  const cudaError_t e = lc.gridBatch == 2
                            ? launchSerialized(k_grid_bricks<2>, dim3(persistentGrid(lc.gridCtasPerSm, L.grid[0], numSMs)), dim3(kThreads), 0, s,
                                               P, b, g, n, err)
                            : launchSerialized(k_grid_bricks<4>, dim3(persistentGrid(lc.gridCtasPerSm, L.grid[1], numSMs)), dim3(kThreads), 0, s,
                                               P, b, g, n, err);
  ++*launches;
  return e;
}

cudaError_t launchGridBricksBatch(const SceneTable& T, uint32_t substep, const BrickBuffers& b, GridBuffers g, uint32_t n, uint32_t* err,
                                  const LaunchConfig& lc, int numSMs, cudaStream_t s, uint64_t* launches) {
  const cudaError_t e = launchSerialized(k_grid_bricks_batch, dim3(persistentGrid(lc.gridCtasPerSm, shapes().gridBatch, numSMs)), dim3(kThreads), 0,
                                         s, T, substep, b, g, n, err);
  ++*launches;
  return e;
}

cudaError_t launchClearBricks(const BrickBuffers& b, GridBuffers g, int numSMs, cudaStream_t s, uint64_t* launches) {
  k_clear_bricks<<<numSMs * 4, kThreads, 0, s>>>(b, g);
  ++*launches;
  return cudaGetLastError();
}

namespace {

template <bool FLIP, bool BATCH, int MS>
cudaError_t launchFused(const LaunchConfig& lc, const SubstepParams& P, const SceneTable& T, StatePtrs cur, const uint32_t* pidCur, StatePtrs nxt,
                        uint32_t* pidNxt, uint32_t n, const BrickBuffers& b, GridBuffers g, float dtStress, uint32_t* err, int numSMs, cudaStream_t s) {
  // Warps per CTA: as asked for, or so that a scene of few rounds has at least
  // four CTAs per SM to spread over the chip: a CTA lands on one SM, and 8,000
  // particles (250 rounds) in CTAs of eight warps would use 32 SMs.
  const uint32_t rounds = (n + 31u) / 32u, fit = rounds / uint32_t(4 * std::max(numSMs, 1));
  const int warps = lc.fusedThreads ? int(lc.fusedThreads / 32u) : fit >= 8u ? 8 : fit >= 4u ? 4 : fit >= 2u ? 2 : 1;
  const int most = persistentGrid(lc.fusedCtasPerSm, shapes().fused[FLIP][BATCH][fusedSlot(warps)], numSMs);
  const int blocks = std::max(1, std::min(most, int((rounds + uint32_t(warps) - 1u) / uint32_t(warps))));
  return launchSerialized(k_g2p2g<FLIP, BATCH, MS>, dim3(blocks), dim3(32 * warps), size_t(warps) * sizeof(WarpRows), s, P, T, cur, pidCur, nxt, pidNxt,
                          n, b, g, dtStress, err);
}

// The instantiation for the transfer and the model set.  Specialised kernels:
// every set for APIC or PIC transfer, the two mixed sets for FLIP (which the
// single-family scenes take too; 85,184 Von Mises particles 676 -> 649 us a step
// of 25 substeps against the any-model kernel), the elastic / Von Mises set
// for batches.
template <bool BATCH>
cudaError_t launchFusedFor(bool flip, int modelSet, const LaunchConfig& lc, const SubstepParams& P, const SceneTable& T, StatePtrs cur,
                           const uint32_t* pidCur, StatePtrs nxt, uint32_t* pidNxt, uint32_t n, const BrickBuffers& b, GridBuffers g, float dtStress,
                           uint32_t* err, int numSMs, cudaStream_t s) {
  if constexpr (!BATCH) {
    if (flip && (modelSet == kModelsElasticVonMises || modelSet == kModelsElastic))
      return launchFused<true, false, kModelsElasticVonMises>(lc, P, T, cur, pidCur, nxt, pidNxt, n, b, g, dtStress, err, numSMs, s);
    if (flip && (modelSet == kModelsElasticDruckerPrager || modelSet == kModelsDruckerPrager))
      return launchFused<true, false, kModelsElasticDruckerPrager>(lc, P, T, cur, pidCur, nxt, pidNxt, n, b, g, dtStress, err, numSMs, s);
  }
  if (flip) return launchFused<true, BATCH, kModelsAny>(lc, P, T, cur, pidCur, nxt, pidNxt, n, b, g, dtStress, err, numSMs, s);
  if (modelSet == kModelsElasticVonMises)
    return launchFused<false, BATCH, kModelsElasticVonMises>(lc, P, T, cur, pidCur, nxt, pidNxt, n, b, g, dtStress, err, numSMs, s);
  if constexpr (!BATCH) {
    if (modelSet == kModelsElastic)
      return launchFused<false, false, kModelsElastic>(lc, P, T, cur, pidCur, nxt, pidNxt, n, b, g, dtStress, err, numSMs, s);
    if (modelSet == kModelsDruckerPrager)
      return launchFused<false, false, kModelsDruckerPrager>(lc, P, T, cur, pidCur, nxt, pidNxt, n, b, g, dtStress, err, numSMs, s);
    if (modelSet == kModelsElasticDruckerPrager)
      return launchFused<false, false, kModelsElasticDruckerPrager>(lc, P, T, cur, pidCur, nxt, pidNxt, n, b, g, dtStress, err, numSMs, s);
  }
  return launchFused<false, BATCH, kModelsAny>(lc, P, T, cur, pidCur, nxt, pidNxt, n, b, g, dtStress, err, numSMs, s);
}

}  // namespace

int modelSetOf(const Material* mats, uint32_t count) {
  bool elastic = count > 0, dp = count > 0, evm = count > 0, edp = count > 0;
  for (uint32_t i = 0; i < count; ++i) {
    const uint32_t m = mats[i].model;
    const bool isDp = m == MAT_DRUCKER_PRAGER || m == MAT_GRANULAR_POWDER;
    elastic = elastic && m == MAT_ELASTIC;
    dp = dp && isDp;
    evm = evm && (m == MAT_ELASTIC || m == MAT_VON_MISES);
    edp = edp && (m == MAT_ELASTIC || isDp);
  }
  return elastic ? kModelsElastic : dp ? kModelsDruckerPrager : evm ? kModelsElasticVonMises : edp ? kModelsElasticDruckerPrager : kModelsAny;
}

cudaError_t launchG2P2G(const SubstepParams& P, int modelSet, StatePtrs cur, const uint32_t* pidCur, StatePtrs nxt, uint32_t* pidNxt, uint32_t n,
                        const BrickBuffers& b, GridBuffers g, float dtStress, uint32_t* err, const LaunchConfig& lc, int numSMs, cudaStream_t s,
                        uint64_t* launches) {
  const cudaError_t e =
      launchFusedFor<false>(P.flip_ratio > 0.01f, modelSet, lc, P, SceneTable{}, cur, pidCur, nxt, pidNxt, n, b, g, dtStress, err, numSMs, s);
  ++*launches;
  return e;
}

cudaError_t launchG2P2GBatch(const SceneTable& T, int modelSet, bool flip, StatePtrs cur, const uint32_t* pidCur, StatePtrs nxt, uint32_t* pidNxt,
                             uint32_t n, const BrickBuffers& b, GridBuffers g, uint32_t* err, const LaunchConfig& lc, int numSMs, cudaStream_t s,
                             uint64_t* launches) {
  const cudaError_t e = launchFusedFor<true>(flip, modelSet == kModelsElasticVonMises || modelSet == kModelsElastic ? kModelsElasticVonMises : kModelsAny,
                                             lc, SubstepParams{}, T, cur, pidCur, nxt, pidNxt, n, b, g, 0.f, err, numSMs, s);
  ++*launches;
  return e;
}

cudaError_t launchUnpermute(StatePtrs in, const uint32_t* pid, StatePtrs out, uint32_t n, cudaStream_t s, uint64_t* launches) {
  if (n == 0) return cudaSuccess;
  k_unpermute<<<blocksFor(n), kThreads, 0, s>>>(in, pid, out, n);
  ++*launches;
  return cudaGetLastError();
}

cudaError_t launchSortedPid(const uint32_t* perm, const uint32_t* pid, uint32_t* out, uint32_t n, cudaStream_t s, uint64_t* launches) {
  if (n == 0) return cudaSuccess;
  k_sorted_pid<<<blocksFor(n), kThreads, 0, s>>>(perm, pid, out, n);
  ++*launches;
  return cudaGetLastError();
}

cudaError_t launchIota(uint32_t* pid, uint32_t n, cudaStream_t s, uint64_t* launches) {
  if (n == 0) return cudaSuccess;
  k_iota<<<blocksFor(n), kThreads, 0, s>>>(pid, n);
  ++*launches;
  return cudaGetLastError();
}

}  // namespace nebula
