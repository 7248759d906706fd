// Uniform-grid counting sort and physical reorder into cell order.
//
// Replaces clearBuffer + countParticles + scanBlocks + scanApply + scatter +
// stagePVA/applyPVA/stageF/applyF (web/js/shaders/simkernels.js:78-186,
// dispatched by web/js/sim.js:223-236) with:
//   k_clear    zeroes the cell counters, water flags and scan descriptors
//   k_count    cell key per particle + warp-aggregated histogram atomics
//   k_scan     single-pass decoupled-lookback exclusive scan of the histogram
//   k_fill     warp-aggregated slot reservation: each cell's members land in
//              its bucket in arbitrary order
//   k_reorder  final slot = bucket start + number of bucket members with a
//              larger previous index (in a crowded cell from counts the fill
//              made per segment of particles), then moves pos/vel/F/state into
//              the slot with the scatter pass's predictor fused in
// The final slot rule reproduces the reference's atomicSub scatter executed
// in invocation order: within a cell, particles are listed by descending
// previous index. Counts, cell starts and the permutation are therefore
// deterministic and bit-identical to that serial order.
#include "chain.cuh"
#include "xpbi_math.cuh"

namespace xpbi {

namespace {

constexpr int kThreads = 256;
constexpr int kScanThreads = 256;
constexpr int kScanItems = (int)kScanTile / kScanThreads;
constexpr uint32_t kLookbackSpinLimit = 1u << 22;

__device__ __forceinline__ uint32_t sceneOfSlot(const Bufs& b, uint32_t i) {
  return b.S > 1 ? (uint32_t)b.sceneOf[i] : 0u;
}

__device__ __forceinline__ uint32_t cellKey(const SceneDev& S, float4 p) {
  I3 c = cellCoord(S, v3(p.x, p.y, p.z));
  return S.cellBase + cellIndex(S, c.x, c.y, c.z);
}

__global__ void __launch_bounds__(kThreads) k_clear(Bufs b) {
  sortClear(b, afterPreviousEager(blockIdx.x * blockDim.x + threadIdx.x));
}

// The crowded ones of a scan thread's cells from `base` on, which end at `end`:
// their counts per segment start at 0, and the mark on their cursor tells the
// fill.
constexpr uint32_t kCrowdMark = 0x80000000u;  // (a handle holds fewer particles)
__device__ __noinline__ void clearCrowds(const uint32_t* cellStart, uint32_t* cursor, uint32_t* crowd, uint32_t n,
                                         uint32_t cells, uint32_t base, uint32_t end) {
  for (uint32_t c = base; c < cells && c < base + kScanItems; ++c) {
    const uint32_t s0 = cellStart[c], s1 = c + 1u < base + kScanItems ? cellStart[c + 1u] : end;
    if (!crowded(n, s0, s1)) continue;
    uint32_t* row = crowdRow(crowd, n, s0);
    for (uint32_t q = 0; q < crowdSegments(n); ++q) row[q] = 0u;
    cursor[c] = s0 | kCrowdMark;
  }
}

// cursor[] was cleared before this launch; on exit it holds cell counts.
__global__ void __launch_bounds__(kThreads) k_count(Bufs b) {
  const uint32_t i = afterPreviousEager(blockIdx.x * blockDim.x + threadIdx.x);
  bool active = i < b.N;
  uint32_t key = 0;
  if (active) {
    const SceneDev& S = b.scenes[sceneOfSlot(b, i)];
    const float4 p = b.pos[i];
    key = cellKey(S, p);
    b.key[i] = key;
    uint32_t mi = 0u;
    if (p.w > 0.f) mi = min((uint32_t)p.w, 7u);
    if (b.mats[S.matBase + mi].kind == kKindWater) b.cellWater[key] = 1u;
  }
  unsigned mask = __ballot_sync(0xffffffffu, active);
  if (!active) return;
  unsigned peers = __match_any_sync(mask, key);
  int lane = threadIdx.x & 31;
  if (lane == __ffs(peers) - 1) atomicAdd(&b.cursor[key], (uint32_t)__popc(peers));
}

// Bounded wait for a look-back descriptor: polls `slot` until its flag
// (high word) is nonzero and returns the descriptor; after `polls` empty
// polls it raises kErrLookback in the error word and returns 0 (no flag),
// and the caller goes on. Nothing waits without a limit.
__device__ __forceinline__ unsigned long long waitDescriptor(const volatile unsigned long long* slot,
                                                             uint32_t polls, int* err) {
  for (uint32_t spins = 0;; ++spins) {
    const unsigned long long w64 = *slot;
    if ((uint32_t)(w64 >> 32) != 0u) return w64;
    if (spins >= polls) {
      atomicOr(err, kErrLookback);
      return 0ull;
    }
    if (spins > 16u) __nanosleep(64);
  }
}

// Exclusive scan of the C counts (plus one zero item, whose prefix is the
// N sentinel) into cellStart[0..C] and cursor[0..C-1]. Tiles take a ticket
// in launch order and look back over earlier tiles' descriptors; a tile only
// waits on tiles holding smaller tickets, which are already running. Each
// wait is bounded: on expiry the error word is raised and the tile goes on.
__global__ void __launch_bounds__(kScanThreads) k_scan(Bufs b) {
  __shared__ uint32_t s_tile, s_excl;
  __shared__ uint32_t s_warp[kScanThreads / 32];
  afterPreviousEager(0u);
  if (threadIdx.x == 0) s_tile = atomicAdd(b.tileTicket, 1u);
  __syncthreads();
  const uint32_t tile = s_tile;
  const uint32_t items = b.C + 1;
  const uint32_t base = tile * kScanTile + threadIdx.x * kScanItems;
  uint32_t v[kScanItems];
  if (base + kScanItems <= b.C) {
    const uint4* src = reinterpret_cast<const uint4*>(b.cursor + base);
#pragma unroll
    for (int k = 0; k < kScanItems / 4; ++k) {
      uint4 q = src[k];
      v[4 * k] = q.x; v[4 * k + 1] = q.y; v[4 * k + 2] = q.z; v[4 * k + 3] = q.w;
    }
  } else {
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) v[k] = (base + k < b.C) ? b.cursor[base + k] : 0u;
  }
  uint32_t sum = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) sum += v[k];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t incl = sum;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    uint32_t n = __shfl_up_sync(0xffffffffu, incl, off);
    if (lane >= off) incl += n;
  }
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    uint32_t w = lane < kScanThreads / 32 ? s_warp[lane] : 0u;
    uint32_t wi = w;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      uint32_t n = __shfl_up_sync(0xffffffffu, wi, off);
      if (lane >= off) wi += n;
    }
    if (lane < kScanThreads / 32) s_warp[lane] = wi - w;  // exclusive warp offsets
    const uint32_t agg = __shfl_sync(0xffffffffu, wi, kScanThreads / 32 - 1);  // tile aggregate
    if (lane == 0) atomicExch(b.tileStatus + tile, ((tile == 0 ? 2ull : 1ull) << 32) | agg);
    uint32_t excl = 0;
    if (tile > 0) {
      // 32 earlier tiles a step, a lane each (a walk of one tile at a time is
      // a chain of L2 round trips): the nearest one that has its prefix, or
      // whose wait expired (error word raised), ends it
      const volatile unsigned long long* status = b.tileStatus;
      for (int last = (int)tile - 1;; last -= 32) {
        const int pred = last - lane;
        const unsigned long long w64 =
            pred >= 0 ? waitDescriptor(status + pred, kLookbackSpinLimit, b.err) : 2ull << 32;
        const unsigned ends = __ballot_sync(0xffffffffu, (uint32_t)(w64 >> 32) != 1u);
        const int stop = ends ? __ffs((int)ends) - 1 : 31;
        excl += __reduce_add_sync(0xffffffffu, lane <= stop ? (uint32_t)w64 : 0u);
        if (ends) break;
      }
      __threadfence();
      if (lane == 0) atomicExch(b.tileStatus + tile, (2ull << 32) | (excl + agg));
    }
    if (lane == 0) s_excl = excl;
  }
  __syncthreads();
  uint32_t run = s_excl + s_warp[warp] + (incl - sum);
  uint32_t out[kScanItems];
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) { out[k] = run; run += v[k]; }
  if (base + kScanItems <= b.C) {
    uint4* d0 = reinterpret_cast<uint4*>(b.cellStart + base);
    uint4* d1 = reinterpret_cast<uint4*>(b.cursor + base);
#pragma unroll
    for (int k = 0; k < kScanItems / 4; ++k) {
      uint4 q = make_uint4(out[4 * k], out[4 * k + 1], out[4 * k + 2], out[4 * k + 3]);
      d0[k] = q;
      d1[k] = q;
    }
  } else {
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
      uint32_t idx = base + k;
      if (idx < items) b.cellStart[idx] = out[k];
      if (idx < b.C) b.cursor[idx] = out[k];
    }
  }
  if (sum > crowdLimit(b.N)) clearCrowds(b.cellStart, b.cursor, b.crowd, b.N, b.C, base, run);
}

// Unordered bucket fill: tmp[cellStart[key] .. +count) receives the members.
__global__ void __launch_bounds__(kThreads) k_fill(Bufs b) {
  const uint32_t i = afterPreviousEager(blockIdx.x * blockDim.x + threadIdx.x);
  bool active = i < b.N;
  uint32_t key = active ? b.key[i] : 0u;
  unsigned mask = __ballot_sync(0xffffffffu, active);
  if (!active) return;
  unsigned peers = __match_any_sync(mask, key);
  int lane = threadIdx.x & 31;
  int leader = __ffs(peers) - 1;
  uint32_t base = 0;
  if (lane == leader) base = atomicAdd(&b.cursor[key], (uint32_t)__popc(peers));
  base = __shfl_sync(mask, base, leader);
  uint32_t rank = __popc(peers & ((1u << lane) - 1u));
  b.tmp[(base & ~kCrowdMark) + rank] = i;
  if ((base & kCrowdMark) && lane == leader)  // (a warp's particles lie in one segment)
    atomicAdd(crowdRow(b.crowd, b.N, b.cellStart[key]) + i / kCrowdSegment, (uint32_t)__popc(peers));
}

// Final slot + physical reorder with the scatter pass's predictor fused in
// (simkernels.js:137-146 and 154-186). A thread per particle in previous
// order: everything it moves is loaded at once, and only its slot waits for
// the chain key -> bucket -> members. (By slot, the chain was one load longer
// and the moved data hung on its end, and crowded buckets had a kernel of
// their own, a block's bitonic sort: the sort of 250k keys 21.3 us.)
__global__ void __launch_bounds__(kThreads) k_reorder(Bufs b, int keepLam) {
  const uint32_t i = afterPrevious(blockIdx.x * blockDim.x + threadIdx.x);
  // both slots of the substep's largest-solid-displacement ring start at 0
  for (uint32_t q = i; q < 2u * b.S; q += gridDim.x * blockDim.x) b.solidDisp[q] = 0u;
  if (i >= b.N) return;
  const uint32_t key = b.key[i];
  const float4 pp = b.pos[i], v = b.vel[i];
  const M3 F = loadM(b.F, b.N, i);
  const float st = b.state[i];
  const uint32_t s0 = b.cellStart[key], s1 = b.cellStart[key + 1];
  const uint32_t s = s0 + rankInBucket(b.tmp, b.key, b.crowd, b.N, s0, s1, i);
  b.sortedIdx[s] = i;
  const SceneDev& S = b.scenes[sceneOfSlot(b, i)];
  // sorted records carry the water flag in the sign bit of pos.w (>= 0)
  uint32_t mi = 0u;
  if (pp.w > 0.f) mi = min((uint32_t)pp.w, 7u);
  const bool water = b.mats[S.matBase + mi].kind == kKindWater;
  b.posS[s] = make_float4(pp.x, pp.y, pp.z, water ? -pp.w : pp.w);
  b.posP[s] = pp.x;
  b.posP[s + b.planeN] = pp.y;
  b.posP[s + 2 * (size_t)b.planeN] = pp.z;
  storeM(b.FS, b.N, s, F);
  float Vn = S.V0 * clampf(det(F), 0.1f, 10.f);
  V3 g = v3(S.grav[0], S.grav[1], S.grav[2]);
  V3 vn = xyz(v) + g * S.dt;
  b.velS[0][s] = make_float4(vn.x, vn.y, vn.z, Vn);
  b.stateS[s] = st;
  b.lam[s] = 0.f;
  if (keepLam) b.lamPrev[s] = b.lamOut[i];
}

inline unsigned grid(uint32_t n, int t) { return (unsigned)((n + t - 1) / t); }

// Test hook: the scan's bounded wait on a descriptor nothing publishes
// (`slot` stays zero), so the wait expires after `polls` polls and raises
// the error word the host reads — the failure path of the look-back without
// a fault. One thread.
__global__ void k_wait_expiry(Bufs b, const unsigned long long* slot, uint32_t polls) {
  waitDescriptor(slot, polls, b.err);
}

}  // namespace

uint32_t scan_tiles(uint32_t cells) { return (cells + 1 + kScanTile - 1) / kScanTile; }

// clears what the whole sort starts from, then counts
void launch_count(const Bufs& b, cudaStream_t st) {
  k_clear<<<grid(sortClearThreads(b), kThreads), kThreads, 0, st>>>(b);
  launch_count_cleared(b, st);
}
void launch_count_cleared(const Bufs& b, cudaStream_t st) {
  launchChained(k_count, grid(b.N, kThreads), kThreads, 0, st, b);
}
void launch_wait_expiry(const Bufs& b, const unsigned long long* slot, uint32_t polls, cudaStream_t st) {
  k_wait_expiry<<<1, 1, 0, st>>>(b, slot, polls);
}
void launch_scan(const Bufs& b, cudaStream_t st) { launchChained(k_scan, b.scanTiles, kScanThreads, 0, st, b); }
void launch_scatter(const Bufs& b, cudaStream_t st) {
  launchChained(k_fill, grid(b.N, kThreads), kThreads, 0, st, b);
}
void launch_reorder(const Bufs& b, bool keepLam, cudaStream_t st) {
  launchChained(k_reorder, grid(b.N, kThreads), kThreads, 0, st, b, keepLam ? 1 : 0);
}

}  // namespace xpbi
