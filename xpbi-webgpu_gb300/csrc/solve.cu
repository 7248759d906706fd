// Neighbour-gather kernels of the XPBI substep, one thread (on small handles
// two or four) per particle slot in cell order. Each restates one compute entry point of
// web/js/shaders/simkernels.js (cited per kernel).
//
// Neighbour lists. Positions do not move between the reorder and the final
// update, so the set of in-support neighbours (b != i, |x_i - x_b|^2 <
// support^2) is the same for computeL, every solveA / solveB iteration, xsph
// and updateF. computeL walks the reference stencil once (dz outer, dy inner,
// candidates ascending over the row-merged range of three x-adjacent cells,
// capped at 384, simkernels.js:62-74) and records the in-support neighbours in
// that order, the slot's own phase (solid or water) from the front of its
// list and the other one from the back, so every later pass sums over exactly
// the reference's terms without rescanning ~216 candidates per particle. A
// warp's 32 lists are interleaved in groups of four entries; loops take two
// neighbours at a time in packed f32x2 arithmetic, and a last odd one is
// paired with the slot itself, whose terms are 0. Lists that do not fit
// kNbrCap fall back to the stencil walk.
//
// PBF passes test predicted positions x + dt v, which change every
// iteration: pbfA records the predicted neighbours with a margin, walks the
// stencil again only after particles moved past it, and both PBF kernels
// iterate that record.
//
// Scans are two-phase: a branch-light candidate test that only sets bits of a
// mask, then a pass over the hits.
//
// Sorted records carry the water flag in the sign bit of pos.w (pos.w is
// material index + colour seed >= 0, so fabsf restores it exactly).
//
// Batched handles: every slot belongs to one scene (sceneOf); its grid, cell
// table range, uniforms and material table come from that scene, and a
// neighbour stencil never leaves the scene's own cells. Passes beyond a
// scene's iteration budget copy velIn to velOut so the shared ping-pong
// parity stays consistent for every scene.
#include <algorithm>

#include "chain.cuh"
#include "xpbi_math.cuh"

namespace xpbi {

namespace {

constexpr int kThreads = 128;

// Launch bounds of the stencil kernels: resident CTAs of kThreads threads per
// SM asked of the register allocator, with one lane per slot and with several
// (ms per launch; one lane on the 4M-particle dam-breach mix): computeL 9 CTAs
// 1.09 (8: 1.11, 7: 1.17, 6: 1.27); with the stored constraint and features
// (the learned solve) 7; pbfA 10: 0.62 (8: 0.66, 9: 0.64, 11: 0.63); pbfB 7:
// 0.047 on the 1M-particle dam breach (8: 0.048, 9: 0.050, 10: 0.054), several
// lanes 8; the update 7: 0.303 (8: 0.337, 6: 0.332, the allocator's choice
// 0.370). With several lanes computeL and pbfA hold 33 KB of shared memory a
// block, so six fit, whatever the registers: 16k solids 199.5 us a substep and
// 27k of a dam breach 154.3 with 6 and 6, 200.5 and 154.1 with the caps of 7
// and 8.
constexpr int kColumnBlocks = 6;
constexpr int minComputeL(int lanes) { return lanes == 1 ? 9 : kColumnBlocks; }
constexpr int minComputeLFeatures(int lanes) { return lanes == 1 ? 7 : kColumnBlocks; }
constexpr int minPbfA(int lanes) { return lanes == 1 ? 10 : kColumnBlocks; }
constexpr int minPbfB(int lanes) { return lanes == 1 ? 7 : 8; }
constexpr int kMinUpdate = 7;
// solveA and solveB are compiled in several launch shapes — the block size
// and the minimum resident CTAs per SM asked of the register allocator (0 =
// its own choice) — and xpbi_autotune picks one per handle by timing them on
// its data. Entry 0 is the default. solveA: 7 CTAs of 128 per SM (72
// registers; the constraint's per-particle tail is a separately compiled
// function): per launch 0.649 ms on the 256-scene batch against 0.681 at 8
// CTAs, 0.724 at 9 and 0.695 at 6; 0.0205 on 113k solids against 0.0229 and
// 0.0241 (one wave: registers beat warps); 0.308 on the 4M-particle
// dam-breach mix against 0.305 and 0.325. solveB: 9 CTAs, 0.333 on that mix
// against 0.354 at 8, 0.351 at 7 and 10; on the batch all of them within 2%.
// The 64-thread shape keeps entry 1's occupancy with blocks of half the size.
constexpr int kSolveAMinB[kSolveAVariants] = {7, 8, 9, 10, 16, 6};
constexpr int kSolveABlock[kSolveAVariants] = {128, 128, 128, 128, 64, 128};
constexpr int kSolveBMinB[kSolveBVariants] = {9, 8, 7, 10, 6};
constexpr int kSolveBBlock[kSolveBVariants] = {128, 128, 128, 128, 128};
struct Ctx {
  const SceneDev* __restrict__ scene;
  const MatDev* __restrict__ mats;  // this scene's 8 materials
};

__device__ __forceinline__ Ctx ctxOf(const Bufs& b, uint32_t i) {
  const uint32_t s = b.S > 1 ? (uint32_t)b.sceneOf[i] : 0u;
  const SceneDev* S = b.scenes + s;
  return Ctx{S, b.mats + S->matBase};
}

// material index stored as a float value in pos.w (simkernels.js:41-44)
__device__ __forceinline__ uint32_t matOfW(float w) {
  w = fabsf(w);
  if (!(w > 0.f)) return 0u;
  const uint32_t m = (uint32_t)w;
  return m > 7u ? 7u : m;
}
__device__ __forceinline__ bool waterW(float w) { return signbit(w); }

struct PV {
  float4 p, v;
};

// The share of the support by which a PBF walk looks further than the pass
// needs: 0.1 against 0.05 (too little for moving water: lists of an 80k dam
// breach rebuilt in most passes) and 0.15 (more pairs to no effect): 3733,
// 3754 and 3768 us per substep of 1M particles, 329, 332 and 328 of 80k.
constexpr float kPbfSkin = 0.1f;
constexpr float kNoRef = 1e30f;  // no slot's pos.w
// The predicted position of slot i for a PBF pass: the record its pair loops
// gather and the coordinate planes pbfA's candidate walk reads. moved: also how
// far it lies from where the last stencil walk saw it, as the scene's maximum
// (pbfA decides by it whether the lists still hold every neighbour).
__device__ __forceinline__ void storeXc(const Bufs& b, uint32_t i, V3 xc, float w, bool moved) {
  b.xc[i] = make_float4(xc.x, xc.y, xc.z, w);
  b.xcP[i] = xc.x;
  b.xcP[i + b.planeN] = xc.y;
  b.xcP[i + 2 * (size_t)b.planeN] = xc.z;
  if (!moved) return;
  const float4 ref = b.xcRef[i];
  if (ref.w == kNoRef) return;  // a solid that no pass pairs
  const float dx = xc.x - ref.x, dy = xc.y - ref.y, dz = xc.z - ref.z;
  const float d2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
  const unsigned act = __activemask();
  const uint32_t sc = b.S > 1 ? (uint32_t)b.sceneOf[i] : 0u;
  const unsigned peers = b.S > 1 ? __match_any_sync(act, sc) : act;
  // (bits of d2 >= 0 order like its values; NaN, whose bits are larger, forces a walk)
  const unsigned mx = __reduce_max_sync(peers, __float_as_uint(d2) & 0x7fffffffu);
  if ((threadIdx.x & 31u) == (unsigned)(__ffs((int)peers) - 1) && mx > b.pbfMoved[sc]) atomicMax(b.pbfMoved + sc, mx);
}

template <class T>
__device__ __forceinline__ T ldg(const T* p) {
  return __ldg(p);
}

// What a slot's own index addresses in the solve kernels: through the read-only
// cache with one lane (1% of a 4M substep), whose launches are plain; several
// lanes are chained to the preceding kernel and need an ordinary load.
template <int G, class T>
__device__ __forceinline__ T loadOwn(const T* p) {
  if constexpr (G == 1)
    return __ldg(p);
  else
    return *p;
}

// Stencil walk over the 9 row-merged ranges (simkernels.js:62-74):
// row(beg, end) is called per in-range row. With G lanes per slot, lane
// `lane` takes the rows r with r % G == lane.
template <int G = 1, class Row>
__device__ __forceinline__ void forRows(const SceneDev& S, const uint32_t* __restrict__ cellStart, V3 x, Row&& row,
                                        uint32_t lane = 0) {
  const I3 cc = cellCoord(S, x);
  const int x0 = max(cc.x - 1, 0);
  const int x1 = min(cc.x + 1, S.dims[0] - 1);
  auto one = [&](int y, int z) {
    const uint32_t c0 = S.cellBase + cellIndex(S, x0, y, z);
    const uint32_t c2 = S.cellBase + cellIndex(S, x1, y, z);
    const uint32_t beg = __ldg(cellStart + c0);
    const uint32_t end = min(__ldg(cellStart + c2 + 1), beg + kRowCap);
    row(beg, end);
  };
  if constexpr (G == 1) {
#pragma unroll 1
    for (int dz = -1; dz <= 1; ++dz) {
      const int z = cc.z + dz;
      if (z < 0 || z >= S.dims[2]) continue;
#pragma unroll 1
      for (int dy = -1; dy <= 1; ++dy) {
        const int y = cc.y + dy;
        if (y < 0 || y >= S.dims[1]) continue;
        one(y, z);
      }
    }
  } else {
#pragma unroll 1
    for (int r = (int)lane; r < 9; r += G) {
      const int z = cc.z + r / 3 - 1, y = cc.y + r % 3 - 1;
      if (z >= 0 && z < S.dims[2] && y >= 0 && y < S.dims[1]) one(y, z);
    }
  }
}

// Neighbour lists. The lists of 32 consecutive slots (a warp's) are
// interleaved by groups of four entries: group q of slot i is one 16-byte
// load at nbrGroups(i)[32 q], and the 32 lanes' loads are contiguous. The
// entries of slot i's own phase (solid or water), the only ones most passes
// visit, come first in stencil order, padded to whole groups with i itself —
// whose distance is 0, so that it adds nothing to a gradient sum and no loop
// tests for its end; computeL puts the other phase's entries at the far end.
// (The list loads are plain ones: computeL and pbfA read what they have just
// written.)
constexpr uint32_t kGroupStride = 32u;
__device__ __forceinline__ uint4* nbrGroups(uint32_t* base, uint32_t i) {
  return reinterpret_cast<uint4*>(base) + (size_t)(i >> 5) * (kNbrCap / 4u * 32u) + (i & 31u);
}
__device__ __forceinline__ uint32_t* nbrEntry(uint32_t* base, uint32_t i, uint32_t e) {
  return reinterpret_cast<uint32_t*>(nbrGroups(base, i) + kGroupStride * (e >> 2)) + (e & 3u);
}
__device__ __forceinline__ uint32_t lane4(const uint4& q, uint32_t s) {
  return s == 0u ? q.x : (s == 1u ? q.y : (s == 2u ? q.z : q.w));
}
// the count word: entries of the slot's own phase, of the other one, and for
// a solid whether its 27 cells hold no water (never set on an overflow)
__device__ __forceinline__ uint32_t sameCount(uint32_t c) { return c & 0xffu; }
__device__ __forceinline__ uint32_t otherCount(uint32_t c) { return (c >> 8) & 0xffu; }
// a PBF list of the neighbours within the support alone
constexpr uint32_t kNbrExact = 0x100u;
__device__ __forceinline__ bool dryCount(uint32_t c) { return (c >> 16) == 1u; }

// Two neighbours at a time over `groups` groups: body(j0, j1, d0, d1) with
// d = gather(j); the list's groups are loaded one group ahead. (Keeping the
// next pair's gathers in flight as well costs 16 registers or more, and the
// resident warps they displace hide more latency: solveA 0.320 ms per launch
// without, 0.331 with, on the 4M-particle mix.)
template <class Gather, class Body>
__device__ __forceinline__ void forPairs(const uint4* L, uint32_t groups, Gather&& gather, Body&& body) {
  if (groups == 0u) return;
  uint4 cur = *(L);
#pragma unroll 1
  for (uint32_t q = 1u; q <= groups; ++q) {
    const uint4 nxt = *(L + kGroupStride * min(q, groups - 1u));
    body(cur.x, cur.y, gather(cur.x), gather(cur.y));
    body(cur.z, cur.w, gather(cur.z), gather(cur.w));
    cur = nxt;
  }
}
// One neighbour at a time: body(j, d) (records of many registers).
template <class Gather, class Body>
__device__ __forceinline__ void forSingles(const uint4* L, uint32_t groups, Gather&& gather, Body&& body) {
  if (groups == 0u) return;
  uint4 cur = *(L);
#pragma unroll 1
  for (uint32_t q = 1u; q <= groups; ++q) {
    const uint4 nxt = *(L + kGroupStride * min(q, groups - 1u));
    body(cur.x, gather(cur.x));
    body(cur.y, gather(cur.y));
    body(cur.z, gather(cur.z));
    body(cur.w, gather(cur.w));
    cur = nxt;
  }
}

// Several lanes per slot run on scenes too small to hide a chain of loads
// behind other warps. What the chain needs and no earlier load decides is
// fetched first: the list's count word and the first two pairs of entries a
// lane visits (the storage holds kNbrCap entries whatever the count; entries
// beyond it are not used).
struct ListHead {
  uint32_t count;
  uint2 e0, e1;
};
__device__ __forceinline__ uint2 pairAt(const uint4* L, uint32_t p) {
  return *(reinterpret_cast<const uint2*>(L + kGroupStride * (p >> 1)) + (p & 1u));
}
// (volatile: not moved behind the branches that follow)
__device__ __forceinline__ uint2 pairNow(const uint4* L, uint32_t p) {
  uint2 e;
  asm volatile("ld.global.v2.u32 {%0, %1}, [%2];"
               : "=r"(e.x), "=r"(e.y)
               : "l"(reinterpret_cast<const uint2*>(L + kGroupStride * (p >> 1)) + (p & 1u)));
  return e;
}
template <int G>
__device__ __forceinline__ ListHead listHead(const uint4* L, const uint32_t* count, uint32_t i, uint32_t lane) {
  ListHead h{};
  if constexpr (G > 1) {
    asm volatile("ld.global.u32 %0, [%1];" : "=r"(h.count) : "l"(count + i));
    h.e0 = pairNow(L, lane);
    h.e1 = pairNow(L, lane + G);
  }
  return h;
}
// Lane `lane` takes the pairs p with p % G == lane of slot i's list, and
// visit(e, d0, d1) gets them in order; kTwo: two pairs in flight.
template <int G, bool kTwo, class Gather, class Visit>
__device__ __forceinline__ void forLanePairs(const uint4* L, const ListHead& h, uint32_t cnt, uint32_t i, uint32_t lane,
                                             Gather&& gather, Visit&& visit) {
  const uint32_t pairs = (cnt + 1u) >> 1;
  // i, by way of the loaded count (whose upper bits are 0 unless it overflowed):
  // a read-only load at i itself could move above a chained kernel's wait
  const uint32_t self = i + (h.count >> 24);
  uint2 e0 = h.e0, e1 = h.e1;
#pragma unroll 1
  for (uint32_t p = lane; p < pairs; p += 2u * G) {
    const uint2 n0 = pairAt(L, min(p + 2u * G, kNbrCap / 2u - 1u)), n1 = pairAt(L, min(p + 3u * G, kNbrCap / 2u - 1u));
    const bool two = p + G < pairs;
    const auto a0 = gather(e0.x), a1 = gather(e0.y);
    if constexpr (kTwo) {
      if (!two) e1 = make_uint2(self, self);  // gathered (one line for neighbouring slots), not visited
      const auto b0 = gather(e1.x), b1 = gather(e1.y);
      visit(e0, a0, a1);
      if (two) visit(e1, b0, b1);
    } else {
      visit(e0, a0, a1);
      if (two) visit(e1, gather(e1.x), gather(e1.y));
    }
    e0 = n0;
    e1 = n1;
  }
}

// A list of `cnt` entries two at a time.
template <int G, class Gather, class Body>
__device__ __forceinline__ void forListPairs(const uint4* L, const ListHead& h, uint32_t cnt, uint32_t i, uint32_t lane,
                                             Gather&& gather, Body&& body) {
  if constexpr (G == 1)
    forPairs(L, (cnt + 3u) >> 2, gather, body);
  else
    forLanePairs<G, true>(L, h, cnt, i, lane, gather,
                          [&](uint2 e, const auto& d0, const auto& d1) { body(e.x, e.y, d0, d1); });
}

// Slot i's neighbours of its own phase, two at a time, over the recorded
// list, or by the stencil walk if it overflowed (a last odd neighbour is
// paired with i itself, whose data self() reads with ordinary loads: its
// address depends on no loaded value, so a chained kernel must not gather it).
//
// Several lanes per slot (small scenes): the G lanes of slot i are
// consecutive in the warp; lane `lane` visits the pairs p with p % G == lane
// (on the walk every G-th candidate of each row) and accumulates a partial
// sum; laneSum adds them over the group.
template <int G, class Gather, class Self, class Body>
__device__ __forceinline__ void forSame(const Bufs& b, const Ctx& cx, const ListHead& h, uint32_t i, V3 xi, bool iWater,
                                        uint32_t lane, Gather&& gather, Self&& self, Body&& body) {
  static_assert(G == 1 || G == 2 || G == 4, "one, two or four lanes per slot");
  const uint32_t c = G == 1 ? b.nbrCount[i] : h.count;
  if (c != kNbrOverflow) {
    forListPairs<G>(nbrGroups(b.nbr, i), h, sameCount(c), i, lane, gather, body);
  } else {
    const SceneDev& S = *cx.scene;
    uint32_t first = i;  // a neighbour waiting for its partner
    forRows(S, b.cellStart, xi, [&](uint32_t beg, uint32_t end) {
#pragma unroll 1
      for (uint32_t j = beg + lane; j < end; j += G) {
        if (j == i) continue;
        const float4 pj = ldg(b.posS + j);
        const V3 d = xi - xyz(pj);
        const float d2 = dot(d, d);
        if (!(d2 < S.support2) || waterW(pj.w) != iWater) continue;
        const bool twin = d2 == 0.f && !iWater;  // paired with i (see coincident)
        if (first == i && !twin) {
          first = j;
          continue;
        }
        const auto p = gather(twin ? j : first);
        auto q = gather(j);
        if (twin) q = self();
        body(twin ? j : first, twin ? i : j, p, q);
        if (!twin) first = i;
      }
    });
    if (first != i) body(first, i, gather(first), self());
  }
}

// A solid's solid neighbours one at a time.
template <int G, class Gather, class Body>
__device__ __forceinline__ void forSameSingles(const Bufs& b, const Ctx& cx, const ListHead& h, uint32_t i, V3 xi,
                                               uint32_t lane, Gather&& gather, Body&& body) {
  const uint32_t c = G == 1 ? b.nbrCount[i] : h.count;
  if (c != kNbrOverflow) {
    const uint4* L = nbrGroups(b.nbr, i);
    if constexpr (G == 1) {
      forSingles(L, (sameCount(c) + 3u) >> 2, gather, body);
    } else {
      // records of 16 floats: two pairs of them only where the scene needs
      // few blocks per SM
      forLanePairs<G, G == 4>(L, h, sameCount(c), i, lane, gather, [&](uint2 e, const auto& d0, const auto& d1) {
        body(e.x, d0);
        body(e.y, d1);
      });
    }
  } else {
    const SceneDev& S = *cx.scene;
    forRows(S, b.cellStart, xi, [&](uint32_t beg, uint32_t end) {
#pragma unroll 1
      for (uint32_t j = beg + lane; j < end; j += G) {
        if (j == i) continue;
        const float4 pj = ldg(b.posS + j);
        const V3 d = xi - xyz(pj);
        if (dot(d, d) < S.support2 && !waterW(pj.w)) body(j, gather(j));
      }
    });
  }
}

// The radial factor of the kernel gradient of two neighbours at offsets
// (dx, dy, dz): gradW = c g (dx, dy, dz) with c = S.gradC = -5 sigW / h^2 and
// g = t^3, t = 1 - r / (2 h). (The Wendland gradient's q / (h r) is 1 / h^2,
// so neither a division by r nor a test for r = 0 is left; neighbours are
// within the support, so t is not negative beyond rounding.)
__device__ __forceinline__ float sqrtFast(float x) {
  float y;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// t = 1 - r / (2 h) from r^2
__device__ __forceinline__ F2 falloff2(const SceneDev& S, F2 r2) {
  return fma2(f2(sqrtFast(lo2(r2)), sqrtFast(hi2(r2))), f2(-S.halfInvH, -S.halfInvH), f2(1.f, 1.f));
}
__device__ __forceinline__ F2 radial2(const SceneDev& S, F2 r2) {
  const F2 t = falloff2(S, r2);
  return mul2(mul2(t, t), t);
}

template <int G>
__device__ __forceinline__ float laneSum(float v) {
  if constexpr (G == 2) {
    const unsigned group = 0x3u << (threadIdx.x & 30u);  // warp lanes 2p, 2p+1
    v += __shfl_xor_sync(group, v, 1);
  } else if constexpr (G == 4) {
    const unsigned group = 0xFu << (threadIdx.x & 28u);  // warp lanes 4p .. 4p+3
    v += __shfl_xor_sync(group, v, 1);
    v += __shfl_xor_sync(group, v, 2);
  }
  return v;
}
template <int G>
__device__ __forceinline__ V3 laneSum(V3 v) {
  return v3(laneSum<G>(v.x), laneSum<G>(v.y), laneSum<G>(v.z));
}
// both halves of a packed sum
__device__ __forceinline__ float sum2(F2 a) { return lo2(a) + hi2(a); }

// Visits, in stencil order, the candidates j != i of the rows around `x`
// whose point in the coordinate planes P (P.x, P.y, P.z of slot j) lies
// within sqrt(s2) of `c`: hit(j).
//
// A walk tests ~216 candidates for ~33 hits and is bound by the L1 data pipe
// and by issue, so its inner loop does nothing but test: four candidates per
// step from three 16-byte loads (aligned down to the planes' groups of four;
// 12 bytes per candidate through the L1 pipe, not the 16 of a position
// record), their distances two per packed instruction with the bound as the
// sums' start value, each sign shifted into a mask of up to 32 candidates.
// The candidates before the row's start and past its end are masked off (the
// planes are padded), and a second loop over the set bits does a hit's work.
struct Planes {
  const float *x, *y, *z;
};
__device__ __forceinline__ Planes planesOf(const float* p, uint32_t stride) {
  return Planes{p, p + stride, p + 2 * (size_t)stride};
}
template <int G = 1, class Hit>
__device__ __forceinline__ void walkCandidates(const SceneDev& S, const uint32_t* __restrict__ cellStart, V3 x,
                                               uint32_t i, Planes P, V3 c, float s2, Hit&& hit, uint32_t lane = 0) {
  const F2 cx = f2(-c.x, -c.x), cy = f2(-c.y, -c.y), cz = f2(-c.z, -c.z), ns2 = f2(-s2, -s2);
  forRows<G>(S, cellStart, x, [&](uint32_t beg, uint32_t end) {
#pragma unroll 1
    for (uint32_t b0 = beg & ~3u; b0 < end; b0 += 32u) {
      const uint32_t n = min(32u, end - b0);
      uint32_t mask = 0;
#pragma unroll 1
      for (uint32_t t = 0; t < n; t += 4u) {
        const ulonglong2 X = ldg(reinterpret_cast<const ulonglong2*>(P.x + b0 + t));
        const ulonglong2 Y = ldg(reinterpret_cast<const ulonglong2*>(P.y + b0 + t));
        const ulonglong2 Z = ldg(reinterpret_cast<const ulonglong2*>(P.z + b0 + t));
        const F2 dx0 = add2(X.x, cx), dy0 = add2(Y.x, cy), dz0 = add2(Z.x, cz);
        const F2 dx1 = add2(X.y, cx), dy1 = add2(Y.y, cy), dz1 = add2(Z.y, cz);
        const F2 r0 = fma2(dz0, dz0, fma2(dy0, dy0, fma2(dx0, dx0, ns2)));
        const F2 r1 = fma2(dz1, dz1, fma2(dy1, dy1, fma2(dx1, dx1, ns2)));
        mask = __funnelshift_l((uint32_t)r0, mask, 1);
        mask = __funnelshift_l((uint32_t)(r0 >> 32), mask, 1);
        mask = __funnelshift_l((uint32_t)r1, mask, 1);
        mask = __funnelshift_l((uint32_t)(r1 >> 32), mask, 1);
      }
      // candidate t of the chunk -> bit 31 - t
      mask <<= 32u - ((n + 3u) & ~3u);
      mask &= 0xffffffffu << (32u - n);
      if (b0 < beg) mask &= 0xffffffffu >> (beg - b0);
      if (i - b0 < 32u) mask &= ~(0x80000000u >> (i - b0));
#pragma unroll 1
      while (mask) {
        const uint32_t t = (uint32_t)__clz((int)mask);
        mask &= ~(0x80000000u >> t);
        hit(b0 + t);
      }
    }
  }, lane);
}

// Exactly coincident solids. The reference's sums see a particle's twin as a
// term of 0, so twins that start alike stay together. The packed sums add even
// and odd neighbours apart, and the twin stands elsewhere in one list than in
// the other: everything behind it would change halves, the sums differ in their
// last bits, and the contact pass drives apart what a rounding separated (a
// doubled body of 2744 particles: 2084 pairs apart after 20 substeps, none with
// the terms in one order). So a list's coincident entries come last, and on the
// stencil walks they are paired with the slot itself.
__device__ __forceinline__ bool coincident(Planes P, uint32_t j, V3 x) {
  return ldg(P.x + j) == x.x && ldg(P.y + j) == x.y && ldg(P.z + j) == x.z;
}
// the n entries at(0), at(1), ... with the coincident ones last, the others in
// their order
template <class At>
__device__ __forceinline__ void coincidentLast(Planes P, V3 x, uint32_t n, At&& at) {
  uint32_t last = n;
#pragma unroll 1
  for (uint32_t e = n; e-- > 0u;) {
    const uint32_t j = *at(e);
    if (!coincident(P, j, x)) continue;
    --last;
#pragma unroll 1
    for (uint32_t q = e; q < last; ++q) *at(q) = *at(q + 1u);
    *at(last) = j;
  }
}
__device__ __noinline__ void coincidentLastInList(Planes P, V3 x, uint32_t n, uint32_t* nbr, uint32_t i) {
  coincidentLast(P, x, n, [&](uint32_t e) { return nbrEntry(nbr, i, e); });
}
// (several lanes: the column of lane 0, whose row holds the slot's own cell and
// whose entries the list starts with)
__device__ __noinline__ void coincidentLastInColumn(Planes P, V3 x, uint32_t n, uint32_t* col, uint32_t* nbr,
                                                    uint32_t i) {
  coincidentLast(P, x, n, [&](uint32_t e) { return col + e * (uint32_t)kThreads; });
  for (uint32_t e = 0; e < n; ++e) *nbrEntry(nbr, i, e) = col[e * (uint32_t)kThreads];
}

// What a walk with several lanes per slot records before the lists are
// written: each lane's hits in a column of shared memory, `same` from the top
// and `other` from the bottom. A lane with more than the column holds loses
// them (the list then counts as overflowed).
template <int G>
struct SubList {
  static constexpr uint32_t kCap = kNbrCap;
  uint32_t* col;  // this thread's column, stride kThreads
  uint32_t same = 0, other = 0;
  bool lost = false;  // of any of the slot's lanes, after totals()
  uint32_t sameAll = 0, otherAll = 0, sameBefore = 0, otherBefore = 0;
  __device__ __forceinline__ uint32_t at(uint32_t e) const { return col[e * kThreads]; }
  __device__ __forceinline__ uint32_t otherAt(uint32_t e) const { return col[(kCap - 1u - e) * kThreads]; }
  __device__ __forceinline__ void add(uint32_t j, bool own) {
    if (same + other >= kCap) {
      lost = true;
      return;
    }
    col[(own ? same : kCap - 1u - other) * kThreads] = j;
    same += own ? 1u : 0u;
    other += own ? 0u : 1u;
  }
  // every lane of the slot together
  __device__ __forceinline__ void totals(uint32_t lane) {
    sameAll = otherAll = sameBefore = otherBefore = anyLost = 0u;
    const uint32_t warpLane = threadIdx.x & 31u, first = warpLane & ~(uint32_t)(G - 1);
    const unsigned group = ((1u << G) - 1u) << first;
#pragma unroll
    for (uint32_t o = 0; o < (uint32_t)G; ++o) {
      const uint32_t v = __shfl_sync(group, same | other << 8 | (lost ? 1u << 16 : 0u), (int)(first + o));
      const uint32_t sv = v & 0xffu, ov = (v >> 8) & 0xffu;
      sameBefore += o < lane ? sv : 0u;
      otherBefore += o < lane ? ov : 0u;
      sameAll += sv;
      otherAll += ov;
      anyLost |= v >> 16;
    }
    lost = anyLost != 0u;
  }
  uint32_t anyLost = 0;
};

// The offsets of two neighbours from xi and what the sums weigh them by:
// (dx, dy, dz) = xi - x_b, w = V_b g (dx, dy, dz), so that V_b gradW_b = c w.
struct Pair {
  F2 dx, dy, dz, r2, wx, wy, wz;
};
__device__ __forceinline__ Pair pairOf(const SceneDev& S, V3 xi, const PV& p, const PV& q) {
  Pair r;
  r.dx = f2(xi.x - p.p.x, xi.x - q.p.x);
  r.dy = f2(xi.y - p.p.y, xi.y - q.p.y);
  r.dz = f2(xi.z - p.p.z, xi.z - q.p.z);
  r.r2 = fma2(r.dz, r.dz, fma2(r.dy, r.dy, mul2(r.dx, r.dx)));
  const F2 s = mul2(radial2(S, r.r2), f2(p.v.w, q.v.w));
  r.wx = mul2(r.dx, s);
  r.wy = mul2(r.dy, s);
  r.wz = mul2(r.dz, s);
  return r;
}

// A += (v_b - v_i) w_b^T for two neighbours: the velocity sum of the
// constraint sweeps, sum V_b (v_b - v_i) gradW_b^T without its factor c. Even
// and odd neighbours add up in the two halves. solveA's sweep and computeL's
// (which stores iteration 0's constraint for it) run these same operations,
// every one with its rounding fixed, so they form the same bits.
struct VelSum {
  F2 a[9];
  __device__ __forceinline__ VelSum() {
#pragma unroll
    for (int k = 0; k < 9; ++k) a[k] = 0ull;
  }
  __device__ __forceinline__ void add(const Pair& r, V3 vi, const float4& v0, const float4& v1) {
    const F2 vx = f2(v0.x - vi.x, v1.x - vi.x), vy = f2(v0.y - vi.y, v1.y - vi.y), vz = f2(v0.z - vi.z, v1.z - vi.z);
    a[0] = fma2(vx, r.wx, a[0]);
    a[1] = fma2(vy, r.wx, a[1]);
    a[2] = fma2(vz, r.wx, a[2]);
    a[3] = fma2(vx, r.wy, a[3]);
    a[4] = fma2(vy, r.wy, a[4]);
    a[5] = fma2(vz, r.wy, a[5]);
    a[6] = fma2(vx, r.wz, a[6]);
    a[7] = fma2(vy, r.wz, a[7]);
    a[8] = fma2(vz, r.wz, a[8]);
  }
  // the sum over the slot's lanes, with the factor c
  template <int G>
  __device__ __forceinline__ M3 total(float c) const {
    M3 m;
#pragma unroll
    for (int k = 0; k < 3; ++k)
      m.c[k] = v3(__fmul_rn(laneSum<G>(__fadd_rn(lo2(a[3 * k]), hi2(a[3 * k]))), c),
                  __fmul_rn(laneSum<G>(__fadd_rn(lo2(a[3 * k + 1]), hi2(a[3 * k + 1]))), c),
                  __fmul_rn(laneSum<G>(__fadd_rn(lo2(a[3 * k + 2]), hi2(a[3 * k + 2]))), c));
    return m;
  }
};

// ---------------------------------------------------------------- computeL
// L of slot i (simkernels.js:198-220) over its recorded neighbours: the
// SVD pseudo-inverse of sum V_b (grad W_b) (x_b - x_i)^T, which is symmetric
// (the gradient points along the offset), so its eigenvectors serve. For a solid (kSolid) the same sweep
// also forms the sums of the constraint passes that no velocity enters —
// s = sum V_b g_b, P = sum (V_b^2 / m_b) g_b g_b^T and the solid neighbour
// count, over the solid neighbours — and stores them in sgP for every
// iteration of the substep. With kVel (a solid, at the velocities iteration 0
// starts from) the sweep also forms that iteration's velocity sum
// Av = sum V_b (v_b - v_i) g_b^T — the constraint sweep's own operations.
template <bool kSolid, bool kVel = false, int G = 1>
__device__ __forceinline__ void bonetLok(const Bufs& b, const Ctx& cx, uint32_t i, V3 xi, M3* velSum = nullptr,
                                         uint32_t lane = 0, const SubList<G>* sub = nullptr) {
  static_assert(kSolid || !kVel, "the velocity sum is a solid's");
  const SceneDev& S = *cx.scene;
  const float4* posS = b.posS;
  const float4* velIn = b.velS[0];  // V^n (.w), which no pass changes; with kVel also v
  V3 vi = splat(0.f);
  if constexpr (kVel) vi = xyz(velIn[i]);
  VelSum Av;
  // sum w dx^T (symmetric) over every neighbour; s and P / c^2 over the solid ones
  F2 a00 = 0ull, a11 = 0ull, a22 = 0ull, a01 = 0ull, a02 = 0ull, a12 = 0ull;
  F2 sx = 0ull, sy = 0ull, sz = 0ull;
  F2 p00 = 0ull, p11 = 0ull, p22 = 0ull, p01 = 0ull, p02 = 0ull, p12 = 0ull;
  uint32_t cnt = 0, zeros = 0;  // the solid neighbours; distances of 0 among them and the padding
  auto gather = [&](uint32_t j) { return PV{ldg(posS + j), ldg(velIn + j)}; };
  auto addA = [&](const Pair& r) {
    a00 = fma2(r.wx, r.dx, a00);
    a11 = fma2(r.wy, r.dy, a11);
    a22 = fma2(r.wz, r.dz, a22);
    a01 = fma2(r.wx, r.dy, a01);
    a02 = fma2(r.wx, r.dz, a02);
    a12 = fma2(r.wy, r.dz, a12);
  };
  auto own = [&](uint32_t, uint32_t, const PV& d0, const PV& d1) {
    const Pair r = pairOf(S, xi, d0, d1);
    addA(r);
    if constexpr (kSolid) {
      if constexpr (kVel) Av.add(r, vi, d0.v, d1.v);
      sx = add2(sx, r.wx);
      sy = add2(sy, r.wy);
      sz = add2(sz, r.wz);
      const F2 m = f2(cx.mats[matOfW(d0.p.w)].invMass, cx.mats[matOfW(d1.p.w)].invMass);
      const F2 ux = mul2(r.wx, m), uy = mul2(r.wy, m), uz = mul2(r.wz, m);
      p00 = fma2(ux, r.wx, p00);
      p11 = fma2(uy, r.wy, p11);
      p22 = fma2(uz, r.wz, p22);
      p01 = fma2(ux, r.wy, p01);
      p02 = fma2(ux, r.wz, p02);
      p12 = fma2(uy, r.wz, p12);
      zeros += (lo2(r.r2) == 0.f ? 1u : 0u) + (hi2(r.r2) == 0.f ? 1u : 0u);
    }
  };
  auto clear = [&] {
    a00 = a11 = a22 = a01 = a02 = a12 = 0ull;
    sx = sy = sz = 0ull;
    p00 = p11 = p22 = p01 = p02 = p12 = 0ull;
    if constexpr (kVel) Av = VelSum();
  };
  // own phase; the other phase's neighbours enter L alone
  const uint32_t c = G == 1 ? b.nbrCount[i] : (sub->lost ? kNbrOverflow : 0u);
  if (c == kNbrOverflow) {
    const PV self{posS[i], velIn[i]};
    forRows<G>(S, b.cellStart, xi, [&](uint32_t beg, uint32_t end) {
#pragma unroll 1
      for (uint32_t j = beg; j < end; ++j) {
        if (j == i) continue;
        const float4 pj = ldg(posS + j);
        const V3 d = xi - xyz(pj);
        if (!(dot(d, d) < S.support2)) continue;
        if (waterW(pj.w) == kSolid) {
          addA(pairOf(S, xi, gather(j), self));
        } else {
          own(j, i, gather(j), self);
          ++cnt;
        }
      }
    }, lane);
  } else if constexpr (G == 1) {
    cnt = sameCount(c);
#pragma unroll 1
    for (bool again = false;; again = true) {
      forPairs(nbrGroups(b.nbr, i), (cnt + 3u) >> 2, gather, own);
      if (!kSolid || again || zeros <= ((0u - cnt) & 3u)) break;
      coincidentLastInList(planesOf(b.posP, b.planeN), xi, cnt, b.nbr, i);
      clear();
    }
    const uint32_t other = (otherCount(c) + 3u) >> 2;
    if (other)
      forPairs(nbrGroups(b.nbr, i) + kGroupStride * (kNbrCap / 4u - other), other, gather,
                  [&](uint32_t, uint32_t, const PV& d0, const PV& d1) { addA(pairOf(S, xi, d0, d1)); });
  } else {
    cnt = sub->same;
    // a last odd one is paired with a copy of itself of no volume
#pragma unroll 1
    for (bool again = false;; again = true) {
#pragma unroll 2
      for (uint32_t e = 0; e < cnt; e += 2u) {
        const bool two = e + 1u < cnt;
        const uint32_t j0 = sub->at(e), j1 = two ? sub->at(e + 1u) : j0;
        const PV d0 = gather(j0);
        PV d1 = gather(j1);
        if (!two) d1.v.w = 0.f;
        own(j0, two ? j1 : i, d0, d1);
      }
      if (!kSolid || again || zeros == 0u || lane != 0) break;
      coincidentLastInColumn(planesOf(b.posP, b.planeN), xi, cnt, sub->col, b.nbr, i);
      clear();
    }
    for (uint32_t e = 0; e < sub->other; e += 2u) {
      const bool two = e + 1u < sub->other;
      const uint32_t j0 = sub->otherAt(e), j1 = two ? sub->otherAt(e + 1u) : j0;
      const PV d0 = gather(j0);
      PV d1 = gather(j1);
      if (!two) d1.v.w = 0.f;
      addA(pairOf(S, xi, d0, d1));
    }
  }
  const float gc = S.gradC;
  auto total = [&](F2 v) { return laneSum<G>(sum2(v)); };
  // x_b - x_i = -(dx, dy, dz)
  const float b00 = -gc * total(a00), b11 = -gc * total(a11), b22 = -gc * total(a22);
  const float b01 = -gc * total(a01), b02 = -gc * total(a02), b12 = -gc * total(a12);
  if constexpr (kVel) *velSum = Av.template total<G>(gc);
  if constexpr (kSolid) {
    const V3 sg = v3(total(sx) * gc, total(sy) * gc, total(sz) * gc);
    const float c2 = gc * gc;
    const float q00 = total(p00) * c2, q11 = total(p11) * c2, q22 = total(p22) * c2;
    const float q01 = total(p01) * c2, q02 = total(p02) * c2, q12 = total(p12) * c2;
    const float count = laneSum<G>((float)cnt);
    if (lane == 0) {
      float4* __restrict__ R = b.sgP + i;
      const size_t N = b.N;
      R[0] = make_float4(sg.x, sg.y, sg.z, count);
      R[N] = make_float4(q00, q11, q22, q01);
      R[2 * N] = make_float4(q02, q12, 0.f, 0.f);
    }
  }
  if (G > 1 && lane != 0) return;  // lane 0 finishes the slot
  // the pseudo-inverse of the symmetric moment matrix
  V3 d;
  M3 V;
  eigSym(Sym3{b00, b11, b22, b01, b02, b12}, d, V);
  const float tol = 0.2f;
  V3 inv = splat(0.f);
  if (fabsf(d.x) > tol) inv.x = __frcp_rn(d.x);
  if (fabsf(d.y) > tol) inv.y = __frcp_rn(d.y);
  if (fabsf(d.z) > tol) inv.z = __frcp_rn(d.z);
  storeM(b.L, b.N, i, diagMul(V, inv, V));
}
// The water particles' L of the last substep, from the same positions,
// neighbour lists and V^n as k_computeL would have used.
__global__ void __launch_bounds__(kThreads, 8) k_computeL_water(Bufs b) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= b.N) return;
  const float4 pi = b.posS[i];
  if (!waterW(pi.w)) return;
  bonetLok<false>(b, ctxOf(b, i), i, xyz(pi));
}

// The record solveB gathers from each solid neighbour, in four float4
// planes (plane f of slot i at Sp[f N + i]) so that one warp-wide gather of
// a field touches as few cache lines as the neighbour indices allow: dlam
// G L columns with the position in .w, then the position predicted with the
// velocities entering this iteration and the mass (the contact pass's
// inputs). The particle's own dv goes to SpSelf.
__device__ __forceinline__ void storeSp(const Bufs& b, uint32_t i, const M3& m, V3 self, V3 x, V3 xc, float mass) {
  float4* __restrict__ R = b.Sp + i;
  const size_t N = b.N;
  R[0] = make_float4(m.c[0].x, m.c[0].y, m.c[0].z, x.x);
  R[N] = make_float4(m.c[1].x, m.c[1].y, m.c[1].z, x.y);
  R[2 * N] = make_float4(m.c[2].x, m.c[2].y, m.c[2].z, x.z);
  R[3 * N] = make_float4(xc.x, xc.y, xc.z, mass);
  b.SpSelf[i] = make_float4(self.x, self.y, self.z, 0.f);
}

// velocityGradient (simkernels.js:224-245) of a solid over its solid
// neighbours, without its factor L^T.
template <int G>
__device__ __forceinline__ M3 velocitySum(const Bufs& b, const Ctx& cx, const ListHead& h, uint32_t i, V3 xi, V3 vi,
                                          const float4* velIn, uint32_t lane) {
  const SceneDev& S = *cx.scene;
  const float4* posS = b.posS;
  // sum dv_b (L g_b)^T = (sum dv_b g_b^T) L^T: L applied once, by the caller
  VelSum A;
  forSame<G>(b, cx, h, i, xi, false, lane, [&](uint32_t j) { return PV{ldg(posS + j), ldg(velIn + j)}; },
             [&] { return PV{posS[i], velIn[i]}; },
             [&](uint32_t, uint32_t, const PV& d0, const PV& d1) { A.add(pairOf(S, xi, d0, d1), vi, d0.v, d1.v); });
  return A.template total<G>(S.gradC);
}

// ---------------------------------------------------------------- solveA
// Inelastic constraint pass A (simkernels.js:248-309) in one neighbour sweep.
//
// The reference sweeps the neighbours twice: once for grad v (to form the
// trial F and the constraint gradient G L) and once for
//   denom = sum_b |g_b|^2 / m_b + |sgrad|^2 / m_i,  sgrad = -sum_b g_b,
//   cdot  = sum_b g_b . v_b + sgrad . v_i,           g_b = V_b (G L) gradW_b.
// With gt_b = L gradW_b (the term grad v already uses) and M = (dC/dF) F^nT,
// g_b = V_b M gt_b, so with the per-sweep sums
//   s = sum_b V_b gt_b,  Q = sum_b (V_b^2 / m_b) gt_b gt_b^T,  grad v = sum_b V_b (v_b - v_i) gt_b^T
// the second sweep reduces exactly to
//   sgrad = -M s,  denom = <M^T M, Q> + |sgrad|^2 / m_i,  cdot = <M, grad v>.
// (The last identity also removes the cancellation of the reference's
// sum_b g_b . v_b against sgrad . v_i when the body moves as a whole.)
// Constraint of a solid slot at the current velocities: the single sweep
// above plus the trial F, SVD, return map and the closed-form sums.
struct Constraint {
  float C;        // sqrt(2 Psi) at the projected state (0 below 1e-7)
  float denom;    // sum |grad C|^2 / m, self term included
  float cdot;     // grad C . v
  M3 GL;          // (dC/dF) F^nT L
  V3 sgrad;       // self gradient (per unit multiplier)
  V3 logSigTr;    // log of the trial singular values (clamped like safeSig)
  float nNbr;     // solid neighbours in the sweep
};

// (Compiled once, not inlined: solveA and computeL with features run the
// same instructions, so iteration 0's stored constraint is bit for bit the
// one solveA would evaluate; inlined, the compiler fuses multiplies and adds
// differently in each kernel. The slot's L, F and sums are loaded in here,
// not handed over through the stack.)
struct TailIn {
  const float *L, *F;
  const float4* sgP;
  uint32_t N, i;
};
__device__ __noinline__ Constraint constraintTail(M3 A, TailIn in, const SceneDev* S, const MatDev* m, float st);

template <int NL = 1>
__device__ __forceinline__ Constraint evalConstraint(const Bufs& b, const Ctx& cx, uint32_t i, float4 pi,
                                                     const float4* velIn, const MatDev* m, float st,
                                                     const ListHead& head = ListHead{}, uint32_t lane = 0) {
  const SceneDev& S = *cx.scene;
  const float4* posS = b.posS;
  const V3 xi = xyz(pi);
  const V3 vi = xyz(loadOwn<NL>(velIn + i));
  // The sum runs over the raw kernel gradients g_b; the correction L is
  // applied once afterwards: with gt_b = L g_b,
  //   G = sum dv_b gt_b^T = A L^T,  s = L sum V_b g_b,  Q = L P L^T,
  // A = sum dv_b g_b^T, P = sum (V_b^2 / m_b) g_b g_b^T (same terms, the L
  // products factored out of the pair loop). s, P and the count do not depend
  // on the velocities: computeL formed them, so the sweep only accumulates A.
  VelSum A;
  forSame<NL>(b, cx, head, i, xi, false, lane, [&](uint32_t j) { return PV{ldg(posS + j), ldg(velIn + j)}; },
              [&] { return PV{posS[i], velIn[i]}; },
              [&](uint32_t, uint32_t, const PV& d0, const PV& d1) { A.add(pairOf(S, xi, d0, d1), vi, d0.v, d1.v); });
  const M3 At = A.template total<NL>(S.gradC);
  if (NL > 1 && lane != 0) return Constraint{};  // lane 0 finishes the slot
  return constraintTail(At, TailIn{b.L, b.FS, b.sgP, b.N, i}, cx.scene, m, st);
}

// The per-particle part of the constraint from the sweep's sum A = sum dv g^T:
// with s = sum V g and P = sum (V^2/m) g g^T over the solid neighbours
// (computeL's sums), the slot's correction L and its F. With G = A L^T and
// M = (dC/dF) F^nT, GL = M L gives every contraction directly:
//   sgrad = -M L s = -GL s,  <M^T M, L P L^T> = <GL^T GL, P>,  <M, A L^T> = <GL, A>.
__device__ __noinline__ Constraint constraintTail(M3 A, TailIn in, const SceneDev* Sp, const MatDev* mp, float st) {
  const SceneDev& S = *Sp;
  const MatDev& m = *mp;
  const M3 Li = loadM(in.L, in.N, in.i), Fn = loadM(in.F, in.N, in.i);
  const float4* R = in.sgP + in.i;
  const float hard = hardening(m, st);
  const float mu = m.mu * hard, lam = m.lam * hard;
  // the trial F minus the identity, which keeps the digits of a small strain
  const M3 Htr = madd(minusIdent(Fn), mscale(mul(mul(A, transpose(Li)), Fn), S.dt));
  V3 eTr;
  bool near;
  const SVD sd = strainSVD(Htr, eTr, near);
  Constraint out;
  out.logSigTr = v3(fmaxf(fmaxf(eTr.x, eTr.y), eTr.z),
                    fmaxf(fminf(eTr.x, eTr.y), fminf(fmaxf(eTr.x, eTr.y), eTr.z)),
                    fminf(fminf(eTr.x, eTr.y), eTr.z));  // descending
  float stOut;
  const Mapped mp2 = returnMap(sd.sig, eTr, m, mu, lam, st, S.dt, stOut);
  const V3 e = mp2.e;
  const float tr = e.x + e.y + e.z;
  out.C = sqrtf(fmaxf(2.f * stvkPsi(e, mu, lam), 0.f));
  const float4 r0 = R[0];
  out.nNbr = r0.w;
  if (out.C < 1e-7f) {
    out.C = 0.f;
    out.denom = 0.f;
    out.cdot = 0.f;
    out.GL = mzero();
    out.sgrad = splat(0.f);
    return out;
  }
  const V3 s = safeSig(mp2.sig);
  const V3 dC = v3((2.f * mu * e.x + lam * tr) / (s.x * out.C), (2.f * mu * e.y + lam * tr) / (s.y * out.C),
                   (2.f * mu * e.z + lam * tr) / (s.z * out.C));
  const M3 Pk = diagMul(sd.U, dC, sd.V);
  out.GL = mul(mul(Pk, transpose(Fn)), Li);
  const float4 r1 = R[in.N], r2 = R[2 * (size_t)in.N];
  out.sgrad = -mul(out.GL, xyz(r0));
  // <GL^T GL, P> = sum over column pairs (a, b) of (GL_a . GL_b) P_ab
  const V3 c0 = out.GL.c[0], c1 = out.GL.c[1], c2 = out.GL.c[2];
  const float denomN = dot(c0, c0) * r1.x + dot(c1, c1) * r1.y + dot(c2, c2) * r1.z +
                       2.f * (dot(c0, c1) * r1.w + dot(c0, c2) * r2.x + dot(c1, c2) * r2.y);
  out.denom = denomN + dot(out.sgrad, out.sgrad) / m.mass;
  out.cdot = dot(c0, A.c[0]) + dot(c1, A.c[1]) + dot(c2, A.c[2]);
  return out;
}

// The iteration-0 constraint of slot i in four float4 planes (plane q of
// slot i at cons0[q N + i]): computeL with features evaluates it at the very
// velocities iteration 0 starts from, so iteration 0 can read it instead of
// sweeping the neighbours again.
__device__ __forceinline__ void storeConstraint(const Bufs& b, uint32_t i, const Constraint& c) {
  float4* __restrict__ R = b.cons0 + i;
  const size_t N = b.N;
  R[0] = make_float4(c.C, c.denom, c.cdot, c.sgrad.x);
  R[N] = make_float4(c.sgrad.y, c.sgrad.z, c.GL.c[0].x, c.GL.c[0].y);
  R[2 * N] = make_float4(c.GL.c[0].z, c.GL.c[1].x, c.GL.c[1].y, c.GL.c[1].z);
  R[3 * N] = make_float4(c.GL.c[2].x, c.GL.c[2].y, c.GL.c[2].z, 0.f);
}
__device__ __forceinline__ Constraint loadConstraint(const Bufs& b, uint32_t i) {
  const float4* __restrict__ R = b.cons0 + i;
  const size_t N = b.N;
  const float4 a = R[0], q = R[N], r = R[2 * N], t = R[3 * N];
  Constraint c;
  c.C = a.x;
  c.denom = a.y;
  c.cdot = a.z;
  c.sgrad = v3(a.w, q.x, q.y);
  c.GL = M3{{v3(q.z, q.w, r.x), v3(r.y, r.z, r.w), v3(t.x, t.y, t.z)}};
  return c;
}

__device__ __forceinline__ bool sceneDone(const Bufs& b, uint32_t i) {
  const uint32_t s = b.S > 1 ? (uint32_t)b.sceneOf[i] : 0u;
  return b.done[s] != 0;
}

// Whether slot i's scene iterates at iteration k: below its budget and not
// stopped, or in the plain re-solve (flags & kRerun) marked for it and below
// its own iteration count.
__device__ __forceinline__ bool iterating(const Bufs& b, const SceneDev& S, uint32_t i, int k, int flags) {
  const uint32_t s = b.S > 1 ? (uint32_t)b.sceneOf[i] : 0u;
  if (flags & kRerun) return b.rerun[s] != 0 && k < S.plainIterations;
  return k < S.iterations && b.done[s] == 0;
}

// Largest solid displacement dt |v| per scene entering iteration k (slot
// k & 1 of solidDisp, cleared by solveB(k - 1) or at the substep's start).
// Called by every thread of the warp before any of them leaves: the lanes of
// one scene combine their values and one of them raises the slot.
__device__ __forceinline__ void recordSolidDisp(const Bufs& b, uint32_t i, int k, float d) {
  const unsigned act = __activemask();
  const uint32_t sc = b.S > 1 ? (uint32_t)b.sceneOf[i] : 0u;
  const unsigned peers = b.S > 1 ? __match_any_sync(act, sc) : act;
  const unsigned mx = __reduce_max_sync(peers, __float_as_uint(d));  // d >= 0: bits order like values
  if ((threadIdx.x & 31u) == (unsigned)(__ffs(peers) - 1) && mx != 0u)
    atomicMax(b.solidDisp + (size_t)(k & 1) * b.S + sc, mx);
}

// ---------------------------------------------------------------- active set
// The learned solve's work skipping (flags kActive / kMarkMoved, never set by
// the reference solve). A slot's constraint depends on its own and its solid
// neighbours' velocities, its contact correction on the predicted positions
// of its solid neighbours: if none of those changed since the slot was last
// evaluated, its residuals are unchanged too. So from iteration 2 on
//   - solveA evaluates only the solids marked as changed (dirty); a solid
//     whose residual is within the scene's per-slot threshold takes no
//     impulse (its multiplier stays), the others update as the reference
//     does and mark their solid neighbours (bmark) for solveB;
//   - solveB visits only the changed or marked slots, updates velocities in
//     place (it reads no neighbour's velocity), applies a contact correction
//     only above the per-slot threshold, and a slot whose velocity changed
//     by more than the scene's velocity scale marks itself and its solid
//     neighbours as changed for the next iteration (as pbfB does);
//   - residuals of slots not visited keep their last values, so the scene's
//     residual sums and the early stop see every slot.
// Iterations 0 and 1 run every slot (iteration 0 moves every particle, so
// skipping in iteration 1 would find nothing to skip); iteration 1 starts
// the marking. The per-slot thresholds (formed once the
// iteration-0 sums are known) give each settled slot an equal share of
// asShare times the scene's residual budget, so settled slots alone can
// never hold the scene above its tolerance. The velocity scale is a quarter
// of that share of tol^2 times the mean squared velocity change of iteration
// 0: a change below it moves a neighbour's residual by less than that
// neighbour's settle threshold, so the kept residuals are exact where nothing
// moved and otherwise off by at most that much (a tracked solve re-measures
// the final state over every slot).
__device__ __forceinline__ void countWarp(uint32_t* ctr) {
  const unsigned m = __activemask();
  if ((threadIdx.x & 31u) == (unsigned)(__ffs(m) - 1)) atomicAdd(ctr, (uint32_t)__popc(m));
}

// flag[j] = 1 for every solid neighbour j of the solid slot i. Plain byte
// stores: concurrent writers store the same value.
__device__ __forceinline__ void markSolidNbrs(const Bufs& b, const Ctx& cx, uint32_t i, V3 xi,
                                              uint8_t* __restrict__ flag) {
  const uint32_t c = b.nbrCount[i];
  if (c != kNbrOverflow) {
    const uint4* L = nbrGroups(b.nbr, i);
    const uint32_t cnt = sameCount(c);
#pragma unroll 1
    for (uint32_t q = 0; 4u * q < cnt; ++q) {
      const uint4 g = *(L + kGroupStride * q);
#pragma unroll
      for (uint32_t t = 0; t < 4u; ++t) {
        const uint32_t e = lane4(g, t);
        if (e != i) flag[e] = 1;
      }
    }
  } else {
    const SceneDev& S = *cx.scene;
    forRows(S, b.cellStart, xi, [&](uint32_t beg, uint32_t end) {
#pragma unroll 1
      for (uint32_t j = beg; j < end; ++j) {
        if (j == i) continue;
        const float4 pj = ldg(b.posS + j);
        const V3 d = xi - xyz(pj);
        if (dot(d, d) < S.support2 && !waterW(pj.w)) flag[j] = 1;
      }
    });
  }
}

__device__ __forceinline__ uint32_t sceneIndex(const Bufs& b, const Ctx& cx) {
  return (uint32_t)(cx.scene - b.scenes);
}

// The iteration a launch works on: its argument, or inside the device loop
// (argument kIterDevice) the loop's current iteration.
__device__ __forceinline__ int iterK(const Bufs& b, int k) {
  return k == kIterDevice ? *reinterpret_cast<volatile const int*>(b.kIter) : k;
}

// Inelastic constraint pass A (simkernels.js:248-309).
//
// flags & kTrackResid: writes r^2 for the residual of the state entering
//   this iteration, r = C + alphaT lambda + gamma dt cdot (the numerator the
//   damped update drives to zero; without the damping term the Jacobi fixed
//   point sits at C + alphaT lambda = -gamma dt cdot, not 0), 0 for an
//   inactive constraint (C = 0), and at iteration 0 the residual at
//   lambda = 0 to c0sq. The tracked variant is a separate instantiation
//   (kTrack) so the plain path carries none of it.
// flags & kWarm (iteration 0): starts from lambda0 = lamWarm instead of 0.
//   Its impulse has not been applied to the velocities this pass sees, so the
//   first correction uses the linearised post-impulse residual: applying
//   lambda0 moves C by denom lambda0 and gamma dt cdot by gamma denom lambda0
//   (the particle's own response, the Jacobi diagonal), so
//     r = C + gamma dt cdot + ((1+gamma) denom + alphaT) lambda0,
//     dlam = -omega r / ((1+gamma) denom + alphaT),
//   and the applied impulse is lambda0 + dlam. A warm value that would not
//   reduce the particle's own residual, |r| >= |C + gamma dt cdot|, is
//   replaced by the plain start lambda0 = 0 (the plain solve stays the
//   fallback). With lambda0 = 0 both updates are the reference's.
// flags & kMeasureOnly: residual only (the pass after the last iteration).
// flags & kStoredC (iteration 0, after computeL with features, one lane per
//   slot): the constraint is the one computeL evaluated at the same
//   velocities; k_solveA_stored applies it without a neighbour sweep.
// G lanes per slot (two or four on small scenes): the lanes split the neighbour
// sweep, lane 0 finishes the slot.
//
// The update of slot i from its constraint c (lane 0 of the slot).
template <bool kTrack, int G = 1>
__device__ __forceinline__ void solveAUpdate(const Bufs& b, const Ctx& cx, uint32_t i, const float4& pi,
                                             const float4* velIn, uint32_t mi, const Constraint& c, int k, bool warm0,
                                             bool measure, bool act = false) {
  const SceneDev& S = *cx.scene;
  constexpr bool track = kTrack;
  const float g = S.kDamp;
  const float stiff = (1.f + g) * c.denom + S.alphaT;  // d(residual) / d(applied multiplier)
  const float r0 = c.C + g * S.dt * c.cdot;            // residual at lambda = 0
  float lam0 = k == 0 ? (warm0 ? b.lamWarm[i] : 0.f) : b.lam[i];
  if (warm0 && !(fabsf(r0 + stiff * lam0) < fabsf(r0))) lam0 = 0.f;
  // the quantity the update drives to zero: r = C + alphaT lambda + gamma dt cdot
  const float lamTerm = warm0 ? stiff * lam0 : S.alphaT * lam0;
  float r2 = 0.f;
  if (track) {
    // an inactive constraint (C below 1e-7: the reference skips the particle
    // and leaves its multiplier alone) has no residual; counting alphaT lambda
    // there would add a term no iteration can change
    const float r = c.C == 0.f ? 0.f : r0 + lamTerm;
    r2 = r * r;
    b.rr[i] = r2;
    if (k == 0) b.c0sq[i] = r0 * r0;
  }
  // an inactive constraint still takes part in the contact pass
  const V3 xi = xyz(pi);
  const V3 xci = xi + S.dt * xyz(loadOwn<G>(velIn + i));
  const float mass = cx.mats[mi].mass;
  if (measure) {  // the contact residual of these velocities, no impulse
    storeSp(b, i, mzero(), splat(0.f), xi, xci, mass);
    return;
  }
  if (kTrack && act && (c.C == 0.f || r2 <= b.thr[3 * sceneIndex(b, cx)])) {
    // settled (or inactive): no impulse (its stamp stays older than k + 1);
    // solveB reads only the predicted position and mass of such a slot
    b.Sp[3 * (size_t)b.N + i] = make_float4(xci.x, xci.y, xci.z, mass);
    return;
  }
  if (c.C == 0.f) {
    if (k == 0) b.lam[i] = lam0;
    storeSp(b, i, mzero(), splat(0.f), xi, xci, mass);
    return;
  }
  const float dlam = S.omega * (-c.C - lamTerm - g * S.dt * c.cdot) / stiff;
  b.lam[i] = lam0 + dlam;
  const float imp = warm0 ? lam0 + dlam : dlam;
  storeSp(b, i, mscale(c.GL, imp), c.sgrad * imp, xi, xci, mass);
  if (kTrack && act) {
    b.imp[i] = (uint8_t)(k + 1);
    // its residual moves with its multiplier even where the velocity change
    // rounds away: evaluate it again next iteration
    b.dirty[(k + 1) & 1][i] = 1;
    markSolidNbrs(b, cx, i, xi, b.bmark);  // their solveB applies this impulse
  }
}

template <bool kTrack, int kMinB, int G, int kBlock = kThreads>
__global__ void __launch_bounds__(kBlock, kMinB) k_solveA(Bufs b, int k, const float4* velIn,
                                                            int flags) {
  const uint32_t t = afterPrevious(blockIdx.x * blockDim.x + threadIdx.x);
  const uint32_t i = t / G, lane = t % G;
  if (i >= b.N) return;
  const ListHead head = listHead<G>(nbrGroups(b.nbr, i), b.nbrCount, i, lane);
  const Ctx cx = ctxOf(b, i);
  const SceneDev& S = *cx.scene;
  constexpr bool track = kTrack;
  const bool measure = kTrack && (flags & kMeasureOnly) != 0;  // measure passes are tracked ones
  const bool warm0 = (flags & kWarm) != 0 && k == 0;
  const float4 pi = b.posS[i];
  const bool active = measure || iterating(b, S, i, k, flags);
  // active set (one lane per slot): from iteration 2 a solid whose inputs
  // did not change keeps its residual and takes no impulse
  const bool act = kTrack && G == 1 && (flags & kActive) != 0 && k > 0;
  bool changed = true;
  if (act && active && !waterW(pi.w)) changed = b.dirty[k & 1][i] != 0;
  const bool counts = active && !waterW(pi.w) && lane == 0 && changed;
  recordSolidDisp(b, i, k, counts ? S.dt * length(xyz(loadOwn<G>(velIn + i))) : 0.f);
  if (!active || waterW(pi.w)) {  // water: its record is never read
    if (track && lane == 0) {
      b.rr[i] = 0.f;
      if (k == 0) b.c0sq[i] = 0.f;
    }
    return;
  }
  if (act) {
    if (!changed) return;
    countWarp(b.actA + k);
  }
  const uint32_t mi = matOfW(pi.w);
  const float st = b.stateS[i];
  const Constraint c = evalConstraint<G>(b, cx, i, pi, velIn, cx.mats + mi, st, head, lane);
  if (G > 1 && lane != 0) return;
  solveAUpdate<kTrack, G>(b, cx, i, pi, velIn, mi, c, k, warm0, measure, act);
}

// Active set, iterations from 2: the changed slots of the scenes still
// iterating, appended to a list (in no particular order: each slot's own
// sums keep their list order, so the results do not depend on it); which = 1
// lists the slots solveB updates (changed or receiving an impulse). Only
// solids are ever marked changed; k_solveA_list skips any water slot. The
// list's length is the iteration's visit count. Each thread reads the flags
// of 16 consecutive slots with one 16-byte load per array (the flag arrays
// are padded to a multiple of 16) and checks the few flagged ones; the
// block appends its slots with one atomic.
constexpr int kCompactSlots = 16;
constexpr int kCompactThreads = 256;
__global__ void __launch_bounds__(kCompactThreads) k_compact(Bufs b, int k, int which) {
  __shared__ uint32_t warpBase[kCompactThreads / 32];
  __shared__ uint32_t blockBase;
  k = iterK(b, k);
  const uint32_t base = (blockIdx.x * blockDim.x + threadIdx.x) * kCompactSlots;
  uint32_t take = 0;
  if (base < b.N) {
    uint4 f = *reinterpret_cast<const uint4*>(b.dirty[k & 1] + base);
    if (which == 1) {
      const uint4 m = *reinterpret_cast<const uint4*>(b.bmark + base);
      f.x |= m.x; f.y |= m.y; f.z |= m.z; f.w |= m.w;
    }
    const uint32_t w[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
    for (int q = 0; q < kCompactSlots; ++q) {
      if (((w[q >> 2] >> (8 * (q & 3))) & 0xffu) == 0u) continue;
      const uint32_t i = base + (uint32_t)q;
      if (i >= b.N) break;
      const uint32_t s = b.S > 1 ? (uint32_t)b.sceneOf[i] : 0u;
      if (k < b.scenes[s].iterations && !b.done[s]) take |= 1u << q;
    }
  }
  const uint32_t cnt = (uint32_t)__popc(take);
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  uint32_t incl = cnt;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t n = __shfl_up_sync(0xffffffffu, incl, off);
    if (lane >= (unsigned)off) incl += n;
  }
  if (lane == 31u) warpBase[warp] = incl;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t run = 0;
#pragma unroll
    for (int q = 0; q < kCompactThreads / 32; ++q) {
      const uint32_t t = warpBase[q];
      warpBase[q] = run;
      run += t;
    }
    blockBase = run ? atomicAdd(which == 0 ? b.actA + k : b.actB + k, run) : 0u;
  }
  __syncthreads();
  if (!take) return;
  uint32_t start = blockBase + warpBase[warp] + incl - cnt;
  uint32_t* out = which == 0 ? b.listA : b.listB;
  while (take) {
    const int q = __ffs(take) - 1;
    take &= take - 1u;
    out[start++] = base + (uint32_t)q;
  }
}

// solveA over listA (iterations k >= 1 of the active set): the listed slots
// with a grid-stride loop over a grid that fills the GPU once, so warps stay
// full however the listed slots are spread.
template <int kMinB, int kBlock>
__global__ void __launch_bounds__(kBlock, kMinB) k_solveA_list(Bufs b, int k, const float4* __restrict__ velIn,
                                                                int flags) {
  k = iterK(b, k);
  const uint32_t cnt = *(volatile const uint32_t*)(b.actA + k);
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < cnt; t += gridDim.x * blockDim.x) {
    const uint32_t i = b.listA[t];
    const float4 pi = b.posS[i];
    if (waterW(pi.w)) continue;  // water takes no constraint (none is ever marked)
    const Ctx cx = ctxOf(b, i);
    const SceneDev& S = *cx.scene;
    recordSolidDisp(b, i, k, S.dt * length(xyz(velIn[i])));
    const uint32_t mi = matOfW(pi.w);
    const float st = b.stateS[i];
    const Constraint c = evalConstraint<1>(b, cx, i, pi, velIn, cx.mats + mi, st);
    solveAUpdate<true>(b, cx, i, pi, velIn, mi, c, k, false, false, true);
  }
  (void)flags;
}

// Iteration 0 after computeL with features: the constraint it stored at
// these velocities (bit-identical to evaluating it), no neighbour sweep — a
// register-light launch at full occupancy in place of the sweep kernel.
template <bool kTrack>
__global__ void __launch_bounds__(kThreads) k_solveA_stored(Bufs b, const float4* __restrict__ velIn, int flags) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= b.N) return;
  const Ctx cx = ctxOf(b, i);
  const SceneDev& S = *cx.scene;
  const bool warm0 = (flags & kWarm) != 0;
  const float4 pi = b.posS[i];
  const bool active = 0 < S.iterations && !sceneDone(b, i);
  recordSolidDisp(b, i, 0, active && !waterW(pi.w) ? S.dt * length(xyz(velIn[i])) : 0.f);
  if (!active || waterW(pi.w)) {
    if (kTrack) {
      b.rr[i] = 0.f;
      b.c0sq[i] = 0.f;
    }
    return;
  }
  solveAUpdate<kTrack>(b, cx, i, pi, velIn, matOfW(pi.w), loadConstraint(b, i), 0, warm0, false);
}

// Network features of every slot at iteration 0 (zeros for water):
//   0-2  log singular values of the trial F
//   3    C = sqrt(2 Psi) at the projected trial state
//   4    alphaT * lambda of the previous substep (same particle)
//   5    alphaT * lambda_1, lambda_1 = -C / (denom + alphaT): the particle's
//        own Newton step, blind to its neighbours
//   6    log10(1 + denom / alphaT): stiffness of the constraint vs compliance
//   7    solid neighbours / 32
//   8-14 material kind one-hot
//   15   log10(mu) - 4.5
__device__ __forceinline__ void fillFeatures(float (&f)[kFeat], const SceneDev& S, const Constraint& c, float lamPrev,
                                             uint32_t kind, float mu) {
  const float aT = S.alphaT;
  f[0] = c.logSigTr.x;
  f[1] = c.logSigTr.y;
  f[2] = c.logSigTr.z;
  f[3] = c.C;
  f[4] = aT * lamPrev;
  f[5] = -c.C * aT / (c.denom + aT);
  f[6] = log10f(1.f + c.denom / aT);
  f[7] = c.nNbr * (1.f / 32.f);
#pragma unroll
  for (uint32_t q = 0; q < 7u; ++q) f[8 + q] = kind == q ? 1.f : 0.f;  // constant indices: f stays in registers
  f[15] = log10f(fmaxf(mu, 1e-6f)) - 4.5f;
}
__device__ __forceinline__ void storeFeatures(const Bufs& b, uint32_t i, const float (&f)[kFeat]) {
  float4* out = reinterpret_cast<float4*>(b.feat + (size_t)i * kFeat);
#pragma unroll
  for (int q = 0; q < kFeat / 4; ++q) out[q] = make_float4(f[4 * q], f[4 * q + 1], f[4 * q + 2], f[4 * q + 3]);
}

// Bonet-Lok correction with SVD pseudo-inverse (simkernels.js:189-221); its
// candidate walk records the substep's neighbour list. kFeatures (the
// learned solve, or features logged): the same sweep forms iteration 0's
// velocity sum, so iteration 0's constraint (the arithmetic solveA's sweep
// would do, from the same sums in the same order) is stored for
// k_solveA_stored here, with the network's features (fillFeatures; zeros
// for water and for scenes without iterations), without a second sweep of
// every solid's neighbours.
// G lanes per slot (small handles): the lanes split the stencil's rows and the
// sums over what they find, lane 0 finishes the slot.
template <bool kFeatures, int G>
__device__ __forceinline__ void computeL(const Bufs& b) {
  __shared__ uint32_t column[G == 1 ? 1 : SubList<G>::kCap * kThreads];
  // blocks run last to first: the pass starts where the reorder ended, on
  // slots whose data is still in L2
  const uint32_t t = afterPrevious((gridDim.x - 1u - blockIdx.x) * blockDim.x + threadIdx.x);
  const uint32_t i = t / G, lane = t % G;
  if (i >= b.N) return;
  const Ctx cx = ctxOf(b, i);
  const SceneDev& S = *cx.scene;
  const float4* __restrict__ posS = b.posS;
  const float4 pi = b.posS[i];
  const V3 xi = xyz(pi);
  const float s2 = S.support2;
  // own phase from the front, the other one from the back (the water flag is
  // the sign bit of pos.w; no load for it in a scene of one phase); a list past
  // the capacity is marked as overflowed and never read, its last entries land
  // anywhere in it
  auto isOwn = [&](uint32_t j) {
    return S.onePhase || ((__float_as_uint(ldg(&posS[j].w)) ^ __float_as_uint(pi.w)) & kWaterBit) == 0u;
  };
  SubList<G> sub;
  uint32_t same = 0, other = 0;
  const Planes planes = planesOf(b.posP, b.planeN);
  if constexpr (G == 1) {
    walkCandidates(S, b.cellStart, xi, i, planes, xi, s2, [&](uint32_t j) {
      const bool own = isOwn(j);
      const uint32_t e = own ? same : ~other;
      *nbrEntry(b.nbr, i, e & (kNbrCap - 1u)) = j;
      same += own ? 1u : 0u;
      other += own ? 0u : 1u;
    });
  } else {
    sub.col = column + threadIdx.x;
    walkCandidates<G>(S, b.cellStart, xi, i, planes, xi, s2, [&](uint32_t j) { sub.add(j, isOwn(j)); }, lane);
    sub.totals(lane);
    same = sub.sameAll;
    other = sub.otherAll;
  }
  const uint32_t same4 = (same + 3u) & ~3u, other4 = (other + 3u) & ~3u;
  const bool fits = same4 + other4 <= kNbrCap && !sub.lost;
  if (fits) {
    if constexpr (G > 1) {
      for (uint32_t e = 0; e < sub.same; ++e) *nbrEntry(b.nbr, i, sub.sameBefore + e) = sub.at(e);
      for (uint32_t e = 0; e < sub.other; ++e)
        *nbrEntry(b.nbr, i, kNbrCap - 1u - sub.otherBefore - e) = sub.otherAt(e);
    }
    if (lane == 0) {
      for (uint32_t e = same; e < same4; ++e) *nbrEntry(b.nbr, i, e) = i;
      for (uint32_t e = other; e < other4; ++e) *nbrEntry(b.nbr, i, kNbrCap - 1u - e) = i;
    }
  }
  if (lane == 0) {
    uint32_t dry = 0u;
    if (S.hasWater && !waterW(pi.w) && fits && other == 0u) {  // for the PBF passes
      const I3 cc = cellCoord(S, xi);
      dry = 1u;
#pragma unroll
      for (int dz = -1; dz <= 1; ++dz)
#pragma unroll
        for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
          for (int dx = -1; dx <= 1; ++dx) {
            const int x = cc.x + dx, y = cc.y + dy, z = cc.z + dz;
            if (x >= 0 && x < S.dims[0] && y >= 0 && y < S.dims[1] && z >= 0 && z < S.dims[2] &&
                __ldg(b.cellWater + S.cellBase + cellIndex(S, x, y, z)) != 0)
              dry = 0u;
          }
    }
    b.nbrCount[i] = fits ? same | other << 8 | dry << 16 : kNbrOverflow;
  }
  // no pass of the substep reads a water particle's correction (every
  // velocity gradient is a solid's): k_computeL_water forms it when the state
  // is read
  if constexpr (kFeatures) {
    float f[kFeat];
#pragma unroll
    for (int q = 0; q < kFeat; ++q) f[q] = 0.f;
    if (!waterW(pi.w)) {
      M3 Av;
      bonetLok<true, true, G>(b, cx, i, xi, &Av, lane, &sub);
      if (G > 1 && lane != 0) return;
      if (S.iterations > 0) {
        const uint32_t mi = matOfW(pi.w);
        const float st = b.stateS[i];
        const MatDev& m = cx.mats[mi];
        const Constraint c = constraintTail(Av, TailIn{b.L, b.FS, b.sgP, b.N, i}, cx.scene, &m, st);
        storeConstraint(b, i, c);
        fillFeatures(f, S, c, b.lamPrev[i], m.kind, m.mu * hardening(m, st));
      }
    }
    if (G > 1 && lane != 0) return;
    storeFeatures(b, i, f);
  } else {
    if (!waterW(pi.w)) bonetLok<true, false, G>(b, cx, i, xi, nullptr, lane, &sub);
  }
}
template <int G>
__global__ void __launch_bounds__(kThreads, minComputeL(G)) k_computeL(Bufs b) {
  computeL<false, G>(b);
}
template <int G>
__global__ void __launch_bounds__(kThreads, minComputeLFeatures(G)) k_computeL_features(Bufs b) {
  computeL<true, G>(b);
}

// lambda_warm = previous multiplier + network output / alphaT (the network
// predicts alphaT times the increment over the previous substep's multiplier)
__global__ void k_warm_from_net(Bufs b) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= b.N) return;
  const Ctx cx = ctxOf(b, i);
  const float4 pi = b.posS[i];
  b.lamWarm[i] = waterW(pi.w) ? 0.f : b.lamPrev[i] + b.netOut[i] / cx.scene->alphaT;
}

// warm start from the previous substep's multiplier alone (no network)
__global__ void k_warm_from_prev(Bufs b) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= b.N) return;
  b.lamWarm[i] = b.lamPrev[i];
}

// Per-scene residual norms, deterministic, in one launch: block (x, s)
// sums the x-th of the scene's residBlocks(n) consecutive slot ranges (at
// least kResidPerBlock slots each, at most kResidBlocks ranges, so a large
// scene fills the GPU with float4 loads in flight and a small one takes few
// blocks) in a fixed order and stores the range's partial sums; the last of
// the scene's blocks to finish (a ticket counter, no waiting) adds the
// partials in range order, so the totals do not depend on which block comes
// last.
// Sums: constraint residual^2, (iteration 0) residual^2 at lambda = 0,
// contact correction^2, (iteration 0) velocity change^2.
// Each thread sums in f32 in a fixed order (a convergence test on sums of
// squares needs nothing finer, and f64 is slow here), then a fixed warp
// butterfly; the warps of a block and the ranges of a scene are added in f64.
//
// k >= 0: the residuals of the state entering iteration k (early stop),
// reduced after iteration k's update; k < 0: after the last iteration (slot
// kMaxResid - 1). A scene stops, skipping iterations k+1.., once both its
// constraint residual and its contact residual are within tol of their
// values entering iteration 0 (an early stop also ends the contact passes,
// which the constraint residual does not see). With a warm start, iteration
// 0's constraint residual is the linearised estimate before the warm impulse
// is applied, so it never stops the solve.
constexpr int kResidSums = 4;
constexpr int kResidThreads = 256;
constexpr uint32_t kResidPerBlock = 4096;
static_assert(kResidBlocks % 32 == 0, "whole lanes of partials in the final sum");
__host__ __device__ __forceinline__ uint32_t residBlocks(uint32_t n) {
  const uint32_t g = (n + kResidPerBlock - 1u) / kResidPerBlock;
  return g < 1u ? 1u : (g > (uint32_t)kResidBlocks ? (uint32_t)kResidBlocks : g);
}
__global__ void __launch_bounds__(kResidThreads) k_resid(Bufs b, int k, int warm) {
  __shared__ float warpSum[kResidThreads / 32][kResidSums];
  __shared__ bool lastBlock;
  k = iterK(b, k);
  const uint32_t s = blockIdx.y;
  const SceneDev& S = b.scenes[s];
  const uint32_t n = S.n, base = S.pBase;
  const uint32_t G = residBlocks(n);
  if (blockIdx.x >= G) return;  // the whole block: this scene needs fewer ranges
  const uint32_t c = blockIdx.x;
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  const uint32_t lo = base + (uint32_t)(((uint64_t)n * c) / G);
  const uint32_t hi = base + (uint32_t)(((uint64_t)n * (c + 1)) / G);
  float a = 0.f, a0 = 0.f, ac = 0.f, av = 0.f;
  const bool velSum = k == 0 && S.asShare > 0.f;  // the active set's velocity-change scale
  if (!b.done[s] || k < 0) {
    // the range's 16-byte-aligned interior as float4 (the arrays start on
    // 256-byte boundaries), its ragged ends (< 4 slots each) as scalars
    const uint32_t lo4 = min(hi, (lo + 3u) & ~3u), hi4 = max(lo4, hi & ~3u);
    if (lo + tid < lo4) {
      a += b.rr[lo + tid];
      ac += b.rc[lo + tid];
      if (k == 0) a0 += b.c0sq[lo + tid];
      if (velSum) av += b.dv0sq[lo + tid];
    }
    if (hi4 + tid < hi) {
      a += b.rr[hi4 + tid];
      ac += b.rc[hi4 + tid];
      if (k == 0) a0 += b.c0sq[hi4 + tid];
      if (velSum) av += b.dv0sq[hi4 + tid];
    }
    const float4* __restrict__ rr4 = reinterpret_cast<const float4*>(b.rr);
    const float4* __restrict__ rc4 = reinterpret_cast<const float4*>(b.rc);
    const float4* __restrict__ c04 = reinterpret_cast<const float4*>(b.c0sq);
#pragma unroll 4
    for (uint32_t q = lo4 / 4u + tid; q < hi4 / 4u; q += kResidThreads) {
      const float4 x = rr4[q], y = rc4[q];
      a += (x.x + x.y) + (x.z + x.w);
      ac += (y.x + y.y) + (y.z + y.w);
      if (k == 0) {
        const float4 z = c04[q];
        a0 += (z.x + z.y) + (z.z + z.w);
      }
      if (velSum) {
        const float4 z = reinterpret_cast<const float4*>(b.dv0sq)[q];
        av += (z.x + z.y) + (z.z + z.w);
      }
    }
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, off);
    a0 += __shfl_xor_sync(0xffffffffu, a0, off);
    ac += __shfl_xor_sync(0xffffffffu, ac, off);
    av += __shfl_xor_sync(0xffffffffu, av, off);
  }
  if (lane == 0) {
    warpSum[warp][0] = a;
    warpSum[warp][1] = a0;
    warpSum[warp][2] = ac;
    warpSum[warp][3] = av;
  }
  __syncthreads();
  if (tid == 0) {
    double t[kResidSums] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int w = 0; w < kResidThreads / 32; ++w)
#pragma unroll
      for (int q = 0; q < kResidSums; ++q) t[q] += (double)warpSum[w][q];
    double* part = b.residPart + ((size_t)s * kResidBlocks + c) * kResidSums;
#pragma unroll
    for (int q = 0; q < kResidSums; ++q) part[q] = t[q];
    __threadfence();  // the partials are visible before this block's ticket
    lastBlock = atomicAdd(b.residTicket + s, 1u) == G - 1u;
  }
  __syncthreads();
  if (!lastBlock || tid >= 32u) return;
  // the scene's last block, one warp: lane l adds ranges l, l + 32, ... in
  // order (loads through L2: the other blocks' partials are not in this
  // SM's L1), then a fixed butterfly combines the lanes
  __threadfence();
  if (lane == 0) b.residTicket[s] = 0u;  // every block of this launch has taken its ticket
  if (k >= 0 && (b.done[s] || k >= S.iterations)) return;
  double ta = 0.0, ta0 = 0.0, tac = 0.0, tav = 0.0;
#pragma unroll
  for (int r = 0; r < kResidBlocks / 32; ++r) {
    const uint32_t q = lane + 32u * (uint32_t)r;
    if (q < G) {
      const double* part = b.residPart + ((size_t)s * kResidBlocks + q) * kResidSums;
      ta += __ldcg(part);
      ta0 += __ldcg(part + 1);
      tac += __ldcg(part + 2);
      tav += __ldcg(part + 3);
    }
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    ta += __shfl_xor_sync(0xffffffffu, ta, off);
    ta0 += __shfl_xor_sync(0xffffffffu, ta0, off);
    tac += __shfl_xor_sync(0xffffffffu, tac, off);
    tav += __shfl_xor_sync(0xffffffffu, tav, off);
  }
  if (lane != 0) return;
  if (k < 0) {
    b.resid[(size_t)s * kMaxResid + (kMaxResid - 1)] = ta;
    b.residC[(size_t)s * kMaxResid + (kMaxResid - 1)] = tac;
    return;
  }
  if (k < kMaxResid - 1) {
    b.resid[(size_t)s * kMaxResid + k] = ta;
    b.residC[(size_t)s * kMaxResid + k] = tac;
  }
  const double tol = (double)S.residTol, tolC = (double)S.residTolC;
  if (k == 0) {
    b.c0[s] = ta0;
    b.cc0[s] = tac;
    // active set: a settled slot may hold up to asShare / nSolid of the
    // scene's squared residual budget (tol^2 of the iteration-0 sums)
    const double share = (double)S.asShare / (double)max(S.nSolid, 1u);
    b.thr[3 * s] = (float)(share * tol * tol * ta0);
    b.thr[3 * s + 1] = (float)(share * tolC * tolC * tac);
    // a velocity change at half the scale the converged solve still makes
    // (the tolerance times iteration 0's) moves a neighbour's residual by
    // less than its own settle threshold: smaller ones do not count as moved.
    // (At the whole scale, changes that add up over the iterations left one
    // particle of a 50k dam breach stale by more than the tolerance.)
    b.thr[3 * s + 2] = (float)(0.25 * share * tol * tol * tav);
  }
  if (tol > 0.0 && ta <= tol * tol * b.c0[s] && tac <= tolC * tolC * b.cc0[s] && !(warm && k == 0)) b.done[s] = 1;
  b.itersUsed[s] = k + 1;
}

// keep this substep's final multipliers for the next substep's features
__global__ void k_keep_lambda(Bufs b) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= b.N) return;
  b.lamOut[i] = b.lam[i];
}

// applyBoundary (simkernels.js:369-404)
__device__ __forceinline__ V3 applyBoundary(const SceneDev& S, V3 xcIn, V3 vIn, V3 xn, float fric) {
  V3 vv = vIn, xq = xcIn;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float lo = S.dmin[k], hi = S.dmax[k];
    if (xq[k] < lo || xq[k] > hi) {
      const float bound = xq[k] < lo ? lo : hi;
      const float vnNew = (bound - xn[k]) / S.dt;
      const float dvn = fabsf(vnNew - vv[k]);
      V3 vt = vv;
      vt[k] = 0.f;
      const float vtl = length(vt);
      if (vtl > 1e-9f) {
        const float drop = fminf(fric * dvn, vtl);
        vv = vv - vt / vtl * drop;
      }
      vv[k] = vnNew;
      xq = xn + S.dt * vv;
    }
  }
  if (S.colActive > 0.5f) {
    const V3 cp = v3(S.colPos[0], S.colPos[1], S.colPos[2]);
    const V3 cv = v3(S.colVel[0], S.colVel[1], S.colVel[2]);
    const V3 d = xq - cp;
    const float dist = length(d);
    if (dist < S.colR && dist > 1e-9f) {
      const V3 n = d / dist;
      const float vOut = dot(vv - cv, n);
      const float vGoal = fminf((S.colR - dist) / S.dt, 0.6f);
      if (vOut < vGoal) vv = vv + n * (vGoal - vOut);
    }
  }
  return vv;
}

struct SBData {
  float4 r0, r1, r2;  // a neighbour's dlam G L columns with its position in .w (the record's first planes)
};
// ... and, with several lanes per slot (small scenes, where a dependent load
// costs more than its bytes), its predicted position and mass
struct SBData4 : SBData {
  float4 r3;
};
template <int G>
__device__ __forceinline__ auto gatherSp(const float4* __restrict__ R, size_t N) {
  if constexpr (G == 1) {
    return SBData{ldg(R), ldg(R + N), ldg(R + 2 * N)};
  } else {
    return SBData4{{ldg(R), ldg(R + N), ldg(R + 2 * N)}, ldg(R + 3 * N)};
  }
}

// sum over the neighbours b of S_b g_b (S_b = dlam G L of b, the kernel
// gradient at x_b - x_i without its factor c). Every rounding is explicit, so
// that solveB and its active-set form add the same bits. add returns the
// squared distance.
struct ImpulseSum {
  V3 dv = V3{0.f, 0.f, 0.f};
  __device__ __forceinline__ float add(const SceneDev& S, V3 xi, const SBData& d) {
    const float dx = __fsub_rn(d.r0.w, xi.x), dy = __fsub_rn(d.r1.w, xi.y), dz = __fsub_rn(d.r2.w, xi.z);
    const float r2 = __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx)));
    const float t = __fmaf_rn(sqrtFast(r2), -S.halfInvH, 1.f);
    const float g = __fmul_rn(__fmul_rn(t, t), t);
    const float wx = __fmul_rn(dx, g), wy = __fmul_rn(dy, g), wz = __fmul_rn(dz, g);
    dv.x = __fmaf_rn(d.r0.x, wx, __fmaf_rn(d.r1.x, wy, __fmaf_rn(d.r2.x, wz, dv.x)));
    dv.y = __fmaf_rn(d.r0.y, wx, __fmaf_rn(d.r1.y, wy, __fmaf_rn(d.r2.y, wz, dv.y)));
    dv.z = __fmaf_rn(d.r0.z, wx, __fmaf_rn(d.r1.z, wy, __fmaf_rn(d.r2.z, wz, dv.z)));
    return r2;
  }
  // k sum + self
  __device__ __forceinline__ V3 total(float k, V3 self) const {
    return v3(__fmaf_rn(dv.x, k, self.x), __fmaf_rn(dv.y, k, self.y), __fmaf_rn(dv.z, k, self.z));
  }
};

// ---------------------------------------------------------------- solveB
// Constraint dv gather + contact correction + boundaries (simkernels.js:315-366).
// When a PBF pass follows, also stores the predicted position x + dt v_out
// that pbfA / pbfB would otherwise recompute for every candidate.
// flags & kTrackResid: writes |contact correction|^2 of the velocities
//   entering this iteration to rc (the contact residual; 0 for water).
// flags & kMeasureOnly: the contact residual only, of every solid slot, no
//   velocity update (the pass after the last iteration).
template <int kMinB, int G, int kBlock = kThreads>
__global__ void __launch_bounds__(kBlock, kMinB) k_solveB(Bufs b, int k, const float4* velIn,
                                                      float4* velOut, int writeXc, int flags) {
  // blocks run last to first: the pass starts where solveA ended, on slots
  // whose data is still in L2
  const uint32_t t = afterPrevious((gridDim.x - 1u - blockIdx.x) * blockDim.x + threadIdx.x);
  const uint32_t i = t / G, lane = t % G;
  for (uint32_t q = t; q < b.S; q += gridDim.x * blockDim.x)  // the next iteration's slot
    b.solidDisp[(size_t)((k + 1) & 1) * b.S + q] = 0u;
  if (i >= b.N) return;
  const ListHead head = listHead<G>(nbrGroups(b.nbr, i), b.nbrCount, i, lane);
  const Ctx cx = ctxOf(b, i);
  const SceneDev& S = *cx.scene;
  const float4* __restrict__ Sp = b.Sp;
  const float4 vi4 = loadOwn<G>(velIn + i);
  const float4 pi = loadOwn<G>(b.posS + i);
  const bool track = (flags & kTrackResid) != 0;
  const bool measure = (flags & kMeasureOnly) != 0;
  if (!measure && !iterating(b, S, i, k, flags)) {
    if (lane == 0) {
      velOut[i] = vi4;
      if (writeXc) {
        const V3 xc = xyz(pi) + S.dt * xyz(vi4);
        storeXc(b, i, xc, pi.w, k > 0);
      }
    }
    return;
  }
  const uint32_t mi = matOfW(pi.w);
  const MatDev& m = cx.mats[mi];
  const V3 xi = xyz(pi);
  V3 dv = splat(0.f), corr = splat(0.f);
  if (!waterW(pi.w)) {
    const size_t N = b.N;
    const float Vi = vi4.w;
    const V3 xci = xi + S.dt * xyz(vi4);
    const float minD = S.minD;
    const float massI = m.mass;
    // A neighbour can be within minD of x_i + dt v_i at the predicted
    // positions only if |x_b - x_i| < minD + dt |v_i| + dt |v_b|, and dt |v_b|
    // is at most the scene's largest solid displacement this iteration
    // (recorded by solveA): farther neighbours skip the contact test and the
    // load of their predicted position. 1% of slack covers the rounding of
    // the predicted positions and of the bound; the test on the pairs that
    // remain is unchanged, so the result is too.
    const float reach = (minD + S.dt * length(xyz(vi4)) +
                         __uint_as_float(loadOwn<G>(b.solidDisp + (size_t)(k & 1) * b.S + (cx.scene - b.scenes)))) *
                        1.01f;
    const float reach2 = reach * reach;
    ImpulseSum sum;
    auto body = [&](uint32_t j, const auto& d) {
      const float r2 = sum.add(S, xi, d);
      if (!(r2 < reach2) || j == i) return;
      float4 r3;
      if constexpr (G == 1)
        r3 = ldg(Sp + 3 * N + j);
      else
        r3 = d.r3;
      const V3 dxc = xci - xyz(r3);
      const float d2 = dot(dxc, dxc);
      if (d2 < minD * minD && d2 > 1e-18f) {
        const float rinv = rsqrtf(d2);
        const float dist = d2 * rinv;
        const float mb = r3.w;
        const float w = mb / (massI + mb);
        corr = corr + dxc * (rinv * ((minD - dist) * w));
      }
    };
    forSameSingles<G>(b, cx, head, i, xi, lane, [&](uint32_t j) { return gatherSp<G>(Sp + j, N); }, body);
    const V3 self = xyz(b.SpSelf[i]);
    const float k = Vi * S.gradC;
    if constexpr (G > 1) {
      sum.dv = laneSum<G>(sum.dv);
      corr = laneSum<G>(corr);
    }
    dv = sum.total(k, self);
  }
  if (G > 1 && lane != 0) return;
  if (track) b.rc[i] = dot(corr, corr);
  if (measure) return;
  V3 dvv = dv / (m.mass * S.dt);
  const float dvl = length(dvv);
  if (dvl > S.dvCap) dvv = dvv * (S.dvCap / dvl);
  V3 v = xyz(vi4) + dvv + corr * (S.contactOmega / S.dt);
  v = applyBoundary(S, xi + S.dt * v, v, xi, m.boundFriction);
  velOut[i] = make_float4(v.x, v.y, v.z, vi4.w);
  if (writeXc) {
    const V3 xc = xi + S.dt * v;
    storeXc(b, i, xc, pi.w, k > 0);
  }
}

// solveB under the active set (one lane per slot; the launch passes
// velOut == velIn: a slot reads only its own velocity, so the update is in
// place and slots not visited keep theirs without a copy). flags & kActive
// (iterations >= 2): only slots marked as changed (dirty) or receiving a
// neighbour's impulse (bmark) run; a changed slot re-evaluates its contact
// correction and applies it only above the scene's per-slot threshold, a
// slot that only receives impulses keeps its (unchanged, unapplied)
// contact correction. A neighbour's impulse record is gathered only if it
// took an impulse (imp); its predicted position and mass (the record's
// fourth plane) are current for every solid. flags & kMarkMoved: a slot
// whose velocity changed marks itself and its solid neighbours as changed
// for iteration k + 1. The scene's solid displacement bound carries into
// the next iteration's slot (solveA raises it for the slots it visits).
// One slot of solveB under the active set; `listed`: the slot came from
// listB (changed or marked), so the flags are only cleared.
__device__ __forceinline__ void solveBActiveSlot(const Bufs& b, int k, float4* __restrict__ vel, int writeXc,
                                                 int flags, uint32_t i, bool listed) {
  const Ctx cx = ctxOf(b, i);
  const SceneDev& S = *cx.scene;
  const float4 pi = b.posS[i];
  if (k >= S.iterations || sceneDone(b, i)) {
    if (writeXc) {
      const float4 vi4 = vel[i];
      const V3 xc = xyz(pi) + S.dt * xyz(vi4);
      storeXc(b, i, xc, pi.w, k > 0);
    }
    return;
  }
  // water: solveB only applies the boundary to it, which after iteration 0
  // the PBF pass that moved it has already done (pbfB folds it in)
  if (k > 0 && waterW(pi.w)) {
    if (writeXc) {
      const float4 vi4 = vel[i];
      const V3 xc = xyz(pi) + S.dt * xyz(vi4);
      storeXc(b, i, xc, pi.w, k > 0);
    }
    return;
  }
  const bool skip = (flags & kActive) != 0 && k > 0;
  bool changed = true;
  if (skip) {
    uint8_t* __restrict__ dk = b.dirty[k & 1];
    changed = dk[i] != 0;
    const bool marked = b.bmark[i] != 0;
    if (changed) dk[i] = 0;
    if (marked) b.bmark[i] = 0;
    if (!changed && !marked) {
      if (writeXc) {
        const float4 vi4 = vel[i];
        const V3 xc = xyz(pi) + S.dt * xyz(vi4);
        storeXc(b, i, xc, pi.w, k > 0);
      }
      return;
    }
    if (!listed) countWarp(b.actB + k);
  }
  const uint8_t stamp = (uint8_t)(k + 1);
  const float4 vi4 = vel[i];
  const uint32_t mi = matOfW(pi.w);
  const MatDev& m = cx.mats[mi];
  const V3 xi = xyz(pi);
  const bool iWater = waterW(pi.w);
  V3 dv = splat(0.f), corr = splat(0.f);
  if (!iWater) {
    const size_t N = b.N;
    const float4* __restrict__ Sp = b.Sp;
    if (!skip || b.imp[i] == stamp) dv = xyz(b.SpSelf[i]);
    const float Vi = vi4.w;
    const V3 xci = xi + S.dt * xyz(vi4);
    const float minD = S.minD;
    const float massI = m.mass;
    const float reach = (minD + S.dt * length(xyz(vi4)) +
                         __uint_as_float(__ldg(b.solidDisp + (size_t)(k & 1) * b.S + sceneIndex(b, cx)))) *
                        1.01f;
    const float reach2 = reach * reach;
    auto contact = [&](const float4& r3) {
      const V3 dxc = xci - xyz(r3);
      const float d2 = dot(dxc, dxc);
      if (d2 < minD * minD && d2 > 1e-18f) {
        const float rinv = rsqrtf(d2);
        const float dist = d2 * rinv;
        const float mb = r3.w;
        const float w = mb / (massI + mb);
        corr = corr + dxc * (rinv * ((minD - dist) * w));
      }
    };
    ImpulseSum sum;
    auto visit = [&](uint32_t j) {
      const bool jImp = !skip || b.imp[j] == stamp;
      if (jImp) {
        const float4* R = Sp + j;
        const float4 r0 = ldg(R), r1 = ldg(R + N), r2 = ldg(R + 2 * N);
        const float d2 = sum.add(S, xi, SBData{r0, r1, r2});
        if (changed && d2 < reach2) contact(ldg(Sp + 3 * N + j));
      } else if (changed) {
        contact(ldg(Sp + 3 * N + j));
      }
    };
    const uint32_t c = b.nbrCount[i];
    if (c != kNbrOverflow) {
      const uint4* L = nbrGroups(b.nbr, i);
      const uint32_t cnt = sameCount(c);
#pragma unroll 1
      for (uint32_t q = 0; 4u * q < cnt; ++q) {
        const uint4 g = *(L + kGroupStride * q);
#pragma unroll
        for (uint32_t t = 0; t < 4u; ++t) {
          const uint32_t e = lane4(g, t);
          if (e != i) visit(e);
        }
      }
    } else {
      forRows(S, b.cellStart, xi, [&](uint32_t beg, uint32_t end) {
#pragma unroll 1
        for (uint32_t j = beg; j < end; ++j) {
          if (j == i) continue;
          const float4 pj = ldg(b.posS + j);
          const V3 d = xi - xyz(pj);
          if (dot(d, d) < S.support2 && !waterW(pj.w)) visit(j);
        }
      });
    }
    dv = sum.total(Vi * S.gradC, dv);
    if (changed) {
      const float c2 = dot(corr, corr);
      b.rc[i] = c2;
      if (skip && c2 <= b.thr[3 * sceneIndex(b, cx) + 1]) corr = splat(0.f);  // settled: left unapplied
    } else {
      corr = splat(0.f);  // unchanged since last evaluated: at or below the threshold, not applied
    }
  } else if (changed) {
    b.rc[i] = 0.f;
  }
  V3 dvv = dv / (m.mass * S.dt);
  const float dvl = length(dvv);
  if (dvl > S.dvCap) dvv = dvv * (S.dvCap / dvl);
  V3 v = xyz(vi4) + dvv + corr * (S.contactOmega / S.dt);
  v = applyBoundary(S, xi + S.dt * v, v, xi, m.boundFriction);
  vel[i] = make_float4(v.x, v.y, v.z, vi4.w);
  if (writeXc) {
    const V3 xc = xi + S.dt * v;
    storeXc(b, i, xc, pi.w, k > 0);
  }
  const V3 dvel = v - xyz(vi4);
  const float dv2 = dot(dvel, dvel);
  if (k == 0) b.dv0sq[i] = iWater ? 0.f : dv2;
  // moved: any change in iteration 0; later, a change above the scene's scale
  if ((flags & kMarkMoved) && (k == 0 ? (v.x != vi4.x || v.y != vi4.y || v.z != vi4.z)
                                      : dv2 > b.thr[3 * sceneIndex(b, cx) + 2])) {
    uint8_t* __restrict__ dn = b.dirty[(k + 1) & 1];
    dn[i] = 1;
    if (!iWater) markSolidNbrs(b, cx, i, xi, dn);
  }
}

// solveB under the active set (one lane per slot; the launch passes one
// velocity array: a slot reads only its own velocity, so the update is in
// place and slots not visited keep theirs without a copy). flags & kActive
// (iterations >= 2): only slots marked as changed (dirty) or receiving a
// neighbour's impulse (bmark) run; a changed slot re-evaluates its contact
// correction and applies it only above the scene's per-slot threshold, a
// slot that only receives impulses keeps its (unchanged, unapplied)
// contact correction. A neighbour's impulse record is gathered only if it
// took an impulse this iteration (its stamp is k + 1); its predicted
// position and mass (the record's fourth plane) are current for every
// solid. flags & kMarkMoved: a slot whose velocity changed (after iteration
// 0: by more than the scene's velocity scale) marks itself and its solid
// neighbours as changed for iteration k + 1. The scene's solid displacement
// bound carries into the next iteration's slot (solveA raises it for the
// slots it visits). With `list` the launch runs over listB (grid-stride),
// else one thread per slot.
template <int kMinB, int kBlock = kThreads>
__global__ void __launch_bounds__(kBlock, kMinB) k_solveB_active(Bufs b, int k, float4* __restrict__ vel, int writeXc,
                                                                 int flags, int list) {
  k = iterK(b, k);
  const uint32_t t0 = blockIdx.x * blockDim.x + threadIdx.x;
  for (uint32_t q = t0; q < b.S; q += gridDim.x * blockDim.x)  // carried into the next iteration's slot
    b.solidDisp[(size_t)((k + 1) & 1) * b.S + q] = b.solidDisp[(size_t)(k & 1) * b.S + q];
  if (list) {
    const uint32_t cnt = *(volatile const uint32_t*)(b.actB + k);
    for (uint32_t t = t0; t < cnt; t += gridDim.x * blockDim.x)
      solveBActiveSlot(b, k, vel, writeXc, flags, b.listB[t], true);
    return;
  }
  const uint32_t i = (gridDim.x - 1u - blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < b.N) solveBActiveSlot(b, k, vel, writeXc, flags, i, false);
}

__device__ __forceinline__ bool pbfActive(const SceneDev& S, int k) {
  return S.hasWater && k < S.pbfUntil;
}

// The PBF pair terms of two predicted neighbours per packed instruction: the
// poly6 kernel of r^2 and the spiky gradient (common.js:81-94, H = support),
// the latter by one reciprocal square root and 0 below r = 1e-9, the
// reference's zero-distance guard (r^2 < 1e-18).
//
// The density solve amplifies rounding: each pass feeds its positions to the
// next, through fourth powers. Sums packed in another order left the
// velocities of a 1M-particle dam with 15 density passes 2.8e-5 (2-norm) from
// the scalar sums after two substeps. So every rounding here is written out,
// and the sums add their terms one neighbour after the other in stencil order
// (with one lane per slot): packing changes no bit. It costs pbfB nothing and
// pbfA 1% against packed accumulators.
struct PbfPair {
  F2 w6, gx, gy, gz;
};
__device__ __forceinline__ float invDist(float r2) { return r2 < 1e-18f ? 0.f : rsqrtf(r2); }
__device__ __forceinline__ PbfPair pbfPair(const SceneDev& S, V3 c, const float4& p, const float4& q) {
  const F2 dx = f2(c.x - p.x, c.x - q.x), dy = f2(c.y - p.y, c.y - q.y), dz = f2(c.z - p.z, c.z - q.z);
  const F2 r2 = fma2(dz, dz, fma2(dx, dx, mul2(dy, dy)));
  const F2 minus = f2(-1.f, -1.f);
  // 0 past the support: the lists also hold neighbours that may come into it
  const F2 x0 = fma2(r2, minus, f2(S.support2, S.support2));
  const F2 x = f2(fmaxf(lo2(x0), 0.f), fmaxf(hi2(x0), 0.f));
  const F2 rinv = f2(invDist(lo2(r2)), invDist(hi2(r2)));
  const F2 t0 = fma2(mul2(r2, rinv), minus, f2(S.support, S.support));
  const F2 t = f2(fmaxf(lo2(t0), 0.f), fmaxf(hi2(t0), 0.f));
  const F2 s = mul2(mul2(mul2(f2(S.spikyC, S.spikyC), t), t), rinv);
  return PbfPair{mul2(mul2(mul2(f2(S.poly6C, S.poly6C), x), x), x), mul2(dx, s), mul2(dy, s), mul2(dz, s)};
}

// ---------------------------------------------------------------- pbfA
// The stencil walk of a PBF pass: slot i's neighbours by predicted position
// within the support (exact) or the support and its skin, recorded in order;
// the count word. Water pairs with everything, a solid with water only (the
// pairs pbfB uses, simkernels.js:457-458; the water flag is the sign bit of
// xc.w, the sorted pos.w).
template <int G>
__device__ __forceinline__ uint32_t pbfWalk(const Bufs& b, const SceneDev& S, uint32_t i, V3 x, const float4& xc4,
                                            bool exact, SubList<G>& sub, uint32_t lane) {
  const float4* __restrict__ xcS = b.xc;
  const V3 xci = xyz(xc4);
  const bool iWater = waterW(xc4.w);
  const Planes P = planesOf(b.xcP, b.planeN);
#pragma unroll 1
  for (;;) {
    const float s2 = exact ? S.support2 : S.support2 * ((1.f + kPbfSkin) * (1.f + kPbfSkin));
    uint32_t cnt = 0;
    sub.same = 0;
    sub.lost = false;
    auto record = [&](uint32_t j) {
      if constexpr (G == 1) {
        *nbrEntry(b.nbrP, i, min(cnt, kNbrCap - 1u)) = j;
        ++cnt;
      } else {
        sub.add(j, true);
      }
    };
    walkCandidates<G>(S, b.cellStart, x, i, P, xci, s2, [&](uint32_t j) {
      if (iWater || waterW(ldg(&xcS[j].w))) record(j);
    }, lane);
    if constexpr (G > 1) {
      sub.totals(lane);
      cnt = sub.sameAll;
    }
    const bool fits = cnt <= kNbrCap && !sub.lost;
    if (!fits && !exact) {
      exact = true;
      continue;
    }
    if (!fits) return kNbrOverflow;
    if constexpr (G > 1)
      for (uint32_t e = 0; e < sub.same; ++e) *nbrEntry(b.nbrP, i, sub.sameBefore + e) = sub.at(e);
    if (lane == 0)  // whole groups
      for (uint32_t e = cnt; e & 3u; ++e) *nbrEntry(b.nbrP, i, e) = i;
    return exact ? cnt | kNbrExact : cnt;
  }
}
// PBF density multiplier (simkernels.js:407-439) over the predicted neighbours,
// which the pass's own walk around the current cell records or an earlier one
// left. G lanes per slot (small handles): the lanes split the stencil's rows and
// the density sums over what they find, lane 0 finishes the slot.
template <int G>
__global__ void __launch_bounds__(kThreads, minPbfA(G)) k_pbfA(Bufs b, int k, int flags) {
  __shared__ uint32_t column[G == 1 ? 1 : SubList<G>::kCap * kThreads];
  const uint32_t t = afterPrevious(blockIdx.x * blockDim.x + threadIdx.x);
  const uint32_t i = t / G, lane = t % G;
  if (i >= b.N) return;
  const Ctx cx = ctxOf(b, i);
  const SceneDev& S = *cx.scene;
  if (!pbfActive(S, k) || ((flags & kRerun) && !b.rerun[sceneIndex(b, cx)])) return;
  const float4* __restrict__ xcS = b.xc;
  const float4 pi = b.posS[i];
  const bool iWater = waterW(pi.w);
  if (!iWater && dryCount(b.nbrCount[i])) {
    // a solid only pairs with water here; its candidates come from its 27
    // cells, and computeL found no water particle in them: nothing to record
    // in any pass of the substep (no water particle pairs with it either)
    if (k == 0 && lane == 0) {
      b.nbrPCount[i] = 0u;
      b.pbfLam[i] = 0.f;
      b.xcRef[i].w = kNoRef;
    }
    return;
  }
  const float4 xc4 = b.xc[i];
  const V3 xci = xyz(xc4);
  const float s2 = S.support2;
  SubList<G> sub;
  sub.col = column + threadIdx.x;
  // One walk serves several passes: it records the neighbours within
  // (1 + skin) times the support, and as long as no particle of the scene has
  // moved half the skin from where that walk saw it (less 2% for rounding),
  // every neighbour within the support is among them. The terms of the others
  // are 0 and the sums add in the same order, so the bits are those of a walk
  // in every pass. A slot with too many of those neighbours keeps to its exact
  // ones and walks in every pass. The walk was two thirds of the kernel: 0.62
  // ms with it and 0.29 without on the 4M-particle mix (pbfB, over a third
  // more pairs, 0.21 -> 0.28); 15 passes of 100k particles 680 -> 524 us.
  const bool still = k > 0 && __uint_as_float(b.pbfMoved[sceneIndex(b, cx)]) <=
                                  S.support2 * (0.49f * 0.49f * kPbfSkin * kPbfSkin);
  const uint32_t before = still ? b.nbrPCount[i] : kNbrOverflow;
  const bool reuse = still && (before & kNbrExact) == 0u;
  uint32_t stored;
  if (reuse) {
    stored = before;
  } else {
    stored = pbfWalk<G>(b, S, i, xyz(pi), xc4, still, sub, lane);
    if (lane == 0) b.nbrPCount[i] = stored;
  }
  if (!still && lane == 0) b.xcRef[i] = xc4;
  if (!iWater) {
    if (lane == 0) {
      b.pbfLam[i] = 0.f;
      b.pbfRec[i] = make_float4(xci.x, xci.y, xci.z, 0.f);
    }
    return;
  }
  const MatDev& m = cx.mats[matOfW(pi.w)];
  const float rho0 = m.density;
  const float invRho0 = __frcp_rn(rho0);
  // a padding entry (i itself) and, on the stencil walk, the second of each
  // pair weigh 0
  float rho = G == 1 || lane == 0 ? m.mass * S.w00 : 0.f;
  V3 gradSum = splat(0.f);
  float grad2 = 0.f;
  auto add = [&](const float4& p, const float4& q, float m0, float m1) {
    const PbfPair r = pbfPair(S, xci, p, q);
    rho = __fmaf_rn(m0, lo2(r.w6), rho);
    rho = __fmaf_rn(m1, hi2(r.w6), rho);
    const F2 k = f2(__fmul_rn(m0, invRho0), __fmul_rn(m1, invRho0));
    const F2 ux = mul2(r.gx, k), uy = mul2(r.gy, k), uz = mul2(r.gz, k);
    gradSum.x = __fadd_rn(__fadd_rn(gradSum.x, lo2(ux)), hi2(ux));
    gradSum.y = __fadd_rn(__fadd_rn(gradSum.y, lo2(uy)), hi2(uy));
    gradSum.z = __fadd_rn(__fadd_rn(gradSum.z, lo2(uz)), hi2(uz));
    const F2 u2 = fma2(uz, uz, fma2(ux, ux, mul2(uy, uy)));
    grad2 = __fadd_rn(__fadd_rn(grad2, lo2(u2)), hi2(u2));
  };
  auto massOf = [&](float w) { return cx.mats[matOfW(w)].mass; };
  auto gather = [&](uint32_t j) { return ldg(xcS + j); };
  // the pairs of the list (with several lanes, of this lane's part of it)
  auto pairs = [&](auto&& body) {
    const uint32_t cnt = stored & 0xffu;
    if constexpr (G == 1) {
      forPairs(nbrGroups(b.nbrP, i), (cnt + 3u) >> 2, gather, body);
    } else if (reuse) {
      const uint4* L = nbrGroups(b.nbrP, i);
      forListPairs<G>(L, listHead<G>(L, b.nbrPCount, i, lane), cnt, i, lane, gather, body);
    } else {
#pragma unroll 2
      for (uint32_t e = 0; e < sub.same; e += 2u) {
        const bool two = e + 1u < sub.same;
        const uint32_t j0 = sub.at(e), j1 = two ? sub.at(e + 1u) : j0;
        body(j0, two ? j1 : i, gather(j0), gather(j1));  // (i weighs 0)
      }
    }
  };
  if (stored != kNbrOverflow) {
    if (S.twoMasses) {  // one water and at most one solid material: the sign of xc.w tells a neighbour's mass
      const float mW = S.massW, mS = S.massS;
      pairs([&](uint32_t j0, uint32_t j1, const float4& p, const float4& q) {
        add(p, q, j0 == i ? 0.f : (waterW(p.w) ? mW : mS), j1 == i ? 0.f : (waterW(q.w) ? mW : mS));
      });
    } else {
      pairs([&](uint32_t j0, uint32_t j1, const float4& p, const float4& q) {
        add(p, q, j0 == i ? 0.f : massOf(p.w), j1 == i ? 0.f : massOf(q.w));
      });
    }
  } else {
    forRows<G>(S, b.cellStart, xyz(pi), [&](uint32_t beg, uint32_t end) {
#pragma unroll 1
      for (uint32_t j = beg; j < end; ++j) {
        if (j == i) continue;
        const float4 c = ldg(xcS + j);
        const V3 d = xci - xyz(c);
        if (dot(d, d) < s2) add(c, c, massOf(c.w), 0.f);
      }
    }, lane);
  }
  if constexpr (G > 1) {
    rho = laneSum<G>(rho);
    gradSum = laneSum<G>(gradSum);
    grad2 = laneSum<G>(grad2);
    if (lane != 0) return;
  }
  const float C = fmaxf(__fmaf_rn(rho, invRho0, -1.f), 0.f);
  const float lam = -C / (grad2 + dot(gradSum, gradSum) + S.pbfEps);
  b.pbfLam[i] = lam;
  b.pbfRec[i] = make_float4(xci.x, xci.y, xci.z, lam);
}

// ---------------------------------------------------------------- pbfB
// PBF position correction with s_corr (simkernels.js:441-477) over pbfA's
// record of predicted neighbours.
template <int G>
__global__ void __launch_bounds__(kThreads, minPbfB(G)) k_pbfB(Bufs b, int k, const float4* velIn, float4* velOut,
                                                               int flags) {
  // blocks run last to first: the pass starts where pbfA ended, on
  // slots whose data is still in L2
  const uint32_t t = afterPrevious((gridDim.x - 1u - blockIdx.x) * blockDim.x + threadIdx.x);
  const uint32_t i = t / G, lane = t % G;
  for (uint32_t q = t; q < b.S; q += gridDim.x * blockDim.x) b.pbfMoved[q] = 0u;  // the next pass's maximum
  if (i >= b.N) return;
  const ListHead head = listHead<G>(nbrGroups(b.nbrP, i), b.nbrPCount, i, lane);
  const Ctx cx = ctxOf(b, i);
  const SceneDev& S = *cx.scene;
  const float4 vi4 = velIn[i];
  const uint32_t word = G == 1 ? b.nbrPCount[i] : head.count;
  const uint32_t cnt = word == kNbrOverflow ? word : word & 0xffu;
  const float4 pi = b.posS[i];
  const bool iWater = waterW(pi.w);
  // no pass, or a solid without pairs: nothing moves it
  if (!pbfActive(S, k) || ((flags & kRerun) && !b.rerun[sceneIndex(b, cx)]) || (cnt == 0u && !iWater)) {
    if (lane == 0) velOut[i] = vi4;
    return;
  }
  const float4* __restrict__ xcS = b.xc;
  const uint32_t mi = matOfW(pi.w);
  const V3 xci = xyz(b.xc[i]);
  const float li = b.pbfLam[i];
  const MatDev& mWi = cx.mats[mi];
  // sum of (lambda_i + lambda_b + s_corr) gradW mpd_b, s_corr = -k (W / W0)^4
  V3 dp = splat(0.f);
  const float nk = -S.sCorrK;
  float reach = 0.f;  // a solid's: > 0 if any of its recorded neighbours is within the support
  auto add = [&](uint32_t j0, uint32_t j1, const float4& p, const float4& q, F2 lb, float mpd0, float mpd1) {
    const PbfPair r = pbfPair(S, xci, p, q);
    if (!iWater) reach = fmaxf(reach, fmaxf(j0 != i ? lo2(r.w6) : 0.f, j1 != i ? hi2(r.w6) : 0.f));
    const F2 w = mul2(r.w6, f2(S.invW0, S.invW0));
    const F2 w2 = mul2(w, w);
    const F2 f = fma2(mul2(w2, w2), f2(nk, nk), add2(f2(li, li), lb));
    const F2 ux = mul2(f, r.gx), uy = mul2(f, r.gy), uz = mul2(f, r.gz);
    dp.x = __fmaf_rn(hi2(ux), mpd1, __fmaf_rn(lo2(ux), mpd0, dp.x));
    dp.y = __fmaf_rn(hi2(uy), mpd1, __fmaf_rn(lo2(uy), mpd0, dp.y));
    dp.z = __fmaf_rn(hi2(uz), mpd1, __fmaf_rn(lo2(uz), mpd0, dp.z));
  };
  // a pair weighs by its water particle's mass / density
  auto mpdOf = [&](float w) { return waterW(w) ? cx.mats[matOfW(w)].massPerDensity : mWi.massPerDensity; };
  if (cnt != kNbrOverflow && S.waterMpd > 0.f) {
    // one water material: every pair weighs by its mass / density, and one
    // gather of pbfA's record (predicted position, multiplier) serves a pair
    const float mpd = S.waterMpd;
    forListPairs<G>(nbrGroups(b.nbrP, i), head, cnt, i, lane, [&](uint32_t j) { return ldg(b.pbfRec + j); },
                    [&](uint32_t j0, uint32_t j1, const float4& p, const float4& q) {
                      add(j0, j1, p, q, f2(p.w, q.w), mpd, mpd);
                    });
  } else if (cnt != kNbrOverflow) {
    forListPairs<G>(nbrGroups(b.nbrP, i), head, cnt, i, lane, [&](uint32_t j) { return ldg(xcS + j); },
                    [&](uint32_t j0, uint32_t j1, const float4& p, const float4& q) {
                      add(j0, j1, p, q, f2(ldg(b.pbfLam + j0), ldg(b.pbfLam + j1)), mpdOf(p.w), mpdOf(q.w));
                    });
  } else {
    forRows<G>(S, b.cellStart, xyz(pi), [&](uint32_t beg, uint32_t end) {
#pragma unroll 1
      for (uint32_t j = beg; j < end; ++j) {
        if (j == i) continue;
        const float4 c = ldg(xcS + j);
        if (!(iWater || waterW(c.w))) continue;
        const V3 d = xci - xyz(c);
        if (dot(d, d) < S.support2) add(j, i, c, c, f2(ldg(b.pbfLam + j), 0.f), mpdOf(c.w), 0.f);
      }
    }, lane);
  }
  if constexpr (G > 1) {
    dp = laneSum<G>(dp);
    reach = laneSum<G>(reach);
    if (lane != 0) return;
  }
  if (!iWater && reach == 0.f) {  // no pair within the support
    velOut[i] = vi4;
    return;
  }
  const float scale = iWater ? 1.f : 0.5f;
  V3 v = xyz(vi4) + dp * (scale / S.dt);
  // active set: a water particle's boundary, which the next solveB would
  // apply to the velocity this pass leaves (its only work on water), is
  // applied here from the same inputs, so that solveB need not visit water
  if ((flags & kInPlace) && iWater) v = applyBoundary(S, xyz(pi) + S.dt * v, v, xyz(pi), mWi.boundFriction);
  velOut[i] = make_float4(v.x, v.y, v.z, vi4.w);
  // active set: the next iteration revisits a solid this pass moved and its
  // solid neighbours, whose constraint and contact inputs it is
  if ((flags & kMarkMoved) && !iWater) {
    const V3 dvel = v - xyz(vi4);
    if (dot(dvel, dvel) > b.thr[3 * (uint32_t)(cx.scene - b.scenes) + 2]) {
      uint8_t* __restrict__ dn = b.dirty[(k + 1) & 1];
      dn[i] = 1;
      markSolidNbrs(b, cx, i, xyz(pi), dn);
    }
  }
}

// ---------------------------------------------------------------- xsph
// simkernels.js:480-507
template <int G>
__global__ void __launch_bounds__(kThreads) k_xsph(Bufs b, const float4* velIn, float4* velOut) {
  const uint32_t t = afterPrevious(blockIdx.x * blockDim.x + threadIdx.x);
  const uint32_t i = t / G, lane = t % G;
  if (i >= b.N) return;
  const ListHead head = listHead<G>(nbrGroups(b.nbr, i), b.nbrCount, i, lane);
  const Ctx cx = ctxOf(b, i);
  const SceneDev& S = *cx.scene;
  const float4* __restrict__ posS = b.posS;
  const float4 pi = b.posS[i];
  const V3 xi = xyz(pi);
  const float4 vi4 = velIn[i];
  const V3 vi = xyz(vi4);
  const bool iWater = waterW(pi.w);
  // W = sigW t^4 (2 q + 1) with t = 1 - q / 2. The two neighbours' terms are
  // formed together and added one after the other, every rounding fixed:
  // the water's next substep amplifies what differs here.
  V3 acc = splat(0.f);
  forSame<G>(b, cx, head, i, xi, iWater, lane, [&](uint32_t j) { return PV{ldg(posS + j), ldg(velIn + j)}; },
             [&] { return PV{pi, vi4}; }, [&](uint32_t, uint32_t, const PV& d0, const PV& d1) {
               const F2 dx = f2(xi.x - d0.p.x, xi.x - d1.p.x), dy = f2(xi.y - d0.p.y, xi.y - d1.p.y),
                        dz = f2(xi.z - d0.p.z, xi.z - d1.p.z);
               const F2 r2 = fma2(dz, dz, fma2(dx, dx, mul2(dy, dy)));
               // (a padding entry is the slot itself: r = 0, dv = 0)
               const F2 rinv = f2(rsqrtf(fmaxf(lo2(r2), 1e-30f)), rsqrtf(fmaxf(hi2(r2), 1e-30f)));
               const F2 q = mul2(mul2(r2, rinv), f2(S.invH, S.invH));
               const F2 t = fma2(q, f2(-0.5f, -0.5f), f2(1.f, 1.f));
               const F2 w = mul2(mul2(mul2(mul2(mul2(f2(S.sigW, S.sigW), t), t), t), t),
                                 fma2(q, f2(2.f, 2.f), f2(1.f, 1.f)));
               const F2 vol = f2(d0.v.w, d1.v.w);
               const F2 ux = mul2(vol, f2(d0.v.x - vi.x, d1.v.x - vi.x));
               const F2 uy = mul2(vol, f2(d0.v.y - vi.y, d1.v.y - vi.y));
               const F2 uz = mul2(vol, f2(d0.v.z - vi.z, d1.v.z - vi.z));
               acc.x = __fmaf_rn(hi2(ux), hi2(w), __fmaf_rn(lo2(ux), lo2(w), acc.x));
               acc.y = __fmaf_rn(hi2(uy), hi2(w), __fmaf_rn(lo2(uy), lo2(w), acc.y));
               acc.z = __fmaf_rn(hi2(uz), hi2(w), __fmaf_rn(lo2(uz), lo2(w), acc.z));
             });
  acc = laneSum<G>(acc);
  if (G > 1 && lane != 0) return;
  float c = S.xsphC;
  if (iWater) c = S.xsphC * 10.f;
  const V3 v = vi + c * acc;
  velOut[i] = make_float4(v.x, v.y, v.z, vi4.w);
}

// ---------------------------------------------------------------- updateF + integrate
// Final F with return mapping (simkernels.js:510-525) fused with the CFL
// clamp and position update (simkernels.js:528-542). Outputs go to the
// "current" arrays, so neighbours still read the unclamped sorted inputs.
// The plastic update of F from the velocity gradient (simkernels.js:510-525):
// trial F, SVD, return map, the projected F. Compiled once, not inlined:
// the update kernel's sweep then keeps its registers (0.424 -> 0.401 ms per
// 4M-particle substep, the same bits).
__device__ __noinline__ M3 plasticUpdate(const SceneDev& S, const M3& gradV, const M3& F0, const MatDev& m, float st,
                                         float& stOut) {
  const M3 Htr = madd(minusIdent(F0), mscale(mul(gradV, F0), S.dt));
  V3 e;
  bool near;
  const SVD sv = strainSVD(Htr, e, near);
  const float hard = hardening(m, st);
  const Mapped mp = returnMap(sv.sig, e, m, m.mu * hard, m.lam * hard, st, S.dt, stOut);
  return withSigma(Htr, sv, safeSig(mp.sig), near);
}
template <int G>
__global__ void __launch_bounds__(kThreads, kMinUpdate) k_updateF_integrate(Bufs b, const float4* __restrict__ velIn) {
  // blocks run last to first: the pass starts where xsph ended, on
  // slots whose data is still in L2
  const uint32_t t = (gridDim.x - 1u - blockIdx.x) * blockDim.x + threadIdx.x;
  const uint32_t i = t / G, lane = t % G;
  if (i >= b.N) return;
  const ListHead head = listHead<G>(nbrGroups(b.nbr, i), b.nbrCount, i, lane);
  const Ctx cx = ctxOf(b, i);
  const SceneDev& S = *cx.scene;
  const float4 pi = b.posS[i];
  const uint32_t mi = matOfW(pi.w);
  const float4 vi4 = velIn[i];
  const bool iWater = waterW(pi.w);
  M3 A = mzero();
  if (!iWater) A = velocitySum<G>(b, cx, head, i, xyz(pi), xyz(vi4), velIn, lane);
  if (G > 1 && lane != 0) return;
  const float st = b.stateS[i];
  M3 Fn = loadM(b.FS, b.N, i);
  float stOut = st;
  if (!iWater)
    Fn = plasticUpdate(S, mul(A, transpose(loadM(b.L, b.N, i))), Fn, cx.mats[mi], st, stOut);
  storeM(b.F, b.N, i, Fn);
  b.state[i] = stOut;
  V3 v = xyz(vi4);
  const float vl = length(v);
  if (vl > S.vmaxCFL) v = v * (S.vmaxCFL / vl);
  b.vel[i] = make_float4(v.x, v.y, v.z, vi4.w);
  V3 x = xyz(pi) + S.dt * v;
  x = v3(clampf(x.x, S.dmin[0], S.dmax[0]), clampf(x.y, S.dmin[1], S.dmax[1]), clampf(x.z, S.dmin[2], S.dmax[2]));
  b.pos[i] = make_float4(x.x, x.y, x.z, fabsf(pi.w));
}

// ---------------------------------------------------------------- device loop
// Whether any scene still iterates at iteration k: not stopped by its
// residuals and below its iteration cap (one block; every thread returns it).
__device__ __forceinline__ bool anyIterating(const Bufs& b, int k) {
  bool run = false;
  for (uint32_t s = threadIdx.x; s < b.S; s += blockDim.x)
    run |= !b.done[s] && k < b.scenes[s].iterations;
  return __syncthreads_or(run) != 0;
}
__global__ void k_loop_begin(Bufs b, int k0, cudaGraphConditionalHandle h) {
  const bool run = anyIterating(b, k0);
  if (threadIdx.x == 0) {
    *b.kIter = k0;
    cudaGraphSetConditional(h, run ? 1u : 0u);
  }
}
__global__ void k_loop_next(Bufs b, cudaGraphConditionalHandle h) {
  const int k = *reinterpret_cast<volatile const int*>(b.kIter) + 1;
  const bool run = anyIterating(b, k);  // its barrier orders every read of kIter before the write
  if (threadIdx.x == 0) {
    *b.kIter = k;
    cudaGraphSetConditional(h, run ? 1u : 0u);
  }
}

// ---------------------------------------------------------------- plain re-solve
// The judge of an early-stopped solve: a scene that did not stop within its
// iteration cap (its residuals never reached the plain solve's tolerances)
// is re-solved with the reference solve from the substep's input. Marks
// those scenes and, inside a graph, sets the condition of the node whose
// body runs the re-solve (nothing runs when every scene stopped).
__global__ void k_judge(Bufs b, cudaGraphConditionalHandle h, int setCond) {
  bool any = false;
  for (uint32_t s = threadIdx.x; s < b.S; s += blockDim.x) {
    const bool fail = b.done[s] == 0 && b.scenes[s].residTol > 0.f && b.scenes[s].plainIterations > 0;
    b.rerun[s] = fail ? 1 : 0;
    any |= fail;
  }
  any = __syncthreads_or(any) != 0;
  if (threadIdx.x == 0 && setCond) cudaGraphSetConditional(h, any ? 1u : 0u);
}
// the re-solved scenes start again from the velocities entering iteration 0
__global__ void k_restore(Bufs b, float4* __restrict__ vel) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= b.N) return;
  const uint32_t s = b.S > 1 ? (uint32_t)b.sceneOf[i] : 0u;
  if (b.rerun[s]) vel[i] = b.vel0[i];
}
// The PBF pass's predicted positions x + dt v of every slot from the
// velocities as they stand: after an active-set iteration over worklists,
// the slots it did not visit and the ones the previous PBF pass moved hold
// older ones. The expression is solveB's when it writes them, so the
// result is the one the per-slot kernels leave.
__global__ void k_predict(Bufs b, const float4* __restrict__ vel) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= b.N) return;
  const SceneDev& S = *ctxOf(b, i).scene;
  const float4 pi = b.posS[i];
  const V3 xc = xyz(pi) + S.dt * xyz(vel[i]);
  storeXc(b, i, xc, pi.w, true);  // (from iteration 2 on)
}
__global__ void k_copy_vel(uint32_t n, const float4* __restrict__ src, float4* __restrict__ dst) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dst[i] = src[i];
}

// One scene's state in the reference layouts, staged in working buffers that
// the next substep rewrites: F in Sp, L in cons0 (12 floats a particle, a zero
// behind each column), aux in SpSelf, the permutation in tmp, the cell
// offsets in cursor, both relative to the scene. A read of the state is then
// one copy per array: it was 26 copies and the transposes on the host, 430 us
// for 10k particles.
__global__ void __launch_bounds__(256) k_stage_state(Bufs b, uint32_t first, uint32_t n, uint32_t firstCell,
                                                     uint32_t cells, uint32_t base, bool F, bool L, bool aux, bool idx,
                                                     bool tab, float volume) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (tab && t < cells) b.cursor[t] = b.cellStart[firstCell + t] - base;
  if (t >= n) return;
  const uint32_t i = first + t;
  auto columns = [&](const float* src, float4* dst) {
    const M3 m = loadM(src, b.N, i);
#pragma unroll
    for (int c = 0; c < 3; ++c) dst[3 * (size_t)t + c] = make_float4(m.c[c].x, m.c[c].y, m.c[c].z, 0.f);
  };
  if (F) columns(b.F, b.Sp);
  if (L) columns(b.L, b.cons0);
  if (aux)  // V^n is vel.w after a substep, V0 before the first
    b.SpSelf[t] = make_float4(volume >= 0.f ? volume : b.vel[i].w, b.lam[i], b.state[i], b.pbfLam[i]);
  if (idx) b.tmp[t] = b.sortedIdx[i] - base;
}

inline unsigned grid(uint32_t n) { return (unsigned)((n + kThreads - 1) / kThreads); }
inline unsigned gridOf(uint32_t n, int block) { return (unsigned)((n + (uint32_t)block - 1) / (uint32_t)block); }

}  // namespace

// The reference schedule's launches are chained (its flags are 0). Those of
// the learned solve stay plain: they follow memsets and conditional nodes or
// form the bodies of conditional nodes. So do those of the one-lane solve, on
// large handles, where a launch's gap does not count.
template <class... P, class... Q>
inline void launchIn(int flags, void (*fn)(P...), unsigned g, unsigned block, cudaStream_t st, Q... q) {
  if (flags == 0)
    launchChained(fn, g, block, 0, st, q...);
  else
    fn<<<g, block, 0, st>>>(q...);
}
void launch_computeL(const Bufs& b, bool features, int lanes, cudaStream_t st) {
  const unsigned g = grid((uint32_t)lanes * b.N);
  if (features) {
    if (lanes == 4) launchChained(k_computeL_features<4>, g, kThreads, 0, st, b);
    else if (lanes == 2) launchChained(k_computeL_features<2>, g, kThreads, 0, st, b);
    else launchChained(k_computeL_features<1>, g, kThreads, 0, st, b);
  } else {
    if (lanes == 4) launchChained(k_computeL<4>, g, kThreads, 0, st, b);
    else if (lanes == 2) launchChained(k_computeL<2>, g, kThreads, 0, st, b);
    else launchChained(k_computeL<1>, g, kThreads, 0, st, b);
  }
}
void launch_computeL_water(const Bufs& b, cudaStream_t st) { k_computeL_water<<<grid(b.N), kThreads, 0, st>>>(b); }
template <int V>
void solveAVariant(const Bufs& b, int k, const float4* velIn, int flags, cudaStream_t st) {
  constexpr int kBlock = kSolveABlock[V];
  if (flags & kTrackResid)
    k_solveA<true, kSolveAMinB[V], 1, kBlock><<<gridOf(b.N, kBlock), kBlock, 0, st>>>(b, k, velIn, flags);
  else
    k_solveA<false, kSolveAMinB[V], 1, kBlock><<<gridOf(b.N, kBlock), kBlock, 0, st>>>(b, k, velIn, flags);
}
void launch_solveA(const Bufs& b, int k, const float4* velIn, int flags, int variant, int lanes, cudaStream_t st) {
  if (flags & kStoredC) {  // iteration 0 after computeL with features (one lane per slot)
    if (flags & kTrackResid)
      k_solveA_stored<true><<<grid(b.N), kThreads, 0, st>>>(b, velIn, flags);
    else
      k_solveA_stored<false><<<grid(b.N), kThreads, 0, st>>>(b, velIn, flags);
    return;
  }
  if (lanes == 4) {  // small scenes: four lanes per slot, the allocator's register choice
    const uint32_t threads = 4u * b.N;
    if (flags & kTrackResid)
      launchIn(flags, k_solveA<true, 0, 4>, grid(threads), kThreads, st, b, k, velIn, flags);
    else
      launchIn(flags, k_solveA<false, 0, 4>, grid(threads), kThreads, st, b, k, velIn, flags);
    return;
  }
  if (lanes == 2) {
    const uint32_t threads = 2u * b.N;
    if (flags & kTrackResid)
      launchIn(flags, k_solveA<true, 0, 2>, grid(threads), kThreads, st, b, k, velIn, flags);
    else
      launchIn(flags, k_solveA<false, 0, 2>, grid(threads), kThreads, st, b, k, velIn, flags);
    return;
  }
  switch (variant) {
    case 1: solveAVariant<1>(b, k, velIn, flags, st); break;
    case 2: solveAVariant<2>(b, k, velIn, flags, st); break;
    case 3: solveAVariant<3>(b, k, velIn, flags, st); break;
    case 4: solveAVariant<4>(b, k, velIn, flags, st); break;
    case 5: solveAVariant<5>(b, k, velIn, flags, st); break;
    default: solveAVariant<0>(b, k, velIn, flags, st); break;
  }
}
void launch_warm_from_net(const Bufs& b, cudaStream_t st) { k_warm_from_net<<<grid(b.N), kThreads, 0, st>>>(b); }
void launch_warm_from_prev(const Bufs& b, cudaStream_t st) { k_warm_from_prev<<<grid(b.N), kThreads, 0, st>>>(b); }
void launch_resid_reduce(const Bufs& b, int k, bool warm, cudaStream_t st) {
  k_resid<<<dim3(residBlocks(b.maxSceneN), b.S), kResidThreads, 0, st>>>(b, k, warm ? 1 : 0);
}
void launch_keep_lambda(const Bufs& b, cudaStream_t st) { k_keep_lambda<<<grid(b.N), kThreads, 0, st>>>(b); }
template <int V>
void solveBVariant(const Bufs& b, int k, const float4* velIn, float4* velOut, int wx, int flags, cudaStream_t st) {
  constexpr int kBlock = kSolveBBlock[V];
  k_solveB<kSolveBMinB[V], 1, kBlock><<<gridOf(b.N, kBlock), kBlock, 0, st>>>(b, k, velIn, velOut, wx, flags);
}
// A grid that fills the GPU once with this kernel's resident blocks (the
// list launches loop over their lists).
inline unsigned fillGrid(const void* fn, int block) {
  int dev = 0, sms = 0, per = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, block, 0);
  return (unsigned)(std::max(1, sms) * std::max(1, per));
}
template <int V>
void solveBActiveVariant(const Bufs& b, int k, float4* vel, int wx, int flags, bool list, cudaStream_t st) {
  auto fn = k_solveB_active<kSolveBMinB[V], kSolveBBlock[V]>;
  const unsigned g = list ? fillGrid((const void*)fn, kSolveBBlock[V]) : gridOf(b.N, kSolveBBlock[V]);
  fn<<<g, kSolveBBlock[V], 0, st>>>(b, k, vel, wx, flags, list ? 1 : 0);
}
template <int V>
void solveAListVariant(const Bufs& b, int k, const float4* velIn, int flags, cudaStream_t st) {
  constexpr int minB = kSolveAMinB[V];
  auto fn = k_solveA_list<minB, kSolveABlock[V]>;
  fn<<<fillGrid((const void*)fn, kSolveABlock[V]), kSolveABlock[V], 0, st>>>(b, k, velIn, flags);
}
void launch_solveB(const Bufs& b, int k, const float4* velIn, float4* velOut, bool writeXc, int flags, int variant,
                   int lanes, cudaStream_t st) {
  const int wx = writeXc ? 1 : 0;
  if (flags & (kInPlace | kActive | kMarkMoved)) {  // the active set: in place, one lane per slot
    float4* vel = velOut;
    switch (variant) {
      case 1: solveBActiveVariant<1>(b, k, vel, wx, flags, false, st); break;
      case 2: solveBActiveVariant<2>(b, k, vel, wx, flags, false, st); break;
      case 3: solveBActiveVariant<3>(b, k, vel, wx, flags, false, st); break;
      case 4: solveBActiveVariant<4>(b, k, vel, wx, flags, false, st); break;
      default: solveBActiveVariant<0>(b, k, vel, wx, flags, false, st); break;
    }
    return;
  }
  if (lanes == 4) {
    launchIn(flags, k_solveB<0, 4>, grid(4u * b.N), kThreads, st, b, k, velIn, velOut, wx, flags);
    return;
  }
  if (lanes == 2) {
    launchIn(flags, k_solveB<0, 2>, grid(2u * b.N), kThreads, st, b, k, velIn, velOut, wx, flags);
    return;
  }
  switch (variant) {
    case 1: solveBVariant<1>(b, k, velIn, velOut, wx, flags, st); break;
    case 2: solveBVariant<2>(b, k, velIn, velOut, wx, flags, st); break;
    case 3: solveBVariant<3>(b, k, velIn, velOut, wx, flags, st); break;
    case 4: solveBVariant<4>(b, k, velIn, velOut, wx, flags, st); break;
    default: solveBVariant<0>(b, k, velIn, velOut, wx, flags, st); break;
  }
}
void launch_loop_begin(const Bufs& b, int k0, cudaGraphConditionalHandle h, cudaStream_t st) {
  k_loop_begin<<<1, 256, 0, st>>>(b, k0, h);
}
void launch_loop_next(const Bufs& b, cudaGraphConditionalHandle h, cudaStream_t st) {
  k_loop_next<<<1, 256, 0, st>>>(b, h);
}
void launch_compact(const Bufs& b, int k, int which, cudaStream_t st) {
  k_compact<<<gridOf((b.N + kCompactSlots - 1) / kCompactSlots, kCompactThreads), kCompactThreads, 0, st>>>(b, k,
                                                                                                       which);
}
void launch_solveA_list(const Bufs& b, int k, const float4* velIn, int flags, int variant, cudaStream_t st) {
  switch (variant) {
    case 1: solveAListVariant<1>(b, k, velIn, flags, st); break;
    case 2: solveAListVariant<2>(b, k, velIn, flags, st); break;
    case 3: solveAListVariant<3>(b, k, velIn, flags, st); break;
    case 4: solveAListVariant<4>(b, k, velIn, flags, st); break;
    case 5: solveAListVariant<5>(b, k, velIn, flags, st); break;
    default: solveAListVariant<0>(b, k, velIn, flags, st); break;
  }
}
void launch_solveB_list(const Bufs& b, int k, float4* vel, int flags, int variant, cudaStream_t st) {
  switch (variant) {
    case 1: solveBActiveVariant<1>(b, k, vel, 0, flags, true, st); break;
    case 2: solveBActiveVariant<2>(b, k, vel, 0, flags, true, st); break;
    case 3: solveBActiveVariant<3>(b, k, vel, 0, flags, true, st); break;
    case 4: solveBActiveVariant<4>(b, k, vel, 0, flags, true, st); break;
    default: solveBActiveVariant<0>(b, k, vel, 0, flags, true, st); break;
  }
}
void launch_pbfA(const Bufs& b, int k, int flags, int lanes, cudaStream_t st) {
  // predicted positions were stored by the preceding solveB
  const unsigned g = grid((uint32_t)lanes * b.N);
  if (lanes == 4) launchIn(flags, k_pbfA<4>, g, kThreads, st, b, k, flags);
  else if (lanes == 2) launchIn(flags, k_pbfA<2>, g, kThreads, st, b, k, flags);
  else launchIn(flags, k_pbfA<1>, g, kThreads, st, b, k, flags);
}
void launch_judge(const Bufs& b, cudaGraphConditionalHandle h, bool setCond, cudaStream_t st) {
  k_judge<<<1, 256, 0, st>>>(b, h, setCond ? 1 : 0);
}
void launch_stage_state(const Bufs& b, uint32_t first, uint32_t n, uint32_t firstCell, uint32_t cells, bool F, bool L,
                        bool aux, bool idx, bool tab, float volume, cudaStream_t st) {
  k_stage_state<<<gridOf(std::max(n, tab ? cells : 0u), 256), 256, 0, st>>>(
      b, first, n, firstCell, cells, n ? first : 0u, F, L, aux, idx, tab, volume);
}
void launch_restore(const Bufs& b, float4* vel, cudaStream_t st) { k_restore<<<grid(b.N), kThreads, 0, st>>>(b, vel); }
void launch_predict(const Bufs& b, const float4* vel, cudaStream_t st) {
  k_predict<<<grid(b.N), kThreads, 0, st>>>(b, vel);
}
void launch_copy_vel(const Bufs& b, const float4* src, float4* dst, cudaStream_t st) {
  k_copy_vel<<<grid(b.N), kThreads, 0, st>>>(b.N, src, dst);
}
void launch_pbfB(const Bufs& b, int k, const float4* velIn, float4* velOut, int flags, int lanes, cudaStream_t st) {
  const unsigned g = grid((uint32_t)lanes * b.N);
  if (lanes == 4) launchIn(flags, k_pbfB<4>, g, kThreads, st, b, k, velIn, velOut, flags);
  else if (lanes == 2) launchIn(flags, k_pbfB<2>, g, kThreads, st, b, k, velIn, velOut, flags);
  else launchIn(flags, k_pbfB<1>, g, kThreads, st, b, k, velIn, velOut, flags);
}
void launch_xsph(const Bufs& b, const float4* velIn, float4* velOut, int flags, int lanes, cudaStream_t st) {
  const unsigned g = grid((uint32_t)lanes * b.N);
  if (lanes == 4) launchIn(flags, k_xsph<4>, g, kThreads, st, b, velIn, velOut);
  else if (lanes == 2) launchIn(flags, k_xsph<2>, g, kThreads, st, b, velIn, velOut);
  else launchIn(flags, k_xsph<1>, g, kThreads, st, b, velIn, velOut);
}
void launch_updateF_integrate(const Bufs& b, const float4* velIn, int lanes, cudaStream_t st) {
  const unsigned g = grid((uint32_t)lanes * b.N);
  if (lanes == 4) k_updateF_integrate<4><<<g, kThreads, 0, st>>>(b, velIn);
  else if (lanes == 2) k_updateF_integrate<2><<<g, kThreads, 0, st>>>(b, velIn);
  else k_updateF_integrate<1><<<g, kThreads, 0, st>>>(b, velIn);
}

}  // namespace xpbi
