// Launches that chain kernels of one stream without a gap (programmatic
// dependent launch), and the clearing of the sort's counters.
//
// A substep is 20 to 100 dependent kernels; on a scene of some ten thousand
// particles each runs for a few microseconds, and draining one grid before
// the next is launched costs about one more. A chained kernel's launch is
// prepared while its predecessor runs; its blocks wait in afterPrevious()
// until the predecessor has completed and its writes are visible. Every
// chained kernel calls it before its first access to memory, so order and
// results are those of plain launches.
//
// The sort's kernels, a few microseconds each, also let the next one's blocks
// take their places early: the sort of 250k keys takes 21 us instead of 45
// (that and one clearing kernel instead of three memsets). The solver's
// kernels must not: blocks that take whatever places come free end up
// unevenly spread over the SMs (16k solids 209 -> 245 us a substep, 113k
// solids 960 -> 1301). Chained without that, 16k solids go from 209 to 204 us.
#pragma once
#include <cuda_runtime.h>

#include <utility>

#include "xpbi_internal.h"

namespace xpbi {

// Waits for the preceding kernel. Returns its argument: an index taken
// through here keeps the loads it addresses behind the wait, if they are
// ordinary loads. Read-only-cache loads (__ldg, and any load through a kernel
// parameter that is const and __restrict__) are not memory operations to the
// assembler's scheduler and do move above the wait (seen in the training
// step's weights): in a chained kernel only addresses formed from data
// loaded behind the wait may be read that way.
__device__ __forceinline__ uint32_t afterPrevious(uint32_t t) {
  asm volatile("griddepcontrol.wait;" : "+r"(t) : : "memory");
  return t;
}
// The same, and the next chained kernel's blocks may take free places (where
// they wait in turn).
__device__ __forceinline__ uint32_t afterPreviousEager(uint32_t t) {
  asm volatile("griddepcontrol.wait;\n\tgriddepcontrol.launch_dependents;" : "+r"(t) : : "memory");
  return t;
}

// Launches fn (which calls afterPrevious) chained to the stream's last kernel.
template <class... P, class... Q>
inline void launchChained(void (*fn)(P...), dim3 grid, unsigned block, size_t smem, cudaStream_t st, Q&&... q) {
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c = {};
  c.gridDim = grid;
  c.blockDim = dim3(block);
  c.dynamicSmemBytes = smem;
  c.stream = st;
  c.attrs = &at;
  c.numAttrs = 1;
  cudaLaunchKernelEx(&c, fn, std::forward<Q>(q)...);
}

// A particle's place in its cell's bucket is the number of members with a
// larger index. Up to crowdLimit members, tmp[s0, s1) is counted through:
// O(L) a member, four members a load where it pays. In a crowded cell (a
// collapsed scene, or one whose positions are all NaN, which the grid clamps
// into its first cell) that would be quadratic in the scene. There the fill
// has counted the cell's members per segment of 8192 consecutive particles:
// those of the later segments are added up, and only the rest of the
// particle's own segment is looked through, by its keys.
// (Everything in one cell, the reorder: 250k particles 0.24 ms against 16.2 of
// comparing all with all, 1M 0.71 against 163, 4M 2.6. The sort of 250k spread
// particles takes 20.5 us with and without.)
__device__ __forceinline__ bool crowded(uint32_t n, uint32_t s0, uint32_t s1) {
  return s1 > s0 && s1 - s0 > crowdLimit(n);
}
// the counts of the crowded cell that starts at s0 (they start more than crowdLimit apart)
__device__ __forceinline__ uint32_t* crowdRow(uint32_t* crowd, uint32_t n, uint32_t s0) {
  return crowd + (size_t)(s0 / crowdLimit(n)) * crowdSegments(n);
}
__device__ __forceinline__ uint32_t rankInCrowd(const uint32_t* key, const uint32_t* row, uint32_t n, uint32_t i) {
  const uint32_t c = key[i], seg = i / kCrowdSegment;
  uint32_t rank = 0, j = i + 1u;
#pragma unroll 4
  for (uint32_t q = seg + 1u; q < crowdSegments(n); ++q) rank += row[q];
  const uint32_t end = min(n, (seg + 1u) * kCrowdSegment);
  for (; j < end && (j & 3u); ++j) rank += key[j] == c ? 1u : 0u;
#pragma unroll 4
  for (; j + 4u <= end; j += 4u) {
    const uint4 m = *reinterpret_cast<const uint4*>(key + j);
    rank += (m.x == c ? 1u : 0u) + (m.y == c ? 1u : 0u) + (m.z == c ? 1u : 0u) + (m.w == c ? 1u : 0u);
  }
  for (; j < end; ++j) rank += key[j] == c ? 1u : 0u;
  return rank;
}
__device__ __forceinline__ uint32_t rankInBucket(const uint32_t* tmp, const uint32_t* key, uint32_t* crowd, uint32_t n,
                                                 uint32_t s0, uint32_t s1, uint32_t i) {
  // (the bound only matters after an expired look-back, whose starts are wrong)
  if (crowded(n, s0, s1)) return min(rankInCrowd(key, crowdRow(crowd, n, s0), n, i), s1 - s0 - 1u);
  uint32_t rank = 0, q = s0;
  if (s1 - s0 > 32u) {
    for (; q & 3u; ++q) rank += tmp[q] > i ? 1u : 0u;
#pragma unroll 4
    for (; q + 4u <= s1; q += 4u) {
      const uint4 m = *reinterpret_cast<const uint4*>(tmp + q);
      rank += (m.x > i ? 1u : 0u) + (m.y > i ? 1u : 0u) + (m.z > i ? 1u : 0u) + (m.w > i ? 1u : 0u);
    }
  }
  for (; q < s1; ++q) rank += tmp[q] > i ? 1u : 0u;
  return min(rank, s1 - s0 - 1u);
}

// Thread t's share of clearing what a sort starts from: cell counters, water
// flags and the scan's control block, in whole 16-byte groups (the buffers
// are padded to them). sortClearThreads() threads clear all of it.
__device__ __forceinline__ void sortClear(const Bufs& b, uint32_t t) {
  const uint4 z = make_uint4(0u, 0u, 0u, 0u);
  if (t < (b.C + 3u) / 4u) reinterpret_cast<uint4*>(b.cursor)[t] = z;
  if (t < (b.C + 15u) / 16u) reinterpret_cast<uint4*>(b.cellWater)[t] = z;
  if (t <= b.scanTiles) reinterpret_cast<unsigned long long*>(b.tileTicket)[t] = 0ull;
}
inline uint32_t sortClearThreads(const Bufs& b) {
  const uint32_t groups = (b.C + 3u) / 4u;
  return groups > b.scanTiles + 1u ? groups : b.scanTiles + 1u;
}

}  // namespace xpbi
