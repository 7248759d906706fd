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

// Number of members of the bucket tmp[s0, s1) with a larger index than i: i's
// place in it. Counting is O(L) a member whatever the bucket's size L; four
// members a load where it pays (9,000 in one cell take 20 us more).
__device__ __forceinline__ uint32_t rankInBucket(const uint32_t* tmp, uint32_t s0, uint32_t s1, uint32_t i) {
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
  return rank;
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
