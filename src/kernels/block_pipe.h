// The order of steps in which the threads of a CTA take tiles through a ring of stages that asynchronous copies
// fill. The kernel runs it over mbarriers and bulk copies (push.cu), the tests over threads and a copy
// that never arrives (tests/cpp/block_pipe_test.cc).
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define TPB_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define TPB_HOST_DEVICE inline
#endif

namespace tpb {
namespace kernels {

// Tiles sent for and tiles taken so far, over all entries of a launch; the same in every thread.
struct TileRing {
  uint32_t stages;
  uint32_t issued, taken;
  bool failed;

  TPB_HOST_DEVICE static uint32_t stageOf(uint32_t tile, uint32_t stages) { return tile % stages; }
  TPB_HOST_DEVICE static uint32_t parityOf(uint32_t tile, uint32_t stages) { return (tile / stages) & 1; }
};

// Tiles first, first + step, ... below numTiles. Every thread of the group calls it with the same arguments and an
// `ops` of its own:
//   issue(tile, stage)            sends for a tile
//   arrived(stage, parity)        waits, within a limit, until the stage is filled; the same answer in all
//                                 threads of a warp, but not necessarily in all warps
//   take(tile, stage)             uses a filled stage
//   anyone(bad)                   a barrier of the whole group that tells whether anybody came with `bad`
// A copy that does not arrive in time ends it for everybody at the same tile, with `failed` set: nothing more
// is sent for, and what is still under way (tiles taken .. issued - 1) is for the caller to wait for.
template <typename Ops>
TPB_HOST_DEVICE void takeTiles(TileRing& ring, uint32_t numTiles, uint32_t first, uint32_t step, Ops& ops) {
  uint32_t ahead = first;  // next tile to send for
  for (uint32_t s = 0; s < ring.stages && ahead < numTiles; ++s, ahead += step)
    ops.issue(ahead, TileRing::stageOf(ring.issued++, ring.stages));
#ifdef __CUDA_ARCH__
#pragma unroll 1
#endif
  for (uint32_t t = first; t < numTiles; t += step) {
    const uint32_t stage = TileRing::stageOf(ring.taken, ring.stages);
    const bool arrived = ops.arrived(stage, TileRing::parityOf(ring.taken, ring.stages));
    if (arrived) ops.take(t, stage);
    if (ops.anyone(!arrived)) {  // everybody is through with this stage
      ring.failed = true;
      return;
    }
    ++ring.taken;
    if (ahead < numTiles) {
      ops.issue(ahead, TileRing::stageOf(ring.issued++, ring.stages));
      ahead += step;
    }
  }
}

// After a failure: waits (wait(stage, parity), bounded) for every copy that is still under way, so that
// none lands in memory that has another use by then.
template <typename Wait>
TPB_HOST_DEVICE void waitForCopiesUnderWay(uint32_t taken, uint32_t issued, uint32_t stages, Wait&& wait) {
  for (uint32_t tile = taken; tile != issued; ++tile) wait(TileRing::stageOf(tile, stages), TileRing::parityOf(tile, stages));
}

}  // namespace kernels
}  // namespace tpb
