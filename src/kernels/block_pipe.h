// The order of steps in which the threads of a CTA take tiles through a ring of stages that asynchronous copies
// fill, and what happens when a copy does not arrive. The tests run it over threads and a copy that never
// arrives (tests/cpp/block_pipe_test.cc); the kernel's loop (BlockTransposer::run) goes through the same steps over mbarriers
// and bulk copies.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define TPB_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define TPB_HOST_DEVICE inline
#endif

namespace tpb {
namespace kernels {

// How far a warp has got, over all entries of a launch: tiles it has sent for and tiles it has seen arrive.
struct TileRing {
  uint32_t stages;
  uint32_t issued, taken;
  bool failed;  // a wait of this warp ran out

  TPB_HOST_DEVICE static uint32_t stageOf(uint32_t tile, uint32_t stages) { return tile % stages; }
  TPB_HOST_DEVICE static uint32_t parityOf(uint32_t tile, uint32_t stages) { return (tile / stages) & 1; }
};

// Tiles first, first + step, ... below numTiles. Every thread of the group calls it with the same arguments and an
// `ops` of its own:
//   issue(tile, stage)            sends for this thread's part of a tile
//   arrived(stage, parity)        waits, within a limit, until the stage is filled; the same answer in all
//                                 threads of a warp, but not necessarily in all warps
//   take(tile, stage)             uses a filled stage
//   barrier()                     a barrier of the whole group
// A warp whose wait runs out sends for nothing more and takes nothing more, but comes to every barrier: nobody is left
// waiting for it, and as it adds nothing to a stage that it has not seen filled, no stage is sent for twice. Warps
// that go on meet stages that are never filled and run out in turn. Whether anybody failed is settled once,
// behind the last entry. (A barrier per tile that tells everybody cost 1 to 3 % of the kernel.)
template <typename Ops>
TPB_HOST_DEVICE void takeTiles(TileRing& ring, uint32_t numTiles, uint32_t first, uint32_t step, Ops& ops) {
  uint32_t ahead = first;  // next tile to send for
  for (uint32_t s = 0; s < ring.stages && ahead < numTiles; ++s, ahead += step)
    if (!ring.failed) ops.issue(ahead, TileRing::stageOf(ring.issued++, ring.stages));
#ifdef __CUDA_ARCH__
#pragma unroll 1
#endif
  for (uint32_t t = first; t < numTiles; t += step) {
    const uint32_t stage = TileRing::stageOf(ring.taken, ring.stages);
    if (!ring.failed) ring.failed = !ops.arrived(stage, TileRing::parityOf(ring.taken, ring.stages));
    if (!ring.failed) {
      ++ring.taken;
      ops.take(t, stage);
    }
    ops.barrier();  // everybody is through with this stage
    if (ahead < numTiles) {
      if (!ring.failed) ops.issue(ahead, TileRing::stageOf(ring.issued++, ring.stages));
      ahead += step;
    }
  }
}

// After a failure: waits (wait(stage, parity), bounded) for every copy that the caller sent for and did not see
// arrive, so that none lands in memory that has another use by then.
template <typename Wait>
TPB_HOST_DEVICE void waitForCopiesUnderWay(uint32_t taken, uint32_t issued, uint32_t stages, Wait&& wait) {
  for (uint32_t tile = taken; tile != issued; ++tile) wait(TileRing::stageOf(tile, stages), TileRing::parityOf(tile, stages));
}

}  // namespace kernels
}  // namespace tpb
