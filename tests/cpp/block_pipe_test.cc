// The block tiles' ring of stages over threads (one per warp) and barriers of memory that behave as mbarriers
// do, with a copy that never arrives or arrives too late for some of the warps. No GPU needed.
#include <condition_variable>
#include <mutex>
#include <set>
#include <thread>
#include <vector>

#include "kernels/block_pipe.h"
#include "test_util.h"

using namespace tpb::kernels;

namespace {

constexpr int kWarps = 8, kIssuers = 4;  // half of the warps send for the copies
constexpr uint32_t kNever = ~0u;

// A stage's barrier: `arrivals` of kIssuers and one copy complete a phase.
struct Stage {
  uint32_t tile = 0;
  int arrivals = 0;
  uint64_t phasesDone = 0;
};

struct Cta {
  std::mutex m;
  std::condition_variable changed;
  std::vector<Stage> stages;
  uint32_t stuckTile = kNever;       // its copy never arrives
  uint32_t lateTile = kNever;        // its copy arrives, but warp `lateWarp` has given up by then
  int lateWarp = -1;
  std::set<uint32_t> sentFor;
  std::vector<std::set<uint32_t>> taken{std::vector<std::set<uint32_t>>(kWarps)};
  std::vector<std::string> violations;
  bool gaveUp = false;               // some warp's wait ran out
  bool left = false;                 // the barrier told everybody
  // the group's barrier
  int waiting = 0;
  uint64_t generation = 0;
  bool bad = false, result = false;
};

struct Warp {
  Cta& cta;
  int id;

  void issue(uint32_t tile, uint32_t stage) {
    if (id >= kIssuers) return;
    std::unique_lock<std::mutex> l(cta.m);
    Stage& s = cta.stages[stage];
    if (cta.left) cta.violations.push_back("tile " + std::to_string(tile) + " sent for after the failure");
    if (s.arrivals == kIssuers) cta.violations.push_back("an arrival beyond what the phase of stage " + std::to_string(stage) + " takes");
    s.tile = tile;
    cta.sentFor.insert(tile);
    if (++s.arrivals == kIssuers && tile != cta.stuckTile) {
      s.arrivals = 0;
      ++s.phasesDone;
      cta.changed.notify_all();
    }
  }
  bool arrived(uint32_t stage, uint32_t parity) {
    std::unique_lock<std::mutex> l(cta.m);
    Stage& s = cta.stages[stage];
    auto filled = [&] { return (s.phasesDone & 1) != parity; };  // what mbarrier.try_wait.parity answers
    auto stuck = [&] { return s.arrivals == kIssuers && s.tile == cta.stuckTile; };
    cta.changed.wait_for(l, std::chrono::milliseconds(20), [&] { return filled() || stuck(); });
    while (!filled() && !stuck()) cta.changed.wait_for(l, std::chrono::milliseconds(20));
    if (filled() && !(s.tile == cta.lateTile && id == cta.lateWarp)) return true;
    cta.gaveUp = true;
    return false;
  }
  void take(uint32_t tile, uint32_t) {
    std::unique_lock<std::mutex> l(cta.m);
    if (cta.left) cta.violations.push_back("a tile taken after the failure");
    cta.taken[id].insert(tile);
  }
  bool anyone(bool bad) {
    std::unique_lock<std::mutex> l(cta.m);
    cta.bad |= bad;
    if (++cta.waiting == kWarps) {
      cta.waiting = 0;
      cta.result = cta.bad;
      cta.left |= cta.bad;
      cta.bad = false;
      ++cta.generation;
      cta.changed.notify_all();
    } else {
      const uint64_t g = cta.generation;
      while (cta.generation == g) cta.changed.wait_for(l, std::chrono::milliseconds(20));
    }
    return cta.result;
  }
};

// Two entries one behind the other, as a launch with two transposed matrices has them.
std::vector<TileRing> runCta(Cta& cta, uint32_t stages, uint32_t tilesOfFirst, uint32_t tilesOfSecond) {
  cta.stages.resize(stages);
  std::vector<TileRing> rings(kWarps, TileRing{stages, 0, 0, false});
  std::vector<std::thread> threads;
  for (int w = 0; w < kWarps; ++w)
    threads.emplace_back([&, w] {
      Warp ops{cta, w};
      takeTiles(rings[w], tilesOfFirst, 0, 1, ops);
      if (!rings[w].failed) takeTiles(rings[w], tilesOfFirst + tilesOfSecond, tilesOfFirst, 1, ops);
    });
  for (auto& t : threads) t.join();
  return rings;
}

}  // namespace

TPB_TEST(Plan, BlockTilesAreAllTakenOnceEach) {
  for (uint32_t stages : {1u, 2u, 3u})
    for (uint32_t first : {0u, 1u, 2u, 3u, 7u}) {
      Cta cta;
      const auto rings = runCta(cta, stages, first, 5);
      EXPECT_EQ(cta.violations.size(), size_t(0));
      for (int w = 0; w < kWarps; ++w) {
        EXPECT_TRUE(!rings[w].failed);
        EXPECT_EQ(rings[w].taken, first + 5);
        EXPECT_EQ(rings[w].issued, first + 5);
        EXPECT_EQ(cta.taken[w].size(), size_t(first + 5));
      }
    }
}

// A copy that does not arrive, or not in time for one of the warps: everybody leaves at that tile, nothing is sent
// for any more, no barrier is arrived on twice, and the copies under way are known.
TPB_TEST(Plan, BlockTilesStopForEverybodyAtACopyThatDoesNotArrive) {
  for (uint32_t stages : {1u, 3u})
    for (uint32_t tile : {0u, 1u, 4u, 5u, 8u})
      for (int late = 0; late < 2; ++late) {
        Cta cta;
        if (late) cta.lateTile = tile, cta.lateWarp = 5;
        else cta.stuckTile = tile;
        const auto rings = runCta(cta, stages, 5, 6);
        EXPECT_EQ(cta.violations.size(), size_t(0));
        EXPECT_TRUE(cta.gaveUp);
        for (int w = 0; w < kWarps; ++w) {
          EXPECT_TRUE(rings[w].failed);
          EXPECT_EQ(rings[w].taken, tile);
          EXPECT_EQ(rings[w].issued, rings[0].issued);
          const bool saw = late && w != 5;
          EXPECT_EQ(cta.taken[w].size(), size_t(tile + (saw ? 1 : 0)));
        }
        // Whoever hands the memory on waits for the tiles that were sent for and not taken, stage by stage.
        std::vector<std::pair<uint32_t, uint32_t>> waits;
        waitForCopiesUnderWay(rings[0].taken, rings[0].issued, stages, [&](uint32_t s, uint32_t p) { waits.emplace_back(s, p); });
        EXPECT_EQ(waits.size(), cta.sentFor.size() - tile);
        EXPECT_EQ(waits.size(), size_t(rings[0].issued - tile));
        EXPECT_TRUE(waits.size() <= stages);
        for (size_t i = 0; i < waits.size(); ++i) {
          EXPECT_EQ(waits[i].first, (tile + uint32_t(i)) % stages);
          EXPECT_EQ(waits[i].second, ((tile + uint32_t(i)) / stages) & 1);
        }
      }
}
