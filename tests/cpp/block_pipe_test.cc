// The block tiles' ring of stages over threads (one per warp) and barriers of memory that behave as mbarriers
// do, with a copy that never arrives or arrives too late for one of the warps. No GPU needed.
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

// A stage's barrier: a phase is complete when every issuer has arrived and all their copies have.
struct Stage {
  uint32_t tile = kNever;
  std::set<int> arrived;  // issuers of the phase that is not complete
  uint64_t phasesDone = 0;
};

struct Cta {
  std::mutex m;
  std::condition_variable changed;
  std::chrono::milliseconds limit{10000};  // of a wait
  std::vector<Stage> stages;
  uint32_t stuckTile = kNever;             // its copies never arrive
  uint32_t lateTile = kNever;              // its copies arrive after warp `lateWarp` has given up
  int lateWarp = -1;
  std::vector<std::vector<uint32_t>> sentFor{std::vector<std::vector<uint32_t>>(kWarps)};
  std::vector<std::vector<uint32_t>> taken{std::vector<std::vector<uint32_t>>(kWarps)};
  std::vector<bool> gaveUp = std::vector<bool>(kWarps, false);
  std::vector<std::string> violations;
  // the group's barrier
  int waiting = 0;
  uint64_t generation = 0;
};

struct Warp {
  Cta& cta;
  int id;

  void issue(uint32_t tile, uint32_t stage) {
    std::unique_lock<std::mutex> l(cta.m);
    if (cta.gaveUp[id]) cta.violations.push_back("tile " + std::to_string(tile) + " sent for after the failure");
    cta.sentFor[id].push_back(tile);
    if (id >= kIssuers) return;
    Stage& s = cta.stages[stage];
    if (!s.arrived.insert(id).second) cta.violations.push_back("stage " + std::to_string(stage) + " sent for twice");
    if (s.arrived.size() > 1 && s.tile != tile) cta.violations.push_back("two tiles in stage " + std::to_string(stage));
    s.tile = tile;
    if (static_cast<int>(s.arrived.size()) == kIssuers && tile != cta.stuckTile) {
      s.arrived.clear();
      ++s.phasesDone;
      cta.changed.notify_all();
    }
  }
  bool arrived(uint32_t stage, uint32_t parity) {
    std::unique_lock<std::mutex> l(cta.m);
    Stage& s = cta.stages[stage];
    auto filled = [&] { return (s.phasesDone & 1) != parity; };  // what mbarrier.try_wait.parity answers
    const bool late = id == cta.lateWarp && cta.taken[id].size() == cta.lateTile;
    if (cta.changed.wait_for(l, cta.limit, filled) && !late) return true;
    cta.gaveUp[id] = true;
    return false;
  }
  void take(uint32_t tile, uint32_t stage) {
    std::unique_lock<std::mutex> l(cta.m);
    if (cta.gaveUp[id]) cta.violations.push_back("a tile taken after the failure");
    if (cta.stages[stage].tile != tile) cta.violations.push_back("another tile in the stage than the one taken");
    cta.taken[id].push_back(tile);
  }
  void barrier() {
    std::unique_lock<std::mutex> l(cta.m);
    if (++cta.waiting == kWarps) {
      cta.waiting = 0;
      ++cta.generation;
      cta.changed.notify_all();
    } else {
      const uint64_t g = cta.generation;
      while (cta.generation == g) cta.changed.wait_for(l, std::chrono::milliseconds(20));
    }
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
      takeTiles(rings[w], tilesOfFirst + tilesOfSecond, tilesOfFirst, 1, ops);
    });
  for (auto& t : threads) t.join();
  return rings;
}

std::vector<uint32_t> upTo(uint32_t n) {
  std::vector<uint32_t> v(n);
  for (uint32_t i = 0; i < n; ++i) v[i] = i;
  return v;
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
        EXPECT_TRUE(cta.taken[w] == upTo(first + 5) && cta.sentFor[w] == upTo(first + 5));
      }
    }
}

// A copy that does not arrive, or not in time for one of the warps: everybody comes to an end, a warp that gave up
// neither sends for nor takes anything more, no stage is sent for twice, and every warp knows what it still has under way.
TPB_TEST(Plan, BlockTilesComeToAnEndWhenACopyDoesNotArrive) {
  constexpr uint32_t kAll = 5 + 6;
  for (uint32_t stages : {1u, 3u})
    for (uint32_t tile : {0u, 4u, 5u, 9u})
      for (int late : {-1, 1, 5}) {  // nobody sees it; one that sends for copies comes too late; one that does not
        Cta cta;
        cta.limit = std::chrono::milliseconds(150);
        if (late < 0) cta.stuckTile = tile;
        else cta.lateTile = tile, cta.lateWarp = late;
        const auto rings = runCta(cta, stages, 5, 6);
        if (!cta.violations.empty()) throw tpbtest::TestFailure(cta.violations[0]);
        for (int w = 0; w < kWarps; ++w) {
          EXPECT_TRUE(cta.taken[w] == upTo(rings[w].taken) && cta.sentFor[w] == upTo(rings[w].issued));
          EXPECT_EQ(rings[w].failed, rings[w].taken < kAll);
          EXPECT_TRUE(rings[w].taken >= tile);
          if (late < 0 || late == w) EXPECT_EQ(rings[w].taken, tile);
          if (late == 5 && w != 5) EXPECT_EQ(rings[w].taken, kAll);  // the others need nothing of it
          if (late == 1 && w != 1) EXPECT_TRUE(rings[w].taken >= std::min(kAll, tile + 1));
          // Before the memory is handed on, a warp waits for the tiles it sent for and did not see, stage by stage.
          std::vector<std::pair<uint32_t, uint32_t>> waits;
          waitForCopiesUnderWay(rings[w].taken, rings[w].issued, stages, [&](uint32_t s, uint32_t p) { waits.emplace_back(s, p); });
          EXPECT_EQ(waits.size(), size_t(rings[w].issued - rings[w].taken));
          EXPECT_TRUE(waits.size() <= stages);
          for (size_t i = 0; i < waits.size(); ++i) {
            const uint32_t t = rings[w].taken + static_cast<uint32_t>(i);
            EXPECT_TRUE(waits[i] == std::make_pair(t % stages, (t / stages) & 1));
          }
        }
      }
}
