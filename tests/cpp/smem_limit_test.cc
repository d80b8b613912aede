// The shared-memory limit of a kernel when several threads raise it at once (no GPU needed: the driver is a
// variable that keeps the last value it was given).
#include <atomic>
#include <chrono>
#include <stdexcept>
#include <thread>
#include <vector>

#include "kernels/smem_limit.h"
#include "test_util.h"

using namespace tpb::kernels;

TPB_TEST(Plan, ASmallerSharedMemoryLimitNeverReplacesALargerOne) {
  // The larger request sits inside its driver call until the smaller one has made its own, or has had time to.
  SmemLimit limit;
  std::atomic<size_t> driver{0};
  std::atomic<bool> inside{false}, smallDone{false};
  std::thread large([&] {
    limit.raise(0, 104472, [&](size_t bytes) {
      driver = bytes;
      inside = true;
      for (int i = 0; i < 300 && !smallDone; ++i) std::this_thread::sleep_for(std::chrono::milliseconds(1));
    });
  });
  std::thread small([&] {
    while (!inside) std::this_thread::yield();
    limit.raise(0, 67584, [&](size_t bytes) { driver = bytes; });
    smallDone = true;
  });
  large.join();
  small.join();
  limit.raise(0, 104472, [&](size_t bytes) { driver = bytes; });  // the next launch of that size
  EXPECT_TRUE(driver >= size_t(104472));
}

TPB_TEST(Plan, EveryThreadFindsTheSharedMemoryItAskedFor) {
  for (int round = 0; round < 50; ++round) {
    SmemLimit limit;
    std::atomic<size_t> driver[2] = {};
    std::atomic<int> refused{0};
    std::vector<std::thread> threads;
    for (int t = 0; t < 8; ++t)
      threads.emplace_back([&, t] {
        for (int i = 0; i < 50; ++i) {
          const int device = i & 1;
          const size_t bytes = 50000 + static_cast<size_t>((t * 7919 + i * 104729 + round) % 60000);
          limit.raise(device, bytes, [&](size_t most) {
            std::this_thread::sleep_for(std::chrono::microseconds(most % 50));  // the calls overlap
            driver[device] = most;
          });
          if (driver[device] < bytes) ++refused;
        }
      });
    for (auto& t : threads) t.join();
    EXPECT_EQ(refused.load(), 0);
  }
}

TPB_TEST(Plan, AFailedLimitIsNotRemembered) {
  SmemLimit limit;
  bool threw = false;
  try {
    limit.raise(3, 1000, [](size_t) { throw std::runtime_error("refused"); });
  } catch (const std::runtime_error&) {
    threw = true;
  }
  EXPECT_TRUE(threw);
  int calls = 0;
  limit.raise(3, 1000, [&](size_t) { ++calls; });
  limit.raise(3, 999, [&](size_t) { ++calls; });
  EXPECT_EQ(calls, 1);
}
