// SmemLimit against a stand-in for the runtime's per-device kernel attribute: what a thread asked for is allowed at its launch,
// on its device, whatever other threads and devices ask for meanwhile.
#include <atomic>
#include <cstdio>
#include <thread>
#include <vector>

#include "../camelid_b200/csrc/smem_limit.h"

int main() {
  int bad = 0;
  {
    cmld::SmemLimit limit;
    int attr[3] = {0, 0, 0}, calls = 0;
    auto ask = [&](int dev, int bytes) { return limit.raise(dev, bytes, [&](int n) { ++calls; attr[dev] = n; return 0; }); };
    ask(0, 100), ask(1, 100), ask(0, 50), ask(0, 200), ask(2, 70), ask(1, 100);
    bad += attr[0] != 200 || attr[1] != 100 || attr[2] != 70 || calls != 4;
    bad += limit.raise(0, 300, [](int) { return 7; }) != 7;  // a failure is reported and not remembered
    ask(0, 300);
    bad += attr[0] != 300;
  }
  std::atomic<int> short_launches{0};
  for (int round = 0; round < 200; ++round) {
    cmld::SmemLimit limit;
    std::atomic<int> attr[2] = {{0}, {0}};
    std::vector<std::thread> threads;
    for (int t = 0; t < 8; ++t)
      threads.emplace_back([&, t] {
        for (int i = 0; i < 50; ++i) {
          const int dev = (t + i) & 1, bytes = 1 + (t * 37 + i * 101) % 1000;
          limit.raise(dev, bytes, [&](int n) { attr[dev] = n; return 0; });
          if (attr[dev] < bytes) ++short_launches;
        }
      });
    for (auto &t : threads) t.join();
  }
  bad += short_launches != 0;
  std::printf("%d failures, %d launches above their limit\n", bad, short_launches.load());
  return bad != 0;
}
