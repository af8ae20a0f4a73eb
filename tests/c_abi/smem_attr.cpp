// raise_smem (csrc/smem_attr.cuh) against a function attribute that several threads raise at once, some to less than others: what is
// granted at the end covers the largest size, a refused size is not noted, and devices are apart.
// Built and run by tests/test_boundary.py::test_shared_memory_sizes_of_several_threads.
#include <atomic>
#include <chrono>
#include <cstdio>
#include <thread>
#include <vector>
#include "smem_attr.cuh"

int main() {
  for (int round = 0; round < 20; ++round) {
    prl::SmemAttr attr = {};
    std::atomic<int> granted[2] = {{0}, {0}}, asked[2] = {{0}, {0}}, failed{0};
    std::vector<std::thread> pool;
    for (int t = 0; t < 8; ++t)
      pool.emplace_back([&, t] {
        const int dev = t & 1, bytes = 64 * 1024 + 8 * 1024 * ((t + round) % 8);
        for (int most = asked[dev].load(); most < bytes && !asked[dev].compare_exchange_weak(most, bytes);) {}
        const int e = prl::raise_smem(attr, dev, bytes, [&](int b) {
          std::this_thread::sleep_for(std::chrono::microseconds(200 * (8 - b / 16384)));      // the smaller, the later
          granted[dev].store(b);
          return 0;
        });
        if (e || granted[dev].load() < bytes) ++failed;
      });
    for (auto& t : pool) t.join();
    for (int dev = 0; dev < 2; ++dev)
      if (granted[dev].load() < asked[dev].load()) ++failed;
    if (failed.load()) { printf("round %d: less is granted than was asked for\n", round); return 1; }
  }
  prl::SmemAttr attr = {};
  int calls = 0;
  auto refuse = [&](int) { ++calls; return 7; };
  if (prl::raise_smem(attr, 3, 100, refuse) != 7 || prl::raise_smem(attr, 3, 100, refuse) != 7 || calls != 2) { printf("a refused size was noted\n"); return 2; }
  printf("ok\n");
  return 0;
}
