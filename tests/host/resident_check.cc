// Several host threads ask for the resident blocks of the same kernels from
// cold: every answer is the one of its kernel, each kernel is queried once,
// and no thread enters the map while another one fills it (a query that dwells
// is alone).
#include <atomic>
#include <chrono>
#include <cstdio>
#include <thread>
#include <vector>

#include "mhc_resident.h"

int main() {
  constexpr int THREADS = 8, KERNELS = 64, ROUNDS = 200;
  static char kernels[KERNELS];
  mhc::ResidentBlocks blocks;
  std::atomic<int> asked{0}, wrong{0}, ready{0}, inside{0}, together{0};
  auto work = [&](int t) {
    ++ready;
    while (ready < THREADS) std::this_thread::yield();
    for (int r = 0; r < ROUNDS; ++r)
      for (int q = 0; q < KERNELS; ++q) {
        const int k = (q + 7 * t) % KERNELS, threads = k % 2 ? 128 : 256;
        const size_t smem = 1024 * (k % 3);
        const int got = blocks.get(kernels + k, threads, smem, [&] {
          ++asked;
          if (++inside > 1) ++together;
          std::this_thread::sleep_for(std::chrono::milliseconds(2));
          --inside;
          return 1 + k % 16;
        });
        if (got != 1 + k % 16) ++wrong;
      }
  };
  std::vector<std::thread> ts;
  for (int t = 0; t < THREADS; ++t) ts.emplace_back(work, t);
  for (auto& t : ts) t.join();
  std::printf("wrong %d together %d asked %d of %d\n", wrong.load(), together.load(), asked.load(), KERNELS);
  return wrong == 0 && together == 0 && asked == KERNELS ? 0 : 1;
}
