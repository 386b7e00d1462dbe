// Resident blocks per SM of the kernels, asked of the runtime once each.
#pragma once
#include <cstddef>
#include <map>
#include <mutex>
#include <tuple>

namespace mhc {

// The answers belong to the process (every device it runs on is the one the
// kernels are compiled for), and host threads that each drive their own case
// or batch ask for them with every launch list: one lock around the map.  A
// lookup takes about 20 ns, a launch some microseconds.
class ResidentBlocks {
  std::mutex mu;
  std::map<std::tuple<const void*, int, size_t>, int> known;

 public:
  // blocks per SM of `kernel` with so many threads and bytes of dynamic shared
  // memory; ask() queries them the first time
  template <class Ask>
  int get(const void* kernel, int threads, size_t smem, Ask ask) {
    const auto key = std::make_tuple(kernel, threads, smem);
    std::lock_guard<std::mutex> lock(mu);
    auto it = known.find(key);
    if (it == known.end()) it = known.emplace(key, ask()).first;
    return it->second;
  }
};

}  // namespace mhc
