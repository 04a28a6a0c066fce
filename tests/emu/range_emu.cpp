// order_emu that also counts, block by block, the member and list words that
// the ordering step loads (test infrastructure): prints the largest count of
// any block after the check's own line.
#include "simt_host.h"
#include "lsb_core.cuh"

#include <atomic>

namespace lsb {
inline std::atomic<uint64_t> g_loads[64];
inline uint32_t counted_ld_cg_u32(const void* p) {
  g_loads[blockIdx.x & 63u].fetch_add(1, std::memory_order_relaxed);
  return ld_cg_u32(p);
}
inline uint4 counted_ld_cg_v4(const void* p) {
  g_loads[blockIdx.x & 63u].fetch_add(4, std::memory_order_relaxed);
  return ld_cg_v4(p);
}
}  // namespace lsb

#define ld_cg_u32 counted_ld_cg_u32
#define ld_cg_v4 counted_ld_cg_v4
#define main order_main
#include "order_emu.cpp"
#undef main

int main(int argc, char** argv) {
  const int rc = order_main(argc, argv);
  uint64_t most = 0;
  for (auto& c : g_loads) most = std::max<uint64_t>(most, c.load());
  std::printf("MOST %llu\n", (unsigned long long)most);
  return rc;
}
