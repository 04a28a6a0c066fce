// window_emu with the probe as the library's default runs it: joins and
// lookups as separate work of the same warps (test infrastructure).  With
// SPLIT_FEW only an eighth of the warps join, which makes them take packed
// 128-op spans.
#include "simt_host.h"
#include "lsb_window.cuh"

namespace lsb {
template <class Tr, bool kGroup, int P, class... Rest>
void phase_probe_split(const TableView& t, const Scratch& sc, const Window<Tr>& w, uint32_t warp,
                       uint32_t nwarps, Rest...) {
  static uint8_t slices[32][kJoinSpan];
#ifdef SPLIT_FEW
  const uint32_t joining = nwarps < 8 ? 1u : nwarps / 8;
#else
  const uint32_t joining = nwarps;
#endif
  const uint32_t lane = threadIdx.x & 31u, back = nwarps - 1 - warp;
  if (back < joining) phase_join<Tr>(sc, w, back, joining, slices[threadIdx.x >> 5]);
  phase_lookup<Tr>(t, sc, w, warp * 32 + lane, nwarps * 32);
}
}  // namespace lsb

#define phase_probe phase_probe_split
#include "window_emu.cpp"
