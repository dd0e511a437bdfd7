// Instantiations and shared-memory layout of the streaming form (dmm_stream.cuh).
#include <algorithm>

#include "dmm_stream.cuh"

namespace dmm {

const void* stream_kernel(bool general) {
  return general ? (const void*)k_stream<true> : (const void*)k_stream<false>;
}

StreamLayout stream_shape(int dl, int st, int bk, int tv) {
  constexpr int T = 4;
  auto al = [](int x) { return (x + 15) & ~15; };
  StreamLayout L{};
  L.v0 = 0;
  L.v1 = al(T * dl);
  L.stage = L.v1 + al(T * dl);
  const int a = L.stage + al(T * st);
  L.b0 = 0;
  L.b1 = 16 + al(T * bk);
  const int bend = L.b1 + 16 + al(T * bk);
  L.total = std::max(std::max(a, bend), al(T * tv));
  return L;
}

}  // namespace dmm
