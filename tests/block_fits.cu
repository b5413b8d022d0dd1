// What a block of a batched launch takes into its shared memory
// (team_sync.cuh), at slot counts whose bytes pass 2^31; on the host.
#include <cstdint>
#include <cstdio>

#include "team_sync.cuh"

int main() {
  using namespace sfr;
  const int left = 231000;
  for (int slots : {0, 6080, 23100, 214748365, 300000000, 429496730, 2147483616}) {
    const bool f10 = block_fits(32, 40, slots, 10, left), f12 = block_fits(32, 40, slots, 12, left);
    Carve a{nullptr, left}, b{nullptr, left};
    a.at = b.at = reinterpret_cast<char *>(64);
    const bool c = a.take<int16_t>(slots) != nullptr, v = b.take<float>(slots) != nullptr;
    std::printf("%d %d %d %d %d %d %d\n", slots, f10, f12, c, v, a.left, b.left);
  }
  return 0;
}
