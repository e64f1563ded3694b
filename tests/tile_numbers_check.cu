// Host-side check of the tiles' device point numbers (number_tiles): ranges of
// adjacent tiles, their alignment, and the refusal of a numbering that does
// not fit 32 bits.  Prints "ok" and exits 0, or prints what is wrong and exits 1.
#include <cstdio>
#include <string>
#include <vector>

#include "tiled_path.cuh"

using namespace insem_b200;

namespace {
int fail(const std::string& what) {
  std::printf("FAIL %s\n", what.c_str());
  return 1;
}

// The points of `tiles` tiles of `edge` edge points and of `halo` halo points, or -1 if refused.
long long stride_of(long long tiles, int edge, int ni, int halo) {
  try {
    return number_tiles(std::vector<int32_t>(tiles, edge), ni, halo).stride;
  } catch (const Error& e) {
    return e.code == INSEM_CUDA_ERR_UNSUPPORTED ? -1 : -2;
  }
}
}  // namespace

int main() {
  for (int ni = 0; ni <= 7; ++ni) {
    std::vector<int32_t> edge;
    for (int q = 0; q < 300; ++q) edge.push_back((q * 37) % 101);
    const TileNumbers t = number_tiles(edge, ni, 13);
    if (t.cbeg.size() != edge.size() + 1 || t.ebeg.size() != edge.size() || t.cbeg[0] != 0) return fail("sizes");
    for (std::size_t q = 0; q < edge.size(); ++q) {
      const std::string id = "ni " + std::to_string(ni) + " tile " + std::to_string(q);
      if (t.cbeg[q] % 32 || t.ebeg[q] % 32) return fail(id + ": range not on a multiple of 32 points");
      if (t.ebeg[q] != t.cbeg[q] + 32 * ni * ni) return fail(id + ": inner rows");
      const int gap = t.cbeg[q + 1] - t.ebeg[q] - edge[q];
      if (gap < 0 || gap > 31) return fail(id + ": edge range");
    }
    if (t.n_complete != t.cbeg.back() || t.stride % 4 || t.stride < t.n_complete + 13 || t.stride > t.n_complete + 16)
      return fail("totals of ni " + std::to_string(ni));
  }
  if (stride_of(0, 0, 3, 0) != 4) return fail("an empty domain has a stride of 4 points");
  // 2^31 - 1 is the last point number; a tile of 1 element at order 8 takes 32 x 49 + 32
  const long long per = 32 * 49 + 32, most = 2147483647LL / per;
  if (stride_of(most, 32, 7, 0) != most * per) return fail("the largest domain that fits was refused or miscounted");
  if (stride_of(most + 1, 32, 7, 0) != -1) return fail("tiles past 2^31 points were not refused");
  const int room = static_cast<int>(2147483647LL - most * per);
  if (stride_of(most, 32, 7, room / 4 * 4) != most * per + room / 4 * 4) return fail("halo points that fit");
  if (stride_of(most, 32, 7, room + 1) != -1) return fail("halo points past 2^31 were not refused");
  if (stride_of(3000000, 4, 7, 0) != -1) return fail("tiles far past 2^31 points were not refused");
  std::printf("ok\n");
  return 0;
}
