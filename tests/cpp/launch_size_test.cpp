// Launch sizes at and around the largest grid, for tiles below, at and above
// a limb.
#include <cstdio>

#include "launch_size.h"

using namespace yell_gb300;

#define CHECK(x) \
  if (!(x)) return std::printf("failed: %s\n", #x), 1

int main() {
  CHECK(tile_ctas(1, 6, 12) == 1 && tile_ctas(64, 6, 12) == 1 && tile_ctas(65, 6, 12) == 2);
  CHECK(tile_ctas(3, 14, 8) == 192);
  // 2^14 in tiles of 2^8: 2^6 CTAs per limb, whose 32-bit product wraps from 2^26 limbs up
  CHECK(one_launch((1u << 25) - 1, 14, 8));
  CHECK(!one_launch(1u << 25, 14, 8));
  CHECK(!one_launch((1u << 26) + 1, 14, 8));  // 64 CTAs if it wrapped
  // 2^20 in tiles of 2^11, and in tiles of 2^12 as many limbs as calls accept
  CHECK(one_launch((1u << 22) - 1, 20, 11) && !one_launch(1u << 22, 20, 11));
  CHECK(one_launch((1u << 23) - 1, 20, 12));
  // one limb per CTA
  CHECK(one_launch((1u << 31) - 1, 7, 7) && !one_launch(1u << 31, 7, 7) && !one_launch(~0u, 3, 3));
  std::printf("OK\n");
  return 0;
}
