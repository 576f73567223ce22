// Launch sizes of the tiled kernels (host only).
#pragma once
#include <cstdint>

namespace yell_gb300 {

// CTAs of a launch over `limbs` limbs of 2^log_n words with 2^tile_log words
// per CTA (several limbs, or a part of one).
constexpr uint64_t tile_ctas(uint32_t limbs, uint32_t log_n, uint32_t tile_log) {
  return (((uint64_t)limbs << log_n) + ((uint64_t(1) << tile_log) - 1)) >> tile_log;
}

// Whether one launch takes them: a grid has at most 2^31 - 1 CTAs, and the
// kernels number theirs in 32 bits.
constexpr bool one_launch(uint32_t limbs, uint32_t log_n, uint32_t tile_log) {
  return tile_ctas(limbs, log_n, tile_log) < (uint64_t(1) << 31);
}

}  // namespace yell_gb300
