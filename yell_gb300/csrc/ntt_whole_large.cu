// Whole-limb variants, degrees 2^9 .. 2^13, and the two-pass variants of
// 2^13, which take every call with more limbs than the small-tile variants:
// two CTAs of 256 threads per SM where the whole-limb 2^13 tile fits one of
// 512 (GB300, polymul of 4096 limbs 837 against 958 us, inverse NTT 342
// against 514).
#include "ntt_kernels.cuh"

namespace yell_gb300 {

void add_whole_variants_large(std::vector<Variant>* by) {
  by[9].push_back(whole_variant<9, 12>());
  by[9].push_back(whole_variant<9, 13>());
  by[10].push_back(whole_variant<10, 12>());
  by[10].push_back(whole_variant<10, 13>());
  by[11].push_back(whole_variant<11, 12>());
  by[11].push_back(whole_variant<11, 13>());
  by[12].push_back(whole_variant<12, 12>());
  by[12].push_back(whole_variant<12, 13>());
  by[13].push_back(whole_variant<13, 13>());
  by[13].push_back(two_pass_variant<13, 6>());
  by[13].back().polymul_at[0] = by[13].back().ntt_at[0] = {1, kAnyLimbs};
  by[13].push_back(two_pass_variant<13, 7>());
}

}  // namespace yell_gb300
