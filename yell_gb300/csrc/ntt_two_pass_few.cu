// Two-pass variants with tiles of 2^10 or 2^11 words and 4 or 8 words per
// thread, for calls whose limbs do not fill the chip with tiles of 2^12: more
// CTAs, and a shorter chain per thread.  Past the bounds the exchanges that
// the narrower rounds add cost more than the idle SMs.  GB300, polymul us
// (tiles of 2^12 -> here): 48 limbs of 2^13 42.9 -> 18.7, 64 of 2^14 46.3 ->
// 36.6, 8 of 2^15 42.3 -> 20.8, 8 of 2^16 50.2 -> 27.0, 4 of 2^17 53.5 -> 28.6,
// 2 of 2^18 55.9 -> 39.5, 1 of 2^20 62.7 -> 54.3; and at the bounds 1024 limbs
// of 2^13 221 against 221, 256 of 2^14 121.7 against 122.2, 128 of 2^15 130.1
// against 128.6, 256 of 2^16 515 against 511, 64 of 2^18 598 against 577.
#include "ntt_kernels.cuh"

namespace yell_gb300 {

void add_two_pass_few_variants(std::vector<Variant>* by) {
  by[13].push_back(upto(two_pass_few_variant<13, 6, 2, 10>(), 64, 0));
  by[13].push_back(upto(two_pass_few_variant<13, 6, 3, 10>(), 768, 0));
  by[14].push_back(upto(two_pass_few_variant<14, 7, 2, 10>(), 40, 56));
  by[14].push_back(upto(two_pass_few_variant<14, 7, 3, 10>(), 224, 160));
  by[15].push_back(upto(two_pass_few_variant<15, 7, 2, 10>(), 22, 32));
  by[15].push_back(upto(two_pass_few_variant<15, 7, 3, 10>(), 112, 64));
  by[16].push_back(upto(two_pass_few_variant<16, 8, 2, 10>(), 8, 16));
  by[16].push_back(upto(two_pass_few_variant<16, 8, 3, 10>(), 192, 28));
  by[17].push_back(upto(two_pass_few_variant<17, 8, 2, 10>(), 6, 8));
  by[17].push_back(upto(two_pass_few_variant<17, 8, 3, 11>(), 96, 12));
  by[18].push_back(upto(two_pass_few_variant<18, 9, 3, 11>(), 32, 8));
  by[19].push_back(upto(two_pass_few_variant<19, 9, 3, 11>(), 24, 4));
  by[20].push_back(upto(two_pass_few_variant<20, 9, 3, 11>(), 12, 4));
}

}  // namespace yell_gb300
