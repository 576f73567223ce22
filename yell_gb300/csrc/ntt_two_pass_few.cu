// Two-pass variants with tiles of 2^10 or 2^11 words and 4 or 8 words per
// thread, for calls whose limbs do not fill the chip with tiles of 2^12: more
// CTAs, and a shorter chain per thread.  Past the bounds the exchanges that
// the narrower rounds add cost more than the idle SMs.  GB300, polymul us
// (tiles of 2^12 -> here): 16 limbs of 2^14 38.6 -> 14.3, 64 46.3 -> 36.6; 8 of
// 2^15 40.4 -> 14.9; 4 of 2^16 42.8 -> 15.7, 8 50.2 -> 27.1; 1 of 2^17 38.2 ->
// 11.8, 4 53.5 -> 28.6; 2 of 2^18 55.9 -> 39.5; 1 of 2^20 62.7 -> 54.3; and past
// the upper bounds 1024 limbs of 2^13 222 against 222, 224 of 2^14 107 against
// 109 (160 85 against 79), 112 of 2^15 112 against 115 (80 90 against 85), 64
// of 2^16 137 against 137 (48 113 against 106), 96 of 2^17 415 against 420 (48
// 221 against 218), 32 of 2^18 307 against 307; NTT of 160 of 2^14 28 against
// 29 (96 22 against 20).
// Between 4 and 8 words per thread the number of CTAs decides, 2^(log_n - 10)
// per limb with 256 or 128 threads.  Up to one per SM the shorter chain wins
// (2 limbs of 2^16 12.2 us against 13.6); at two and three per SM CTAs of 4
// words get one more than their share on some SMs (4 limbs of 2^16 21.8
// against 16.3, 9 of 2^15 20.9 against 15.6); at four and five the 8-word ones
// do (15 limbs of 2^15 25.2 against 33.0, 9 of 2^16 27.2 against 35.7).  NTTs
// keep 4 words in those ranges: alone in a loop 8 are as much better (12 limbs
// of 2^15 8.7 us against 10.4), among other kernels they are not (encryptions
// of 2 x 7 limbs of 2^15, whole sequence: 50.5 us with 4 words, 55.1 with 8).
#include "ntt_kernels.cuh"

namespace yell_gb300 {

void add_two_pass_few_variants(std::vector<Variant>* by) {
  by[13].push_back(upto(two_pass_few_variant<13, 6, 2, 10>(), 19, 0, {57, 64}));
  by[13].push_back(upto(two_pass_few_variant<13, 6, 3, 10>(), 768, 0));
  by[14].push_back(upto(two_pass_few_variant<14, 7, 2, 10>(), 0, 56, {29, 40}));
  by[14].push_back(upto(two_pass_few_variant<14, 7, 3, 10>(), 192, 128));
  by[15].push_back(upto(two_pass_few_variant<15, 7, 2, 10>(), 4, 32, {15, 22}));
  by[15].push_back(upto(two_pass_few_variant<15, 7, 3, 10>(), 96, 64));
  by[16].push_back(upto(two_pass_few_variant<16, 8, 2, 10>(), 2, 16, {8, 10}));
  by[16].push_back(upto(two_pass_few_variant<16, 8, 3, 10>(), 64, 28));
  by[17].push_back(upto(two_pass_few_variant<17, 8, 2, 10>(), 1, 8, {3, 5}));
  by[17].push_back(upto(two_pass_few_variant<17, 8, 3, 11>(), 64, 12));
  by[18].push_back(upto(two_pass_few_variant<18, 9, 3, 11>(), 32, 8));
  by[19].push_back(upto(two_pass_few_variant<19, 9, 3, 11>(), 24, 4));
  by[20].push_back(upto(two_pass_few_variant<20, 9, 3, 11>(), 12, 4));
}

}  // namespace yell_gb300
