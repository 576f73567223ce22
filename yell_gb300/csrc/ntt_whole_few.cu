// Whole-limb variants with one limb per CTA and 4 or 8 words per thread, for
// calls with few limbs: a 4096-word tile of several limbs leaves most SMs
// idle, and 16 words per thread make a thread's chain of butterflies four
// times as long.  Past the bounds the wider tiles win, which exchange less
// per butterfly.  GB300, polymul us (tile of 2^12 -> here): 64 limbs of 2^6
// 13.6 -> 5.7, of 2^8 14.4 -> 6.3; at the bounds 4096 limbs of 2^6 14.4 ->
// 12.4 (16384: 20.6 against 32.8), 4096 of 2^9 49.4 -> 45.4 (16384: 161.8
// against 168.2); 2^10, 96 limbs 15.9 -> 6.4 at 4 words, 256 limbs 16.0 ->
// 12.4 at 4 words and 9.2 at 8, 1024 limbs 30.8 -> 26.8 at 8 words (4096: 92.9
// against 101.6); 2^10 forward NTT, 64 limbs 7.6 -> 3.7, 256 7.8 -> 5.9.
#include "ntt_kernels.cuh"

namespace yell_gb300 {

void add_few_limb_variants(std::vector<Variant>* by) {
  by[6].push_back(upto(whole_variant<6, 6, 2>(), 4096, 4096));
  by[7].push_back(upto(whole_variant<7, 7, 2>(), 16384, kAnyLimbs));
  by[8].push_back(upto(whole_variant<8, 8, 2>(), 4096, kAnyLimbs));
  by[9].push_back(upto(whole_variant<9, 9, 2>(), 4096, 16384));
  by[10].push_back(upto(whole_variant<10, 10, 2>(), 160, 1024));
  by[10].push_back(upto(whole_variant<10, 10, 3>(), 2048, 0));
}

}  // namespace yell_gb300
