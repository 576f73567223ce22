// Cluster variants, degrees 2^10 .. 2^14 (k1 = column stages), for calls with
// few limbs.  GB300, us (before -> here), polymul / forward NTT: 1 limb of
// 2^10 14.5 -> 5.8 / 8.2 -> 3.8; 8 limbs of 2^12 20.5 -> 6.9 / 10.9 -> 4.6; 12
// of 2^13 36.9 -> 8.6 / 16.5 -> 5.3; 12 of 2^14 38.7 -> 14.1 / 10.8 -> 7.0.  The
// bounds are where the next variant is as fast: 2^10 at 64 limbs 8.5 against
// 8.3 whole-limb; 2^11 at 2048 103.6 against 100.3; 2^12, 16 limbs on 8 CTAs
// 8.1 against 7.9 on 4, and 1024 limbs 115.9 against 107.8 whole-limb; 2^13,
// 40 limbs 21.2 against 18.8 two-pass; 2^14, 16 limbs 22.9 against 19.9.
#include "ntt_cluster.cuh"

namespace yell_gb300 {

void add_cluster_variants(std::vector<Variant>* by) {
  by[10].push_back(upto(cluster_variant<10, 5, 2, 2>(), 48, 256));
  by[11].push_back(upto(cluster_variant<11, 5, 2, 2>(), 1024, 1024));
  by[12].push_back(upto(cluster_variant<12, 6, 2, 3>(), 12, 160));
  by[12].push_back(upto(cluster_variant<12, 6, 2, 2>(), 640, 1024));
  by[13].push_back(upto(cluster_variant<13, 6, 2, 3>(), 32, 12));
  by[13].push_back(upto(cluster_variant<13, 6, 3, 3>(), 0, 320));
  by[14].push_back(upto(cluster_variant<14, 7, 2, 3>(), 12, 12));
}

}  // namespace yell_gb300
