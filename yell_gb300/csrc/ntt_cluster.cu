// Cluster variants, degrees 2^10 .. 2^14 (k1 = column stages), for calls with
// few limbs.  GB300, us (before -> here), polymul / forward NTT: 1 limb of
// 2^10 14.5 -> 5.5 (its NTTs run one limb per CTA); 8 limbs of 2^12 20.5 -> 6.7 /
// 10.9 -> 4.2; 10 of 2^13 36.9 -> 8.2 / 16.5 -> 4.7; 15 of 2^13 36.9 -> 9.9; 11 of
// 2^14 38.7 -> 13.5 / 10.8 -> 6.4.  The
// ranges end where another variant is as fast: 2^10 polymul at 96 limbs 7.1
// against 6.4 with one limb per CTA; 2^11 at 2048 103.6 against 100.3; 2^12 on
// 8 CTAs and on 4: polymul at 16 limbs 7.7 and 7.6, NTT at 64 6.0 and 5.7, at
// 128 8.2 and 10.4 (four CTAs on some SMs); 2^12 polymul at 1024 limbs 115.9
// against 107.8 whole-limb; 2^13 polymul at 16 limbs 12.0 against 10.4
// two-pass, at 20 12.4 against 13.2, at 34 14.3 against 13.5, at 48 (8 words
// per thread) 16.4 against 17.8; 2^13 NTT at 56 limbs 11.1 with 4 words per
// thread and 8.6 with 8, at 512 41.6 against 39.1 two-pass; 2^14 at 12 limbs,
// whose clusters no longer find 8 free SMs each, 18.0 against 14.7 and 8.3
// against 7.0.
#include "ntt_cluster.cuh"

namespace yell_gb300 {

void add_cluster_variants(std::vector<Variant>* by) {
  by[10].push_back(upto(cluster_variant<10, 5, 2, 2>(), 80, 0));
  by[11].push_back(upto(cluster_variant<11, 5, 2, 2>(), 1024, 1024));
  by[12].push_back(upto(cluster_variant<12, 6, 2, 3>(), 12, 48, {}, {115, 144}));
  by[12].push_back(upto(cluster_variant<12, 6, 2, 2>(), 640, 1024));
  by[13].push_back(upto(cluster_variant<13, 6, 2, 3>(), 15, 52, {20, 33}));
  by[13].push_back(upto(cluster_variant<13, 6, 3, 3>(), 0, 320, {40, 48}));
  by[14].push_back(upto(cluster_variant<14, 7, 2, 3>(), 11, 11));
}

}  // namespace yell_gb300
