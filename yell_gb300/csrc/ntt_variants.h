// Launch variants of the NTT / fused polymul per degree (internal).
//
// Each degree has one or more variants that apply exactly the same
// butterflies (so produce the same words) with a different split of the work:
// the tile size of the whole-limb path (limbs per CTA) or the number of
// column stages k1 of the two-pass path (columns of 2^k1 words, rows of
// 2^(log_n - k1) words), or one limb per thread-block cluster.  A degree for
// which no variant was selected, or variant 0 was, takes the one registered
// for the call's number of limbs (polymul_at, ntt_at), else variant 0; the
// autotuner times every variant of a degree but those for few limbs on the
// current device and selects the fastest, which then runs at every number of
// limbs that no variant for few limbs is registered for.  Another variant
// selected by hand runs at every number of limbs; the last of each degree is
// variant 0 once more, for that.
#pragma once
#include <vector>

#include "kernels.h"

namespace yell_gb300 {

struct LimbRange {
  uint32_t least = 1, most = 0;  // none
};

struct Variant {
  char name[96] = {};
  cudaError_t (*ntt)(const LimbSet&, const DevMod*, NttDir, cudaStream_t) = nullptr;
  cudaError_t (*polymul)(const LimbSet&, const ConstLimbSet&, const ConstLimbSet&, const DevMod*,
                         uint64_t* scratch, uint64_t* const* scratch_ptrs, cudaStream_t) = nullptr;
  cudaError_t (*set_attrs)() = nullptr;
  // Whether the current device can place the kernels' clusters (nullptr: no
  // clusters).  Asked once per device, after set_attrs.
  bool (*placeable)() = nullptr;
  uint32_t ntt_launches = 0;
  uint32_t polymul_launches = 0;
  uint32_t tile_log = 0;  // log2 of the words of its smallest tile (words per CTA)
  bool polymul_scratch = false;  // the polymul needs one operand's worth of scratch words
  // Chosen without a selection for calls whose number of limbs lies in one of
  // these ranges; among several variants, the one whose range ends first.
  LimbRange polymul_at[2], ntt_at[2];
  // One of the variants for few limbs: never the stand-in for a polymul
  // called without scratch.
  bool few_limbs = false;
  // Variant 0 once more: selected, it runs at every number of limbs.
  bool again = false;
};

constexpr uint32_t kAnyLimbs = 0xFFFFFFFFu;

// A variant for few limbs: polymuls of up to polymul_limbs, NTTs of up to
// ntt_limbs, and one further range of each.
inline Variant upto(Variant v, uint32_t polymul_limbs, uint32_t ntt_limbs, LimbRange polymul_also = {},
                    LimbRange ntt_also = {}) {
  v.polymul_at[0] = {1, polymul_limbs};
  v.polymul_at[1] = polymul_also;
  v.ntt_at[0] = {1, ntt_limbs};
  v.ntt_at[1] = ntt_also;
  v.few_limbs = true;
  return v;
}

// Registration, one per translation unit (by_degree has kMaxLogN + 1 entries).
void add_whole_variants_small(std::vector<Variant>* by_degree);  // 2^3 .. 2^8
void add_whole_variants_large(std::vector<Variant>* by_degree);  // 2^9 .. 2^13 (and two-pass 2^13)
void add_two_pass_variants_a(std::vector<Variant>* by_degree);   // 2^14, 2^15
void add_two_pass_variants_b(std::vector<Variant>* by_degree);   // 2^16, 2^17
void add_two_pass_variants_c(std::vector<Variant>* by_degree);   // 2^18 .. 2^20
void add_two_pass_variants_d(std::vector<Variant>* by_degree);   // more 2^16 splits and round widths
void add_two_pass_variants_e(std::vector<Variant>* by_degree);   // pipelined polymul, 2^16

void add_few_limb_variants(std::vector<Variant>* by_degree);     // 2^6 .. 2^10, whole-limb, fewer words per thread
void add_two_pass_few_variants(std::vector<Variant>* by_degree); // 2^13 .. 2^20, small tiles
void add_cluster_variants(std::vector<Variant>* by_degree);      // 2^10 .. 2^14, one limb per cluster

// Variant table of a degree.
const std::vector<Variant>& variants_of(uint32_t log_n);
// The variant selected on a device (0 when none was), and its selection by the
// autotuner or by hand.  By hand, 0 ends a selection, and the tuner's last
// choice stands as if the tuner had selected it: selecting what
// selected_variant returned earlier restores the dispatch of that time.
uint32_t selected_variant(int device, uint32_t log_n);
void select_tuned_variant(int device, uint32_t log_n, uint32_t v);
void select_variant(int device, uint32_t log_n, uint32_t v);
// The variant that a transform (polymul: a fused polymul with scratch) of so
// many limbs runs on the current device.
const Variant& variant_for(uint32_t log_n, uint32_t limbs, bool polymul);

}  // namespace yell_gb300
