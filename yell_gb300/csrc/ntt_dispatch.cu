// Host dispatch of the NTT / polymul variants, the element-wise kernels,
// and the autotuner.
#include <array>
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <fstream>
#include <mutex>
#include <sstream>
#include <string>
#include <vector>

#include "kernels.h"
#include "launch_size.h"
#include "ntt_variants.h"
#include "profiler.h"
#include "runtime.h"
#include "yell_gb300.h"

namespace yell_gb300 {

namespace {

// plain, as in the transforms (ntt_kernels.cuh)
__device__ __forceinline__ ulonglong2 ld_pair(const uint64_t* p) {
  return *reinterpret_cast<const ulonglong2*>(p);
}

__device__ __forceinline__ void st_pair(uint64_t* p, uint64_t a, uint64_t b) {
  *reinterpret_cast<ulonglong2*>(p) = make_ulonglong2(a, b);
}

// ===========================================================================
// Element-wise ops, a grid of up to kEwCtasPerSm CTAs per SM striding over
// 16-byte pairs.  Bound by HBM (24 or 32 bytes per word).  addmod and submod
// keep two pairs per operand in flight per thread; the Barrett products need
// the registers for resident warps instead.  A grid of 8 CTAs per SM is a
// whole and a partial wave at their occupancy (5 or 6 CTAs per SM); many
// short CTAs level that out, while one per 256 pairs adds launch work.
// GB300, 512 limbs of 2^16 (us, 8 CTAs per SM and one pair -> here -> one CTA
// per 256 pairs): mulmod 138 -> 122 -> 135, muladd 156 -> 154 -> 163, addmod
// 130 -> 118 -> 127, negate 85 -> 83 -> 96 (two pairs 88); 108 limbs of 2^15:
// muladd 20.4 -> 18.1, addmod 16.4 -> 14.5.
// ===========================================================================
constexpr uint32_t kEwCtasPerSm = 24;
constexpr bool ew_product(int op) { return op == (int)EwOp::kMulmod || op == (int)EwOp::kMuladd; }

template <int OP>
__global__ void __launch_bounds__(256) k_elementwise(LimbSet dst, ConstLimbSet a, ConstLimbSet b,
                                                     uint32_t log_n, const DevMod* __restrict__ mods) {
  constexpr bool kBinary = OP != (int)EwOp::kNegate;
  constexpr int kPairs = ew_product(OP) || !kBinary ? 1 : 2;
  constexpr bool kAcc = OP == (int)EwOp::kMuladd;
  grid_dep_launch();
  grid_dep_wait();  // the caller's words, and its limb and modulus lists, come after
  const size_t pairs = ((size_t)dst.count << log_n) >> 1;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  const uint32_t nmask = (1u << log_n) - 1u;
  for (size_t i0 = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i0 < pairs; i0 += kPairs * stride) {
    ulonglong2 x[kPairs], y[kPairs], acc[kPairs];
    uint64_t* d[kPairs];
    uint64_t p[kPairs], pn[kPairs];
#pragma unroll
    for (int u = 0; u < kPairs; ++u) {
      const size_t v = (i0 + u * stride) * 2;
      if (i0 + u * stride < pairs) {
        const uint32_t limb = (uint32_t)(v >> log_n), off = (uint32_t)v & nmask;
        x[u] = ld_pair(a.limb(limb, log_n) + off);
        if (kBinary) y[u] = ld_pair(b.limb(limb, log_n) + off);
        d[u] = dst.limb(limb, log_n) + off;
        if (kAcc) acc[u] = *reinterpret_cast<const ulonglong2*>(d[u]);
        const DevMod* m = mods + dst.cm(limb);
        p[u] = __ldg(&m->p);
        pn[u] = __ldg(&m->pn);
      }
    }
#pragma unroll
    for (int u = 0; u < kPairs; ++u) {
      if (i0 + u * stride < pairs) {
        uint64_t r0, r1;
        if (OP == (int)EwOp::kNegate) {
          r0 = p[u] - x[u].x;
          r1 = p[u] - x[u].y;
        } else if (OP == (int)EwOp::kAddmod) {
          r0 = addmod(x[u].x, y[u].x, p[u]);
          r1 = addmod(x[u].y, y[u].y, p[u]);
        } else if (OP == (int)EwOp::kSubmod) {
          r0 = submod(x[u].x, y[u].x, p[u]);
          r1 = submod(x[u].y, y[u].y, p[u]);
        } else if (OP == (int)EwOp::kMulmod) {
          r0 = mulmod_barrett(x[u].x, y[u].x, p[u], pn[u]);
          r1 = mulmod_barrett(x[u].y, y[u].y, p[u], pn[u]);
        } else {
          r0 = muladd_barrett(acc[u].x, x[u].x, y[u].x, p[u], pn[u]);
          r1 = muladd_barrett(acc[u].y, x[u].y, y[u].y, p[u], pn[u]);
        }
        st_pair(d[u], r0, r1);
      }
    }
  }
}

int g_num_sms = 0;

int num_sms() {
  if (g_num_sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_num_sms, cudaDevAttrMultiProcessorCount, dev);
    if (g_num_sms <= 0) g_num_sms = 1;
  }
  return g_num_sms;
}

std::vector<Variant> g_table[kMaxLogN + 1];
std::once_flag g_table_once;
// Selected variant + 1, with kTuned when the autotuner selected it, or 0 when
// none was selected; and the tuner's last choice + 1, or 0.
constexpr uint32_t kTuned = 0x80;
std::array<std::array<std::atomic<uint8_t>, kMaxLogN + 1>, 64> g_selected{}, g_tuned{};

// Variants whose clusters the device cannot place, one bit each: never taken
// for a call's number of limbs (selected by hand, their launch fails).
std::array<std::array<std::atomic<uint64_t>, kMaxLogN + 1>, 64> g_unplaceable{};

void build_table() {
  add_whole_variants_small(g_table);
  add_whole_variants_large(g_table);
  add_two_pass_variants_a(g_table);
  add_two_pass_variants_b(g_table);
  add_two_pass_variants_c(g_table);
  add_two_pass_variants_d(g_table);
  add_two_pass_variants_e(g_table);
  // after the others: a variant keeps its index
  add_few_limb_variants(g_table);
  add_two_pass_few_variants(g_table);
  add_cluster_variants(g_table);
  for (uint32_t n = kMinLogN; n <= kMaxLogN; ++n) {
    Variant v = g_table[n][0];
    v.again = true;
    std::strncat(v.name, ", for every call", sizeof(v.name) - std::strlen(v.name) - 1);
    g_table[n].push_back(v);
  }
}

int current_device() {
  int d = 0;
  cudaGetDevice(&d);
  return (d >= 0 && d < 64) ? d : 0;
}

}  // namespace

// The variant a call of `limbs` limbs runs: the selected one, else the one
// registered for that many limbs, else the first.  A variant that the
// autotuner selected takes the first one's place, behind those for few limbs:
// it was timed at one size (2^14 tuned at 32 limbs picked 4 words per thread,
// at which an NTT of 512 limbs took 99 us against 77).
const Variant& variant_for(uint32_t log_n, uint32_t limbs, bool polymul) {
  LimbRange(Variant::*const ranges)[2] = polymul ? &Variant::polymul_at : &Variant::ntt_at;
  const std::vector<Variant>& vs = variants_of(log_n);
  const int dev = current_device();
  const uint32_t sel = g_selected[dev][log_n].load(std::memory_order_relaxed);
  const uint64_t unplaceable = g_unplaceable[dev][log_n].load(std::memory_order_relaxed);
  const bool tuned = (sel & kTuned) != 0;
  if (sel != 0 && !tuned) return vs[sel - 1];
  const Variant* best = &vs[tuned ? (sel & ~kTuned) - 1 : 0];
  uint64_t most = ~0ull;
  for (const Variant& v : vs)
    for (const LimbRange& r : v.*ranges)
      if ((!tuned || v.few_limbs) && r.least <= limbs && limbs <= r.most && r.most < most &&
          !(unplaceable >> (&v - vs.data()) & 1)) {
        best = &v;
        most = r.most;
      }
  return *best;
}

const std::vector<Variant>& variants_of(uint32_t log_n) {
  std::call_once(g_table_once, build_table);
  return g_table[log_n];
}

uint32_t selected_variant(int device, uint32_t log_n) {
  const uint32_t sel = g_selected[device][log_n].load(std::memory_order_relaxed);
  return sel != 0 ? (sel & ~kTuned) - 1 : 0;
}

void select_tuned_variant(int device, uint32_t log_n, uint32_t v) {
  g_tuned[device][log_n].store((uint8_t)(v + 1), std::memory_order_relaxed);
  g_selected[device][log_n].store((uint8_t)((v + 1) | kTuned), std::memory_order_relaxed);
}

void select_variant(int device, uint32_t log_n, uint32_t v) {
  uint32_t sel = v != 0 ? v + 1 : 0;
  if (g_tuned[device][log_n].load(std::memory_order_relaxed) == v + 1) sel = (v + 1) | kTuned;
  g_selected[device][log_n].store((uint8_t)sel, std::memory_order_relaxed);
}

cudaError_t init_kernel_attributes() {
  const int dev = current_device();
  for (uint32_t n = kMinLogN; n <= kMaxLogN; ++n) {
    uint64_t unplaceable = 0;
    for (const Variant& v : variants_of(n)) {
      const cudaError_t e = v.set_attrs();
      if (e != cudaSuccess) return e;
      if (v.placeable && !v.placeable()) unplaceable |= uint64_t(1) << (&v - variants_of(n).data());
    }
    g_unplaceable[dev][n].store(unplaceable, std::memory_order_relaxed);
  }
  return cudaSuccess;
}

uint32_t ntt_launch_count(uint32_t log_n, uint32_t limbs) { return variant_for(log_n, limbs, false).ntt_launches; }
uint32_t polymul_launch_count(uint32_t log_n, uint32_t limbs) {
  return variant_for(log_n, limbs, true).polymul_launches;
}

// The words a polymul of this degree may need, whichever variant is selected
// (the selection can change between the caller's allocation and its call).
size_t polymul_scratch_words(uint32_t count, uint32_t log_n, const NttShape&) {
  if (log_n < kMinLogN || log_n > kMaxLogN) return 0;
  for (const Variant& v : variants_of(log_n))
    if (v.polymul_scratch) return (size_t)count << log_n;
  return 0;
}

// True when some variant of this degree runs its polymul without scratch.
bool polymul_scratch_optional(uint32_t log_n) {
  if (log_n < kMinLogN || log_n > kMaxLogN) return true;
  for (const Variant& v : variants_of(log_n))
    if (!v.polymul_scratch && !v.few_limbs) return true;
  return false;
}

cudaError_t launch_ntt(const LimbSet& ls, uint32_t log_n, const DevMod* mods, NttDir dir,
                       const NttShape&, cudaStream_t st) {
  if (ls.count == 0) return cudaSuccess;
  if (log_n < kMinLogN || log_n > kMaxLogN) return cudaErrorInvalidValue;
  const Variant& v = variant_for(log_n, ls.count, false);
  if (!one_launch(ls.count, log_n, v.tile_log)) return cudaErrorInvalidConfiguration;
  return v.ntt(ls, mods, dir, st);
}

cudaError_t launch_polymul(const LimbSet& c, const ConstLimbSet& a, const ConstLimbSet& b,
                           uint32_t log_n, const DevMod* mods, uint64_t* scratch,
                           const NttShape&, cudaStream_t st, uint64_t* const* scratch_ptrs) {
  if (c.count == 0) return cudaSuccess;
  if (log_n < kMinLogN || log_n > kMaxLogN) return cudaErrorInvalidValue;
  const Variant* v = &variant_for(log_n, c.count, true);
  if (v->polymul_scratch && scratch == nullptr && scratch_ptrs == nullptr) {
    // Without scratch, the first (selection order) variant that needs none.
    v = nullptr;
    for (const Variant& w : variants_of(log_n))
      if (!w.polymul_scratch && !w.few_limbs) {
        v = &w;
        break;
      }
    if (!v) return cudaErrorInvalidValue;
  }
  if (!one_launch(c.count, log_n, v->tile_log)) return cudaErrorInvalidConfiguration;
  return v->polymul(c, a, b, mods, scratch, scratch_ptrs, st);
}

cudaError_t launch_elementwise(EwOp op, const LimbSet& dst, const ConstLimbSet& a,
                               const ConstLimbSet& b, uint32_t log_n, const DevMod* mods,
                               cudaStream_t st) {
  if (dst.count == 0) return cudaSuccess;
  const size_t pairs = ((size_t)dst.count << log_n) >> 1;
  const size_t want = (pairs + 255) / 256;
  const size_t cap = (size_t)num_sms() * kEwCtasPerSm;
  const uint32_t grid = (uint32_t)(want < cap ? want : cap);
  LaunchScope ps("elementwise", st);
  switch (op) {
    case EwOp::kMulmod: launch_dependent(k_elementwise<0>, grid, 256, 0, st, dst, a, b, log_n, mods); break;
    case EwOp::kAddmod: launch_dependent(k_elementwise<1>, grid, 256, 0, st, dst, a, b, log_n, mods); break;
    case EwOp::kSubmod: launch_dependent(k_elementwise<2>, grid, 256, 0, st, dst, a, b, log_n, mods); break;
    case EwOp::kMuladd: launch_dependent(k_elementwise<3>, grid, 256, 0, st, dst, a, b, log_n, mods); break;
    case EwOp::kNegate: launch_dependent(k_elementwise<4>, grid, 256, 0, st, dst, a, b, log_n, mods); break;
  }
  g_kernel_launches += 1;
  return cudaGetLastError();
}

}  // namespace yell_gb300
