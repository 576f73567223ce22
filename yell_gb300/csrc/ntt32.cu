// 32-bit moduli mode of the hot path (the reference built with
// -DYELL_USE_32BITS_MODULI: include/yell/params_32.hpp, 291 30-bit primes,
// uint32 words and uint64 products, degrees up to kMaxPolyDegree = 2^15).
//
// The kernels reuse the tile engine of the 64-bit path at 32-bit words.  Up to
// 2^13 a CTA can hold whole limbs in shared memory (2^T words, T =
// max(log_n, 11), several limbs per CTA below 2^11); every word is read from
// HBM once and written once.  That fused polymul keeps one operand tile in
// shared memory at a time: NTT(a) leaves its last forward round in registers
// and parks the reduced words in the output limb (the same thread reads them
// back, so they stay in L2), NTT(b) then runs in the same buffer, and the
// product, inverse rounds and scaled last layer follow.  From 2^10 up a limb
// can also be split over a cluster (the 64-bit path's cluster kernels at
// 32-bit words), by the number of limbs up to 2^13 and always above
// (kCluster32).  The butterflies, their order and their twiddle indices are
// the reference's, so lazy words match it exactly.
#include <algorithm>
#include <array>
#include <atomic>
#include <cstring>
#include <memory>
#include <mutex>
#include <string>
#include <utility>
#include <vector>

#include <cooperative_groups.h>

#include "async_copy.cuh"
#include "kernels.h"
#include "ntt_cluster.cuh"
#include "ntt_tile.cuh"
#include "profiler.h"
#include "runtime.h"
#include "yell_gb300.h"

namespace yell_gb300 {
namespace {

constexpr uint32_t kMaxModuli32 = 291;   // params_32.hpp kMaxNbModuli
constexpr uint32_t kLogMaxDegree32 = 15; // kMaxPolyDegree = 2^15
constexpr uint32_t kMinLogN32 = 3;

// ---- prime table -------------------------------------------------------------
// params_32.hpp:15-34: p = 2^30 - j * 2^16 + 1 for increasing j, kept when
// prime (the stated 2^14 step, restricted to p = 1 mod 2^16 so that a
// primitive 2^16-th root exists); Pn = low word of floor(2^64 / p);
// primitive_roots[cm] = g^((p - 1) / 2^16), g the least primitive root.
struct Prime32 {
  uint32_t p, pn, root;
};

uint32_t pow32(uint64_t b, uint64_t e, uint32_t m) {
  uint64_t r = 1;
  b %= m;
  while (e) {
    if (e & 1) r = r * b % m;
    b = b * b % m;
    e >>= 1;
  }
  return (uint32_t)r;
}

bool is_prime32(uint32_t n) {
  if (n < 2) return false;
  for (uint32_t q : {2u, 7u, 61u})
    if (n % q == 0) return n == q;
  uint32_t d = n - 1;
  int s = 0;
  while (!(d & 1)) d >>= 1, ++s;
  for (uint32_t a : {2u, 7u, 61u}) {
    uint64_t x = pow32(a, d, n);
    if (x == 1 || x == n - 1) continue;
    bool comp = true;
    for (int r = 1; r < s && comp; ++r) {
      x = x * x % n;
      if (x == n - 1) comp = false;
    }
    if (comp) return false;
  }
  return true;
}

uint32_t least_primitive_root32(uint32_t p) {
  std::vector<uint32_t> f;
  uint32_t m = p - 1;
  for (uint32_t q = 2; q * q <= m; ++q)
    if (m % q == 0) {
      f.push_back(q);
      while (m % q == 0) m /= q;
    }
  if (m > 1) f.push_back(m);
  for (uint32_t g = 2;; ++g) {
    bool ok = true;
    for (uint32_t q : f) ok = ok && pow32(g, (p - 1) / q, p) != 1;
    if (ok) return g;
  }
}

const std::vector<Prime32>& primes32() {
  static std::vector<Prime32> table = [] {
    std::vector<Prime32> t;
    for (uint32_t j = 1; t.size() < kMaxModuli32; ++j) {
      const uint32_t p = (1u << 30) - j * (1u << 16) + 1;
      if (!is_prime32(p)) continue;
      t.push_back({p, (uint32_t)(~0ull / p), pow32(least_primitive_root32(p), (p - 1) >> 16, p)});
    }
    return t;
  }();
  return table;
}

uint32_t shoupify32(uint32_t x, uint32_t p) { return (uint32_t)(((uint64_t)x << 32) / p); }

// details/ntt.hpp:28-77 at 32-bit words: psi = root^(2^(15 - log_n)); phi and
// invphi powers with Shoup forms, bit-reversed; N^-1 and N^-1 * invphi[1].
void build_host_tables32(uint32_t log_n, uint32_t cm, uint32_t* out4n, uint32_t* sc4) {
  const Prime32& pe = primes32()[cm];
  const uint32_t p = pe.p, n = 1u << log_n;
  uint32_t psi = pe.root;
  for (uint32_t i = 0; i < kLogMaxDegree32 - log_n; ++i) psi = (uint32_t)((uint64_t)psi * psi % p);
  const uint32_t ipsi = pow32(psi, 2ull * n - 1, p);
  uint32_t a = 1, b = 1;
  for (uint32_t i = 0; i < n; ++i) {
    uint32_t r = 0;
    for (uint32_t k = 0; k < log_n; ++k) r |= ((i >> k) & 1u) << (log_n - 1 - k);
    out4n[r] = a;
    out4n[n + r] = shoupify32(a, p);
    out4n[2 * n + r] = b;
    out4n[3 * n + r] = shoupify32(b, p);
    a = (uint32_t)((uint64_t)a * psi % p);
    b = (uint32_t)((uint64_t)b * ipsi % p);
  }
  const uint32_t inv_n = pow32(n % p, p - 2, p);
  const uint32_t inv_n_iphi = (uint32_t)((uint64_t)inv_n * out4n[2 * n + 1] % p);
  sc4[0] = inv_n;
  sc4[1] = shoupify32(inv_n, p);
  sc4[2] = inv_n_iphi;
  sc4[3] = shoupify32(inv_n_iphi, p);
}

// ---- device tables -------------------------------------------------------------
struct DeviceTables32 {
  std::mutex mu;
  DevMod32* mods[kLogMaxDegree32 + 1] = {};
  std::vector<uint8_t> built[kLogMaxDegree32 + 1];
};

DeviceTables32& tables_of(int device) {
  static std::mutex mu;
  static std::vector<std::unique_ptr<DeviceTables32>> all;
  std::lock_guard<std::mutex> g(mu);
  if ((int)all.size() <= device) all.resize(device + 1);
  if (!all[device]) all[device].reset(new DeviceTables32);
  return *all[device];
}

int ensure32(int device, uint32_t log_n, uint32_t cm0, uint32_t L, const DevMod32** out) {
  DeviceTables32& t = tables_of(device);
  std::lock_guard<std::mutex> g(t.mu);
  std::vector<uint8_t>& built = t.built[log_n];
  if (built.empty()) built.assign(kMaxModuli32, 0);
  cudaError_t e;
  if (!t.mods[log_n]) {
    // [cm]: transforms and element-wise ops; [kMaxModuli32 + cm]: the fused
    // polymul (Montgomery product, inverse scaled by N^-1 * 2^32)
    e = lib_malloc(&t.mods[log_n], 2 * kMaxModuli32 * sizeof(DevMod32));
    if (e != cudaSuccess) {
      t.mods[log_n] = nullptr;
      return fail_cuda(e, "cudaMalloc(DevMod32 table)");
    }
    e = upload_zeros(t.mods[log_n], 2 * kMaxModuli32 * sizeof(DevMod32));
    if (e != cudaSuccess) return fail_cuda(e, "cudaMemset(DevMod32 table)");
  }
  const uint32_t n = 1u << log_n;
  std::vector<uint32_t> host(4 * (size_t)n), packed(4 * (size_t)n);
  for (uint32_t cm = cm0; cm < cm0 + L; ++cm) {
    if (built[cm]) continue;
    uint32_t sc[4];
    build_host_tables32(log_n, cm, host.data(), sc);
    for (uint32_t k = 0; k < n; ++k) {  // {w, w'} pairs: fwd then inv
      packed[2 * k] = host[k];
      packed[2 * k + 1] = host[n + k];
      packed[2 * (size_t)n + 2 * k] = host[2 * n + k];
      packed[2 * (size_t)n + 2 * k + 1] = host[3 * n + k];
    }
    uint32_t* d = nullptr;
    e = lib_malloc(&d, packed.size() * sizeof(uint32_t));
    if (e != cudaSuccess) return fail_cuda(e, "cudaMalloc(twiddles32)");
    e = upload(d, packed.data(), packed.size() * sizeof(uint32_t));
    if (e != cudaSuccess) return fail_cuda(e, "upload twiddles32");
    DevMod32 m;
    m.fwd = reinterpret_cast<const uint2*>(d);
    m.inv = reinterpret_cast<const uint2*>(d + 2 * (size_t)n);
    m.p = primes32()[cm].p;
    m.pn = primes32()[cm].pn;
    m.inv_n = sc[0];
    m.inv_n_s = sc[1];
    m.inv_n_iphi = sc[2];
    m.inv_n_iphi_s = sc[3];
    e = upload(t.mods[log_n] + cm, &m, sizeof m);
    if (e != cudaSuccess) return fail_cuda(e, "upload DevMod32");
    DevMod32 pm = m;
    uint32_t inv = m.p;  // p * p = 1 mod 8; Newton's iteration doubles the correct low bits
    for (int i = 0; i < 4; ++i) inv *= 2u - m.p * inv;
    const uint64_t r32 = (1ull << 32) % m.p;
    pm.pn = 0u - inv;
    pm.inv_n = (uint32_t)(m.inv_n * r32 % m.p);
    pm.inv_n_s = shoupify32(pm.inv_n, m.p);
    pm.inv_n_iphi = (uint32_t)(m.inv_n_iphi * r32 % m.p);
    pm.inv_n_iphi_s = shoupify32(pm.inv_n_iphi, m.p);
    e = upload(t.mods[log_n] + kMaxModuli32 + cm, &pm, sizeof pm);
    if (e != cudaSuccess) return fail_cuda(e, "upload DevMod32");
    built[cm] = 1;
  }
  *out = t.mods[log_n];
  return kOk;
}

// ---- kernels -------------------------------------------------------------------
// Tile geometry per degree: whole limbs, 2^LOGE words per thread.
template <int LOGN>
struct Cfg32 {
  static constexpr int T = LOGN > 11 ? LOGN : 11;
  static constexpr int LOGE = LOGN < 4 ? LOGN : 4;
  using C = TileCfg<T, LOGN, 0, LOGE>;
  static constexpr size_t kSmem = Smem<uint32_t>::words(1u << T) * sizeof(uint32_t);
};

struct Limbs32 {
  uint32_t count, L, cm0;
  __device__ __forceinline__ uint32_t cm(uint32_t k) const { return cm0 + k % L; }
};

// Tile <- limbs limb0 .. (16-byte global loads and shared stores), in two
// halves: a thread's loads, all of them before its first store, and the stores.
// A kernel requests its first tile before the modulus' constants (2048 limbs of
// 2^13 forward 55.3 us against 56.8, 4096 of 2^12 polymul 142.2 against 145.0).
template <class C>
constexpr int kStage32 = (1 << C::T) / (C::THREADS * 4);
template <class C>
__device__ __forceinline__ void stage_load32(uint4* d, const uint32_t* g, uint32_t limb0, uint32_t count) {
  static_assert(kStage32<C> * C::THREADS * 4 == (1 << C::T), "tile not a whole number of 16-byte chunks per thread");
#pragma unroll
  for (int i = 0; i < kStage32<C>; ++i) {
    const uint32_t v = (threadIdx.x + i * C::THREADS) * 4;
    const uint32_t limb = limb0 + (v >> C::K);
    if (limb < count)
      d[i] = ld_quad(g + ((size_t)limb << C::K) + (v & ((1u << C::K) - 1u)));
  }
}
template <class C>
__device__ __forceinline__ void stage_store32(uint32_t* s, const uint4* d, uint32_t limb0, uint32_t count) {
#pragma unroll
  for (int i = 0; i < kStage32<C>; ++i) {
    const uint32_t v = (threadIdx.x + i * C::THREADS) * 4;
    if (limb0 + (v >> C::K) < count) *reinterpret_cast<uint4*>(s + Smem<uint32_t>::idx(v)) = d[i];
  }
}

template <class C>
__device__ __forceinline__ void stage_out32(const uint32_t* s, uint32_t* g, uint32_t limb0, const Limbs32& ls,
                                            const DevMod32* __restrict__ mods, bool reduce) {
  for (uint32_t v = threadIdx.x * 4; v < (1u << C::T); v += C::THREADS * 4) {
    const uint32_t limb = limb0 + (v >> C::K);
    if (limb < ls.count) {
      uint4 d = *reinterpret_cast<const uint4*>(s + Smem<uint32_t>::idx(v));
      if (reduce) {
        const uint32_t p = __ldg(&mods[ls.cm(limb)].p), p2 = p << 1;
        d.x = fwd_correct(d.x, p, p2);
        d.y = fwd_correct(d.y, p, p2);
        d.z = fwd_correct(d.z, p, p2);
        d.w = fwd_correct(d.w, p, p2);
      }
      *reinterpret_cast<uint4*>(g + ((size_t)limb << C::K) + (v & ((1u << C::K) - 1u))) = d;
    }
  }
}

// DIR: 0 forward (reduced to [0, p)), 1 forward lazy ([0, 4p)), 2 backward.
template <class C, int DIR>
__global__ void __launch_bounds__(C::THREADS, 1024 / C::THREADS) k32_ntt(uint32_t* data, Limbs32 ls, const DevMod32* __restrict__ mods) {
  extern __shared__ __align__(16) uint32_t smem32[];
  constexpr int NR = C::NR;
  grid_dep_wait();  // the stream's previous kernel may produce or read data
  grid_dep_launch();
  const uint32_t tid = threadIdx.x;
  const uint32_t limb0 = blockIdx.x << (C::T - C::K);
  const uint32_t my_limb = limb0 + C::sub(tid);
  const bool active = my_limb < ls.count;
  uint4 d[kStage32<C>];
  stage_load32<C>(d, data, limb0, ls.count);
  const DevMod32 m = load_mod(mods, ls.cm(active ? my_limb : 0));
  stage_store32<C>(smem32, d, limb0, ls.count);
  __syncthreads();
  if constexpr (DIR != 2) {
    fwd_rounds<C, 0, NR>(smem32, tid, 0, 0, m.fwd, m.p, active);
  } else {
    inv_rounds<C, NR - 1, -1, true>(smem32, tid, (uint32_t)C::K, 0, 0, m, active);
  }
  stage_out32<C>(smem32, data, limb0, ls, mods, DIR == 0);
}

// c = INTT(NTT(a) * NTT(b)) per limb; c must not alias a or b.
template <class C>
__global__ void __launch_bounds__(C::THREADS, 1024 / C::THREADS) k32_polymul(uint32_t* c, const uint32_t* a, const uint32_t* b,
                                                          Limbs32 ls, const DevMod32* __restrict__ mods) {
  extern __shared__ __align__(16) uint32_t smem32[];
  constexpr int NR = C::NR, E = 1 << C::LOGE;
  using RB = Round<C, NR - 1>;
  static_assert(RB::R == C::LOGE && RB::BETA == 0 && RB::EB == 0, "bottom round must own contiguous words");
  grid_dep_wait();  // the stream's previous kernel may produce a or b, or read c
  grid_dep_launch();
  const uint32_t tid = threadIdx.x;
  const uint32_t limb0 = blockIdx.x << (C::T - C::K);
  const uint32_t my_limb = limb0 + C::sub(tid);
  const bool active = my_limb < ls.count;
  uint4 d[kStage32<C>];
  stage_load32<C>(d, a, limb0, ls.count);
  const DevMod32 m = load_mod(mods, ls.cm(active ? my_limb : 0));
  const uint32_t p = m.p, p2 = p << 1;
  const uint32_t bb = RB::base(tid);
  // the thread's E contiguous words of the output tile (in limb my_limb)
  uint32_t* park = c + ((size_t)my_limb << C::K) + (bb & ((1u << C::K) - 1u));
  uint32_t x[E];
  // NTT(a), parked in c
  stage_store32<C>(smem32, d, limb0, ls.count);
  __syncthreads();
  fwd_rounds<C, 0, NR - 1>(smem32, tid, 0, 0, m.fwd, p, active);
  if (active) {
    smem_load<RB>(x, smem32, bb);
    ct_round<RB>(x, m.fwd, (uint32_t)RB::HI, RB::gr(bb, 0), p);
#pragma unroll
    for (int i = 0; i < E; i += 4)
      *reinterpret_cast<uint4*>(park + i) =
          make_uint4(csub(x[i], p2), csub(x[i + 1], p2), csub(x[i + 2], p2), csub(x[i + 3], p2));
  }
  // NTT(b), product, inverse
  __syncthreads();
  stage_load32<C>(d, b, limb0, ls.count);
  stage_store32<C>(smem32, d, limb0, ls.count);
  __syncthreads();
  fwd_rounds<C, 0, NR - 1>(smem32, tid, 0, 0, m.fwd, p, active);
  if (active) {
    smem_load<RB>(x, smem32, bb);
    ct_round<RB>(x, m.fwd, (uint32_t)RB::HI, RB::gr(bb, 0), p);
#pragma unroll
    for (int i = 0; i < E; i += 4) {
      const uint4 ah = *reinterpret_cast<const uint4*>(park + i);  // written above by this thread
      x[i] = mont_mul(ah.x, csub(x[i], p2), p, m.pn);
      x[i + 1] = mont_mul(ah.y, csub(x[i + 1], p2), p, m.pn);
      x[i + 2] = mont_mul(ah.z, csub(x[i + 2], p2), p, m.pn);
      x[i + 3] = mont_mul(ah.w, csub(x[i + 3], p2), p, m.pn);
    }
    gs_round<RB, NR == 1>(x, (uint32_t)C::K, (uint32_t)RB::BETA, RB::gr(bb, 0), m);
    smem_store<RB>(x, smem32, bb);
  }
  __syncthreads();
  inv_rounds<C, NR - 2, -1, true>(smem32, tid, (uint32_t)C::K, 0, 0, m, active);
  stage_out32<C>(smem32, c, limb0, ls, mods, false);
}


// ---- polymul at 2^15 by a CTA pair with staged operands ------------------------
// One limb is split over the two CTAs of a cluster, each holding half of it.
// The forward stage that pairs words N/2 apart (stage 0, twiddle w[1]) is
// applied to the raw operand: each CTA brings the whole limb and keeps the
// butterfly output of its own half.  Stages 1 .. log N - 1 stay inside a half
// (group G = the CTA's rank).  The inverse's last layer (N^-1 scaling fused)
// pairs the halves again: after a cluster barrier each CTA reads the peer's
// words through distributed shared memory and writes its own half of the
// outputs.  One CTA of 1024 threads per SM, so 76 limbs are one wave; used
// only around that size (kCluster32).
//
// The stages inside a half limb of 2^H words run as two tiles of the engine:
// the top KTOP (pair distances 2^(H-1) .. 2^(H-KTOP)) across the CTA (CA:
// columns of stride 2^(H-KTOP), CTA barriers), the other H - KTOP in rows of
// 2^(H-KTOP) words (CB), each row held by the threads of one warp, so the
// rounds inside a row need only warp barriers.  The bottom round gives each
// thread 2^LOGE consecutive words.
template <int H, int LOGE, int KTOP>
struct HalfSplit {
  using CA = TileCfg<H, KTOP, H - KTOP, LOGE>;
  using CB = TileCfg<H, H - KTOP, 0, LOGE>;
  static constexpr int KB = H - KTOP, KTOP_STAGES = KTOP;
  static_assert(CA::THREADS == CB::THREADS && CB::LOCAL_BARRIER == 1, "rows must stay inside a warp");
  // Row index within the whole limb (the sub-transform group of CB's top stage).
  __device__ static __forceinline__ uint32_t row_group(uint32_t r, uint32_t tid) {
    return (r << KTOP) + CB::sub(tid);
  }
};

// Geometry: 1024-thread CTAs of 16 words per thread at 64 registers, the top 7
// stages across the CTA and rows of 128 words (6 or 8 stages across the CTA
// measured 0 and 2% slower, 512 threads of 32 words 2 to 15%).
struct PairGeom32 {
  static constexpr int H = 14, LOGE = 4, KTOP = 7;
  using C = TileCfg<H, H, 0, LOGE>;
  using S = HalfSplit<H, LOGE, KTOP>;
};

// Inverse stages inside the half limb from the bottom-round registers x:
// rows (warp barriers), then the top KTOP across the CTA; the words end in
// shared memory.  CB's last round is followed by a CTA barrier.
template <class PC>
__device__ __forceinline__ void pair_inverse(uint32_t* x, uint32_t* smem32, uint32_t tid, uint32_t r,
                                             uint32_t bb, const DevMod32& m) {
  using C = typename PC::C;
  using S = typename PC::S;
  using CA = typename S::CA;
  using CB = typename S::CB;
  using RBB = Round<CB, CB::NR - 1>;
  constexpr uint32_t log_n = C::K + 1;
  const uint32_t G = S::row_group(r, tid);
  gs_round<RBB, false>(x, log_n, (uint32_t)RBB::BETA, RBB::gr(bb, G), m);
  smem_store<RBB>(x, smem32, bb);
  round_barrier<CB, CB::LOCAL_BARRIER>(tid);
  inv_rounds<CB, CB::NR - 2, 0, false, CB::LOCAL_BARRIER>(smem32, tid, log_n, 0, G, m, true);
  inv_rounds<CB, 0, -1, false>(smem32, tid, log_n, 0, G, m, true);  // CTA barrier after
  inv_rounds<CA, CA::NR - 1, -1, false>(smem32, tid, log_n, S::KB, r, m, true);
}

// Last inverse layer across the pair with the N^-1 scaling: u = word i
// (rank 0), w = word i + N/2 (rank 1); each CTA writes its own half.
template <class PC, bool UNROLL>
__device__ __forceinline__ void pair_last_layer(uint32_t* dst, const uint32_t* smem32, const uint32_t* peer,
                                                uint32_t tid, uint32_t r, const DevMod32& m) {
  using C = typename PC::C;
  constexpr int IT = (int)((1u << C::K) / (C::THREADS * 4));
  const uint32_t p2 = m.p << 1;
#pragma unroll(UNROLL ? IT : 1)
  for (int i = 0; i < IT; ++i) {
    const uint32_t v = (tid + i * C::THREADS) * 4;
    const uint4 own = *reinterpret_cast<const uint4*>(smem32 + Smem<uint32_t>::idx(v));
    const uint4 oth = *reinterpret_cast<const uint4*>(peer + Smem<uint32_t>::idx(v));
    const uint32_t o[4] = {own.x, own.y, own.z, own.w}, q[4] = {oth.x, oth.y, oth.z, oth.w};
    uint32_t res[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint32_t u = r == 0 ? o[k] : q[k], w = r == 0 ? q[k] : o[k];
      res[k] = r == 0 ? mulmod_shoup(u + w, m.inv_n, m.inv_n_s, m.p)
                      : mulmod_shoup(u - w + p2, m.inv_n_iphi, m.inv_n_iphi_s, m.p);
    }
    *reinterpret_cast<uint4*>(dst + v) = make_uint4(res[0], res[1], res[2], res[3]);
  }
}

// The operands move by bulk asynchronous copies (cp.async.bulk, completion
// counted on an mbarrier): both halves of a's limb land in a raw staging area S of shared memory; the
// stage-0 butterflies read them from there; then b's copy into S starts and
// runs while a's remaining stages compute.  a's reduced NTT stays in the work
// tile W where its bottom round left it, and b is transformed in place in S
// (its own-half outputs overwrite the raw words once every thread has read
// its pairs).  Shared memory: W (half limb) + S (whole limb) + the mbarrier.
// Every wait on the mbarrier is bounded; one that runs out records
// YELL_ERR_TIMEOUT in g_k32_wait_status and the kernel carries on, so that
// every thread still reaches every barrier.
__device__ uint32_t g_k32_wait_status;

// Bounded wait on the staged kernel's mbarrier; a wait that runs out records
// YELL_ERR_TIMEOUT in g_k32_wait_status.
__device__ __forceinline__ bool mbar_wait32(uint64_t* mbar, uint32_t parity,
                                            uint64_t timeout_ns = 1000000000ull) {
  return mbar_wait(mbar, parity, &g_k32_wait_status, (uint32_t)YELL_ERR_TIMEOUT, timeout_ns);
}

// Check of that bounded wait: one CTA announces 16 bytes of copies on an
// mbarrier, starts none, and waits on it the way the staged kernel does; the
// wait runs out after timeout_ns and records YELL_ERR_TIMEOUT.  No copy is in
// flight when the CTA exits.
__global__ void k32_wait_check(uint64_t timeout_ns) {
  __shared__ uint64_t mbar;
  if (threadIdx.x == 0) {
    mbar_init(&mbar, 1);
    mbar_expect(&mbar, 16);
  }
  __syncthreads();
  mbar_wait32(&mbar, 0, timeout_ns);
}

// Stage 0 (pairs N/2 apart, twiddle w[1]) from the raw halves of a limb in
// S_lo and S_hi into this CTA's half in `dst` (swizzled tile layout).  With
// IN_PLACE, dst overlaps S_lo: every thread keeps its outputs in registers
// until all raw words are read.
// Ends with a CTA barrier.
template <class PC, bool IN_PLACE>
__device__ __forceinline__ void stage0_from_smem(uint32_t* dst, const uint32_t* S_lo, const uint32_t* S_hi,
                                                 uint32_t tid, uint32_t r, uint32_t p, uint2 w1) {
  using C = typename PC::C;
  constexpr uint32_t half = 1u << C::K;
  constexpr int IT = (int)(half / (C::THREADS * 4));
  const uint32_t p2 = p << 1, np = 0u - p;
  uint4 out[IN_PLACE ? IT : 1];
#pragma unroll
  for (int i = 0; i < IT; ++i) {
    const uint32_t v = (tid + i * C::THREADS) * 4;
    const uint4 lo = *reinterpret_cast<const uint4*>(S_lo + v);
    const uint4 hi = *reinterpret_cast<const uint4*>(S_hi + v);
    uint32_t u0[4] = {lo.x, lo.y, lo.z, lo.w}, u1[4] = {hi.x, hi.y, hi.z, hi.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) ct_bfly(u0[k], u1[k], w1.x, w1.y, np, p2);
    const uint4 o = r == 0 ? make_uint4(u0[0], u0[1], u0[2], u0[3]) : make_uint4(u1[0], u1[1], u1[2], u1[3]);
    if constexpr (IN_PLACE) out[i] = o;
    else *reinterpret_cast<uint4*>(dst + Smem<uint32_t>::idx(v)) = o;
  }
  if constexpr (IN_PLACE) {
    __syncthreads();
#pragma unroll
    for (int i = 0; i < IT; ++i)
      *reinterpret_cast<uint4*>(dst + Smem<uint32_t>::idx((tid + i * C::THREADS) * 4)) = out[i];
  }
  __syncthreads();
}

// Stages 1 .. log N - 1 of the half limb in `work` (after stage 0), the last
// round into the registers x.
template <class PC>
__device__ __forceinline__ void pair_forward_rounds(uint32_t* x, uint32_t* work, uint32_t tid, uint32_t r,
                                                    const DevMod32& m) {
  using C = typename PC::C;
  using S = typename PC::S;
  using CA = typename S::CA;
  using CB = typename S::CB;
  using RBB = Round<CB, CB::NR - 1>;
  constexpr uint32_t s_rows = 1 + S::KTOP_STAGES;
  fwd_rounds<CA, 0, CA::NR>(work, tid, 1, r, m.fwd, m.p, true);
  const uint32_t G = S::row_group(r, tid);
  fwd_rounds<CB, 0, CB::NR - 1, CB::LOCAL_BARRIER>(work, tid, s_rows, G, m.fwd, m.p, true);
  const uint32_t bb = RBB::base(tid);
  smem_load<RBB>(x, work, bb);
  ct_round<RBB>(x, m.fwd, s_rows + RBB::HI, RBB::gr(bb, G), m.p);
}

struct Staged32 {
  static constexpr int THREADS = PairGeom32::C::THREADS;
  static constexpr size_t kSmem = 3 * (size_t(1) << PairGeom32::H) * sizeof(uint32_t) + 16;  // W, S, mbarrier
};

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(Staged32::THREADS, 1)
    k32_polymul_staged(uint32_t* c, const uint32_t* a, const uint32_t* b, Limbs32 ls,
                       const DevMod32* __restrict__ mods) {
  namespace cg = cooperative_groups;
  using PC = PairGeom32;
  using C = typename PC::C;
  extern __shared__ __align__(128) uint32_t smem_st[];
  constexpr int H = C::K, NR = C::NR, E = 1 << C::LOGE;
  constexpr uint32_t log_n = H + 1, half = 1u << H;
  using RB = Round<C, NR - 1>;
  static_assert(RB::R == C::LOGE && RB::BETA == 0 && RB::EB == 0, "bottom round must own contiguous words");
  uint32_t* W = smem_st;             // a's tile, then a's parked NTT
  uint32_t* S = smem_st + half;      // raw limb (2 halves); b's tile after its stage 0
  uint64_t* mbar = reinterpret_cast<uint64_t*>(smem_st + 3 * half);
  cg::cluster_group cluster = cg::this_cluster();
  const uint32_t r = cluster.block_rank();
  const uint32_t limb = blockIdx.x >> 1;
  const uint32_t tid = threadIdx.x;
  const DevMod32 m = load_mod(mods, ls.cm(limb));
  const uint32_t p = m.p, p2 = p << 1;
  const uint2 w1 = __ldg(m.fwd + 1);
  const size_t lbase = (size_t)limb << log_n;
  const uint32_t bb = RB::base(tid);
  grid_dep_wait();  // the stream's previous kernel may produce a or b, or read c
  grid_dep_launch();
  if (tid == 0) {
    mbar_init(mbar, 1);
    mbar_expect(mbar, 2 * half * (uint32_t)sizeof(uint32_t));
    bulk_g2s(S, a + lbase, half * (uint32_t)sizeof(uint32_t), mbar);
    bulk_g2s(S + half, a + lbase + half, half * (uint32_t)sizeof(uint32_t), mbar);
  }
  __syncthreads();  // the mbarrier is initialised before anyone polls it
  mbar_wait32(mbar, 0);
  stage0_from_smem<PC, false>(W, S, S + half, tid, r, p, w1);
  if (tid == 0) {
    // S was read through the generic proxy; the copies write it through the async one
    fence_proxy_async();
    mbar_expect(mbar, 2 * half * (uint32_t)sizeof(uint32_t));
    bulk_g2s(S, b + lbase, half * (uint32_t)sizeof(uint32_t), mbar);
    bulk_g2s(S + half, b + lbase + half, half * (uint32_t)sizeof(uint32_t), mbar);
  }
  uint32_t x[E];
  pair_forward_rounds<PC>(x, W, tid, r, m);
  // park a's words (in [0, 2p)) where its bottom round read them (only this thread's positions)
#pragma unroll
  for (int i = 0; i < E; ++i) x[i] = csub(x[i], p2);
  smem_store<RB>(x, W, bb);
  mbar_wait32(mbar, 1);
  stage0_from_smem<PC, true>(S, S, S + half, tid, r, p, w1);
  pair_forward_rounds<PC>(x, S, tid, r, m);
  {
    const uint32_t ib = Smem<uint32_t>::idx(bb);
#pragma unroll
    for (int i = 0; i < E; i += 4) {
      const uint4 ah = *reinterpret_cast<const uint4*>(W + (ib ^ (uint32_t)i));
      x[i] = mont_mul(ah.x, csub(x[i], p2), p, m.pn);
      x[i + 1] = mont_mul(ah.y, csub(x[i + 1], p2), p, m.pn);
      x[i + 2] = mont_mul(ah.z, csub(x[i + 2], p2), p, m.pn);
      x[i + 3] = mont_mul(ah.w, csub(x[i + 3], p2), p, m.pn);
    }
  }
  pair_inverse<PC>(x, S, tid, r, bb, m);
  cluster.sync();
  pair_last_layer<PC, true>(c + lbase + r * half, S, cluster.map_shared_rank(S, (int)(r ^ 1u)), tid, r, m);
  cluster.sync();  // the peer may still be reading this CTA's shared memory
}

template <int OP>
__global__ void k32_elementwise(uint32_t* dst, const uint32_t* a, const uint32_t* b, size_t total, uint32_t log_n,
                                Limbs32 ls, const DevMod32* __restrict__ mods) {
  grid_dep_launch();
  grid_dep_wait();  // as above
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < total; k += (size_t)gridDim.x * blockDim.x) {
    const uint32_t cm = ls.cm((uint32_t)(k >> log_n));
    const uint32_t p = __ldg(&mods[cm].p);
    if constexpr (OP == YELL_OP_MULMOD) dst[k] = mulmod_barrett(a[k], b[k], p, __ldg(&mods[cm].pn));
    else if constexpr (OP == YELL_OP_ADDMOD) dst[k] = addmod(a[k], b[k], p);
    else if constexpr (OP == YELL_OP_SUBMOD) dst[k] = submod(a[k], b[k], p);
    else if constexpr (OP == YELL_OP_MULADD) dst[k] = muladd_barrett(dst[k], a[k], b[k], p, __ldg(&mods[cm].pn));
    else dst[k] = p - a[k];
  }
}

// ---- launch ----------------------------------------------------------------------
// Degrees of the one-CTA kernels; larger ones run on clusters only.
// At 2^13 clusters take every inverse and polymul where one of 2 can be placed
// (512 limbs, us: polymul 39.6 and 47.3 with one CTA, inverse 16.7 and 17.6).
constexpr int kLogMaxOneCta32 = 13;
// Host-pointer calls up to this degree run in place on the context's pinned,
// device-mapped host buffer.
constexpr uint32_t kSmallCall32LogN = 13;

template <int LOGN>
cudaError_t set_attrs32() {
  using C = typename Cfg32<LOGN>::C;
  const int smem = (int)Cfg32<LOGN>::kSmem;
  cudaError_t e = cudaSuccess;
  for (auto k : {k32_ntt<C, 0>, k32_ntt<C, 1>, k32_ntt<C, 2>})
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k32_polymul<C>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  return e;
}

// As programmatic dependents, like the 64-bit kernels (GB300, polymul, us:
// 1 limb of 2^9 8.2 -> 5.3, 1024 of 2^9 10.3 -> 7.5, 2000 of 2^12 75.8 -> 73.8;
// forward NTT of 1024 limbs of 2^9 6.2 -> 4.0).
template <int LOGN>
cudaError_t launch32(int kind, uint32_t* c, const uint32_t* a, const uint32_t* b, const Limbs32& ls,
                     const DevMod32* mods, cudaStream_t st) {
  using CF = Cfg32<LOGN>;
  using C = typename CF::C;
  const uint32_t blocks = (ls.count + (1u << (C::T - LOGN)) - 1) >> (C::T - LOGN);
  if (kind == 0) launch_dependent(k32_ntt<C, 0>, blocks, C::THREADS, CF::kSmem, st, c, ls, mods);
  else if (kind == 1) launch_dependent(k32_ntt<C, 1>, blocks, C::THREADS, CF::kSmem, st, c, ls, mods);
  else if (kind == 2) launch_dependent(k32_ntt<C, 2>, blocks, C::THREADS, CF::kSmem, st, c, ls, mods);
  else launch_dependent(k32_polymul<C>, blocks, C::THREADS, CF::kSmem, st, c, a, b, ls, mods + kMaxModuli32);
  return cudaGetLastError();
}

// Contiguous 32-bit limbs for the cluster kernels (the interface of LimbSet).
template <class P>
struct LimbSet32 {
  P* base;
  uint32_t count, L, cm0;
  __device__ __forceinline__ P* limb(uint32_t k, uint32_t log_n) const { return base + ((size_t)k << log_n); }
  __device__ __forceinline__ uint32_t cm(uint32_t k) const { return cm0 + k % L; }
  __device__ __forceinline__ uint32_t ordered(uint32_t i) const {  // modulus-major, as LimbSet
    const uint32_t polys = count / L;
    return (i % polys) * L + i / polys;
  }
};
using Out32 = LimbSet32<uint32_t>;
using In32 = LimbSet32<const uint32_t>;

template <class CC>
cudaError_t cluster_ntt32(int kind, uint32_t* c, const Limbs32& ls, const DevMod32* mods, cudaStream_t st) {
  const Out32 o{c, ls.count, ls.L, ls.cm0};
  if (kind == 0) launch_cluster<CC>(k_ntt_cluster<CC, 0, Out32, DevMod32>, ls.count, 2 * CC::kTileBytes, st, o, mods);
  else if (kind == 1)
    launch_cluster<CC>(k_ntt_cluster<CC, 1, Out32, DevMod32>, ls.count, 2 * CC::kTileBytes, st, o, mods);
  else launch_cluster<CC>(k_ntt_cluster<CC, 2, Out32, DevMod32>, ls.count, 2 * CC::kTileBytes, st, o, mods);
  return cudaGetLastError();
}
template <class CC>
cudaError_t cluster_polymul32(uint32_t* c, const uint32_t* a, const uint32_t* b, const Limbs32& ls,
                              const DevMod32* mods, cudaStream_t st) {
  launch_cluster<CC>(k_polymul_cluster<CC, Out32, In32, DevMod32>, ls.count, 4 * CC::kTileBytes, st,
                     Out32{c, ls.count, ls.L, ls.cm0}, In32{a, ls.count, ls.L, ls.cm0},
                     In32{b, ls.count, ls.L, ls.cm0}, mods + kMaxModuli32);
  return cudaGetLastError();
}
template <class CC>
cudaError_t attrs_ntt32() {
  constexpr size_t bytes = 2 * CC::kTileBytes;
  cudaError_t e = set_smem(k_ntt_cluster<CC, 0, Out32, DevMod32>, bytes);
  if (e == cudaSuccess) e = set_smem(k_ntt_cluster<CC, 1, Out32, DevMod32>, bytes);
  return e == cudaSuccess ? set_smem(k_ntt_cluster<CC, 2, Out32, DevMod32>, bytes) : e;
}
template <class CC>
cudaError_t attrs_polymul32() {
  return set_smem(k_polymul_cluster<CC, Out32, In32, DevMod32>, 4 * CC::kTileBytes);
}
cudaError_t staged_polymul32(uint32_t* c, const uint32_t* a, const uint32_t* b, const Limbs32& ls,
                             const DevMod32* mods, cudaStream_t st) {
  launch_dependent(k32_polymul_staged, 2 * ls.count, Staged32::THREADS, Staged32::kSmem, st, c, a, b, ls,
                   mods + kMaxModuli32);
  return cudaGetLastError();
}
cudaError_t attrs_staged32() { return set_smem(k32_polymul_staged, Staged32::kSmem); }
// Cluster of 2 (compiled into the kernel), as ClusterCfg names it.
struct StagedPair {
  static constexpr int CL = 1, THREADS = Staged32::THREADS;
};
template <class CC>
bool placeable_ntt32() {
  return cluster_placeable<CC>(k_ntt_cluster<CC, 0, Out32, DevMod32>, 2 * CC::kTileBytes);
}
template <class CC>
bool placeable_polymul32() {
  return cluster_placeable<CC>(k_polymul_cluster<CC, Out32, In32, DevMod32>, 4 * CC::kTileBytes);
}
bool placeable_staged32() { return cluster_placeable<StagedPair>(k32_polymul_staged, Staged32::kSmem); }

// Cluster kernels (one limb per cluster of 2^CL CTAs) by degree and number of
// limbs: a call takes the entry of its degree with the smallest bound that
// its limbs do not exceed, else the one-CTA kernels above (2^3 .. 2^13).  The
// polymul shares every twiddle load between its operands, where the one-CTA
// kernels transform one after the other; with few limbs a limb spread over
// 2, 4 or 8 SMs is a shorter chain.  Past the bounds the one-CTA kernels win,
// which exchange nothing between CTAs.  The last template argument is the
// CTAs per SM that the polymul is compiled for: registers against residency.
//
// GB300, us (one-CTA and CTA-pair kernels -> here), polymul / forward /
// inverse: 8 limbs of 2^13 16.5 -> 6.0 / 8.2 -> 5.3 / 8.2 -> 5.4; 24 of 2^14
// 21.3 -> 9.5 / 10.3 -> 7.5 / 12.3 -> 7.3; 512 of 2^13 51.2 -> 40.2 / 19.6 ->
// 18.6 / 20.7 -> 17.1; 512 of 2^14 90.8 -> 84.9 / 39.2 -> 35.0 / 39.2 -> 32.5;
// 512 of 2^15 200 -> 188 / 82 -> 72 / 76 -> 66.  At the bounds: 1024 limbs of
// 2^11 polymul 20.6 -> 19.8 (1536: 28.9 against 32.7), 1536 of 2^12 61.2 -> 59.3
// (2048: 77.1 against 79.4), 768 of 2^13 forward 27.1 -> 26.8 (1536: 45.7
// against 47.8).  57 to 76 limbs of 2^15 are one wave of the staged CTA pair
// (28 us), but two of the three clusters' worth of SMs that 8 CTAs each need
// (32 to 34 us).
struct Cluster32 {
  uint32_t log_n;
  uint32_t polymul_upto, fwd_upto, inv_upto;  // 0: never
  cudaError_t (*ntt)(int, uint32_t*, const Limbs32&, const DevMod32*, cudaStream_t);
  cudaError_t (*polymul)(uint32_t*, const uint32_t*, const uint32_t*, const Limbs32&, const DevMod32*, cudaStream_t);
  cudaError_t (*ntt_attrs)();
  cudaError_t (*polymul_attrs)();
  bool (*placeable)();  // on the current device
};
template <int LOGN, int K1, int LOGE, int CL, int PB = 0>
using CC32 = ClusterCfg<LOGN, K1, LOGE, CL, uint32_t, PB>;
template <class CC>
constexpr Cluster32 polymul_route32(uint32_t upto) {
  return {CC::LOGN, upto, 0, 0, nullptr, cluster_polymul32<CC>, nullptr, attrs_polymul32<CC>,
          placeable_polymul32<CC>};
}
template <class CC>
constexpr Cluster32 ntt_route32(uint32_t fwd, uint32_t inv) {
  return {CC::LOGN, 0, fwd, inv, cluster_ntt32<CC>, nullptr, attrs_ntt32<CC>, nullptr, placeable_ntt32<CC>};
}
constexpr uint32_t kAny32 = 0xFFFFFFFFu;
constexpr Cluster32 kCluster32[] = {
    polymul_route32<CC32<10, 5, 3, 1>>(1024),
    ntt_route32<CC32<10, 5, 3, 1>>(1024, 1024),
    polymul_route32<CC32<11, 5, 3, 1>>(1024),
    ntt_route32<CC32<11, 5, 3, 1>>(768, 512),
    polymul_route32<CC32<12, 6, 3, 1>>(224),
    polymul_route32<CC32<12, 6, 4, 1, 4>>(1536),
    ntt_route32<CC32<12, 6, 3, 2>>(288, 288),
    ntt_route32<CC32<12, 6, 3, 1>>(1536, 768),
    polymul_route32<CC32<13, 6, 3, 2>>(100),
    polymul_route32<CC32<13, 6, 4, 1, 3>>(kAny32),
    ntt_route32<CC32<13, 6, 3, 2>>(400, 400),
    ntt_route32<CC32<13, 6, 4, 1>>(768, kAny32),
    polymul_route32<CC32<14, 7, 4, 2, 2>>(76),
    polymul_route32<CC32<14, 7, 4, 2, 3>>(kAny32),
    ntt_route32<CC32<14, 7, 4, 3>>(200, 200),
    ntt_route32<CC32<14, 7, 4, 2>>(kAny32, kAny32),
    polymul_route32<CC32<15, 8, 4, 3, 2>>(32),
    polymul_route32<CC32<15, 8, 4, 3, 3>>(57),
    {15, 76, 0, 0, nullptr, staged_polymul32, nullptr, attrs_staged32, placeable_staged32},
    polymul_route32<CC32<15, 8, 4, 3, 3>>(kAny32),
    ntt_route32<CC32<15, 8, 4, 3>>(kAny32, kAny32),
    // where no clusters of 4 or 8 can be placed (GB300, 512 limbs, us, the
    // entries above -> these, polymul / forward / inverse: 2^14 86 -> 104 / 34 ->
    // 37 / 32 -> 33; 2^15 187 -> 199 / 71 -> 90 / 65 -> 81)
    polymul_route32<CC32<14, 7, 4, 1>>(kAny32),
    ntt_route32<CC32<14, 7, 4, 1>>(kAny32, kAny32),
    {15, kAny32, 0, 0, nullptr, staged_polymul32, nullptr, nullptr, placeable_staged32},
    ntt_route32<CC32<15, 8, 4, 1>>(kAny32, kAny32),
};
constexpr size_t kRoutes32 = sizeof(kCluster32) / sizeof(kCluster32[0]);
// Per device, the entries whose clusters it can place, one bit each.
std::array<std::atomic<uint64_t>, 64> g_placeable32{};
static_assert(kRoutes32 <= 64, "a bit per entry");

// The entry of kCluster32 for a call, the first of those with the same bound,
// or nullptr.
const Cluster32* route32(int device, uint32_t log_n, int kind, uint32_t limbs) {
  const uint64_t placeable = g_placeable32[device].load(std::memory_order_relaxed);
  const auto bound = kind == 3 ? &Cluster32::polymul_upto : (kind == 2 ? &Cluster32::inv_upto : &Cluster32::fwd_upto);
  const Cluster32* best = nullptr;
  for (const Cluster32& r : kCluster32)
    if (r.log_n == log_n && (placeable >> (&r - kCluster32) & 1) && r.*bound >= limbs && (!best || r.*bound < best->*bound)) best = &r;
  return best;
}

template <int... L>
cudaError_t dispatch32(std::integer_sequence<int, L...>, uint32_t log_n, int kind, uint32_t* c, const uint32_t* a,
                       const uint32_t* b, const Limbs32& ls, const DevMod32* mods, cudaStream_t st) {
  cudaError_t e = cudaErrorInvalidValue;
  ((log_n == (uint32_t)(L + kMinLogN32) ? (e = launch32<L + kMinLogN32>(kind, c, a, b, ls, mods, st), 0) : 0), ...);
  return e;
}

template <int... L>
cudaError_t attrs32(std::integer_sequence<int, L...>) {
  cudaError_t e = cudaSuccess;
  ((e = (e == cudaSuccess ? set_attrs32<L + kMinLogN32>() : e)), ...);
  return e;
}

// The degrees of the one-CTA kernels.
using OneCta32 = std::make_integer_sequence<int, kLogMaxOneCta32 - kMinLogN32 + 1>;

int prepare32(uint32_t log_n, uint32_t cm0, uint32_t L, DeviceContext** ctx, const DevMod32** mods) {
  if (log_n < kMinLogN32 || log_n > kLogMaxDegree32)
    return fail(kUnsupportedDegree, "32-bit moduli: log_n must be in [3, 15]");
  if (L == 0 || cm0 >= kMaxModuli32 || L > kMaxModuli32 - cm0)
    return fail(kInvalidModulus, "32-bit moduli: indices must lie in [0, 291)");
  int st = kOk;
  *ctx = DeviceContext::current(&st);
  if (!*ctx) return st;
  {
    static std::mutex mu;
    static std::vector<int> done;
    std::lock_guard<std::mutex> g(mu);
    const int dev = (*ctx)->device();
    if (std::find(done.begin(), done.end(), dev) == done.end()) {
      cudaError_t e = attrs32(OneCta32{});
      for (const Cluster32& r : kCluster32) {
        if (e == cudaSuccess && r.ntt_attrs) e = r.ntt_attrs();
        if (e == cudaSuccess && r.polymul_attrs) e = r.polymul_attrs();
      }
      uint64_t placeable = 0;
      for (size_t i = 0; i < kRoutes32 && e == cudaSuccess; ++i)
        if (kCluster32[i].placeable()) placeable |= uint64_t(1) << i;
      g_placeable32[dev].store(placeable, std::memory_order_relaxed);
      if (e != cudaSuccess) return fail_cuda(e, "32-bit kernel attributes");
      done.push_back(dev);
    }
  }
  return ensure32((*ctx)->device(), log_n, cm0, L, mods);
}

int aligned16(const void* p, const char* what) {
  return reinterpret_cast<uintptr_t>(p) % 16 ? fail(kInvalidArgument, std::string(what) + " is not 16-byte aligned")
                                             : kOk;
}

int run32(int kind, uint32_t* c, const uint32_t* a, const uint32_t* b, uint32_t count, uint32_t L, uint32_t log_n,
          uint32_t cm0, void* stream) {
  DeviceContext* ctx;
  const DevMod32* mods;
  int st = check_limbs(count, L, log_n, nullptr);
  if (st != kOk) return st;
  st = prepare32(log_n, cm0, L, &ctx, &mods);
  if (st != kOk) return st;
  if ((st = aligned16(c, "output")) != kOk) return st;
  if (a && (st = aligned16(a, "a")) != kOk) return st;
  if (b && (st = aligned16(b, "b")) != kOk) return st;
  const Limbs32 ls{count * L, L, cm0};
  cudaStream_t s = stream ? static_cast<cudaStream_t>(stream) : ctx->stream();
  static const char* names[4] = {"ntt32_forward", "ntt32_forward_lazy", "ntt32_backward", "polymul32"};
  LaunchScope ps(names[kind], s);
  const Cluster32* r = route32(ctx->device(), log_n, kind, ls.count);
  const cudaError_t e = !r ? dispatch32(OneCta32{}, log_n, kind, c, a, b, ls, mods, s)
                        : kind == 3 ? r->polymul(c, a, b, ls, mods, s)
                                    : r->ntt(kind, c, ls, mods, s);
  g_kernel_launches += 1;
  return e == cudaSuccess ? kOk : fail_cuda(e, names[kind]);
}

// Host-memory single-limb transform through the staging buffer.
int host_ntt32(int kind, uint32_t* op, uint32_t log_n, uint32_t cm) {
  if (!op) return fail(kInvalidArgument, "null pointer");
  DeviceContext* ctx;
  const DevMod32* mods;
  int st = prepare32(log_n, cm, 1, &ctx, &mods);
  if (st != kOk) return st;
  const size_t n = (size_t)1 << log_n;
  cudaStream_t s = ctx->stream();
  if (log_n <= kSmallCall32LogN) {
    // small call: one launch in place on the mapped host buffer
    std::lock_guard<std::mutex> g(ctx->small.lock);
    st = ctx->small.ensure();
    if (st != kOk) return st;
    uint32_t* h = reinterpret_cast<uint32_t*>(ctx->small.host);
    std::memcpy(h, op, n * 4);
    st = run32(kind, reinterpret_cast<uint32_t*>(ctx->small.dev), nullptr, nullptr, 1, 1, log_n, cm, s);
    if (st != kOk) return st;
    const cudaError_t e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return fail_cuda(e, "synchronize");
    std::memcpy(op, h, n * 4);
    return kOk;
  }
  std::lock_guard<std::mutex> g(ctx->staging.lock);
  st = ctx->staging.reserve(n);
  if (st != kOk) return st;
  uint32_t* d = reinterpret_cast<uint32_t*>(ctx->staging.ptr);
  cudaError_t e = cudaMemcpyAsync(d, op, n * 4, cudaMemcpyHostToDevice, s);
  if (e != cudaSuccess) return fail_cuda(e, "H2D");
  st = run32(kind, d, nullptr, nullptr, 1, 1, log_n, cm, s);
  if (st != kOk) return st;
  e = cudaMemcpyAsync(op, d, n * 4, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  return e == cudaSuccess ? kOk : fail_cuda(e, "D2H");
}

}  // namespace
}  // namespace yell_gb300

using namespace yell_gb300;

extern "C" {

uint32_t yell32_max_moduli(void) { return kMaxModuli32; }
uint32_t yell32_max_log_degree(void) { return kLogMaxDegree32; }
uint32_t yell32_prime(uint32_t cm) { return cm < kMaxModuli32 ? primes32()[cm].p : 0; }
uint32_t yell32_prime_pn(uint32_t cm) { return cm < kMaxModuli32 ? primes32()[cm].pn : 0; }
uint32_t yell32_primitive_root(uint32_t cm) { return cm < kMaxModuli32 ? primes32()[cm].root : 0; }

int yell32_ntt_tables(uint32_t log_n, uint32_t cm, uint32_t* out4n, uint32_t* scalars4) {
  if (!out4n || !scalars4) return fail(kInvalidArgument, "null output");
  if (log_n < 1 || log_n > kLogMaxDegree32) return fail(kUnsupportedDegree, "log_n must be in [1, 15]");
  if (cm >= kMaxModuli32) return fail(kInvalidModulus, "modulus index out of range");
  build_host_tables32(log_n, cm, out4n, scalars4);
  return kOk;
}

int yell32_init_ntt_tables(uint32_t log_n, uint32_t cm0, uint32_t L) {
  DeviceContext* ctx;
  const DevMod32* mods;
  return prepare32(log_n, cm0, L, &ctx, &mods);
}

int yell32_ntt_forward(uint32_t* op, uint32_t log_n, uint32_t cm) { return host_ntt32(0, op, log_n, cm); }
int yell32_ntt_forward_lazy(uint32_t* op, uint32_t log_n, uint32_t cm) { return host_ntt32(1, op, log_n, cm); }
int yell32_ntt_backward(uint32_t* op, uint32_t log_n, uint32_t cm) { return host_ntt32(2, op, log_n, cm); }

int yell32_dev_ntt(uint32_t* d_polys, uint32_t count, uint32_t L, uint32_t log_n, uint32_t cm0, int direction,
                   void* stream) {
  if (!d_polys || count == 0) return fail(kInvalidArgument, "null pointer or zero count");
  if (direction < 0 || direction > 2) return fail(kInvalidArgument, "bad direction");
  return run32(direction, d_polys, nullptr, nullptr, count, L, log_n, cm0, stream);
}

int yell32_dev_polymul(uint32_t* d_c, const uint32_t* d_a, const uint32_t* d_b, uint32_t pairs, uint32_t L,
                       uint32_t log_n, uint32_t cm0, void* stream) {
  if (!d_c || !d_a || !d_b || pairs == 0) return fail(kInvalidArgument, "null pointer or zero pairs");
  if (d_c == d_a || d_c == d_b) return fail(kInvalidArgument, "the product may not overwrite an operand");
  return run32(3, d_c, d_a, d_b, pairs, L, log_n, cm0, stream);
}

int yell32_wait_check(uint64_t timeout_ns, uint32_t* status) {
  if (!status) return fail(kInvalidArgument, "null output");
  if (timeout_ns == 0 || timeout_ns > 10'000'000'000ull) return fail(kInvalidArgument, "timeout must be in (0, 10 s]");
  int st = kOk;
  DeviceContext* ctx = DeviceContext::current(&st);
  if (!ctx) return st;
  k32_wait_check<<<1, 32, 0, ctx->stream()>>>(timeout_ns);
  g_kernel_launches += 1;
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail_cuda(e, "wait check");
  return yell32_wait_status(status);
}

int yell32_wait_status(uint32_t* status) {
  if (!status) return fail(kInvalidArgument, "null output");
  int st = kOk;
  DeviceContext* ctx = DeviceContext::current(&st);
  if (!ctx) return st;
  cudaError_t e = cudaDeviceSynchronize();
  if (e != cudaSuccess) return fail_cuda(e, "synchronize");
  uint32_t v = 0;
  e = cudaMemcpyFromSymbol(&v, g_k32_wait_status, sizeof(v));
  if (e != cudaSuccess) return fail_cuda(e, "read wait status");
  if (v != 0) {
    void* word = nullptr;
    e = cudaGetSymbolAddress(&word, g_k32_wait_status);
    if (e == cudaSuccess) e = upload_zeros(word, sizeof(v));
    if (e != cudaSuccess) return fail_cuda(e, "clear wait status");
  }
  *status = v;
  return kOk;
}

int yell32_dev_elementwise(int op, uint32_t* d_dst, const uint32_t* d_a, const uint32_t* d_b, uint32_t count,
                           uint32_t L, uint32_t log_n, uint32_t cm0, void* stream) {
  if (!d_dst || !d_a || (op != YELL_OP_NEGATE && !d_b) || count == 0)
    return fail(kInvalidArgument, "null pointer or zero count");
  if (op < YELL_OP_MULMOD || op > YELL_OP_NEGATE) return fail(kInvalidArgument, "bad op");
  DeviceContext* ctx;
  const DevMod32* mods;
  int st = check_limbs(count, L, log_n, nullptr);
  if (st != kOk) return st;
  st = prepare32(log_n, cm0, L, &ctx, &mods);
  if (st != kOk) return st;
  cudaStream_t s = stream ? static_cast<cudaStream_t>(stream) : ctx->stream();
  const size_t total = ((size_t)count * L) << log_n;
  const Limbs32 ls{count * L, L, cm0};
  const int grid = (int)std::min<size_t>((total + 255) / 256, 152 * 16);
  LaunchScope ps("elementwise32", s);
  switch (op) {
    case YELL_OP_MULMOD: launch_dependent(k32_elementwise<YELL_OP_MULMOD>, grid, 256, 0, s, d_dst, d_a, d_b, total, log_n, ls, mods); break;
    case YELL_OP_ADDMOD: launch_dependent(k32_elementwise<YELL_OP_ADDMOD>, grid, 256, 0, s, d_dst, d_a, d_b, total, log_n, ls, mods); break;
    case YELL_OP_SUBMOD: launch_dependent(k32_elementwise<YELL_OP_SUBMOD>, grid, 256, 0, s, d_dst, d_a, d_b, total, log_n, ls, mods); break;
    case YELL_OP_MULADD: launch_dependent(k32_elementwise<YELL_OP_MULADD>, grid, 256, 0, s, d_dst, d_a, d_b, total, log_n, ls, mods); break;
    default: launch_dependent(k32_elementwise<YELL_OP_NEGATE>, grid, 256, 0, s, d_dst, d_a, d_b, total, log_n, ls, mods); break;
  }
  g_kernel_launches += 1;
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? kOk : fail_cuda(e, "elementwise32");
}

// ---- host-memory poly<N> drop-ins (limb pointer arrays, moduli 0 .. L-1) ----
// The reference's poly<N> members in 32-bit mode (details/poly.hpp:118-186 and
// the operators of include/yell/poly.hpp:163-168): limbs staged through device memory,
// one launch over all limbs, copied back; synchronous.

static int host_poly32(int kind, int op, uint32_t* const* dst, const uint32_t* const* a, const uint32_t* const* b,
                       uint32_t L, uint32_t log_n) {
  // kind 0..2: NTT of dst in place; kind 3: element-wise op
  if (!dst || L == 0) return fail(kInvalidArgument, "null limb array or zero limbs");
  const bool binary = kind == 3 && op != YELL_OP_NEGATE;
  if (kind == 3 && (!a || (binary && !b))) return fail(kInvalidArgument, "null limb array");
  for (uint32_t l = 0; l < L; ++l)
    if (!dst[l] || (kind == 3 && !a[l]) || (binary && !b[l])) return fail(kInvalidArgument, "null limb pointer");
  DeviceContext* ctx;
  const DevMod32* mods;
  int st = prepare32(log_n, 0, L, &ctx, &mods);
  if (st != kOk) return st;
  const size_t n = (size_t)1 << log_n, w = n * L;
  cudaStream_t s = ctx->stream();
  const bool need_dst = kind != 3 || op == YELL_OP_MULADD;
  if (log_n <= kSmallCall32LogN && w <= 2 * DeviceContext::kSmallCallWords) {
    // small call: the kernel works on the mapped host buffer (three operands
    // of w 32-bit words fit its 3 x kSmallCallWords 64-bit words)
    std::lock_guard<std::mutex> g(ctx->small.lock);
    st = ctx->small.ensure();
    if (st != kOk) return st;
    uint32_t* hd = reinterpret_cast<uint32_t*>(ctx->small.host);
    uint32_t* ha = hd + w;
    uint32_t* hb = ha + w;
    for (uint32_t l = 0; l < L; ++l) {
      if (need_dst) std::memcpy(hd + l * n, dst[l], n * 4);
      if (kind == 3) std::memcpy(ha + l * n, a[l], n * 4);
      if (binary) std::memcpy(hb + l * n, b[l], n * 4);
    }
    uint32_t* vd = reinterpret_cast<uint32_t*>(ctx->small.dev);
    st = kind == 3 ? yell32_dev_elementwise(op, vd, vd + w, binary ? vd + 2 * w : nullptr, 1, L, log_n, 0, s)
                   : run32(kind, vd, nullptr, nullptr, 1, L, log_n, 0, s);
    if (st != kOk) return st;
    const cudaError_t e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return fail_cuda(e, "synchronize");
    for (uint32_t l = 0; l < L; ++l) std::memcpy(dst[l], hd + l * n, n * 4);
    return kOk;
  }
  std::lock_guard<std::mutex> g(ctx->staging.lock);
  st = ctx->staging.reserve((3 * w + 1) / 2);  // three uint32 operands in uint64 words
  if (st != kOk) return st;
  uint32_t* dd = reinterpret_cast<uint32_t*>(ctx->staging.ptr);
  uint32_t* da = dd + w;
  uint32_t* db = da + w;
  cudaError_t e = cudaSuccess;
  for (uint32_t l = 0; l < L && e == cudaSuccess; ++l) {
    if (need_dst) e = cudaMemcpyAsync(dd + l * n, dst[l], n * 4, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess && kind == 3) e = cudaMemcpyAsync(da + l * n, a[l], n * 4, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess && binary) e = cudaMemcpyAsync(db + l * n, b[l], n * 4, cudaMemcpyHostToDevice, s);
  }
  if (e != cudaSuccess) return fail_cuda(e, "H2D limbs");
  st = kind == 3 ? yell32_dev_elementwise(op, dd, da, binary ? db : nullptr, 1, L, log_n, 0, s)
                 : run32(kind, dd, nullptr, nullptr, 1, L, log_n, 0, s);
  if (st != kOk) return st;
  for (uint32_t l = 0; l < L && e == cudaSuccess; ++l)
    e = cudaMemcpyAsync(dst[l], dd + l * n, n * 4, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  return e == cudaSuccess ? kOk : fail_cuda(e, "D2H limbs");
}

int yell32_poly_forward(uint32_t* const* limbs, uint32_t L, uint32_t log_n) {
  return host_poly32(0, 0, limbs, nullptr, nullptr, L, log_n);
}
int yell32_poly_forward_lazy(uint32_t* const* limbs, uint32_t L, uint32_t log_n) {
  return host_poly32(1, 0, limbs, nullptr, nullptr, L, log_n);
}
int yell32_poly_backward(uint32_t* const* limbs, uint32_t L, uint32_t log_n) {
  return host_poly32(2, 0, limbs, nullptr, nullptr, L, log_n);
}
int yell32_poly_mulmod(uint32_t* const* dst, const uint32_t* const* a, const uint32_t* const* b, uint32_t L,
                       uint32_t log_n) {
  return host_poly32(3, YELL_OP_MULMOD, dst, a, b, L, log_n);
}
int yell32_poly_addmod(uint32_t* const* dst, const uint32_t* const* a, const uint32_t* const* b, uint32_t L,
                       uint32_t log_n) {
  return host_poly32(3, YELL_OP_ADDMOD, dst, a, b, L, log_n);
}
int yell32_poly_submod(uint32_t* const* dst, const uint32_t* const* a, const uint32_t* const* b, uint32_t L,
                       uint32_t log_n) {
  return host_poly32(3, YELL_OP_SUBMOD, dst, a, b, L, log_n);
}
int yell32_poly_add_product_of(uint32_t* const* acc, const uint32_t* const* a, const uint32_t* const* b, uint32_t L,
                               uint32_t log_n) {
  return host_poly32(3, YELL_OP_MULADD, acc, a, b, L, log_n);
}
int yell32_poly_negate(uint32_t* const* limbs, uint32_t L, uint32_t log_n) {
  return host_poly32(3, YELL_OP_NEGATE, limbs, limbs, nullptr, L, log_n);
}

}  // extern "C"
