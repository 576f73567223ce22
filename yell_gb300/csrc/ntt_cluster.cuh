// Cluster NTT and fused polymul: one limb per thread-block cluster, for calls
// with few limbs.
//
// The one-tile-per-CTA kernels (ntt_kernels.cuh) give a thread 16 words of a
// 4096-word tile: the fewest exchanges per butterfly, but a call of a few
// limbs then runs on a few SMs, and its two-pass kernels follow one another
// through HBM.  Here a limb of N = 2^LOGN words is split over the 2^CL CTAs
// of one cluster, 2^(LOGN - CL) words each, and a thread holds 2^LOGE = 4 or
// 8 words, so a limb occupies 2^CL SMs and every step of it has a quarter or
// half of the serial work per thread.  Both passes run in one launch: CTA r
// owns columns [r, r + 1) * 2^(LOGB - CL) during the column stages and rows
// [r, r + 1) * 2^(K1 - CL) during the row stages (K1 column stages, rows of
// 2^LOGB words), and the words change owners once per direction through
// distributed shared memory (st.shared::cluster), with a cluster barrier.
// The butterflies, their pairing and their twiddles are the same as
// everywhere else, so the words are too.
//
// What bounds it: at few limbs the latency of the dependent stages and of the
// barriers; once the limbs fill the chip, the 64-bit multiplier, where the
// 16-word tiles win because they exchange less (the bounds in ntt_cluster.cu).
#pragma once
#include <cstdlib>

#include "ntt_kernels.cuh"

namespace yell_gb300 {
namespace {

__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// Shared-window address of `smem_addr` (this CTA's shared::cta address) in
// CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t map_rank(uint32_t smem_addr, uint32_t rank) {
  uint32_t a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_addr), "r"(rank));
  return a;
}
__device__ __forceinline__ void st_cluster(uint32_t addr, uint64_t v) {
  asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(addr), "l"(v) : "memory");
}
__device__ __forceinline__ void st_cluster(uint32_t addr, uint32_t v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void st_cluster2(uint32_t addr, uint32_t v0, uint32_t v1) {
  asm volatile("st.shared::cluster.v2.u32 [%0], {%1, %2};" ::"r"(addr), "r"(v0), "r"(v1) : "memory");
}
__device__ __forceinline__ void st_cluster2(uint32_t addr, uint64_t v0, uint64_t v1) {
  asm volatile("st.shared::cluster.v2.u64 [%0], {%1, %2};" ::"r"(addr), "l"(v0), "l"(v1) : "memory");
}

template <int LOGN_, int K1_, int LOGE_, int CL_, class W_ = uint64_t, int PB_ = 0>
struct ClusterCfg {
  static constexpr int kPolymulBlocks = PB_;  // CTAs per SM that the polymul is compiled for (0: any)
  using W = W_;
  static constexpr int LOGN = LOGN_, K1 = K1_, LOGE = LOGE_, CL = CL_;
  static constexpr int LOGB = LOGN - K1;  // words per row
  static constexpr int T = LOGN - CL;     // words per CTA
  static constexpr int LB = T - K1;       // columns per CTA
  using Col = TileCfg<T, K1, LB, LOGE>;
  using Row = TileCfg<T, LOGB, 0, LOGE>;
  static constexpr int THREADS = Col::THREADS;
  static constexpr uint32_t kTileWords = Smem<W>::words(1u << T);
  static constexpr size_t kTileBytes = kTileWords * sizeof(W);
  static_assert(LB >= 1 && K1 >= CL, "every CTA owns whole columns and whole rows");
};

// Words of column round RG, at tile indices base_v + off (row c of the limb =
// index >> LB), to the CTAs that own their rows.  dst: the receiving tile.
template <class CC, class RG, class W>
__device__ __forceinline__ void send_to_rows(const W* x, const W* dst, uint32_t base_v, uint32_t rank) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
#pragma unroll
  for (int ex = 0; ex < RG::E; ++ex)
#pragma unroll
    for (int j = 0; j < (1 << RG::R); ++j) {
      const uint32_t v = base_v + RG::off(ex, j);
      const uint32_t c = v >> CC::LB, col = (rank << CC::LB) | (v & ((1u << CC::LB) - 1u));
      const uint32_t u = ((c & ((1u << (CC::K1 - CC::CL)) - 1u)) << CC::LOGB) | col;
      st_cluster(map_rank(d + (uint32_t)sizeof(W) * Smem<W>::idx(u), c >> (CC::K1 - CC::CL)), x[(ex << RG::R) | j]);
    }
}

// Words of row round RG, at tile indices base_v + off (column = index mod
// 2^LOGB), to the CTAs that own their columns.
template <class CC, class RG, class W>
__device__ __forceinline__ void send_to_cols(const W* x, const W* dst, uint32_t base_v, uint32_t rank) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  auto address = [&](uint32_t u) {
    const uint32_t col = u & ((1u << CC::LOGB) - 1u);
    const uint32_t c = (rank << (CC::K1 - CC::CL)) | (u >> CC::LOGB);
    return map_rank(d + (uint32_t)sizeof(W) * Smem<W>::idx((c << CC::LB) | (col & ((1u << CC::LB) - 1u))), col >> CC::LB);
  };
  if constexpr (RG::PAIRS) {  // adjacent columns of one CTA (LB >= 1)
#pragma unroll
    for (int m = 0; m < RG::E / 2; ++m)
#pragma unroll
      for (int j = 0; j < (1 << RG::R); ++j)
        st_cluster2(address(base_v + RG::off(2 * m, j)), x[((2 * m) << RG::R) | j], x[((2 * m + 1) << RG::R) | j]);
  } else {
#pragma unroll
    for (int ex = 0; ex < RG::E; ++ex)
#pragma unroll
      for (int j = 0; j < (1 << RG::R); ++j)
        st_cluster(address(base_v + RG::off(ex, j)), x[(ex << RG::R) | j]);
  }
}

// DIR: 0 forward (reduced), 1 forward lazy, 2 backward.  In place: every CTA
// of the cluster has its words in registers or shared memory before the
// cluster barrier, and stores only after it.
template <class CC, int DIR, class LS, class M>
__global__ void __launch_bounds__(CC::THREADS) k_ntt_cluster(LS ls, const M* __restrict__ mods) {
  extern __shared__ __align__(16) uint64_t smem_c[];
  using W = typename CC::W;
  W* smem = reinterpret_cast<W*>(smem_c);
  using Col = typename CC::Col;
  using Row = typename CC::Row;
  constexpr uint32_t log_n = CC::LOGN;
  constexpr int E = 1 << CC::LOGE;
  W* sc = smem;                   // column tile
  W* sr = smem + CC::kTileWords;  // row tile
  cluster_arrive();  // the peers have started: awaited before the first word is sent
  grid_dep_wait();  // as in k_col_pass
  grid_dep_launch();
  const uint32_t tid = threadIdx.x;
  const uint32_t rank = blockIdx.x & ((1u << CC::CL) - 1u);  // of a one-dimensional cluster
  const uint32_t limb = ls.ordered(blockIdx.x >> CC::CL);
  W* data = ls.limb(limb, log_n);
  const M m = load_mod(mods, ls.cm(limb));
  const uint32_t G = (rank << (CC::K1 - CC::CL)) + Row::sub(tid);
  W x[E];
  using C0 = Round<Col, 0>;
  using CL_ = Round<Col, Col::NR - 1>;
  using R0 = Round<Row, 0>;
  using RL = Round<Row, Row::NR - 1>;
  const uint32_t c0 = C0::base(tid), cl = CL_::base(tid), r0 = R0::base(tid), rl = RL::base(tid);
  if constexpr (DIR != 2) {
    gload_cols<C0, CC::LOGB>(x, (const W*)data + (rank << CC::LB), c0);
    ct_round<C0>(x, m.fwd, C0::HI, C0::gr(c0, 0), m.p);
    if constexpr (Col::NR > 1) {
      smem_store<C0>(x, sc, c0);
      __syncthreads();
      fwd_rounds<Col, 1, Col::NR - 1>(sc, tid, 0, 0, m.fwd, m.p, true);
      smem_load<CL_>(x, sc, cl);
      ct_round<CL_>(x, m.fwd, CL_::HI, CL_::gr(cl, 0), m.p);
    }
    cluster_wait();
    send_to_rows<CC, CL_>(x, sr, cl, rank);
    cluster_arrive();
    cluster_wait();
    fwd_rounds<Row, 0, Row::NR - 1, Row::LOCAL_BARRIER>(sr, tid, CC::K1, G, m.fwd, m.p, true);
    smem_load<RL>(x, sr, rl);
    ct_round<RL>(x, m.fwd, CC::K1 + RL::HI, RL::gr(rl, G), m.p);
    if constexpr (DIR == 0) {
#pragma unroll
      for (int i = 0; i < E; ++i) x[i] = fwd_correct(x[i], m.p, (W)(m.p << 1));
    }
    gstore_rows<RL>(x, data + ((size_t)rank << CC::T), rl);
  } else {
    gload_rows<RL>(x, (const W*)data + ((size_t)rank << CC::T), rl);
    gs_round<RL, false>(x, log_n, RL::BETA, RL::gr(rl, G), m);
    if constexpr (Row::NR > 1) {
      smem_store<RL>(x, sr, rl);
      round_barrier<Row, Row::LOCAL_BARRIER>(tid);
      inv_rounds<Row, Row::NR - 2, 0, false, Row::LOCAL_BARRIER>(sr, tid, log_n, 0, G, m, true);
      smem_load<R0>(x, sr, r0);
      gs_round<R0, false>(x, log_n, R0::BETA, R0::gr(r0, G), m);
    }
    cluster_wait();
    send_to_cols<CC, R0>(x, sc, r0, rank);
    cluster_arrive();
    cluster_wait();
    inv_rounds<Col, Col::NR - 1, 0, false>(sc, tid, log_n, CC::LOGB, 0, m, true);
    smem_load<C0>(x, sc, c0);
    gs_round<C0, true>(x, log_n, CC::LOGB + C0::BETA, C0::gr(c0, 0), m);
    gstore_cols<C0, CC::LOGB>(x, data + (rank << CC::LB), c0);
  }
}

// c = INTT(NTT(a) * NTT(b)) per limb, without scratch.
template <class CC, class LS, class CLS, class M>
__global__ void __launch_bounds__(CC::THREADS, CC::kPolymulBlocks)
    k_polymul_cluster(LS c, CLS a, CLS b, const M* __restrict__ mods) {
  extern __shared__ __align__(16) uint64_t smem_c[];
  using W = typename CC::W;
  W* smem = reinterpret_cast<W*>(smem_c);
  using Col = typename CC::Col;
  using Row = typename CC::Row;
  constexpr uint32_t log_n = CC::LOGN;
  constexpr int E = 1 << CC::LOGE;
  constexpr uint32_t TW = CC::kTileWords;
  constexpr int BK = Row::LOCAL_BARRIER;
  W *sa = smem, *sb = smem + TW;              // column tiles
  W *ra = smem + 2 * TW, *rb = smem + 3 * TW;  // row tiles
  cluster_arrive();
  grid_dep_wait();  // as in k_col_pass
  grid_dep_launch();
  const uint32_t tid = threadIdx.x;
  const uint32_t rank = blockIdx.x & ((1u << CC::CL) - 1u);
  const uint32_t limb = c.ordered(blockIdx.x >> CC::CL);
  const M m = load_mod(mods, c.cm(limb));
  const W np = (W)(0 - m.p), p2 = (W)(m.p << 1);
  const uint32_t G = (rank << (CC::K1 - CC::CL)) + Row::sub(tid);
  W xa[E], xb[E];
  using C0 = Round<Col, 0>;
  using CL_ = Round<Col, Col::NR - 1>;
  using R0 = Round<Row, 0>;
  using RB = Round<Row, Row::NR - 1>;
  const uint32_t c0 = C0::base(tid), cl = CL_::base(tid), r0 = R0::base(tid), rb0 = RB::base(tid);
  gload_cols<C0, CC::LOGB>(xa, a.limb(limb, log_n) + (rank << CC::LB), c0);
  gload_cols<C0, CC::LOGB>(xb, b.limb(limb, log_n) + (rank << CC::LB), c0);
  ct_stages2<C0::R, C0::E>(xa, xb, m.fwd, C0::HI, C0::gr(c0, 0), np, p2);
  if constexpr (Col::NR > 1) {
    smem_store<C0>(xa, sa, c0);
    smem_store<C0>(xb, sb, c0);
    __syncthreads();
    fwd_rounds2<Col, 1, Col::NR - 1>(sa, sb, tid, 0, 0, m.fwd, m.p, true);
    smem_load<CL_>(xa, sa, cl);
    smem_load<CL_>(xb, sb, cl);
    ct_stages2<CL_::R, CL_::E>(xa, xb, m.fwd, CL_::HI, CL_::gr(cl, 0), np, p2);
  }
  cluster_wait();
  send_to_rows<CC, CL_>(xa, ra, cl, rank);
  send_to_rows<CC, CL_>(xb, rb, cl, rank);
  cluster_arrive();
  const auto w0 = fused_w0<Row>(rb0, CC::K1, G, m);
  cluster_wait();
  fwd_rounds2<Row, 0, Row::NR - 1, BK>(ra, rb, tid, CC::K1, G, m.fwd, m.p, true);
  smem_load<RB>(xa, ra, rb0);
  smem_load<RB>(xb, rb, rb0);
  fused_product<Row, false>(xa, xb, rb0, log_n, CC::K1, G, m, w0);
  if constexpr (Row::NR > 1) {
    smem_store<RB>(xa, ra, rb0);
    round_barrier<Row, BK>(tid);
    inv_rounds<Row, Row::NR - 2, 0, false, BK>(ra, tid, log_n, 0, G, m, true);
    smem_load<R0>(xa, ra, r0);
    gs_round<R0, false>(xa, log_n, R0::BETA, R0::gr(r0, G), m);
  }
  // the column tiles are free: every CTA of the cluster is past its column stages
  send_to_cols<CC, R0>(xa, sa, r0, rank);
  cluster_arrive();
  cluster_wait();
  inv_rounds<Col, Col::NR - 1, 0, false>(sa, tid, log_n, CC::LOGB, 0, m, true);
  smem_load<C0>(xa, sa, c0);
  gs_round<C0, true>(xa, log_n, CC::LOGB + C0::BETA, C0::gr(c0, 0), m);
  gstore_cols<C0, CC::LOGB>(xa, c.limb(limb, log_n) + (rank << CC::LB), c0);
}

// Whether the current device can place a cluster of the kernel's CTAs: a small
// partition may have no 8 SMs side by side.  YELL_GB300_MAX_CLUSTER bounds the
// clusters of a process that shares its device with other work.
template <class CC, typename... KArgs>
bool cluster_placeable(void (*kernel)(KArgs...), size_t smem) {
  const char* bound = std::getenv("YELL_GB300_MAX_CLUSTER");
  if (bound && *bound && std::atoi(bound) < (1 << CC::CL)) return false;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1u << CC::CL;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(1u << CC::CL);
  cfg.blockDim = dim3(CC::THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int clusters = 0;
  if (cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) != cudaSuccess) {
    (void)cudaGetLastError();
    return false;
  }
  return clusters > 0;
}

// Launch of a cluster kernel, as a programmatic dependent like the two-pass
// kernels.
template <class CC, typename... KArgs, typename... Args>
void launch_cluster(void (*kernel)(KArgs...), uint32_t limbs, size_t smem, cudaStream_t st, Args... args) {
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1u << CC::CL;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(limbs << CC::CL);
  cfg.blockDim = dim3(CC::THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = g_dependent_launches ? 2 : 1;
  (void)cudaLaunchKernelEx(&cfg, kernel, args...);  // errors surface through cudaGetLastError
}

template <class CC>
cudaError_t launch_cluster_ntt(const LimbSet& ls, const DevMod* mods, NttDir dir, cudaStream_t st) {
  LaunchScope ps(dir == NttDir::kBackward ? "ntt_cluster_inv" : "ntt_cluster_fwd", st);
  switch (dir) {
    case NttDir::kForward: launch_cluster<CC>(k_ntt_cluster<CC, 0, LimbSet, DevMod>, ls.count, 2 * CC::kTileBytes, st, ls, mods); break;
    case NttDir::kForwardLazy:
      launch_cluster<CC>(k_ntt_cluster<CC, 1, LimbSet, DevMod>, ls.count, 2 * CC::kTileBytes, st, ls, mods);
      break;
    case NttDir::kBackward: launch_cluster<CC>(k_ntt_cluster<CC, 2, LimbSet, DevMod>, ls.count, 2 * CC::kTileBytes, st, ls, mods); break;
  }
  g_kernel_launches += 1;
  return cudaGetLastError();
}

template <class CC>
cudaError_t launch_cluster_polymul(const LimbSet& c, const ConstLimbSet& a, const ConstLimbSet& b, const DevMod* mods,
                                   uint64_t*, uint64_t* const*, cudaStream_t st) {
  mods += kPolymulConsts;  // the fused polymul's copy of the constants
  LaunchScope ps("polymul_cluster", st);
  launch_cluster<CC>(k_polymul_cluster<CC, LimbSet, ConstLimbSet, DevMod>, c.count, 4 * CC::kTileBytes, st, c, a, b, mods);
  g_kernel_launches += 1;
  return cudaGetLastError();
}

template <class CC>
cudaError_t set_attrs_cluster() {
  constexpr size_t ntt = 2 * CC::kTileBytes, polymul = 4 * CC::kTileBytes;
  cudaError_t e;
  if ((e = set_smem(k_ntt_cluster<CC, 0, LimbSet, DevMod>, ntt)) != cudaSuccess) return e;
  if ((e = set_smem(k_ntt_cluster<CC, 1, LimbSet, DevMod>, ntt)) != cudaSuccess) return e;
  if ((e = set_smem(k_ntt_cluster<CC, 2, LimbSet, DevMod>, ntt)) != cudaSuccess) return e;
  return set_smem(k_polymul_cluster<CC, LimbSet, ConstLimbSet, DevMod>, polymul);
}

template <class CC>
bool cluster_variant_placeable() {
  return cluster_placeable<CC>(k_ntt_cluster<CC, 0, LimbSet, DevMod>, 2 * CC::kTileBytes) &&
         cluster_placeable<CC>(k_polymul_cluster<CC, LimbSet, ConstLimbSet, DevMod>, 4 * CC::kTileBytes);
}

template <int LOGN, int K1, int LOGE, int CL>
Variant cluster_variant() {
  using CC = ClusterCfg<LOGN, K1, LOGE, CL>;
  Variant v;
  std::snprintf(v.name, sizeof(v.name), "cluster of %d k1=%d (%d threads, %d words per thread)", 1 << CL, K1,
                CC::THREADS, 1 << LOGE);
  v.ntt = &launch_cluster_ntt<CC>;
  v.polymul = &launch_cluster_polymul<CC>;
  v.set_attrs = &set_attrs_cluster<CC>;
  v.placeable = &cluster_variant_placeable<CC>;
  v.ntt_launches = 1;
  v.polymul_launches = 1;
  v.tile_log = CC::T;
  return v;
}

}  // namespace
}  // namespace yell_gb300
