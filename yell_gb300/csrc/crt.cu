// RNS -> big-integer lifting (CRT) on the device: gmp::poly2mpz of the
// reference (include/yell/gmp.hpp:42-70, tables lib/gmp.cpp:6-51).
//
// For residues r_j mod q_j (j < L), the lifted value is the unique
// x in [0, Q), Q = prod q_j, with x = r_j mod q_j.  The reference sums
// r_j * lift_j (lift_j = ((Q/q_j)^-1 mod q_j) * Q/q_j) and reduces the sum mod
// Q with a Shoup quotient; for residues below their moduli that returns x.
// Here, per coefficient:
//   y_j = r_j * ((Q/q_j)^-1 mod q_j) mod q_j          (Shoup product, exact)
//   v   = floor(sum_j y_j / q_j), estimated with 64-bit fractions
//         f_j = floor(y_j * floor(2^125 / q_j) / 2^61); the estimate is v or v - 1
//   x   = sum_j y_j * (Q/q_j) - v * Q, minus Q once more when still >= Q
// sum_j y_j * (Q/q_j) = Q * sum_j y_j / q_j, so with the exact v this is x.
// With 4 to 32 moduli the sums run on the tensor cores (crt_mma.cuh).  Below
// and above that the multi-word sums run over 32-bit digits: a thread owns one
// coefficient
// and keeps its y_j in shared memory; the cofactor digits are staged per tile
// of output digits and shared by the block; x is written as W little-endian
// words per coefficient, W = words of Q, coefficient-major.
#include <cstring>
#include <map>
#include <memory>
#include <tuple>
#include <mutex>
#include <set>
#include <utility>
#include <vector>

#include "common.cuh"
#include "crt_mma.cuh"
#include "kernels.h"
#include "profiler.h"
#include "runtime.h"
#include "yell_gb300.h"

using namespace yell_gb300;

namespace {

typedef unsigned __int128 u128;

constexpr uint32_t kMmaMinModuli = 4;    // see crt_lift
constexpr uint32_t kCrtMaxModuli = 400;  // 32 threads * 400 words * 8 B = 100 KB of y per block

// Per (device, cm0, L) constants, device resident:
//   mods[j] = {q_j, inv_j, inv_j', c_j} with inv_j = (Q/q_j)^-1 mod q_j, inv_j' its
//   Shoup companion floor(inv_j * 2^64 / q_j), c_j = floor(2^125 / q_j);
//   words[j * W + w] = word w of Q/q_j; qwords[w] = word w of Q.
struct CrtConst {
  uint64_t q, inv, inv_s, c;
};

struct CrtTables {
  uint32_t W = 0;
  CrtConst* mods = nullptr;
  uint64_t* cofactors = nullptr;
  uint64_t* q = nullptr;
  // the tensor-core kernel's (kMmaMinModuli <= L <= crt_mma::kMaxL)
  crt_mma::Mod* mma_mods = nullptr;
  uint4* image = nullptr;
};

// Host big integers: little-endian 64-bit words.
using Big = std::vector<uint64_t>;

void big_mul_small(Big& a, uint64_t m) {
  uint64_t carry = 0;
  for (uint64_t& w : a) {
    const u128 t = (u128)w * m + carry;
    w = (uint64_t)t;
    carry = (uint64_t)(t >> 64);
  }
  if (carry) a.push_back(carry);
}

// a / m (exact or not), remainder returned.
uint64_t big_divmod_small(const Big& a, uint64_t m, Big* quot) {
  quot->assign(a.size(), 0);
  u128 rem = 0;
  for (size_t i = a.size(); i-- > 0;) {
    const u128 cur = (rem << 64) | a[i];
    (*quot)[i] = (uint64_t)(cur / m);
    rem = cur % m;
  }
  while (!quot->empty() && quot->back() == 0) quot->pop_back();
  return (uint64_t)rem;
}

uint64_t pow_mod(uint64_t b, uint64_t e, uint64_t m) {
  uint64_t r = 1;
  b %= m;
  while (e) {
    if (e & 1) r = (uint64_t)((u128)r * b % m);
    b = (uint64_t)((u128)b * b % m);
    e >>= 1;
  }
  return r;
}

// The first D balanced base-256 digits (-128 .. 127) of a modulo 256^D.
std::vector<int> balanced_digits(const Big& a, uint32_t D) {
  std::vector<int> out(D, 0);
  int carry = 0;
  for (uint32_t d = 0; d < D; ++d) {
    const int byte = d / 8 < a.size() ? (int)((a[d / 8] >> (8 * (d % 8))) & 255u) : 0;
    int v = byte + carry;
    carry = v > 127 ? 1 : 0;
    out[d] = v - 256 * carry;
  }
  return out;
}

// An integer of magnitude below 2048 * 2 as a 16-bit float (exact).
uint16_t f16_bits(int v) {
  if (v == 0) return 0;
  const uint32_t sign = v < 0 ? 0x8000u : 0u;
  uint32_t m = (uint32_t)(v < 0 ? -v : v), e = 0;
  while ((m >> e) > 1) ++e;  // 2^e <= m
  return (uint16_t)(sign | ((e + 15) << 10) | ((e <= 10 ? m << (10 - e) : m >> (e - 10)) & 0x3FFu));
}

// The constant matrix of the tensor-core kernel in its shared-memory layout:
// column d, row (j, i) = digit d of (Q/q_j) * 256^i, eight moduli per chunk;
// the tail's rows are the digits of -Q (factor v), 3072 (factor 4096) and
// (factor 1) the digits of minus what the accumulators' offset and the bit
// patterns' exponents add to the epilogue's sum, modulo 256^D: 2^22 at every
// digit and 0x4B000000 at digits 0 and 2 of every four.
std::vector<uint8_t> mma_image(uint32_t L, uint32_t W, const std::vector<uint64_t>& cof, const Big& Q) {
  using namespace crt_mma;
  const uint32_t N = columns(W), D = 8 * W;
  std::vector<uint8_t> img(image_bytes(L, N), 0);
  auto put = [&](size_t at, int v) {
    const uint16_t h = f16_bits(v);
    std::memcpy(img.data() + at, &h, 2);
  };
  for (uint32_t j = 0; j < L; ++j) {
    const Big c(cof.begin() + (size_t)j * W, cof.begin() + (size_t)(j + 1) * W);
    const std::vector<int> dig = balanced_digits(c, D);
    const size_t chunk = (size_t)(j / kChunkMods) * image_chunk(N);
    for (uint32_t i = 0; i < 8; ++i)
      for (uint32_t d = i; d < D; ++d)
        put(chunk + swizzle128(d * 128 + ((j % kChunkMods) * 8 + i) * 2), dig[d - i]);
  }
  const size_t tail = (size_t)chunks(L) * image_chunk(N);
  Big neg(W), off(W);
  uint64_t borrow = 0, carry = 0;
  std::vector<uint64_t> sums(D + 8, 0);
  for (uint32_t d = 0; d < D; ++d) {
    sums[d + 2] += 0x40;                     // 2^22 = 0x40 * 256^2
    if (d % 2 == 0) sums[d + 3] += 0x4B;     // 0x4B000000 = 0x4B * 256^3
  }
  for (uint32_t w = 0; w < W; ++w) {
    uint64_t word = 0;
    for (uint32_t k = 0; k < 8; ++k) {
      carry += sums[8 * w + k];
      word |= (carry & 255u) << (8 * k);
      carry >>= 8;
    }
    off[w] = word;
  }
  auto negate = [&](const Big& a, Big* out) {
    borrow = 0;
    for (uint32_t w = 0; w < W; ++w) {
      const uint64_t v = w < a.size() ? a[w] : 0;
      (*out)[w] = 0 - v - borrow;
      borrow = (v | borrow) ? 1 : 0;
    }
  };
  negate(Q, &neg);
  const std::vector<int> nq = balanced_digits(neg, D);
  Big noff(W);
  negate(off, &noff);
  for (uint32_t d = 0; d < N; ++d) {
    put(tail + swizzle32(d * 32), d < D ? nq[d] : 0);
    put(tail + swizzle32(d * 32 + 2), 3072);
    put(tail + swizzle32(d * 32 + 4), d < D ? (int)((noff[d / 8] >> (8 * (d % 8))) & 255u) : 0);
  }
  return img;
}

int build_crt_tables(uint32_t cm0, uint32_t L, CrtTables* t) {
  Big Q{1};
  for (uint32_t j = 0; j < L; ++j) big_mul_small(Q, prime_entry(cm0 + j).p);
  const uint32_t W = (uint32_t)Q.size();
  std::vector<CrtConst> mods(L);
  std::vector<uint64_t> cof((size_t)L * W, 0);
  for (uint32_t j = 0; j < L; ++j) {
    const uint64_t q = prime_entry(cm0 + j).p;
    Big m;
    const uint64_t rem = big_divmod_small(Q, q, &m);
    if (rem != 0) return fail(kInvalidArgument, "CRT: modulus does not divide the product");
    uint64_t mq;
    {
      Big unused;
      mq = big_divmod_small(m, q, &unused);
    }
    const uint64_t inv = pow_mod(mq, q - 2, q);  // q prime
    mods[j].q = q;
    mods[j].inv = inv;
    mods[j].inv_s = (uint64_t)(((u128)inv << 64) / q);
    mods[j].c = (uint64_t)(((u128)1 << 125) / q);
    for (size_t w = 0; w < m.size(); ++w) cof[(size_t)j * W + w] = m[w];
  }
  cudaError_t e = lib_malloc(&t->mods, L * sizeof(CrtConst));
  if (e == cudaSuccess) e = lib_malloc(&t->cofactors, cof.size() * 8);
  if (e == cudaSuccess) e = lib_malloc(&t->q, (size_t)W * 8);
  if (e == cudaSuccess) e = upload(t->mods, mods.data(), L * sizeof(CrtConst));
  if (e == cudaSuccess) e = upload(t->cofactors, cof.data(), cof.size() * 8);
  if (e == cudaSuccess) e = upload(t->q, Q.data(), (size_t)W * 8);
  if (e == cudaSuccess && L >= kMmaMinModuli && L <= crt_mma::kMaxL) {
    std::vector<crt_mma::Mod> mm(L);
    for (uint32_t j = 0; j < L; ++j)
      mm[j] = {mods[j].q, mods[j].inv, mods[j].inv_s, (int64_t)(((u128)1 << 88) / mods[j].q)};
    const std::vector<uint8_t> img = mma_image(L, W, cof, Q);
    e = lib_malloc(&t->mma_mods, L * sizeof(crt_mma::Mod));
    if (e == cudaSuccess) e = lib_malloc(&t->image, img.size());
    if (e == cudaSuccess)
      e = upload(t->mma_mods, mm.data(), L * sizeof(crt_mma::Mod));
    if (e == cudaSuccess) e = upload(t->image, img.data(), img.size());
  }
  if (e != cudaSuccess) {
    cudaFree(t->mods);
    cudaFree(t->cofactors);
    cudaFree(t->q);
    cudaFree(t->mma_mods);
    cudaFree(t->image);
    return fail_cuda(e, "CRT tables");
  }
  t->W = W;
  return kOk;
}

int crt_tables(int device, uint32_t cm0, uint32_t L, const CrtTables** out) {
  static std::mutex mu;
  static std::map<std::tuple<int, uint32_t, uint32_t>, CrtTables> cache;
  std::lock_guard<std::mutex> g(mu);
  const auto key = std::make_tuple(device, cm0, L);
  auto it = cache.find(key);
  if (it == cache.end()) {
    CrtTables t;
    const int st = build_crt_tables(cm0, L, &t);
    if (st != kOk) return st;
    it = cache.emplace(key, t).first;
  }
  *out = &it->second;
  return kOk;
}

uint32_t crt_words(uint32_t cm0, uint32_t L) {
  // bits of Q = sum of bit lengths, up to one less per product; exact count
  // from the product itself (cheap on the host).
  Big Q{1};
  for (uint32_t j = 0; j < L; ++j) big_mul_small(Q, prime_entry(cm0 + j).p);
  return (uint32_t)Q.size();
}

// 32-bit digit d of a little-endian word array of `words` words (0 outside).
__device__ __forceinline__ uint32_t digit(const uint64_t* w, int d, uint32_t words) {
  return (d >= 0 && (uint32_t)d < 2 * words) ? __ldg(reinterpret_cast<const uint32_t*>(w) + d) : 0u;
}

// (r0, r1, r2) += a * b, a 64-bit product into a 96-bit accumulator.
__device__ __forceinline__ void mac32(uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t a, uint32_t b) {
  asm("mad.lo.cc.u32 %0, %3, %4, %0;\n\t"
      "madc.hi.cc.u32 %1, %3, %4, %1;\n\t"
      "addc.u32 %2, %2, 0;"
      : "+r"(r0), "+r"(r1), "+r"(r2)
      : "r"(a), "r"(b));
}

// d = a - b - bin (32-bit), returns the borrow out.
__device__ __forceinline__ uint32_t sub_borrow32(uint32_t a, uint32_t b, uint32_t bin, uint32_t* d) {
  const uint32_t t = a - b;
  *d = t - bin;
  return (uint32_t)(a < b) | (uint32_t)(t < bin);
}

__device__ __forceinline__ uint32_t sub_borrow(uint64_t a, uint64_t b, uint32_t bin, uint64_t* d) {
  const uint64_t t = a - b;
  *d = t - bin;
  return (uint32_t)(a < b) | (uint32_t)(t < (uint64_t)bin);
}

// Output digits are produced in tiles of kDigitTile 32-bit digits.  For one
// tile the block stages digits [e0 - 1, e0 + kDigitTile) of every cofactor in
// shared memory; each thread then runs over j once, adding
// y_j[0] * C_j[d] + y_j[1] * C_j[d - 1] into one 96-bit accumulator per digit
// d of the tile (independent chains), and finally resolves the carries digit
// by digit, subtracting v * Q on the way.
constexpr int kDigitTile = 8;  // 8: 72 registers, 0.77 ms at L = 32; 16: 114 registers, 0.87 ms

template <int T>
__global__ void __launch_bounds__(T) k_crt_lift(uint64_t* out, const uint64_t* in,
                                                uint32_t count, uint32_t L, uint32_t log_n,
                                                const CrtConst* __restrict__ mods, const uint64_t* __restrict__ cof,
                                                const uint64_t* __restrict__ qw, uint32_t W) {
  extern __shared__ __align__(16) uint64_t smem_crt[];
  uint64_t* ys = smem_crt;                                          // [L][T]
  uint32_t* cs = reinterpret_cast<uint32_t*>(smem_crt + (size_t)L * T);  // [L][kDigitTile + 1]
  constexpr int CT = kDigitTile + 1;
  grid_dep_wait();  // the caller's words are read and written below
  grid_dep_launch();
  const uint64_t coeffs = (uint64_t)count << log_n;
  const uint64_t g = (uint64_t)blockIdx.x * T + threadIdx.x;
  const bool live = g < coeffs;
  const uint64_t poly = g >> log_n;
  const uint64_t i = g & ((1ull << log_n) - 1);
  const uint64_t n = 1ull << log_n;

  // y_j and the 64-bit-fraction sum of y_j / q_j
  uint64_t f_lo = 0, f_hi = 0;
  for (uint32_t j = 0; j < L; ++j) {
    uint64_t y = 0;
    if (live) {
      const CrtConst m = mods[j];
      y = mulmod_shoup(in[(poly * L + j) * n + i], m.inv, m.inv_s, m.q);
      const uint64_t pl = y * m.c, ph = __umul64hi(y, m.c);
      const uint64_t f = (pl >> 61) | (ph << 3);  // floor(y c / 2^61) < 2^64
      asm("add.cc.u64 %0, %0, %2;\n\taddc.u64 %1, %1, 0;" : "+l"(f_lo), "+l"(f_hi) : "l"(f));
    }
    ys[j * T + threadIdx.x] = y;
  }
  const uint64_t v = f_hi;
  const uint32_t v0 = (uint32_t)v, v1 = (uint32_t)(v >> 32);

  uint64_t* dst = out + g * W;
  const int digits = 2 * (int)W + 2;  // two digits past Q for the borrow chains
  uint64_t cx = 0, cq = 0;            // carries of sum y_j (Q/q_j) and of v Q, in digits
  uint32_t br = 0, bq = 0, lo_digit = 0;
  for (int e0 = 0; e0 < digits; e0 += kDigitTile) {
    __syncthreads();  // previous tile's cofactor digits are no longer read
    for (uint32_t k = threadIdx.x; k < L * CT; k += T) {
      const uint32_t j = k / CT;
      const int d = e0 - 1 + (int)(k - j * CT);
      cs[k] = digit(cof + (size_t)j * W, d, W);
    }
    __syncthreads();
    if (live) {
      uint32_t r0[kDigitTile], r1[kDigitTile], r2[kDigitTile];
#pragma unroll
      for (int t = 0; t < kDigitTile; ++t) r0[t] = r1[t] = r2[t] = 0;
      for (uint32_t j = 0; j < L; ++j) {
        const uint64_t y = ys[j * T + threadIdx.x];
        const uint32_t y0 = (uint32_t)y, y1 = (uint32_t)(y >> 32);
        const uint32_t* c = cs + j * CT;  // c[t + 1] = C_j[e0 + t]
        uint32_t prev = c[0];
#pragma unroll
        for (int t = 0; t < kDigitTile; ++t) {
          const uint32_t cur = c[t + 1];
          mac32(r0[t], r1[t], r2[t], y0, cur);
          mac32(r0[t], r1[t], r2[t], y1, prev);
          prev = cur;
        }
      }
#pragma unroll
      for (int t = 0; t < kDigitTile; ++t) {
        const int d = e0 + t;
        if (d < digits) {
          // x digit: accumulator + carry
          uint64_t xl = ((uint64_t)r1[t] << 32 | r0[t]);
          const uint64_t s = xl + cx;
          const uint64_t xh = (uint64_t)r2[t] + (s < xl ? 1u : 0u);
          const uint32_t xd = (uint32_t)s;
          cx = (s >> 32) | (xh << 32);
          // (v Q) digit
          const uint32_t qd0 = digit(qw, d, W), qd1 = digit(qw, d - 1, W);
          const uint64_t pq = (uint64_t)v0 * qd0, pq2 = (uint64_t)v1 * qd1;
          const uint64_t sq = pq + pq2;
          const uint64_t sq2 = sq + cq;
          const uint64_t qh = (uint64_t)(sq < pq) + (uint64_t)(sq2 < sq);
          const uint32_t qd = (uint32_t)sq2;
          cq = (sq2 >> 32) | (qh << 32);
          uint32_t rd, ad;
          br = sub_borrow32(xd, qd, br, &rd);
          bq = sub_borrow32(rd, qd0, bq, &ad);
          if (d < 2 * (int)W) {
            if (d & 1) dst[d >> 1] = (uint64_t)rd << 32 | lo_digit;
            else lo_digit = rd;
          }
        }
      }
    }
  }
  if (live && bq == 0) {  // x - vQ >= Q: the estimate of v was one short
    uint32_t b = 0;
    for (uint32_t w = 0; w < W; ++w) {
      uint64_t d;
      b = sub_borrow(dst[w], __ldg(&qw[w]), b, &d);
      dst[w] = d;
    }
  }
}

size_t crt_smem(uint32_t L, int threads) {
  return (size_t)L * threads * sizeof(uint64_t) + (size_t)L * (kDigitTile + 1) * sizeof(uint32_t);
}

// First status of a bounded wait of the tensor-core kernel, for the lifts of
// device arrays; a host call has a word of its own.
__device__ uint32_t g_crt_wait_status;

cudaError_t launch_crt_mma(uint64_t* d_out, const uint64_t* d_in, uint64_t coeffs, uint32_t L, uint32_t log_n,
                           const CrtTables* t, cudaStream_t st, int device, uint32_t* own_status) {
  using namespace crt_mma;
  static constexpr decltype(&k_crt_mma<1>) kKernels[] = {k_crt_mma<1>, k_crt_mma<2>, k_crt_mma<3>, k_crt_mma<4>};
  static_assert(sizeof(kKernels) / sizeof(kKernels[0]) == chunks(kMaxL), "a kernel per number of chunks");
  static std::mutex mu;
  static std::map<int, std::pair<uint32_t, uint32_t*>> devices;  // SMs and the status word's address
  uint32_t sms = 0;
  uint32_t* status = own_status;
  {
    std::lock_guard<std::mutex> g(mu);
    auto it = devices.find(device);
    if (it == devices.end()) {
      int n = 0;
      void* p = nullptr;
      cudaError_t e = cudaSuccess;
      for (auto k : kKernels)
        if (e == cudaSuccess)
          e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes(kMaxL, 256));
      if (e == cudaSuccess) e = cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device);
      if (e == cudaSuccess) e = cudaGetSymbolAddress(&p, g_crt_wait_status);
      if (e != cudaSuccess) return e;
      it = devices.emplace(device, std::make_pair((uint32_t)n, static_cast<uint32_t*>(p))).first;
    }
    sms = it->second.first;
    if (!status) status = it->second.second;
  }
  const uint64_t tiles = (coeffs + kRows - 1) / kRows;
  const uint32_t grid = (uint32_t)(tiles < sms ? tiles : sms);
  LaunchScope ps("crt_lift_mma", st);
  launch_dependent(kKernels[chunks(L) - 1], grid, kThreads, smem_bytes(L, columns(t->W)), st, d_out, d_in, coeffs, L, log_n,
                   (const Mod*)t->mma_mods, (const uint4*)t->image, (const uint64_t*)t->q, t->W, status);
  g_kernel_launches += 1;
  return cudaGetLastError();
}

// Reads a word that waits are recorded in, after the work queued on `st`, and
// clears it.
cudaError_t take_status(uint32_t* word, cudaStream_t st, uint32_t* status) {
  uint32_t v = 0;
  cudaError_t e = cudaMemcpyAsync(&v, word, sizeof(v), cudaMemcpyDeviceToHost, st);
  const cudaError_t se = cudaStreamSynchronize(st);  // v is written until then
  if (e == cudaSuccess) e = se;
  if (e == cudaSuccess && v != 0) {
    e = cudaMemsetAsync(word, 0, sizeof(v), st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  }
  *status = v;
  return e;
}

// own_status: the word of device memory that a wait of the tensor-core kernel
// which runs out is recorded in, nullptr for the device's.
int crt_lift(uint64_t* d_out, const uint64_t* d_in, uint32_t count, uint32_t L, uint32_t log_n, uint32_t cm0,
             cudaStream_t st, int device, uint32_t* own_status) {
  const CrtTables* t = nullptr;
  int s = crt_tables(device, cm0, L, &t);
  if (s != kOk) return s;
  // From 4 moduli up the tensor-core kernel is the faster one at every number
  // of coefficients (GB300, us, digit kernel -> tensor cores: 2^20
  // coefficients, L = 3: 33 -> 41, 4: 53 -> 38, 8: 117 -> 47, 16: 286 -> 78,
  // 32: 762 -> 137; 2^13, L = 3: 3.7 -> 4.1, 32: 35 -> 5.7); its digits are exact
  // up to kMaxL moduli.
  if (t->image) {
    const cudaError_t me = launch_crt_mma(d_out, d_in, (uint64_t)count << log_n, L, log_n, t, st, device, own_status);
    return me == cudaSuccess ? kOk : fail_cuda(me, "crt_lift");
  }
  // 64 threads per block while their y_j fit in 160 KB of shared memory, else 32
  // (128-thread blocks measured 2% slower at L = 32)
  const int threads = crt_smem(L, 64) <= (160u << 10) ? 64 : 32;
  const size_t smem = crt_smem(L, threads);
  cudaError_t e = cudaSuccess;
  {
    // the shared-memory limit is a per-device attribute of each kernel
    static std::mutex mu;
    static std::set<int> done;
    std::lock_guard<std::mutex> g(mu);
    if (!done.count(device)) {
      e = cudaFuncSetAttribute(k_crt_lift<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(160u << 10));
      if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_crt_lift<32>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)crt_smem(kCrtMaxModuli, 32));
      if (e != cudaSuccess) return fail_cuda(e, "crt attributes");
      done.insert(device);
    }
  }
  const uint64_t coeffs = (uint64_t)count << log_n;
  const uint32_t blocks = (uint32_t)((coeffs + threads - 1) / threads);
  {
    LaunchScope ps("crt_lift", st);
    // A dependent for few moduli (GB300, 2 moduli, 2^15 coefficients 6.1 -> 3.8
    // us, 2^20 28.5 -> 25.6).  With more than 32 its long CTAs, placed while the
    // previous kernel's hold their SMs, pack unevenly: 2^16 coefficients, 33
    // moduli, 76 us plainly and 102 as a dependent.
    const bool dependent = g_dependent_launches;
    g_dependent_launches = dependent && L < kMmaMinModuli;
    if (threads == 64)
      launch_dependent(k_crt_lift<64>, blocks, 64, smem, st, d_out, d_in, count, L, log_n, t->mods, t->cofactors, t->q, t->W);
    else
      launch_dependent(k_crt_lift<32>, blocks, 32, smem, st, d_out, d_in, count, L, log_n, t->mods, t->cofactors, t->q, t->W);
    g_dependent_launches = dependent;
    g_kernel_launches += 1;
  }
  e = cudaGetLastError();
  return e == cudaSuccess ? kOk : fail_cuda(e, "crt_lift");
}

int check_crt_args(uint32_t L, uint32_t log_n, uint32_t cm0) {
  int st = check_degree(log_n);
  if (st != kOk) return st;
  st = check_moduli(cm0, L);
  if (st != kOk) return st;
  if (L > kCrtMaxModuli) return fail(kInvalidArgument, "CRT lifting takes at most 400 moduli");
  return kOk;
}

}  // namespace

extern "C" {

int yell_crt_words(uint32_t L, uint32_t cm0, uint32_t* words) {
  if (!words) return fail(kInvalidArgument, "null output");
  const int st = check_moduli(cm0, L);
  if (st != kOk) return st;
  *words = crt_words(cm0, L);
  return kOk;
}

int yell_dev_crt_lift(uint64_t* d_out, const uint64_t* d_in, uint32_t count, uint32_t L, uint32_t log_n,
                      uint32_t cm0, void* stream) {
  if (!d_out || !d_in || count == 0) return fail(kInvalidArgument, "null pointer or zero count");
  int st = check_crt_args(L, log_n, cm0);
  if (st != kOk) return st;
  st = check_limbs(count, L, log_n, nullptr);
  if (st != kOk) return st;
  DeviceContext* ctx = DeviceContext::current(&st);
  if (!ctx) return st;
  return crt_lift(d_out, d_in, count, L, log_n, cm0, stream ? static_cast<cudaStream_t>(stream) : ctx->stream(),
                  ctx->device(), nullptr);
}

int yell_crt_wait_status(uint32_t* status) {
  if (!status) return fail(kInvalidArgument, "null output");
  int st = kOk;
  DeviceContext* ctx = DeviceContext::current(&st);
  if (!ctx) return st;
  cudaError_t e = cudaDeviceSynchronize();
  void* word = nullptr;
  if (e == cudaSuccess) e = cudaGetSymbolAddress(&word, g_crt_wait_status);
  if (e == cudaSuccess) e = take_status(static_cast<uint32_t*>(word), ctx->stream(), status);
  return e == cudaSuccess ? kOk : fail_cuda(e, "read wait status");
}

int yell_crt_wait_check(uint64_t timeout_ns, uint32_t* status) {
  if (!status) return fail(kInvalidArgument, "null output");
  if (timeout_ns == 0 || timeout_ns > 10'000'000'000ull) return fail(kInvalidArgument, "timeout must be in (0, 10 s]");
  int st = kOk;
  DeviceContext* ctx = DeviceContext::current(&st);
  if (!ctx) return st;
  void* word = nullptr;
  cudaError_t e = cudaGetSymbolAddress(&word, g_crt_wait_status);
  if (e != cudaSuccess) return fail_cuda(e, "wait check");
  crt_mma::k_crt_wait_check<<<1, 64, 0, ctx->stream()>>>((uint32_t)(timeout_ns >> 10) + 1, static_cast<uint32_t*>(word));
  g_kernel_launches += 1;
  e = cudaGetLastError();
  if (e != cudaSuccess) return fail_cuda(e, "wait check");
  return yell_crt_wait_status(status);
}

int yell_poly_to_bigint(uint64_t* out, const uint64_t* const* limbs, uint32_t L, uint32_t log_n) {
  if (!out || !limbs) return fail(kInvalidArgument, "null pointer");
  int st = check_crt_args(L, log_n, 0);
  if (st != kOk) return st;
  for (uint32_t j = 0; j < L; ++j)
    if (!limbs[j]) return fail(kInvalidArgument, "null limb pointer");
  DeviceContext* ctx = DeviceContext::current(&st);
  if (!ctx) return st;
  const size_t n = (size_t)1 << log_n;
  const uint32_t W = crt_words(0, L);
  std::lock_guard<std::mutex> g(ctx->staging.lock);
  st = ctx->staging.reserve(n * L + n * W + 1);
  if (st != kOk) return st;
  cudaStream_t s = ctx->stream();
  uint64_t* d_in = ctx->staging.ptr;
  uint64_t* d_out = d_in + n * L;
  uint32_t* d_status = reinterpret_cast<uint32_t*>(d_out + n * W);
  uint32_t status = kOk;
  cudaError_t e = cudaMemsetAsync(d_status, 0, sizeof(status), s);
  for (uint32_t j = 0; j < L && e == cudaSuccess; ++j)
    e = cudaMemcpyAsync(d_in + j * n, limbs[j], n * 8, cudaMemcpyHostToDevice, s);
  if (e != cudaSuccess) return fail_cuda(e, "H2D limbs");
  st = crt_lift(d_out, d_in, 1, L, log_n, 0, s, ctx->device(), d_status);
  if (st != kOk) return st;
  e = cudaMemcpyAsync(out, d_out, n * W * 8, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = take_status(d_status, s, &status);
  if (e != cudaSuccess) return fail_cuda(e, "D2H / synchronize");
  return status == kOk ? kOk : fail((int)status, "CRT lift: a wait on the device ran out, the words are undefined");
}

}  // extern "C"
