// RNS -> big-integer lifting as a tensor-core contraction (crt.cu has the
// mathematics and the tables' meaning).
//
// With y_j the cofactor-scaled residues and v the quotient, the lifted value is
// x = sum_j y_j * (Q/q_j) - v * Q.  In digits of base 256 that is a matrix
// product: a coefficient's row holds the 8 digits of every y_j and the digit
// v; row (j, i) of the constant matrix holds the digits of (Q/q_j) * 256^i,
// its last rows those of -Q and an offset; column d of the product is the sum
// of weight 256^d.  Digits are balanced (-128 .. 127), so 16-bit floats hold
// them exactly, and with at most kMaxL = 32 moduli a column's sum stays below
// 2^22 in magnitude (32 * (7 * 128 * 128 + 65 * 128) + 33 * 128 + 255), so the
// 32-bit float accumulators are exact integers whatever the order of the
// additions.  The offset 2^23 + 2^22 puts every accumulator into
// [2^23, 2^24), where a float's low 23 bits are the integer minus 2^23: the
// epilogue reads digits m_d out of the bit patterns without a conversion.  The
// second offset row holds the digits that cancel what the offset (and the bit
// patterns' exponents) add to the sum modulo 2^(64 W), so that
// x = sum_d m_d * 256^d modulo 2^(64 W).
//
// The quotient v = floor(sum_j y_j / q_j) is estimated from 57-bit fixed
// point terms (y_j >> 31) * floor(2^88 / q_j), minus a bias that makes the
// estimate v or v - 1, v - 1 only when the fraction lies within
// L * (2^32 + 2^27) of wrapping; those rows are marked, and their thread
// compares the stored x with Q and subtracts Q if needed.  y_j is taken in
// [-q_j, q_j) (Shoup product minus q_j), which changes v accordingly.
//
// One CTA per SM, persistent over tiles of 128 coefficients; the constant
// matrix (up to 264 x 256 values, 136 KB) stays in shared memory.  16
// producer warps (4 threads per coefficient) compute y_j, split it into
// digits and write the left operand in chunks of 8 moduli (64 digits, 128
// bytes per row, 128-byte swizzle) into a ring of kRing chunks; one warp
// issues the tcgen05.mma of each chunk; two groups of 4 epilogue warps (a
// thread per coefficient), one for each of two accumulators in TMEM, resolve
// the carries while the other accumulator fills, and write the words through
// shared memory in segments of 64 bytes.
//
// What bounds it: no one unit.  Per tile at L = 32 the tensor cores need 2190
// cycles, HBM (63 words per coefficient) 3000, and a tile takes about 5000;
// the counters have issue slots at 49%, the tensor pipe at 38%, DRAM at 23%,
// and warps waiting on long scoreboards, fixed latencies and the barriers
// between them.  GB300, 16 x 2^16 coefficients, L = 32, calls in a row: 136 to
// 142 us, 3.8 TB/s (762 us for the kernel with 32-bit multiply-add chains);
// one call by itself 151.  On the way: one-lane issue loop 166 us, TMEM loads of 32
// columns two deep (spills) 339 us, producers' own proxy fences 181 us.
#pragma once
#include <cuda_fp16.h>

#include "async_copy.cuh"
#include "common.cuh"
#include "yell_gb300.h"

namespace yell_gb300 {
namespace crt_mma {

constexpr uint32_t kMaxL = 32;
constexpr uint32_t kRows = 128;                 // coefficients per tile
constexpr uint32_t kChunkMods = 8;              // moduli per chunk: 64 digits = 128 bytes per row
constexpr uint32_t kRing = 3;
constexpr uint32_t kParts = 4;                  // producer threads per coefficient
constexpr uint32_t kTails = 3, kFlags = 8;       // tails and marks in flight
constexpr uint32_t kMine = kChunkMods / kParts; // moduli of a chunk per producer thread
constexpr uint32_t kEpilogueWarps = 8, kProducerWarps = kParts * kRows / 32;
constexpr uint32_t kThreads = 32 * (kEpilogueWarps + kProducerWarps + 1);
constexpr uint32_t kChunkBytes = kRows * 128;   // one chunk of the left operand
constexpr uint32_t kTailBytes = kRows * 32;     // its last 16 columns: v, the offsets' factors, zeros
constexpr uint32_t kStageWords = 8, kStageStride = 9;

// A modulus: q, inv = (Q/q)^-1 mod q and its Shoup companion, floor(2^88 / q).
struct alignas(16) Mod {
  uint64_t q, inv, inv_s;
  int64_t c;
};

__host__ __device__ constexpr uint32_t columns(uint32_t W) { return (8 * W + 31) / 32 * 32; }
__host__ __device__ constexpr uint32_t chunks(uint32_t L) { return (L + kChunkMods - 1) / kChunkMods; }
// Byte offsets into the constant matrix' image: chunk c, then the tail.
__host__ __device__ constexpr uint32_t image_chunk(uint32_t N) { return N * 128; }
__host__ __device__ constexpr uint32_t image_bytes(uint32_t L, uint32_t N) { return chunks(L) * N * 128 + N * 32; }
// The 128- and 32-byte swizzles of tcgen05 shared-memory operands (rows of 128
// and 32 bytes): byte offset in the operand -> byte offset in memory.
__host__ __device__ constexpr uint32_t swizzle128(uint32_t o) { return o ^ (((o >> 7) & 7u) << 4); }
__host__ __device__ constexpr uint32_t swizzle32(uint32_t o) { return o ^ (((o >> 7) & 1u) << 4); }

// Shared memory, from a 1024-byte boundary.
struct Layout {
  uint32_t ring, tail_b, tail_a, stage, mods, part, flags, bars, bytes;
};
__host__ __device__ constexpr Layout layout(uint32_t L, uint32_t N) {
  Layout l{};
  l.ring = chunks(L) * image_chunk(N);  // the constant chunks start at 0
  l.tail_b = l.ring + kRing * kChunkBytes;
  l.tail_a = l.tail_b + N * 32;
  l.stage = l.tail_a + kTails * kTailBytes;
  l.mods = l.stage + kEpilogueWarps * 32 * kStageStride * 8;
  l.part = l.mods + kMaxL * (uint32_t)sizeof(Mod);
  l.flags = l.part + 2 * kParts * kRows * 8;
  l.bars = l.flags + kFlags * kRows;
  l.bytes = l.bars + 256;
  return l;
}
constexpr uint32_t smem_bytes(uint32_t L, uint32_t N) { return layout(L, N).bytes + 1024; }  // room to align
static_assert(smem_bytes(kMaxL, 256) <= (227u << 10), "the largest lift fits one SM");

// ---- tcgen05 ------------------------------------------------------------------
__device__ __forceinline__ uint64_t operand_desc(uint32_t smem_addr, uint32_t stride_bytes, uint32_t swizzle) {
  return (uint64_t)((smem_addr >> 4) & 0x3FFFu) | (1ull << 16) | ((uint64_t)(stride_bytes >> 4) << 32) | (1ull << 46) |
         ((uint64_t)swizzle << 61);
}
constexpr uint32_t kSwizzle128 = 2, kSwizzle32 = 6;

__device__ __forceinline__ void mma_f16(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t* mbar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(mbar))
               : "memory");
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld16(uint32_t addr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(addr));
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void mbar_arrive(uint64_t* mbar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"((uint32_t)__cvta_generic_to_shared(mbar)) : "memory");
}

__device__ __forceinline__ int64_t mad_wide(int32_t a, int32_t b, int64_t c) {
  int64_t r;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
  return r;
}

__device__ __forceinline__ uint64_t mad_wide_u(uint32_t a, uint32_t b, uint64_t c) {
  uint64_t r;
  asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
  return r;
}

// The 8 balanced digits of y (|y| < 2^62) as 16-bit floats: each byte b of
// y + 0x80..80 is a digit plus 128; 0x6400 | b is the float 1024 + b.
__device__ __forceinline__ uint4 digits_f16(int64_t y) {
  const uint64_t z = (uint64_t)y + 0x8080808080808080ull;
  const uint32_t lo = (uint32_t)z, hi = (uint32_t)(z >> 32);
  auto pair = [](uint32_t w, uint32_t sel) {
    const uint32_t v = __byte_perm(w, 0x64646464u, sel);
    const __half2 d = __hsub2(*reinterpret_cast<const __half2*>(&v), __half2half2(__ushort_as_half(0x6480)));
    return *reinterpret_cast<const uint32_t*>(&d);
  };
  return make_uint4(pair(lo, 0x4140), pair(lo, 0x4342), pair(hi, 0x4140), pair(hi, 0x4342));
}

struct Bars {
  uint64_t full[kRing], empty[kRing], tail_full[kTails], tail_empty[kTails], acc_full[2], acc_empty[2], done;
  uint32_t tmem, gave_up, limit;  // limit: wait<0>
};
static_assert(sizeof(Bars) <= 256, "barrier block");

// A bounded wait (1 s).  The first one to run out records YELL_ERR_TIMEOUT
// and lets the CTA's other waits return at once: the CTA still reaches its
// end, with its output undefined.  Only time in which the wait polls counts:
// what it waits for is done by warps of the same CTA, which stand still with
// it while a debugger or another process has the device.
constexpr uint32_t kWaitLimit = 1000000000u >> 10;  // in units of 1024 ns
// LIMIT 0: the limit is b->limit (read from shared memory it costs the lift of
// 32 moduli a spill).
template <uint32_t LIMIT>
__device__ __noinline__ void wait_slow(Bars* b, uint64_t* mbar, uint32_t parity, uint32_t* status) {
  if (*(volatile uint32_t*)&b->gave_up && mbar != &b->done) return;  // work in flight is waited for in any case
  if (!mbar_wait_running(mbar, parity, status, (uint32_t)YELL_ERR_TIMEOUT, LIMIT ? LIMIT : b->limit))
    *(volatile uint32_t*)&b->gave_up = 1;
}
template <uint32_t LIMIT = kWaitLimit>
__device__ __forceinline__ void wait(Bars* b, uint64_t* mbar, uint32_t parity, uint32_t* status) {
  if (!mbar_test(mbar, parity)) wait_slow<LIMIT>(b, mbar, parity, status);
}

// The TMEM address that the issuing warp's allocation left.  All threads of the
// CTA meet here, so that no bounded wait runs while another kernel on this SM
// still has the columns.
__device__ __forceinline__ uint32_t tmem_address(Bars* b) {
  fence_before();
  asm volatile("bar.sync 2, %0;" ::"n"(kThreads) : "memory");
  fence_after();
  return *(volatile uint32_t*)&b->tmem;
}

// Check of the bounded wait: one CTA waits twice on a barrier at which nobody
// arrives.  The first wait runs out and records YELL_ERR_TIMEOUT, the second
// returns at once.
__global__ void k_crt_wait_check(uint32_t limit, uint32_t* status) {
  __shared__ Bars bars;
  if (threadIdx.x == 0) {
    mbar_init(&bars.full[0], 1);
    bars.gave_up = 0;
    bars.limit = limit;
  }
  __syncthreads();
  wait<0>(&bars, &bars.full[0], 0, status);
  __syncthreads();
  wait<0>(&bars, &bars.full[0], 0, status);
}

// image: image_bytes(L, N) bytes in operand layout; mods: L entries.
template <uint32_t NC>  // chunks(L)
__global__ void __launch_bounds__(kThreads, 1)
    k_crt_mma(uint64_t* out, const uint64_t* in, uint64_t coeffs, uint32_t L, uint32_t log_n,
              const Mod* __restrict__ mods, const uint4* __restrict__ image, const uint64_t* __restrict__ qw,
              uint32_t W, uint32_t* status) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t N = columns(W);
  const Layout lay = layout(L, N);
  uint8_t* s = smem_raw + ((1024u - ((uint32_t)__cvta_generic_to_shared(smem_raw) & 1023u)) & 1023u);
  const uint32_t s_addr = (uint32_t)__cvta_generic_to_shared(s);
  Bars* bars = reinterpret_cast<Bars*>(s + lay.bars);
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
  const uint32_t tmem_cols = N <= 16 ? 32u : (N <= 32 ? 64u : (N <= 64 ? 128u : (N <= 128 ? 256u : 512u)));
  const uint32_t tiles = (uint32_t)((coeffs + kRows - 1) / kRows);

  // once per CTA: constant matrix, moduli, barriers, TMEM
  {
    uint4* b = reinterpret_cast<uint4*>(s);
    const uint32_t nb = NC * image_chunk(N) / 16;
    for (uint32_t i = tid; i < nb; i += kThreads) b[i] = __ldg(image + i);
    uint4* t = reinterpret_cast<uint4*>(s + lay.tail_b);
    for (uint32_t i = tid; i < N * 2; i += kThreads) t[i] = __ldg(image + nb + i);
    uint4* m = reinterpret_cast<uint4*>(s + lay.mods);
    for (uint32_t i = tid; i < L * 2; i += kThreads) m[i] = __ldg(reinterpret_cast<const uint4*>(mods) + i);
  }
  if (tid == 0) {
    for (uint32_t i = 0; i < kRing; ++i) {
      mbar_init(&bars->full[i], kProducerWarps);
      mbar_init(&bars->empty[i], 1);
    }
    for (uint32_t i = 0; i < kTails; ++i) {
      mbar_init(&bars->tail_full[i], kRows / 32);
      mbar_init(&bars->tail_empty[i], 1);
    }
    for (uint32_t i = 0; i < 2; ++i) {
      mbar_init(&bars->acc_full[i], 1);
      mbar_init(&bars->acc_empty[i], kEpilogueWarps / 2);
    }
    mbar_init(&bars->done, 1);
    bars->gave_up = 0;
  }
  fence_proxy_async();
  __syncthreads();
  grid_dep_wait();  // the caller's words are read and written below

  if (warp >= kEpilogueWarps && warp < kEpilogueWarps + kProducerWarps) {
    // ---- producers: thread (row, part) takes moduli 8 c + kMine part .. of each chunk c
    const uint32_t pt = tid - kEpilogueWarps * 32, row = pt & (kRows - 1), part = pt / kRows;
    const Mod* sm = reinterpret_cast<const Mod*>(s + lay.mods) + kMine * part;
    int64_t* parts = reinterpret_cast<int64_t*>(s + lay.part);
    const uint64_t n_mask = (1ull << log_n) - 1, n = 1ull << log_n;
    const int32_t last = (int32_t)L - (int32_t)((NC - 1) * kChunkMods + kMine * part);  // moduli in the last chunk
    // a tile's words are requested a tile ahead
    uint64_t r[NC][kMine];
    const uint64_t* src = nullptr;
    bool live = false;
    auto locate = [&](uint64_t tile) {
      const uint64_t g = tile * kRows + row;
      live = tile < tiles && g < coeffs;
      if (live) src = in + (((g >> log_n) * L + kMine * part) << log_n) + (g & n_mask);
    };
    auto fetch = [&](uint32_t c) {
#pragma unroll
      for (int i = 0; i < (int)kMine; ++i)
        r[c][i] = live && (c + 1 < NC || i < last) ? src[i * n] : 0;
      src += kChunkMods * n;
    };
    locate(blockIdx.x);
#pragma unroll
    for (uint32_t c = 0; c < NC; ++c) fetch(c);
    (void)tmem_address(bars);
    uint32_t slot = 0, round = 0, t = 0, ts = 0, tr = 0;
    // this thread's 16-byte units of a chunk row
    uint8_t* unit[kMine];
#pragma unroll
    for (uint32_t i = 0; i < kMine; ++i) unit[i] = s + lay.ring + row * 128 + (((kMine * part + i) ^ (row & 7u)) << 4);
    for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x, ++t) {
      locate((uint64_t)tile + gridDim.x);
      int64_t acc = 0;
#pragma unroll
      for (uint32_t c = 0; c < NC; ++c) {
        uint64_t w[kMine];
#pragma unroll
        for (uint32_t i = 0; i < kMine; ++i) w[i] = r[c][i];
        fetch(c);
        uint4 d[kMine];
#pragma unroll
        for (int i = 0; i < (int)kMine; ++i) {
          d[i] = make_uint4(0, 0, 0, 0);
          if (c + 1 < NC || i < last) {
            const Mod m = sm[c * kChunkMods + i];
            const int64_t y = (int64_t)(shoup_lazy(w[i], m.inv, m.inv_s, 0 - m.q) - m.q);
            acc = mad_wide((int32_t)(y >> 31), (int32_t)m.c, acc);
            d[i] = digits_f16(y);
          }
        }
        wait(bars, &bars->empty[slot], (round & 1u) ^ 1u, status);
#pragma unroll
        for (uint32_t i = 0; i < kMine; ++i) *reinterpret_cast<uint4*>(unit[i] + slot * kChunkBytes) = d[i];
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->full[slot]);
        if (++slot == kRing) {
          slot = 0;
          ++round;
        }
      }
      {
        // the quotient, from the parts of the row
        const uint32_t b = t & 1u;
        parts[(b * kParts + part) * kRows + row] = acc;
        asm volatile("bar.sync 1, %0;" ::"n"(kProducerWarps * 32) : "memory");
        if (part == 0) {
          int64_t sum = -(int64_t)L * (1ll << 31);
#pragma unroll
          for (uint32_t k = 0; k < kParts; ++k) sum += parts[(b * kParts + k) * kRows + row];
          const int32_t v = (int32_t)(sum >> 57);
          const uint64_t frac = (uint64_t)sum & ((1ull << 57) - 1);
          const uint32_t flag = frac >= (1ull << 57) - (uint64_t)L * ((1ull << 32) + (1ull << 27)) ? 1u : 0u;
          wait(bars, &bars->tail_empty[ts], (tr & 1u) ^ 1u, status);
          // kFlags tiles ago: read, as the ring has been refilled since and the
          // tensor cores have started a later tile of the same accumulator
          s[lay.flags + (t & (kFlags - 1)) * kRows + row] = (uint8_t)flag;
          uint8_t* ta = s + lay.tail_a + ts * kTailBytes;
          const uint32_t vh = __half_as_ushort(__int2half_rn(v));
          // 4096 (times 3072 = 2^23 + 2^22) and 1 (times the cancelling digits)
          *reinterpret_cast<uint4*>(ta + swizzle32(row * 32)) = make_uint4(vh | (0x6C00u << 16), 0x3C00u, 0, 0);
          *reinterpret_cast<uint4*>(ta + swizzle32(row * 32 + 16)) = make_uint4(0, 0, 0, 0);
          __syncwarp();
          if (lane == 0) mbar_arrive(&bars->tail_full[ts]);
        }
        if (++ts == kTails) {
          ts = 0;
          ++tr;
        }
      }
    }
  } else if (warp == kEpilogueWarps + kProducerWarps) {
    // ---- one warp issues the tensor-core work.  All its lanes run the loop on
    // the same values, so the operand descriptors stay in uniform registers,
    // and one lane issues: with the whole loop inside a one-lane branch an MMA
    // took 220 cycles to issue (128 to run) beside the producers' warps.
    //
    // TMEM is taken only now, while the producers start: a CTA that holds columns
    // while it waits could keep them from a CTA of the kernel that it waits for.
    // For the same reason the next kernel may start only once this CTA has them.
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(&bars->tmem)),
                 "r"(tmem_cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    const uint32_t tmem = tmem_address(bars);
    grid_dep_launch();
    const uint32_t idesc = (1u << 4) | ((N >> 3) << 17) | ((kRows >> 4) << 24);  // f16 x f16 -> f32, both K-major
    const uint64_t desc_a = operand_desc(s_addr + lay.ring, 1024, kSwizzle128);
    const uint64_t desc_b = operand_desc(s_addr, 1024, kSwizzle128);
    const uint64_t desc_ta = operand_desc(s_addr + lay.tail_a, 256, kSwizzle32);
    const uint64_t desc_tb = operand_desc(s_addr + lay.tail_b, 256, kSwizzle32);
    const uint32_t last_steps = (L - (NC - 1) * kChunkMods + 1) / 2;  // 2 moduli per step
    const uint32_t acc0 = __shfl_sync(0xFFFFFFFFu, tmem, 0);
    const bool leader = lane == 0;
    uint32_t slot = 0, round = 0, t = 0, ts = 0, tr = 0;
    for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x, ++t) {
      const uint32_t b = t & 1u, d = acc0 + b * N;
      wait(bars, &bars->acc_empty[b], ((t >> 1) & 1u) ^ 1u, status);
#pragma unroll
      for (uint32_t c = 0; c < NC; ++c) {
        wait(bars, &bars->full[slot], round & 1u, status);
        // The producers' generic writes before the tensor cores' reads.  Their
        // arrivals release the writes and this wait acquires them; a proxy
        // fence orders the two proxies wherever it stands between the write
        // and the read in causality order (PTX memory consistency model), so
        // one here serves all producers, whose own would each also wait for
        // their words in flight.
        fence_proxy_async();
        fence_after();
        const uint64_t a0 = desc_a + slot * (kChunkBytes >> 4), b0 = desc_b + c * (image_chunk(N) >> 4);
        if (leader) {
#pragma unroll
          for (uint32_t k = 0; k < kChunkMods / 2; ++k)
            if (c + 1 < NC || k < last_steps) mma_f16(d, a0 + 2 * k, b0 + 2 * k, idesc, (c | k) != 0);
          mma_commit(&bars->empty[slot]);
        }
        __syncwarp();
        if (++slot == kRing) {
          slot = 0;
          ++round;
        }
      }
      wait(bars, &bars->tail_full[ts], tr & 1u, status);
      fence_proxy_async();
      fence_after();
      if (leader) {
        mma_f16(d, desc_ta + ts * (kTailBytes >> 4), desc_tb, idesc, 1);
        mma_commit(&bars->tail_empty[ts]);
        mma_commit(&bars->acc_full[b]);
      }
      __syncwarp();
      if (++ts == kTails) {
        ts = 0;
        ++tr;
      }
    }
    if (leader) mma_commit(&bars->done);
    __syncwarp();
    wait(bars, &bars->done, 0, status);
    __syncwarp();
  } else {
    // ---- epilogue: warps 4 b .. 4 b + 3 take the tiles of accumulator b; thread
    // = coefficient row 32 * quarter + lane = TMEM lane
    const uint32_t tmem = tmem_address(bars);
    const uint32_t quarter = warp & 3u, b = warp >> 2, row = quarter * 32 + lane;
    uint64_t* stage = reinterpret_cast<uint64_t*>(s + lay.stage) + warp * 32 * kStageStride;
    uint32_t kt = 0, t = b;
    for (uint64_t tile = blockIdx.x + (uint64_t)b * gridDim.x; tile < tiles; tile += 2 * gridDim.x, kt ^= 1u, t += 2) {
      const uint64_t g0 = tile * kRows + quarter * 32;
      wait(bars, &bars->acc_full[b], kt, status);
      fence_after();
      const uint32_t flag = *(volatile const uint8_t*)(s + lay.flags + (t & (kFlags - 1)) * kRows + row);
      const uint32_t base = tmem + b * N + ((quarter * 32) << 16);
      const uint32_t rows = g0 >= coeffs ? 0u : (coeffs - g0 < 32 ? (uint32_t)(coeffs - g0) : 32u);
      uint32_t carry = 0, carry_bit = 0;
      uint32_t cols[2][16];
      tmem_ld16(base, cols[0]);
      for (uint32_t w0 = 0; w0 < W; w0 += kStageWords) {
        const uint32_t nw = W - w0 < kStageWords ? W - w0 : kStageWords;
#pragma unroll
        for (uint32_t q = 0; q < kStageWords / 2; ++q) {
          // 16 columns = 2 words; the next ones load meanwhile
          uint32_t* m = cols[q & 1u];
          tmem_ld_wait();
          if (8 * w0 + 16 * (q + 1) < N) tmem_ld16(base + 8 * w0 + 16 * (q + 1), cols[(q + 1) & 1u]);
          if (2 * q < nw) {
            // 4 digits of weight 256^(4 e): with bits = 0x4B000000 + m_d, << 8
            // drops the constant; the constants that p[0] and p[2] keep are
            // cancelled by the offset row.  The sums' upper halves are added
            // to the next position in one carry chain.
            uint32_t l[4], h[4];
#pragma unroll
            for (uint32_t e = 0; e < 4; ++e) {
              const uint32_t* p = m + 4 * e;
              const uint32_t lo = (p[1] << 8) + p[0], hi = (p[3] << 8) + p[2];
              const uint64_t x = mad_wide_u(hi, 1u << 16, (uint64_t)lo);
              l[e] = (uint32_t)x;
              h[e] = (uint32_t)(x >> 32);
            }
            // carry: upper half of the position below, and its carry bit (0 or 1)
            asm("add.cc.u32 %5, %5, 0xFFFFFFFF;\n\t"
                "addc.cc.u32 %0, %0, %4;\n\taddc.cc.u32 %1, %1, %6;\n\taddc.cc.u32 %2, %2, %7;\n\t"
                "addc.cc.u32 %3, %3, %8;\n\taddc.u32 %5, 0, 0;"
                : "+r"(l[0]), "+r"(l[1]), "+r"(l[2]), "+r"(l[3]), "+r"(carry), "+r"(carry_bit)
                : "r"(h[0]), "r"(h[1]), "r"(h[2]));
            carry = h[3];
            uint64_t* st = stage + lane * kStageStride + 2 * q;
            st[0] = (uint64_t)l[1] << 32 | l[0];
            st[1] = (uint64_t)l[3] << 32 | l[2];
          }
        }
        __syncwarp();
        // out: four rows of up to 8 words per step
        const uint32_t k = lane & 7u, r0 = lane >> 3;
        if (k < nw) {
          uint64_t* o = out + (g0 + r0) * W + w0 + k;
          const uint64_t* st = stage + r0 * kStageStride + k;
          if (rows == 32) {
#pragma unroll
            for (uint32_t r = 0; r < 32; r += 4, o += 4 * (size_t)W) *o = st[r * kStageStride];
          } else {
            for (uint32_t r = 0; r0 + r < rows; r += 4, o += 4 * (size_t)W) *o = st[r * kStageStride];
          }
        }
        __syncwarp();
      }
      tmem_ld_wait();
      fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->acc_empty[b]);
      if (flag && lane < rows) {
        // x or x - Q: the words hold x modulo 2^(64 W), x / Q within 2^-20 of 1
        uint64_t* x = out + (g0 + lane) * W;
        const uint64_t top = x[W - 1], qtop = __ldg(&qw[W - 1]);
        bool ge = true;
        for (uint32_t w = W; w-- > 0;) {
          const uint64_t a = x[w], q = __ldg(&qw[w]);
          if (a != q) {
            ge = a > q;
            break;
          }
        }
        if ((qtop >> 63) && top < (1ull << 62)) ge = true;  // x passed 2^(64 W)
        if (ge) {
          uint32_t br = 0;
          for (uint32_t w = 0; w < W; ++w) {
            const uint64_t a = x[w], q = __ldg(&qw[w]), d = a - q;
            x[w] = d - br;
            br = (uint32_t)(a < q) | (uint32_t)(d < br);
          }
        }
      }
    }
    fence_before();
  }
  __syncthreads();
  if (warp == kEpilogueWarps + kProducerWarps) {
    fence_after();
    const uint32_t tmem = *(volatile uint32_t*)&bars->tmem;
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tmem_cols) : "memory");
  }
}

}  // namespace crt_mma
}  // namespace yell_gb300
