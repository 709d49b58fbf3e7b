// Device helpers shared by the split-precision GEMMs (split.cu, split8.cu):
// mbarriers with bounded waits, shared-memory matrix descriptors, exact
// conversion of the integer diagonal sums, and the fixed-point cut of FP64 rows.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace gi {
namespace {

__device__ __forceinline__ uint32_t sptr(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t* b, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(sptr(b)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* b, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(sptr(b)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ uint32_t mbar_try(uint64_t* b, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      "selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(sptr(b)), "r"(parity)
      : "memory");
  return ok;
}
__device__ __forceinline__ uint64_t gtimer() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;\n" : "=l"(t));
  return t;
}
// Try-wait with cluster-scope acquire: phases completed by the peer CTA's
// arrivals or TMA bytes.
__device__ __forceinline__ uint32_t mbar_try_cl(uint64_t* b, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n.reg .pred p;\nmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
      "selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(sptr(b)), "r"(parity)
      : "memory");
  return ok;
}
// Bounded wait on an mbarrier phase.  Returns false when the CTA is aborting
// (another warp timed out) or this wait exceeded its time limit (then it
// raises the abort itself and records the error).
// `sleep_ns` backs the poll off so that a waiting warp leaves the issue slots of
// its SM sub-partition to the MMA-issuing warp.
// CL: cluster-scope acquire (barriers that the peer CTA of a pair completes).
template <bool CL = false>
__device__ bool mbar_wait(uint64_t* b, uint32_t parity, volatile int* abort_flag, int* err,
                          int code, unsigned sleep_ns = 0) {
  uint64_t t0 = 0;
  for (uint32_t it = 1;; ++it) {
    if (CL ? mbar_try_cl(b, parity) : mbar_try(b, parity)) return true;
    if (sleep_ns) __nanosleep(sleep_ns);
    if ((it & 63) == 0) {
      if (*abort_flag) return false;
      if (*reinterpret_cast<volatile int*>(err)) {  // another CTA timed out: stop waiting
        *abort_flag = 1;
        return false;
      }
      const uint64_t t = gtimer();
      if (t0 == 0) {
        t0 = t;
      } else if (t - t0 > 4000000000ull) {  // 4 s: far beyond any tile's work
        *abort_flag = 1;
        atomicExch(err, code);
        return false;
      }
    }
  }
}
// v * 2^E for an integer |v| < 2^53 (so the double is exact), built from the
// bits with integer instructions: FP64 throughput is low on this GPU and the
// epilogues convert every output element.  Results outside the normal range
// take ldexp.
__device__ __forceinline__ double scaled_int_body(long long v, int E) {
  if (v == 0) return 0.0;
  const unsigned long long sgn = v < 0 ? (1ull << 63) : 0ull;
  const unsigned long long a = v < 0 ? 0ull - (unsigned long long)v : (unsigned long long)v;
  const int msb = 63 - __clzll((long long)a);
  const int ex = 1023 + msb + E;
  if (msb > 52 || ex <= 0 || ex >= 2047) return ldexp((double)v, E);
  const unsigned long long mant = (a << (52 - msb)) & ((1ull << 52) - 1);
  return __longlong_as_double((long long)(sgn | ((unsigned long long)ex << 52) | mant));
}
// The epilogues call these instead of inlining the conversion: inlined into
// the unrolled column chunks, it made the pass-1 epilogue of the half-ls GEMM
// a long stretch of straight-line code that ran out of the instruction cache
// once per tile (39 us of a 265 us tile, against 21 us called, measured with
// per-tile clock stamps).
__device__ __noinline__ double scaled_int(long long v, int E) { return scaled_int_body(v, E); }
// a0 * 2^ea0 + b0 * 2^eb0 and the same for a second element, in one call (the
// two parts of a two-pass tile's exact sums, added in FP64; the conversions of
// the two elements interleave)
__device__ __noinline__ double2 scaled_pair2(long long a0, int ea0, long long b0, int eb0,
                                             long long a1, int ea1, long long b1, int eb1) {
  double2 r;
  r.x = scaled_int_body(a0, ea0) + scaled_int_body(b0, eb0);
  r.y = scaled_int_body(a1, ea1) + scaled_int_body(b1, eb1);
  return r;
}
// Shared-memory matrix descriptor of a K-major bf16 tile whose rows are 32
// bytes (16 elements) with the 32-byte swizzle: 8-row groups 256 bytes apart.
__device__ __forceinline__ uint64_t sdesc_sw32(uint32_t addr) {
  uint64_t d = 0;
  d |= (uint64_t)((addr >> 4) & 0x3FFF);          // start address
  d |= (uint64_t)1 << 16;                          // leading byte offset (unused here)
  d |= (uint64_t)((256 >> 4) & 0x3FFF) << 32;      // stride byte offset: 8 rows x 32 B
  d |= (uint64_t)1 << 46;                          // descriptor version (tcgen05)
  d |= (uint64_t)6 << 61;                          // SWIZZLE_32B
  return d;
}
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
          sptr(bar))
      : "memory");
}
__device__ __forceinline__ void tmem_wait_ld() {
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
}

// Row exponent from the largest magnitude's bit pattern: 2^(e-1) <= max < 2^e.
__device__ __forceinline__ int row_exponent(unsigned long long maxbits) {
  if (maxbits == 0) return 0;
  const int eb = (int)(maxbits >> 52);
  return eb ? eb - 1022 : -1021 - (__clzll((long long)maxbits) - 12);
}

__device__ __forceinline__ long long fixed_point(double x, int e, int ws) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const int eb = (int)((b >> 52) & 0x7FF);
  const long long mant = (long long)(b & 0xFFFFFFFFFFFFFull) | (eb ? (1ll << 52) : 0ll);
  const int sh = (eb ? eb : 1) - 1075 - e + ws;  // x 2^(ws-e) = mant 2^sh
  long long X;
  if (sh >= 0) {
    X = mant << sh;
  } else if (sh > -54) {
    X = (mant + (1ll << (-sh - 1))) >> (-sh);  // round half up
  } else {
    X = 0;
  }
  return (b >> 63) ? -X : X;
}

}  // namespace
}  // namespace gi
