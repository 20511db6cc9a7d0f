// Device helpers shared by the tensor-core kernels: bounded barrier waits and
// the integer side of the fixed-point operands and results.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "vl1_tc.cuh"

namespace vl1 {

constexpr uint32_t kSleepNs = 200000;      // suspend hint of one barrier test
constexpr uint32_t kWaitLimitUs = 2000000; // a wait gives up after 2 s

__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Wait for `phase` of `bar`.  Gives up (returns false) when another role has
// set the abort flag, or after `limit_us` microseconds (then it sets the
// flag itself); both are looked at every 32 tests.  A warp whose test fails
// sleeps between tests, so that waiting warps leave the issue slots of
// their scheduler to the producer warps that share it: with `backoff` the
// sleep doubles from 32 ns to 256 ns (warps with slack: producers, readout);
// without it, it stays at 32 ns (the tensor-core issuer and the table
// loader, whose reaction time is on the pipeline's critical path).
__device__ __forceinline__ bool wait_or_abort(uint64_t *bar, uint32_t phase,
                                              volatile int *abort_flag, uint32_t limit_us,
                                              bool backoff) {
  if (tc::mbar_try_wait_sleep(bar, phase, kSleepNs)) return true;
  const uint64_t t0 = global_ns();
  uint32_t ns = 32;
  for (uint32_t i = 1;; ++i) {
    __nanosleep(ns);
    if (backoff) ns = ns < 256 ? 2 * ns : ns;
    if (tc::mbar_try_wait_sleep(bar, phase, kSleepNs)) return true;
    if ((i & 31u) == 0u) {
      if (*abort_flag) return false;
      if (global_ns() - t0 > (uint64_t)limit_us * 1000ull) break;
    }
  }
  *abort_flag = 1;
  return false;
}

// Wait for `phase` of `bar` regardless of the abort flag, at most
// `limit_us`: used after an abort for operations already issued (bulk copies
// into this CTA's shared memory, MMAs into its TMEM), which complete on
// their own, before the CTA releases its TMEM and exits.
__device__ __forceinline__ bool wait_bounded(uint64_t *bar, uint32_t phase, uint32_t limit_us) {
  const uint64_t t0 = global_ns();
  while (!tc::mbar_try_wait_sleep(bar, phase, kSleepNs)) {
    if (global_ns() - t0 > (uint64_t)limit_us * 1000ull) return false;
    __nanosleep(256);
  }
  return true;
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc::smem_addr(bar)) : "memory");
}

// A kernel launched with launch_overlapped may start once every CTA of the
// kernel before it in the stream has called grid_dep_launch (or exited), and
// runs up to its grid_dep_wait beside that kernel's last CTAs: the launch, the
// barriers' and TMEM's set-up and the work item's records are then off the
// stream's path (2 to 4 us a boundary: digits and FP64 kernel 233 -> 229 us on
// the adaptive 3D tree, exponents, planes and mixed kernel 114.5 -> 109.7 us).  grid_dep_wait returns when the kernel
// before has completed and its writes are visible; without the overlap both are
// no-ops.
__device__ __forceinline__ void grid_dep_launch() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void grid_dep_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

inline cudaError_t launch_overlapped(const void *fn, dim3 grid, dim3 block, void **args,
                                     size_t smem, cudaStream_t s) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelExC(&cfg, fn, args);
}

// exponent e with |v| < 2^e, as frexp returns it (-1074 for v == 0), from the
// IEEE-754 fields
__device__ __forceinline__ int scale_exponent(double v) {
  const unsigned long long mag =
      static_cast<unsigned long long>(__double_as_longlong(v)) & 0x7FFFFFFFFFFFFFFFull;
  if (mag == 0) return -1074;
  const int ef = (int)(mag >> 52);
  if (ef) return ef - 1022;
  return (64 - __clzll((long long)mag)) - 1074;   // subnormal
}

// v * 2^k rounded once to FP64 (nearest, ties to even), with integer
// operations only while the result is a normal number
__device__ __forceinline__ double scaled_i64_to_double(long long v, int k) {
  if (v == 0) return 0.0;
  const unsigned long long sgn = v < 0 ? (1ull << 63) : 0ull;
  const unsigned long long mag =
      v < 0 ? (unsigned long long)(-(v + 1)) + 1ull : (unsigned long long)v;
  const int lz = __clzll((long long)mag);
  const unsigned long long m = mag << lz;   // leading one at bit 63
  unsigned long long frac = m >> 11;        // 53 significant bits
  const unsigned long long rem = m & 0x7FFull;
  int ex = 63 - lz + k;                     // v * 2^k = (m / 2^63) * 2^ex
  if (rem > 0x400ull || (rem == 0x400ull && (frac & 1ull))) {
    ++frac;
    if (frac == (1ull << 53)) {
      frac >>= 1;
      ++ex;
    }
  }
  const int biased = ex + 1023;
  if (biased >= 1 && biased <= 2046)
    return __longlong_as_double((long long)(sgn | ((unsigned long long)biased << 52) |
                                            (frac & 0xFFFFFFFFFFFFFull)));
  return ldexp((double)v, k);   // subnormal or overflowing results
}

// The same without a branch when the result is zero or a normal number;
// otherwise `rare` is set and the value is to come from scaled_i64_to_double.
// For threads that convert many independent values: their dependent chains
// overlap, which the branches above (for zero, for the rounding's carry, for
// the exponent range) prevent.  The rounded 53 bits, leading one included,
// are added to the exponent field, so that the rounding's carry moves into
// the exponent.
__device__ __forceinline__ double scaled_i64_select(long long v, int k, bool &rare) {
  const long long sg = v >> 63;
  const unsigned long long mag = (unsigned long long)((v ^ sg) - sg);
  const int lz = __clzll((long long)(mag | 1ull));
  const unsigned long long m = mag << lz;   // leading one at bit 63
  const unsigned lo = (unsigned)m;
  const unsigned up = ((lo & 0x7FFu) + 0x3FFu + ((lo >> 11) & 1u)) >> 11;
  const unsigned field = mag == 0ull ? 0u : (unsigned)(1085 - lz + k);   // biased exponent - 1
  const unsigned long long bits = (m >> 11) + up + ((unsigned long long)field << 52);
  rare |= field >= 2046u;
  return __longlong_as_double(
      (long long)(bits | ((unsigned long long)sg & 0x8000000000000000ull)));
}

}  // namespace vl1
