// Helpers of the 8D kernels that walk pursuer poses with an evader block in
// shared memory (world8d_fast.cu, world8d_column_exact.cu).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace pe {
namespace {

// e / d as __umulhi(e, m), m = ceil(2^32 / d): exact for e * (m*d - 2^32) <
// 2^32, which holds for e < 2^24 and d < 256 and, in general, for e < 2^32/d.
struct Divisor {
  uint32_t m;
  int d;
};

Divisor make_divisor(int d) {
  return {(uint32_t)((((uint64_t)1 << 32) + (uint64_t)d - 1) / (uint64_t)d), d};
}

__device__ __forceinline__ int split(int e, Divisor v, int &rem) {
  const int q = (int)__umulhi((uint32_t)e, v.m);
  rem = e - q * v.d;
  return q;
}

enum AxisKind { kExtrapolated = 0, kPeriodic = 1, kInward = 2 };

// Window offsets (in cells) of positions p-2, p-1, p+1, p+2 along an axis of
// stride s: clamped to the ends, or wrapped when periodic.
__device__ __forceinline__ void window_offsets(int p, int n, int s, bool periodic,
                                               int &om2, int &om1, int &op1, int &op2) {
  if (periodic) {
    om1 = p > 0 ? -s : (n - 1) * s;
    om2 = p > 1 ? -2 * s : (n - 2) * s;
    op1 = p < n - 1 ? s : -(n - 1) * s;
    op2 = p < n - 2 ? 2 * s : -(n - 2) * s;
  } else {
    om1 = p > 0 ? -s : 0;
    om2 = p > 1 ? -2 * s : om1;
    op1 = p < n - 1 ? s : 0;
    op2 = p < n - 2 ? 2 * s : op1;
  }
}

__device__ __forceinline__ void cp_async4(float *dst, const float *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;" ::: "memory");
}
__device__ __forceinline__ void cp_async_wait_one() {
  asm volatile("cp.async.wait_group 1;" ::: "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.wait_all;" ::: "memory");
}

}  // namespace
}  // namespace pe
