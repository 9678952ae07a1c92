// Quotient and remainder by a number that is fixed at launch.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define LLMCTL_HD __host__ __device__ __forceinline__
#else
#define LLMCTL_HD inline
#endif

namespace llmctl {

// A multiplication and a shift (Granlund and Montgomery, "Division by invariant integers using multiplication") for numbers below 2^31 and
// divisors of 1 to 2^31; a division by a kernel argument takes some 200 clocks, three of them before each work item's first load.
struct FastDiv {
  uint32_t d, mul, shift;
  explicit FastDiv(uint32_t divisor) : d(divisor), mul(0), shift(0) {
    while (shift < 31 && (1u << shift) < d) ++shift;
    mul = static_cast<uint32_t>((((1ull << shift) - d) << 32) / d + 1);
  }
  LLMCTL_HD uint32_t divide(uint32_t n, uint32_t& rem) const {
#ifdef __CUDA_ARCH__
    const uint32_t hi = __umulhi(n, mul);
#else
    const uint32_t hi = static_cast<uint32_t>((static_cast<uint64_t>(n) * mul) >> 32);
#endif
    const uint32_t q = (hi + n) >> shift;
    rem = n - q * d;
    return q;
  }
};

}  // namespace llmctl
