// Exact n / d for 0 <= n < 2^31 with one high multiply (Granlund and Montgomery, "Division by invariant integers using
// multiplication", 1994).  Every role of a persistent kernel decodes its next tile at the head of its chain, and a runtime
// 32-bit division is 100 to 250 cycles there: three of them in front of every tile took each role of the GEMM 790 cycles (14 %
// of a short-K tile), with this 310.
#pragma once

#include <stdint.h>

#ifndef __CUDACC__
#define HB_HD inline
#else
#define HB_HD __host__ __device__ __forceinline__
#endif

namespace hb {

struct FastDiv {
  uint32_t mul, shift, d;
};
inline FastDiv make_fast_div(uint32_t d) {
  FastDiv f;
  f.d = d;
  f.shift = 0;
  while ((1ull << f.shift) < d) ++f.shift;
  f.mul = static_cast<uint32_t>((((1ull << f.shift) - d) << 32) / d + 1);
  return f;
}
HB_HD int fast_div(int n, const FastDiv& f) {
  const uint32_t u = static_cast<uint32_t>(n);
  const uint32_t hi = static_cast<uint32_t>((static_cast<uint64_t>(u) * f.mul) >> 32);
  return static_cast<int>((hi + u) >> f.shift);
}

}  // namespace hb
