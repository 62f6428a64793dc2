// Division by a launch-time constant as multiply-high + shift (dividends below 2^31): every role of the persistent kernels
// decodes a tile index per tile and the producers a filter tap per k-block; with small tiles the hardware's divisions were a
// quarter of a microsecond per tile.
#pragma once

#include <stdint.h>

struct FastDiv {
  uint32_t mul, shr, d;
};
static inline FastDiv make_fastdiv(uint32_t d) {
  FastDiv f;
  f.d = d ? d : 1;
  uint32_t l = 0;
  while ((1u << l) < f.d) l++;
  f.shr = l;
  f.mul = (uint32_t)((((uint64_t)1 << 32) * (((uint64_t)1 << l) - f.d)) / f.d + 1);
  return f;
}
#ifdef __CUDACC__
__device__ __forceinline__ uint32_t fdiv(const FastDiv& f, uint32_t n) { return (__umulhi(f.mul, n) + n) >> f.shr; }
#endif
