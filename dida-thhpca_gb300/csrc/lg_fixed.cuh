// lg_fixed.cuh -- fixed-point numbers of the FP64 path's reduction and
// reflections (lg_tri.cu, lg_ft.cu): 64-bit integers held as h 2^30 + l with
// -2^29 <= l < 2^29, so that products are 32 x 32 -> 64-bit multiply-adds.
#pragma once
#include <cuda_runtime.h>

namespace lg {

// (l, h) <-> h 2^30 + l
__device__ inline long long fixed_join(int2 v) { return (long long)v.y * (1 << 30) + v.x; }
__device__ inline int2 fixed_split(long long v) {
  const int h = (int)((v + (1 << 29)) >> 30);
  return make_int2((int)v - (int)((unsigned)h << 30), h);
}

// v 2^ex rounded to nearest-even; results below the normal range become 0
__device__ inline double fixed_to_double(long long v, int ex) {
  if (v == 0) return 0.0;
  const bool neg = v < 0;
  const unsigned long long m = neg ? 0ull - (unsigned long long)v : (unsigned long long)v;
  const int z = __clzll((long long)m);
  const unsigned long long t = m << z;  // leading one at bit 63
  unsigned long long mant = t >> 11;
  const unsigned rest = (unsigned)t & 0x7ffu;
  mant += (rest > 0x400u || (rest == 0x400u && (mant & 1))) ? 1 : 0;
  const int e = 63 - z + ex + 1023 - 1;  // the leading one adds 1
  if (e < 0) return 0.0;
  const unsigned long long bits = ((unsigned long long)e << 52) + mant;
  return __longlong_as_double((long long)(bits | (neg ? 0x8000000000000000ull : 0ull)));
}

}  // namespace lg
