// warp_sum.cuh -- sum of one double per lane over a warp by integer reductions
// (the QR's dot products, linalg.cu).
#pragma once
#include <cuda_runtime.h>

namespace pqmc {

// The sum of v over the warp, to every lane, as 58-bit integers in units of
// 2^-57 of the largest, each rounded to the nearest: errors of 0.36e-16 of sum
// |v| rms over a wide range of magnitudes, 0.74e-16 for a tree of FP64
// additions.  Five levels of a tree cost 140 cycles each, 64 of them the
// addition; this is four warp-wide integer reductions and some thirty integer
// instructions, 300 cycles.  A NaN or infinity makes it NaN; a sum below
// 2^-1022 is 0.
__device__ __forceinline__ double warp_sum(double v) {
  const unsigned full = 0xffffffffu;
  const int hi = __double2hiint(v), e = (hi >> 20) & 0x7ff;
  const int top = __reduce_max_sync(full, e);
  unsigned long long f = (((unsigned long long)(unsigned)((hi & 0xfffff) | (e ? 0x100000 : 0))) << 32) | (unsigned)__double2loint(v);
  f = (((f << 5) >> min(top - e, 63)) + 1) >> 1;
  const long long g = hi < 0 ? -(long long)f : (long long)f;
  const unsigned lo = __reduce_add_sync(full, (unsigned)g & 0xffffffu);
  const unsigned mid = __reduce_add_sync(full, (unsigned)(g >> 24) & 0xffffffu);
  const int up = __reduce_add_sync(full, (int)(g >> 48));
  const double t = (double)((long long)lo + ((long long)mid << 24) + ((long long)up << 48));
  const int ht = __double2hiint(t), et = ((ht >> 20) & 0x7ff) + top - 1079;   // units of 2^(top - 1075 - 4)
  if (top == 0x7ff) return __hiloint2double(0x7ff80000, 0);
  if (et <= 0) return 0.0;   // t = 0 too: its exponent field is 0
  if (et >= 0x7ff) return __hiloint2double((ht & (int)0x80000000) | 0x7ff00000, 0);
  return __hiloint2double(ht + ((top - 1079) << 20), __double2loint(t));
}

}  // namespace pqmc
