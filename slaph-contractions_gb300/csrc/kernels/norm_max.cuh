// Largest norm of a column of complex entries without the FP64 units.
//
// |v|^2 in FP64 is three operations per entry on units that issue two per cycle
// and SM, which bounds a scan of the eigenvectors at 2.5 TB/s.  The norms are
// taken in FP32 from mantissas cut to 23 bits instead: the largest |v|^2 then
// lies between n2 (1 - 2^-20) and n2 (1 + 2^-20), which settles its exponent
// unless those two differ in theirs (or the entries leave the FP32 range).
#pragma once

#include <cuda_runtime.h>

#include "kernels.cuh"

namespace slaph {
namespace dev {

// |v| as a float, the mantissa cut to 23 bits: integer operations on the two
// words, for 2^-126 <= |v| < 2^128 (smaller gives zero).  hi: the high word.
__device__ __forceinline__ float abs_cut(double v, unsigned int &hi) {
  hi = static_cast<unsigned int>(__double2hiint(v)) & 0x7FFFFFFFu;
  int const t = static_cast<int>(hi) - (896 << 20);
  return t < (1 << 20) ? 0.f
                       : __uint_as_float(__funnelshift_l(static_cast<unsigned int>(__double2loint(v)),
                                                         static_cast<unsigned int>(t), 3));
}
__device__ __forceinline__ void norm_max(NormMax &m, double2 v) {
  unsigned int h0, h1;
  float const p = abs_cut(v.x, h0), q = abs_cut(v.y, h1);
  m.top = max(m.top, max(h0, h1));
  m.n2 = max(m.n2, __float_as_uint(fmaf(p, p, q * q)));  // non-negative: order of the bits
}
// The warp's largest into *m (all 32 lanes call).
__device__ __forceinline__ void norm_max_add(NormMax *m, NormMax const &x) {
  unsigned int const top = __reduce_max_sync(0xffffffffu, x.top);
  unsigned int const n2 = __reduce_max_sync(0xffffffffu, x.n2);
  if (threadIdx.x % 32 == 0) {
    atomicMax(&m->top, top);
    atomicMax(&m->n2, n2);
  }
}

}  // namespace dev
}  // namespace slaph
