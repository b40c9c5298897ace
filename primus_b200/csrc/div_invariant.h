// Quotients by a divisor that is the same for many numerators (host and device).
#pragma once
#include <cmath>

#ifdef __CUDACC__
#define PB_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define PB_HOST_DEVICE inline
#endif

namespace pb {

// a / b, correctly rounded, for 0 <= b <= 1 and r = 1 / b correctly rounded (an invariant b: the caller has it once).
// An estimate, its remainder (fma) and two corrections: the first brings any estimate to within one step of the last
// place, from there the second gives the correctly rounded quotient (P. Markstein, "Computation of elementary functions on
// the IBM RISC System/6000 processor", 1990), whose premise the estimate alone does not meet for every b.  The remainder is
// exact while its last place, that of a times 2^-47, is no subnormal; numerators below (m, v of an element that hardly ever
// sees a gradient) and quotients that could overflow take the division.  Zeros are common and keep their sign.
PB_HOST_DEVICE float div_invariant(float a, float b, float r) {
  const float q = a * r;
  const float c = fmaf(fmaf(-q, b, a), r, q);
  const float d = fmaf(fmaf(-c, b, a), r, c);
  if (fabsf(a) >= 0x1p-100f && fabsf(q) <= 0x1p126f) return d;
  return a == 0.f ? q : a / b;
}

}  // namespace pb
