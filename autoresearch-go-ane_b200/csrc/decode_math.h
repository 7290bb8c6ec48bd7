// Divisions and square roots of the persistent decode kernels, from a constant of the host or from the hardware's approximation.
// A division, like an IEEE square root, is a long run of dependent instructions, and where it is reached once in a phase they come
// from beyond the instruction cache: between the sum of squares and the first normalised column, 1 / sqrtf(x / dim) took 2000 cycles.
// Plain C++, for host compilers too.
#pragma once
#include <math.h>
#include <stdint.h>

#ifdef __CUDACC__
#define ANE_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define ANE_HOST_DEVICE inline
#endif

namespace ane {

// n / d for 0 <= n < 2^16 and 1 <= d < 2^16 with magic = quotient_magic(d): n * magic / 2^32 is n / d and at most n / 2^32 more, too
// little to reach the next whole number.
inline unsigned quotient_magic(unsigned d) { return 0xffffffffu / d + 1u; }
ANE_HOST_DEVICE int quotient(int n, int d, unsigned magic) {
#ifdef __CUDA_ARCH__
  return d == 1 ? n : (int)__umulhi((unsigned)n, magic);
#else
  return d == 1 ? n : (int)((uint64_t)n * magic >> 32);
#endif
}

// 1 / x from an approximation within two ulps: one step of Newton's method.
ANE_HOST_DEVICE float newton_inverse(float x, float approx) { return fmaf(approx, fmaf(-x, approx, 1.f), approx); }
// o / x from such an inverse: the remainder of the first quotient is exact, and what its share of the inverse's error leaves is 2^-46,
// so that it is rounded as IEEE division rounds it but where o / x is that near to the middle between two numbers.  An infinite o
// stays infinite (it has no remainder).
ANE_HOST_DEVICE float divide(float o, float x, float inverse) {
  const float q = o * inverse;
  return fabsf(q) < INFINITY ? fmaf(fmaf(-x, q, o), inverse, q) : q;
}
// 1 / sqrt(x) from an approximation within two ulps: one step of Newton's method leaves the rounding of x * approx, half of which
// passes on, and its own: 1.01 ulp (1.f / sqrtf(x): 1.49).  1 / sqrt(inf) stays 0, as in the norms of the forward pass (the step
// alone would make it NaN).  x * approx in two parts, for 0.51 ulp, took registers: one sequence 13.7 -> 14.3 ms.
ANE_HOST_DEVICE float newton_inverse_sqrt(float x, float approx) {
  const float y = approx;
  return y == 0.f ? y : fmaf(0.5f * y, fmaf(-x * y, y, 1.f), y);
}

}  // namespace ane
