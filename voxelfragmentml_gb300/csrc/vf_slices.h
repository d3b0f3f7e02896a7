// vf_slices.h -- where a coordinate lies among the slice planes of the tetrahedra.
#pragma once
#include <cmath>
#include <cstdint>

#ifdef __CUDACC__
#define VF_SLICE_FN __host__ __device__ __forceinline__
#else
#define VF_SLICE_FN inline
#endif

// The first of n planes above v, or n (also for NaN, which no plane is above).  The
// planes are -1, -1 + 2 / n, ... added up, so one is near (v + 1) n / 2 and its
// neighbours are looked at from there.  The guess is brought into range as a float:
// v is any coordinate of a mesh in units of the box the caller gave.
template <class Planes>
VF_SLICE_FN uint32_t slice_above(const Planes& a, uint32_t n, float v) {
  const float guess = (v + 1.0f) * (0.5f * (float)n) + 1.0f;
  uint32_t i = (uint32_t)fmaxf(fminf(guess, (float)n), 0.0f);
  while (i > 0 && a[i - 1] > v) --i;
  while (i < n && !(a[i] > v)) ++i;
  return i;
}
