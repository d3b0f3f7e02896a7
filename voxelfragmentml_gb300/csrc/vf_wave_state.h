// vf_wave_state.h -- the two state planes of the flood's rows (vf_flood.cu).
//
// A row is 32 voxels along the words' axis, bit by bit in the planes A and B:
//
//   A B
//   1 0   EMPTY
//   0 1   U, occupied and not claimed yet
//   0 0   E0, claimed by a wave of odd number (a seed: wave -1)
//   1 1   E1, claimed by a wave of even number
//
// Wave t reads the rows around a row while their owners claim voxels in them, and
// a reader may see a row's words from different times: a vector access is a set of
// 32-bit ones in no order.  A claim of wave t changes U into E((t + 1) & 1), which
// is one bit of ONE plane, so no mix of old and new words shows a bit in E(t & 1)
// that was not there before the wave, nor in U.  (With EMPTY 00 and E0 10 a claim
// of an odd wave changes both planes, and the new A with the old B reads as E1:
// claimed by the wave before.)  All that is asked of the hardware is that a 32-bit
// word is read as it was before or after a store.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define VF_WAVE_FN __host__ __device__ __forceinline__
#else
#define VF_WAVE_FN inline
#endif

// the planes of a row with these voxels occupied, none claimed
VF_WAVE_FN uint32_t wave_empty_a(uint32_t occupied) { return ~occupied; }
VF_WAVE_FN uint32_t wave_empty_b(uint32_t occupied) { return occupied; }

VF_WAVE_FN uint32_t wave_unclaimed(uint32_t a, uint32_t b) { return b & ~a; }
VF_WAVE_FN uint32_t wave_claimed(uint32_t a, uint32_t b) { return ~(a ^ b); }
// E(t & 1): what wave t dilates
VF_WAVE_FN uint32_t wave_front(uint32_t a, uint32_t b, uint32_t t) {
  const uint32_t m = t & 1u ? 0u : ~0u;
  return (a ^ m) & (b ^ m);
}
// wave t claims the unclaimed voxels n
VF_WAVE_FN void wave_claim(uint32_t& a, uint32_t& b, uint32_t n, uint32_t t) {
  if (t & 1u) b &= ~n; else a |= n;
}
