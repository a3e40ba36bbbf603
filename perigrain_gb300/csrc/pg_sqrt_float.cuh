// (float)sqrt(x), the FP64 square root rounded again, without the FP64 root: c = sqrtf((float)x) is at
// most one float off, and the exact remainder x - c c tells on which side of the halfway point between
// two floats the root lies. Only within 2^-18 ulp of that point (where the second rounding could matter),
// at a power of two and outside 1e-30..1e30 is the FP64 root itself taken. 300 cycles against 760: an
// FP64 operation has a latency of 63 cycles here, and a square root chains ten.
//
// Host and device share the code, so the margins are tested on the host, with the quotient's estimate
// (two units in the last place on the GPU) scaled by PG_SQRT_FLOAT_EST_SCALE.
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>

#ifndef PG_SQRT_FLOAT_EST_SCALE
#define PG_SQRT_FLOAT_EST_SCALE 1.0f
#endif

namespace pg {

#ifdef __CUDACC__
__host__ __device__ __forceinline__
#else
inline
#endif
    float
    sqrt_to_float(double x) {
  const float a = (float)x;
  const float c = sqrtf(a);
  uint32_t cb;
  float est, up;
#ifdef __CUDA_ARCH__
  cb = __float_as_uint(c);
  up = __uint_as_float(cb + 1u) - c;
  est = __fdividef(0.5f, c);
  // c as a double by its bits (the conversion runs on the FP64 pipe); only a normal c is used below
  const double cd = __longlong_as_double((long long)(((uint64_t)(cb >> 23) + 896u) << 52 |
                                                     (uint64_t)(cb & 0x7fffffu) << 29));
#else
  std::memcpy(&cb, &c, 4);
  const uint32_t ub = cb + 1u;
  std::memcpy(&up, &ub, 4);
  up -= c;
  est = 0.5f / c * PG_SQRT_FLOAT_EST_SCALE;
  const double cd = c;
#endif
  const float off = (float)fma(-cd, cd, x) * est;  // sqrt(x) - c
  const float h = 0.5f * up, ao = fabsf(off);
  if (a > 1e-30f && a < 1e30f && (cb & 0x7fffffu) > 1u && (cb & 0x7fffffu) < 0x7ffffeu) {
    if (ao < h * 0.999996f) return c;
    if (ao > h * 1.000004f && ao < 1.4f * up) {
      const uint32_t rb = off > 0.f ? cb + 1u : cb - 1u;
      float r;
#ifdef __CUDA_ARCH__
      r = __uint_as_float(rb);
#else
      std::memcpy(&r, &rb, 4);
#endif
      return r;
    }
  }
  return (float)sqrt(x);
}

}  // namespace pg
