// Layout of the mixed path's FP32 hi/lo vectors (Dev::dref, Dev::xref and the gradient tape's
// displacements): x = hi + lo. 2D: one float4 per node, [hi.xy, lo.xy]. 3D: a float4 [hi.xyz, lo.x]
// per node, then a float2 [lo.yz] per node from float 4 np on (np: nodes padded to whole chunks).
//
// Displacements and reference positions sit in arrays of their own: the k-th neighbours of a warp's
// 32 nodes are mostly consecutive, so a 16-byte gather touches 512 consecutive bytes, four
// wavefronts of the L1 data pipe. As one 32-byte record the two halves took eight each (the pipe
// 55 % busy in the 2D force kernel, 40 % as it stands), and 3D in 12 planes of single floats took 12
// loads a bond. Step times, records and planes against this: 3D spheres 99.0 -> 91.2 us, settling
// 22.3 -> 21.4, two disks 15.8 -> 15.7, collision ensemble 72.5 -> 73.1.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace pg {

template <int D>
constexpr uint32_t HL_FLOATS = D == 2 ? 4u : 6u;  // floats per node

template <int D>
__device__ __forceinline__ void ld_hl(const float* __restrict__ a, uint32_t np, uint32_t i, float (&h)[D],
                                      float (&l)[D]) {
  const float4 p = __ldg(reinterpret_cast<const float4*>(a) + i);
  h[0] = p.x;
  h[1] = p.y;
  if constexpr (D == 2) {
    l[0] = p.z;
    l[1] = p.w;
  } else {
    const float2 q = __ldg(reinterpret_cast<const float2*>(a + 4ull * np) + i);
    h[2] = p.z;
    l[0] = p.w;
    l[1] = q.x;
    l[2] = q.y;
  }
}
template <int D>
__device__ __forceinline__ void st_hl(float* a, uint32_t np, uint32_t i, const float (&h)[D], const float (&l)[D]) {
  if constexpr (D == 2) {
    reinterpret_cast<float4*>(a)[i] = make_float4(h[0], h[1], l[0], l[1]);
  } else {
    reinterpret_cast<float4*>(a)[i] = make_float4(h[0], h[1], h[2], l[0]);
    reinterpret_cast<float2*>(a + 4ull * np)[i] = make_float2(l[1], l[2]);
  }
}

}  // namespace pg
