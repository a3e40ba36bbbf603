// Host-side entry points of the mixed-precision kernels (pg_kernels_mixed.cu).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "pg_device.cuh"
#include "pg_kernels.h"

namespace pg {

cudaError_t kernels_mixed_init();
// The parts of a mixed-precision step, as in pg_kernels.h.
void launch_mixed_predict(const Dev& P, cudaStream_t s, uint64_t* launches, bool pdl);
void launch_mixed_body(const Dev& P, const LaunchCfg& L, cudaStream_t s, uint64_t* launches, bool pdl,
                       bool rec = false, cudaEvent_t e0 = nullptr, cudaEvent_t e1 = nullptr);
void launch_mixed_finalize(const Dev& P, cudaStream_t s, uint64_t* launches, bool pdl);

}  // namespace pg
