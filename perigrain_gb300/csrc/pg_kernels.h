// Host-side entry points of the device kernels (pg_kernels.cu, pg_kernels_mixed.cu).
#pragma once
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>

#include "pg_device.cuh"

namespace pg {

struct LaunchCfg {
  uint32_t force_block = 128;   // threads per block of the fused force kernel (multiple of 32, <= 128)
  uint32_t cells_per_node = 4;  // grid capacity per node of an instance
};

// Per-thread local memory of this process's context at least `bytes` (cudaLimitStackSize), so
// kernels with local frames above the default limit find room for them.
inline cudaError_t ensure_local_bytes(size_t bytes) {
  size_t cur = 0;
  cudaError_t e = cudaDeviceGetLimit(&cur, cudaLimitStackSize);
  if (e != cudaSuccess || cur >= bytes) return e;
  return cudaDeviceSetLimit(cudaLimitStackSize, (bytes + 255) / 256 * 256);
}
// The largest local frame (cudaFuncAttributes::localSizeBytes) among the kernels `fs`; asked for once
// (*known, 0 before), as it is a constant of the compiled code and the 144 force kernels take a tenth of a
// small handle's creation to ask.
inline cudaError_t max_local_bytes(const void* const* fs, int n, std::atomic<size_t>* known, size_t* out) {
  size_t m = known->load(std::memory_order_relaxed);
  if (m) {
    *out = m;
    return cudaSuccess;
  }
  for (int k = 0; k < n; ++k) {
    cudaFuncAttributes a;
    const cudaError_t e = cudaFuncGetAttributes(&a, fs[k]);
    if (e != cudaSuccess) return e;
    m = a.localSizeBytes > m ? a.localSizeBytes : m;
  }
  known->store(m, std::memory_order_relaxed);
  *out = m;
  return cudaSuccess;
}

// Blocks of 128 threads per SM the force kernels are compiled for that suit a handle of n_chunks
// warps: a warp holds its slot for its whole chunk, so the time grows with the number of rounds of
// resident warps times the warps that share an SM in each, rounds * bps; the smallest product wins,
// the larger register budget on a tie. The product picks the fastest of those measured but is no model
// of the times: an SM is not 1.4 times as fast with 7 blocks as with 5, and a last round is seldom full.
// Mixed, us a step at 5 / 6 / 7 blocks (product): collision ensemble (80 warps an SM) 70 / 71 / 62
// (25 / 24 / 21), 3D spheres (26) 87 / 110 / 86 (10 / 12 / 7), settling (24) 20.7 / 17.9 / 19.0
// (10 / 6 / 7), two disks (1) 12.5 / 13.9 / 14.0 (5 / 6 / 7).
inline int force_bps(uint32_t n_chunks, uint32_t sms) {
  int best = 5;
  uint64_t best_cost = ~0ull;
  for (int b = 5; b <= 7; ++b) {
    const uint64_t slots = (uint64_t)sms * 4 * b, cost = (n_chunks + slots - 1) / slots * b;
    if (cost < best_cost) {
      best_cost = cost;
      best = b;
    }
  }
  return best;
}

// Whether the mixed force kernel puts a team of four warps on a chunk (candidate lists and the default
// block of 128 threads only): where all teams are resident at once, 4 blocks of 128 threads (128
// registers) an SM. us a step, a warp / a team a chunk: settling 179 chunks 11.9 / 8.0, 544 11.9 / 9.5,
// 726 12.1 / 14.0, 1089 12.6 / 14.9; 3D spheres 242 chunks 27.8 / 16.6, 545 28.0 / 21.7, 847 30.1 /
// 38.0; two disks (79 chunks) 13.3 / 9.7.
inline bool force_team(const Dev& P, uint32_t block) {
  return P.cand_q && block == 128 && P.n_chunks <= P.n_sms * 4u;
}

cudaError_t kernels_init();
// The parts of an FP64 step, each enqueued on stream s: the position update; the grid build and the
// force kernels; the end of the step. Add the number of kernel launches to *launches. pdl:
// programmatic dependent launch behind the kernel before. With rec the force kernel also records
// the step's contact and wall masks (Dev::rec_*); e0/e1 (may be null) are recorded around the force
// kernels (pdl must be false then).
void launch_predict(const Dev& P, cudaStream_t s, uint64_t* launches, bool pdl);
void launch_body(const Dev& P, const LaunchCfg& L, cudaStream_t s, uint64_t* launches, bool pdl, bool rec = false,
                 cudaEvent_t e0 = nullptr, cudaEvent_t e1 = nullptr);
void launch_finalize(const Dev& P, cudaStream_t s, uint64_t* launches, bool pdl);
// Blocks of the cooperative grid build (k_grid_coop): every block resident at once (occupancy x
// SMs), no more than the work needs; 0 when the device has no cooperative launch.
uint32_t grid_coop_blocks(const Dev& P, int device);
// out[i] = op(a[i], b[i]) through the integer FP64 routines (pg_ieee64.cuh), op a pg_ieee_op;
// device pointers, n < 2^31 * 256.
cudaError_t launch_ieee64_check(int32_t op, const double* a, const double* b, int64_t n, double* out,
                                cudaStream_t s);

}  // namespace pg
