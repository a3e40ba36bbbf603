// On-device post-processing of a snapshot (C ABI pg_postprocess of include/perigrain.h): the
// per-grain and per-instance quantities the reference's scripts compute by reading every
// tc_%05u.h5 / wall_%05u.h5 back into numpy --
//   damage per node (deg0 - deg) / deg0 and its grain mean   read_sim_output.py:126-133,
//                                                            gen_damage_data.py:55-66
//   grain means of vel, acc, CurrPos; grain sum of force     read_sim_output.py:201-232
//   sum of vol * rho * acc                                   read_sim_output.py:305-312
//   volume fraction = grain volume / wall box volume        read_sim_output.py:183-196
// -- from the state already in HBM, so a run's time series needs no snapshot download. One block
// per grain reduces its nodes in a fixed order (deterministic); only the per-grain sums leave the
// device.
#include <cuda_runtime.h>

#include <cmath>
#include <vector>

#include "pg_common.cuh"
#include "pg_device.cuh"
#include "pg_handle.h"
#include "pg_ieee64.cuh"

using namespace pg;

namespace {

constexpr int POST_THREADS = 256;
constexpr int POST_WARPS = POST_THREADS / 32;

// per grain: sum vel[D], sum acc[D], sum CurrPos[D], sum force[D], sum vol*rho*acc[D],
// sum damage, sum vol; then the node count and the instance, as numbers
template <int D>
__host__ __device__ constexpr int post_ns() {
  return 5 * D + 2;
}
template <int D>
__host__ __device__ constexpr int post_nq() {
  return post_ns<D>() + 2;
}

// Damage of each node, at its place in the input's order: intact bonds now against bonds at
// creation (each bond sits in both endpoints' rows). A pass of its own, a lane a device node: a
// warp's nodes share their chunk's bond words, so the words are broadcast loads and enough warps are
// in flight to hide them, which the grain sums' few warps did not (68 us with the sums for 390k nodes
// in 512 grains; 8 us here and 29 there now, where the FP64 pipe adds).
__global__ void __launch_bounds__(256) k_post_damage(const Dev P, double* q) {
  const uint32_t i = blockIdx.x * 256 + threadIdx.x;
  if (i >= P.N) return;
  const uint32_t lane = i & 31, deg0 = P.node_deg[i];
  const uint32_t* w = P.alive + P.chunk_word[i >> 5];
  uint32_t deg = 0;
#pragma unroll 8
  for (uint32_t k = 0; k < deg0; ++k) deg += (w[k] >> lane) & 1u;
  double v = 0.0;
  if (deg != deg0 || !deg0) v = ieee64::div_rn((double)deg0 - (double)deg, (double)deg0);  // 0/0 -> NaN, as numpy
  q[orig_of(P, i)] = v;
}

template <int D>
struct PostNode {
  double v[D], x[D], a[D], f[D], vol, q;
  __device__ __forceinline__ void load(const Dev& P, const double* vel, const double* damage, uint32_t o) {
    const uint32_t i = at_of(P, o);
    ldv<D>(vel, i, v);
    ldv<D>(P.cur, i, x);
    if (P.acc_f) {
      constexpr uint32_t SF = D == 2 ? 2 : 4;
#pragma unroll
      for (int c = 0; c < D; ++c) {
        a[c] = ieee64::widen_f32(P.acc_f[(size_t)i * SF + c]);
        f[c] = ieee64::widen_f32(P.force_f[(size_t)i * SF + c]);
      }
    } else {
      ldv<D>(P.acc, i, a);
      ldv<D>(P.force, i, f);
    }
    vol = P.vol[i];
    q = damage[o];
  }
};

// The sums of a grain, one block a grain: thread t adds the nodes t, t + 256, ... of the input's order,
// and the 256 partial sums are folded by halves, a warp a quantity. The next node is loaded while one
// is added. Block b also copies its share of the walls and the device status behind the grains' sums,
// so that one copy brings the host all it needs.
template <int D>
__global__ void __launch_bounds__(POST_THREADS) k_post(const Dev P, const double* vel, const double* damage,
                                                       double* out) {
  constexpr int NS = post_ns<D>(), NQ = post_nq<D>();
  __shared__ double red[NS][POST_THREADS];
  const uint32_t g = blockIdx.x, tid = threadIdx.x, lane = tid & 31;
  if (g < P.G) {
    const GrainDev& gr = P.grain[g];
    const double rho = gr.rho;
    const uint32_t end = gr.node_end;
    double s[NS];
#pragma unroll
    for (int k = 0; k < NS; ++k) s[k] = 0.0;
    PostNode<D> n, m;
    uint32_t o = gr.node_begin + tid;
    if (o < end) n.load(P, vel, damage, o);
    for (; o < end; o += POST_THREADS) {
      if (o + POST_THREADS < end) m.load(P, vel, damage, o + POST_THREADS);
#pragma unroll
      for (int c = 0; c < D; ++c) {
        s[c] += n.v[c];
        s[D + c] += n.a[c];
        s[2 * D + c] += n.x[c];
        s[3 * D + c] += n.f[c];
        s[4 * D + c] += (n.vol * rho) * n.a[c];
      }
      s[5 * D] += n.q;
      s[5 * D + 1] += n.vol;
      n = m;
    }
#pragma unroll
    for (int k = 0; k < NS; ++k) red[k][tid] = s[k];
    __syncthreads();
    double* sum = out + (size_t)g * NQ;
    for (int k = (int)(tid >> 5); k < NS; k += POST_WARPS) {
      double r[POST_WARPS];
#pragma unroll
      for (int j = 0; j < POST_WARPS; ++j) r[j] = red[k][32 * j + lane];
#pragma unroll
      for (int w = POST_WARPS / 2; w > 0; w >>= 1)
#pragma unroll
        for (int j = 0; j < w; ++j) r[j] += r[j + w];
#pragma unroll
      for (int w = 16; w > 0; w >>= 1) r[0] += __shfl_down_sync(0xffffffffu, r[0], w);
      if (lane == 0) sum[k] = r[0];
    }
    if (tid == 0) {
      sum[NS] = (double)(end - gr.node_begin);
      sum[NS + 1] = (double)gr.inst;
    }
  }
  double* rest = out + (size_t)P.G * NQ;
  const uint32_t walls = P.I * 2 * D;
  for (uint32_t k = g * POST_THREADS + tid; k < walls; k += gridDim.x * POST_THREADS)
    rest[k] = P.inst[k / (2 * D)].wall[k % (2 * D)];
  if (g == 0 && tid == 0) rest[walls] = (double)*P.status;
}

}  // namespace

extern "C" int pg_postprocess(pg_handle* h, const pg_post* out) {
  if (!h || !out) return pg_fail(PG_EINVAL, "null argument");
  Dev P = h->P;
  P.cur = h->cur();
  const uint32_t D = h->dim, G = P.G, I = P.I, N = P.N, NS = 2 * D;
  const int NQ = (D == 2) ? post_nq<2>() : post_nq<3>();
  const size_t n_out = (size_t)G * NQ + (size_t)I * NS + 1;  // sums, walls, status
  if (!h->post_sum) CU(h->dalloc(&h->post_sum, n_out));
  if (!h->post_damage) CU(h->dalloc(&h->post_damage, N));
  const double* vel = h->vel_parity == 0 ? h->vel_a : h->vel_b;
  if (N) k_post_damage<<<(N + 255) / 256, 256, 0, h->stream>>>(P, h->post_damage);
  if (D == 2) {
    k_post<2><<<G ? G : 1, POST_THREADS, 0, h->stream>>>(P, vel, h->post_damage, h->post_sum);
  } else {
    k_post<3><<<G ? G : 1, POST_THREADS, 0, h->stream>>>(P, vel, h->post_damage, h->post_sum);
  }
  CU(cudaGetLastError());
  std::vector<double> gs(n_out);
  CU(cudaMemcpyAsync(gs.data(), h->post_sum, n_out * 8, cudaMemcpyDeviceToHost, h->stream));
  CU(cudaStreamSynchronize(h->stream));
  const int32_t st = (int32_t)gs[n_out - 1];
  if (st == PG_ETIMEOUT) h->halted = true;
  int rc = device_status_fail(st);
  if (rc) return rc;
  if (out->node_damage && N) {
    CU(cudaMemcpyAsync(out->node_damage, h->post_damage, (size_t)N * 8, cudaMemcpyDeviceToHost, h->stream));
    CU(cudaStreamSynchronize(h->stream));
  }
  std::vector<double> inert((size_t)I * D, 0.0), vol((size_t)I, 0.0);
  for (uint32_t g = 0; g < G; ++g) {
    const double* q = &gs[(size_t)g * NQ];
    const double n = q[5 * D + 2];
    const size_t inst = (size_t)q[5 * D + 3];
    for (uint32_t c = 0; c < D; ++c) {
      if (out->grain_mean_vel) out->grain_mean_vel[(size_t)g * D + c] = q[c] / n;
      if (out->grain_mean_acc) out->grain_mean_acc[(size_t)g * D + c] = q[D + c] / n;
      if (out->grain_mean_currpos) out->grain_mean_currpos[(size_t)g * D + c] = q[2 * D + c] / n;
      if (out->grain_force) out->grain_force[(size_t)g * D + c] = q[3 * D + c];
      inert[inst * D + c] += q[4 * D + c];  // per instance, grains in order
    }
    if (out->grain_damage) out->grain_damage[g] = q[5 * D] / n;
    vol[inst] += q[5 * D + 1];
  }
  if (out->inertial_force)
    for (size_t k = 0; k < inert.size(); ++k) out->inertial_force[k] = inert[k];
  if (out->volume_fraction)
    for (uint32_t k = 0; k < I; ++k) {
      const double* wi = &gs[(size_t)G * NQ + (size_t)k * NS];
      // the wall box volume of extract_bulk (read_sim_output.py:183-196), its index pairing kept
      const double wv = (D == 2) ? (wi[1] - wi[0]) * (wi[2] - wi[3])
                                 : (wi[1] - wi[0]) * (wi[3] - wi[2]) * (wi[5] - wi[4]);
      out->volume_fraction[k] = vol[k] / wv;
    }
  return PG_OK;
}
