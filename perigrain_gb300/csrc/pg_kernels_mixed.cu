// GB300 (sm_103a) kernels of the PeriDEM time step, mixed precision (PG_MIXED).
//
// State that accumulates over time stays FP64: disp, vel, pos and CurrPos. Everything per bond and
// per contact pair is FP32:
//   * the bond reference vector xi = x_j - x_i and the deformation eta = u_j - u_i are formed from
//     FP32 hi/lo pairs of the FP64 values, (hi_j - hi_i) + (lo_j - lo_i), which keeps ~48 bits of
//     the FP64 difference without an FP64 instruction;
//   * the stretch is evaluated without cancellation,
//       s = (|xi + eta| - |xi|) / |xi| = (2 xi.eta + eta.eta) / (|xi| (|xi + eta| + |xi|)),
//     so its relative error stays ~1e-7 even for stretches of 1e-6, where the reference form
//     would lose every digit in FP32;
//   * forces accumulate per node in FP32; the velocity update adds them to the FP64 state.
// The bond stream is the neighbour index plus one alive bit (4.125 B per directed bond; the FP64
// path also streams xi_norm). Compiled with FMA contraction on.
#include <cuda_runtime.h>

#include <cmath>

#include "pg_common.cuh"
#include "pg_device.cuh"
#include "pg_hilo.cuh"
#include "pg_kernels_mixed.h"

namespace pg {

// FP64 <-> FP32 moves done with integer instructions: GB300 executes FP64 arithmetic and the
// F2F conversions on its narrow FP64 pipe (~1/64 of the FP32 rate), so the per-node hi/lo split
// and the float->double widening below use bit manipulation on the INT pipe instead.
//
// trunc_f32: x truncated to 24 significant bits, as a float and (exactly) as a double. Values
// below the FP32 normal range become 0 (their size is < 1.2e-38); inf/NaN take the converting
// path so they propagate.
__device__ __forceinline__ float trunc_f32(double x, double* as_double) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const unsigned int hw = (unsigned int)(b >> 32);
  const int e = (int)((hw >> 20) & 0x7ffu);
  const unsigned int sgn = hw & 0x80000000u;
  if (e < 1023 - 126) {  // below the FP32 normal range: 0
    *as_double = 0.0;
    return __uint_as_float(sgn);
  }
  if (e > 1023 + 127) {  // beyond FP32 (inf/NaN included): inf or NaN, and lo = x - x
    *as_double = x;
    const bool nan = (e == 0x7ff) && ((b & 0xfffffffffffffull) != 0);
    return __uint_as_float(sgn | 0x7f800000u | (nan ? 0x400000u : 0u));
  }
  *as_double = __longlong_as_double((long long)(b & ~((1ull << 29) - 1)));
  return __uint_as_float(sgn | ((unsigned int)(e - 896) << 23) | (unsigned int)((b >> 29) & 0x7fffffu));
}
// Exact widening of a float; subnormal floats become a signed zero.
__device__ __forceinline__ double widen(float f) {
  const unsigned int b = __float_as_uint(f);
  const unsigned int e = (b >> 23) & 0xffu;
  const unsigned long long sgn = (unsigned long long)(b & 0x80000000u) << 32;
  if (e == 0) return __longlong_as_double((long long)sgn);
  const unsigned long long ee = (e == 0xff) ? 0x7ffull : (unsigned long long)(e + 896);
  return __longlong_as_double((long long)(sgn | (ee << 52) | ((unsigned long long)(b & 0x7fffffu) << 29)));
}
// hi/lo pair: x = hi + lo + O(2^-47 |x|); hi = trunc_f32(x), lo = trunc_f32(x - hi). When hi is an
// FP32 normal number the difference x - hi is exactly x's low 29 mantissa bits, so lo is formed
// from them with integer instructions (identical bits, no FP64 subtraction); otherwise the FP64
// route.
__device__ __forceinline__ void split_hl(double x, float* hi, float* lo) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const unsigned int hw = (unsigned int)(b >> 32);
  const int e = (int)((hw >> 20) & 0x7ffu);
  if (e < 1023 - 126 || e > 1023 + 127) {
    double hd, ld;
    *hi = trunc_f32(x, &hd);
    *lo = trunc_f32(x - hd, &ld);
    return;
  }
  const unsigned int sgn = hw & 0x80000000u;
  *hi = __uint_as_float(sgn | ((unsigned int)(e - 896) << 23) | (unsigned int)((b >> 29) & 0x7fffffu));
  const unsigned int r = (unsigned int)(b & ((1ull << 29) - 1));
  if (r == 0) {  // x - hi = +0
    *lo = 0.0f;
    return;
  }
  const int p = 31 - __clz(r);  // leading bit of the remainder
  const int ed = e + p - 52;     // biased FP64 exponent of x - hi
  if (ed < 1023 - 126) {         // below the FP32 normal range: signed zero
    *lo = __uint_as_float(sgn);
    return;
  }
  const unsigned int frac = (p <= 23) ? ((r << (23 - p)) & 0x7fffffu) : ((r >> (p - 23)) & 0x7fffffu);
  *lo = __uint_as_float(sgn | ((unsigned int)(ed - 896) << 23) | frac);
}

template <int D>
__device__ __forceinline__ void ldvf(const float* a, uint32_t i, float (&v)[D]) {
  if constexpr (D == 2) {
    float2 t = reinterpret_cast<const float2*>(a)[i];
    v[0] = t.x;
    v[1] = t.y;
  } else {
    float4 t = reinterpret_cast<const float4*>(a)[i];
    v[0] = t.x;
    v[1] = t.y;
    v[2] = t.z;
  }
}
template <int D>
__device__ __forceinline__ void stvf(float* a, uint32_t i, const float (&v)[D]) {
  if constexpr (D == 2) {
    reinterpret_cast<float2*>(a)[i] = make_float2(v[0], v[1]);
  } else {
    reinterpret_cast<float4*>(a)[i] = make_float4(v[0], v[1], v[2], 0.f);
  }
}
template <int D>
__device__ __forceinline__ float dotf(const float (&a)[D], const float (&b)[D]) {
  float s = a[0] * b[0];
  for (int c = 1; c < D; ++c) s = fmaf(a[c], b[c], s);
  return s;
}

// CurrPos of node d from its displacement, its FP32 images, and either the list-rebuild check or the
// node's grid key.
template <int D>
__device__ __forceinline__ void place_node_mx(const Dev& P, uint32_t d, const InstDev& in, const double (&dp)[D],
                                              const double (&ps)[D], const float (&db)[D], double* cur, float* curf,
                                              float* dref, uint32_t* rebuild, double (&cu)[D]) {
  float dh[D], dl[D];
  for (int c = 0; c < D; ++c) split_hl(dp[c], &dh[c], &dl[c]);
  st_hl<D>(dref, P.np, d, dh, dl);
  for (int c = 0; c < D; ++c) cu[c] = ps[c] + dp[c];
  stv<D>(cur, d, cu);
  // the FP32 position image: offset from the fixed frame with candidate lists, else from this step's
  // grid origin; formed in FP32 from the truncated CurrPos (integer instructions) -- an FP64
  // subtraction here would run on the narrow FP64 pipe, and the image only feeds the cell keys and
  // the FP32 prefilter
  float rf[D];
  bool ok = true;
  for (int c = 0; c < D; ++c) {
    if (((__double_as_longlong(cu[c]) >> 52) & 0x7ff) == 0x7ff) ok = false;  // inf or NaN
    double cut;
    rf[c] = trunc_f32(cu[c], &cut) - in.org_f[c];
  }
  if (!ok) set_status(P.status, PG_ENAN);
  stf<D>(curf, d, rf);
  if (P.cand_q) {
    // rebuild once any node has moved 0.45 skin since the last build
    float m2 = 0.f;
    for (int c = 0; c < D; ++c) {
      double dpt;
      const float dd = trunc_f32(dp[c], &dpt) - db[c];  // truncation (integer ops), not an FP64 conversion
      m2 += dd * dd;
    }
    if (m2 > in.skin_lim2) *rebuild = 1;
  } else {
    int32_t ci[3] = {0, 0, 0};
    for (int c = 0; c < D; ++c) ci[c] = cell_coord(rf[c] + in.frame_off_f[c], in.inv_cell_f, in.dims[c]);
    const uint32_t key =
        in.table_off + ((uint32_t)ci[2] * in.dims[1] + (uint32_t)ci[1]) * in.dims[0] + (uint32_t)ci[0];
    P.cell_key[d] = key;
    P.cell_rank[d] = atomicAdd(&P.cell_count[key], 1u);
  }
}

// disp += dt*v + (dt*dt/2)*a: the increment is formed in FP32 (relative error ~1e-7 of a step's
// motion); the accumulation into disp stays FP64
template <int D>
__device__ __forceinline__ void advance_mx(const Dev& P, const double (&v)[D], const float (&a)[D], double (&dp)[D]) {
  double vd;
  for (int c = 0; c < D; ++c) {
    const float vf = trunc_f32(v[c], &vd);
    dp[c] = dp[c] + widen(fmaf(P.dt_f, vf, P.hdt2_f * a[c]));
  }
}

// ---------------------------------------------------------------------------------------------
// position update: FP64 disp and CurrPos, plus their FP32 hi/lo images and the grid key
// ---------------------------------------------------------------------------------------------
template <int D>
__global__ void __launch_bounds__(256) k_predict_mx(const Dev P) {
  pdl_enter();
  const uint32_t d = blockIdx.x * blockDim.x + threadIdx.x;
  const bool act = d < P.N;
  uint32_t g = 0;
  double cu[D];
  for (int c = 0; c < D; ++c) cu[c] = 0.0;
  if (act) {
    // every per-node load is issued before the grain's flags are known, so they overlap
    g = P.node_grain[d];
    double dp[D], ps[D], v[D];
    float a[D], db[D];
    ldv<D>(P.disp, d, dp);
    ldv<D>(P.vel_in, d, v);
    ldvf<D>(P.acc_f, d, a);
    ldv<D>(P.pos, d, ps);
    for (int c = 0; c < D; ++c) db[c] = 0.f;
    if (P.cand_q) ldf<D>(P.disp_b, d, db);
    const bool pend = P.clamp_pending[d] != 0;
    const GrainDev& gr = P.grain[g];
    const bool mov = gr.flags & GF_MOVABLE;
    if (pend) {
      for (int c = 0; c < D; ++c) dp[c] = 0.0;
      P.clamp_pending[d] = 0;
    }
    if (mov) advance_mx<D>(P, v, a, dp);
    if (mov || pend) stv<D>(P.disp, d, dp);
    place_node_mx<D>(P, d, P.inst[gr.inst], dp, ps, db, P.cur, P.curf, P.dref, P.rebuild, cu);
  }
  grow_box<D>(P.bbox, g, act, cu);
}

// One bond: stretch s = (2 xi.eta + eta.eta) / (|xi| (|xi+eta| + |xi|)), force density
// cnot * s * vol_j * (xi+eta)/|xi+eta| added to f when `use`. cv = cnot * vol_j.
template <int D>
__device__ __forceinline__ void bond_term(const float (&dh)[D], const float (&dl)[D], const float (&xh)[D],
                                          const float (&xl)[D], const float (&jdh)[D], const float (&jdl)[D],
                                          const float (&jxh)[D], const float (&jxl)[D], float cv, bool use,
                                          float (&f)[D], float* str_out) {
  float xi[D], et[D], y[D];
  for (int c = 0; c < D; ++c) {
    xi[c] = (jxh[c] - xh[c]) + (jxl[c] - xl[c]);
    et[c] = (jdh[c] - dh[c]) + (jdl[c] - dl[c]);
    y[c] = xi[c] + et[c];
  }
  const float xx = dotf<D>(xi, xi), yy = dotf<D>(y, y);
  const float ixn = rsqrtf(xx), iyn = rsqrtf(yy);
  const float num = fmaf(2.f, dotf<D>(xi, et), dotf<D>(et, et));
  const float str = __fdividef(num * ixn, fmaf(yy, iyn, xx * ixn));
  const float sc = use ? cv * str * iyn : 0.f;
  for (int c = 0; c < D; ++c) f[c] = fmaf(sc, y[c], f[c]);
  *str_out = str;
}

// ---------------------------------------------------------------------------------------------
// fused force + integrate, FP32 forces
// ---------------------------------------------------------------------------------------------
// The input's index of device node i in a force kernel: PERM (the handle's node layout differs
// from the input order) looks it up, otherwise the layout is the input order and i is it.
template <bool PERM>
__device__ __forceinline__ uint32_t input_index(const Dev& P, uint32_t i) {
  if constexpr (PERM) return P.node_orig[i];
  return i;
}

template <int D, bool REC, bool GC, bool PERM, bool LIST, int BPS>
__global__ void __launch_bounds__(128, BPS) k_force_mx(const Dev P) {
  pdl_enter();
  pdl_release();
  const uint32_t d = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t chunk = d >> 5;
  if (chunk >= P.n_chunks) return;
  const bool act = d < P.N;
  const uint32_t t = *P.step;
  const uint32_t g = act ? P.node_grain[d] : 0;
  const GrainDev gr = P.grain[g];
  const bool mov = act && (gr.flags & GF_MOVABLE);

  float f[D];
  for (int c = 0; c < D; ++c) f[c] = 0.f;
  double vpd[D];
  if (act) ldv<D>(P.vel_in, d, vpd);
  // per-node inputs of the epilogue: in 2D loaded up front so their latency hides behind the bond
  // loop; in 3D where they are used (the extra live registers spill there and measured slower)
  constexpr int DE = (D == 2) ? D : 1;
  float ef_in[DE], ao_in[DE];
  bool clamped_in = false;
  if constexpr (D == 2) {
    if (mov) {
      ldvf<D>(P.extf_f, d, ef_in);
      ldvf<D>(P.acc_f, d, ao_in);
      clamped_in = P.clamped[d] != 0;
    }
  }

  const bool brk = P.enable_fracture && (gr.flags & GF_BREAKABLE) && (gr.flags & GF_BREAK_BONDS);
  const float cnot = gr.cnot_f, snot = brk ? gr.snot_f : INFINITY;  // never exceeded without the break test
  const uint32_t cdeg = P.chunk_deg[chunk];
  const uint32_t slot0 = P.chunk_slot[chunk] + lane;
  const uint32_t w0 = P.chunk_word[chunk];
  {
    // bond forces and bond breaking (particle2.h:102-232): two bonds per iteration, both
    // neighbour gathers issued before either is used
    float dh[D], dl[D], xh[D], xl[D];
    if (mov) {
      ld_hl<D>(P.dref, P.np, d, dh, dl);
      ld_hl<D>(P.xref, P.np, d, xh, xl);
    }
    if constexpr (REC) {
      if (mov && P.rec_df) st_hl<D>(P.rec_df, P.np, d, dh, dl);
    }
    // The alive words and neighbour indices are loaded two pairs ahead (they stream from memory, the
    // longest latency of the loop; one pair ahead took the collision ensemble's step from 59.6 to
    // 62.3 us and the 3D spheres' from 81.4 to 85.4), so only the neighbour gathers wait in an
    // iteration. A lane past the last node (d >= N in the last chunk) gathers its own index for bonds
    // it never uses: dref, xref and vol_f are allocated in whole chunks (zero padding), so those
    // reads stay inside the arrays.
    auto ahead = [&](uint32_t k, uint32_t& w, uint32_t& c) {
      w = 0u;
      c = d;
      if (k < cdeg) {
        w = P.alive[w0 + k];
        c = P.bcol[slot0 + 32u * k];
      }
    };
    uint32_t wa_n, wb_n, ca_n, cb_n, wa_m, wb_m, ca_m, cb_m;
    ahead(0, wa_n, ca_n);
    ahead(1, wb_n, cb_n);
    ahead(2, wa_m, ca_m);
    ahead(3, wb_m, cb_m);
    for (uint32_t k = 0; k < cdeg; k += 2) {
      const bool two = (k + 1) < cdeg;
      const uint32_t wa = wa_n, wb = wb_n, ca = ca_n, cb = cb_n;
      wa_n = wa_m;
      wb_n = wb_m;
      ca_n = ca_m;
      cb_n = cb_m;
      if (k + 4 < cdeg) {
        wa_m = P.alive[w0 + k + 4];
        ca_m = P.bcol[slot0 + 32u * (k + 4)];
      }
      ahead(k + 5, wb_m, cb_m);
      bool ba = (wa >> lane) & 1u, bb = (wb >> lane) & 1u;
      const bool ua = mov && ba, ub = mov && bb;
      const uint32_t sa = slot0 + 32u * k, sb = sa + 32u;
      const uint32_t ja = ua ? ca : d;
      const uint32_t jb = ub ? cb : d;
      float adh[D], adl[D], axh[D], axl[D], bdh[D], bdl[D], bxh[D], bxl[D];
      ld_hl<D>(P.dref, P.np, ja, adh, adl);
      ld_hl<D>(P.xref, P.np, ja, axh, axl);
      ld_hl<D>(P.dref, P.np, jb, bdh, bdl);
      ld_hl<D>(P.xref, P.np, jb, bxh, bxl);
      const float va = P.vol_f[ja], vb = P.vol_f[jb];
      float stra, strb;
      bond_term<D>(dh, dl, xh, xl, adh, adl, axh, axl, cnot * va, ua, f, &stra);
      bond_term<D>(dh, dl, xh, xl, bdh, bdl, bxh, bxl, cnot * vb, ub, f, &strb);
      // the alive words change only where a bond of the warp breaks: one vote a pair instead of two
      // ballots and two conditional stores (step times: collision ensemble 74.9 -> 72.5 us, settling
      // 23.7 -> 22.3, 3D spheres 104.4 -> 99.0, two disks 16.8 -> 15.8)
      const bool xa = ua && stra > snot, xb = ub && strb > snot;
      if (!__any_sync(0xffffffffu, xa || xb)) continue;
      if (xa) {
        ba = false;
        P.break_step[sa] = t;
      }
      if (xb) {
        bb = false;
        P.break_step[sb] = t;
      }
      const uint32_t na = __ballot_sync(0xffffffffu, ba);
      const uint32_t nb = __ballot_sync(0xffffffffu, bb);
      if (lane == 0) {
        if (na != wa) P.alive[w0 + k] = na;
        if (two && nb != wb) P.alive[w0 + k + 1] = nb;
      }
    }
  }
  __syncwarp();
  __syncwarp();

  unsigned long long my_pairs = 0, my_hash = 0, my_close = 0;
  uint32_t rent[REC ? MAX_CAND : 1];  // recorded contact entries of this node (REC only)
  uint32_t nrec = 0, wbits = 0;
  const InstDev& in = P.inst[gr.inst];
  const bool p_bdry = !P.nl_bdry_only || (act && P.bdry_rank[d] != NONE);
  const bool selfc = mov && P.enable_fracture && (gr.flags & GF_BREAKABLE) && P.self_contact;
  const bool other = mov && (P.worm || (gr.flags & GF_STOPPABLE));

  // with candidate lists a node whose list is empty has no contact this step
  const uint32_t ncl = (LIST && act) ? (uint32_t)P.cand_n[d] : 0u;
  if ((selfc || other) && p_bdry && (!LIST || ncl > 0)) {
    double bmn[D], bmx[D];
    grain_box<D>(P, g, bmn, bmx);
    float ph[D];
    ldf<D>(P.curf, d, ph);
    const float thr2 = in.pre_f * in.pre_f;
    // does candidate q pass the FP32 prefilter, the contact rules and the grain-box test? (the box
    // test of the grain asked about last is kept: a list is sorted by grain)
    uint32_t box_g = NONE;
    bool box_ok = false;
    auto passes = [&](uint32_t q) {
      float qf[D];
      ldf<D>(P.curf, q, qf);
      const uint32_t gq = P.node_grain[q];  // issued with the position, used after the prefilter
      float d2 = 0.f;
      for (int c = 0; c < D; ++c) {
        float dd = qf[c] - ph[c];
        d2 = fmaf(dd, dd, d2);
      }
      if (d2 > thr2) return false;
      const bool same = (gq == g);
      if (same ? !selfc : !other) return false;
      if (P.nl_bdry_only && P.bdry_rank[q] == NONE) return false;
      if (same) return true;
      if (gq != box_g) {
        double qmn[D], qmx[D];
        grain_box<D>(P, gq, qmn, qmx);
        box_g = gq;
        box_ok = boxes_touch<D>(bmn, bmx, qmn, qmx, in.contact_rad);
      }
      return box_ok;
    };
    // the contacts of this step in the reference's visit order: with candidate lists (LIST) a bit per
    // entry of the list, which is in that order; else the grid search's nodes sorted by key
    const size_t cbase = (size_t)chunk * P.cand_cap * 32 + lane;
    uint32_t hits = 0;
    uint32_t idx[LIST ? 1 : MAX_CAND];
    int nc = 0;
    if constexpr (LIST) {
      uint32_t qn = P.cand_q[cbase];  // the next entry is loaded one candidate ahead
      for (uint32_t k = 0; k < ncl; ++k) {
        const uint32_t q = qn;
        if (k + 1 < ncl) qn = P.cand_q[cbase + (size_t)(k + 1) * 32];
        if (!passes(q)) continue;
        if (nc >= (int)P.max_cand) {
          set_status(P.status, PG_ECAPACITY);
          break;
        }
        hits |= 1u << k;
        ++nc;
      }
    } else {
      unsigned long long keys[MAX_CAND];
      int32_t cc[3] = {0, 0, 0};
      for (int c = 0; c < D; ++c) cc[c] = cell_coord(ph[c] + in.frame_off_f[c], in.inv_cell_f, in.dims[c]);
      const int z0 = (D == 3) ? max(cc[2] - 1, 0) : 0, z1 = (D == 3) ? min(cc[2] + 1, (int)in.dims[2] - 1) : 0;
      const int y0 = max(cc[1] - 1, 0), y1 = min(cc[1] + 1, (int)in.dims[1] - 1);
      const int x0 = max(cc[0] - 1, 0), x1 = min(cc[0] + 1, (int)in.dims[0] - 1);
      for (int z = z0; z <= z1; ++z)
        for (int y = y0; y <= y1; ++y) {
          const uint32_t row = in.table_off + ((uint32_t)z * in.dims[1] + (uint32_t)y) * in.dims[0];
          const uint32_t b0 = P.cell_start[row + x0], b1 = P.cell_start[row + x1 + 1];
          for (uint32_t b = b0; b < b1; ++b) {
            const uint32_t q = P.sorted[b];
            if (q == d || !passes(q)) continue;
            const uint32_t gq = P.node_grain[q];
            const unsigned long long key =
                ((unsigned long long)(gq == g ? 0u : 1u) << 63) | ((unsigned long long)gq << 32) | P.node_sub[q];
            insert_cand<D>(keys, idx, nc, key, q, P);
          }
        }
    }
    const uint32_t mydeg = P.node_deg[d];
    // the pair log hashes input indices (the node's own looked up once; recorded runs only)
    const unsigned long long od_hash = P.record_pairs ? ((unsigned long long)input_index<PERM>(P, d) << 32) : 0ull;
    const float Kn0 = (float)in.normal_stiffness;
    const float mu0 = (float)in.friction_coefficient, zeta0 = (float)in.damping_ratio;
    const float rho = (float)gr.rho, dtf = (float)P.dt;
    double xp64[D];
    if (nc) ldv<D>(P.cur, d, xp64);
    for (int ci = 0; ci < nc; ++ci) {
      uint32_t q;
      if constexpr (LIST) {
        q = P.cand_q[cbase + (size_t)(__ffs(hits) - 1) * 32];
        hits &= hits - 1;
      } else {
        q = idx[ci];
      }
      const uint32_t gqi = P.node_grain[q];
      const bool same = gqi == g;
      // The contact decision |x_q - x_p| <= R_c' is made with the reference's FP64 arithmetic:
      // contact damping switches on at full strength at that boundary, so a decision flipped by
      // FP32 rounding would kick a node by metres per second.
      double xq64[D], dir64[D];
      ldv<D>(P.cur, q, xq64);
      for (int c = 0; c < D; ++c) dir64[c] = xq64[c] - xp64[c];
      double n2 = dir64[0] * dir64[0];
      for (int c = 1; c < D; ++c) n2 = n2 + dir64[c] * dir64[c];
      // dn64 <= R_c' <= contact_rad needs n2 <= contact_s_max (the same outcome as the sqrt
      // test): candidates beyond it skip the square root and the bonded-neighbour scan
      if (!(n2 <= in.contact_s_max)) continue;
      const double dn64 = sqrt(n2);
      double Rc64 = in.contact_rad;
      float Kn = Kn0, zeta = zeta0, mu = mu0;
      if constexpr (GC) {
        const GrainDev& gq = P.grain[gqi];
        Kn = (float)((gr.kn + gq.kn) * 0.5);
        zeta = (float)((gr.zeta + gq.zeta) * 0.5);
        mu = (float)((gr.mu + gq.mu) * 0.5);
      }
      if (same) {
        bool bonded = false;
        for (uint32_t k = 0; k < mydeg && !bonded; ++k) {
          if (((P.alive[w0 + k] >> lane) & 1u) && P.bcol[slot0 + 32u * k] == q) bonded = true;
        }
        if (bonded) continue;
        double pp[D], pq[D], r[D];
        ldv<D>(P.pos, d, pp);
        ldv<D>(P.pos, q, pq);
        for (int c = 0; c < D; ++c) r[c] = pp[c] - pq[c];
        double r2 = r[0] * r[0];
        for (int c = 1; c < D; ++c) r2 = r2 + r[c] * r[c];
        const double ref = sqrt(r2);
        Rc64 = ref < in.contact_rad ? ref : in.contact_rad;
        Kn = (float)(gr.cnot / Rc64);
      }
      if (!(dn64 <= Rc64)) continue;
      const float Rc = (float)Rc64, dn = (float)dn64;
      float dir[D];
      for (int c = 0; c < D; ++c) dir[c] = (float)dir64[c];
      if (P.record_pairs) {
        my_pairs += 1;
        my_hash += splitmix64(od_hash | input_index<PERM>(P, q));
      }
      if (dn == 0.f) my_close += 1;
      const float inv = 1.f / dn;
      float u[D];
      for (int c = 0; c < D; ++c) u[c] = dir[c] * inv;
      const float nvol = P.vol_f[q];
      const float s1 = -Kn * (Rc - dn) * nvol;
      for (int c = 0; c < D; ++c) f[c] = fmaf(s1, u[c], f[c]);
      const float cfn = fabsf(s1);
      uint32_t fr = 0;
      if (P.allow_damping || P.allow_friction) {
        double vqd[D];
        ldv<D>(P.vel_in, q, vqd);
        float rv[D];
        for (int c = 0; c < D; ++c) rv[c] = (float)(vpd[c] - vqd[c]);
        const float rvp = dotf<D>(rv, u);
        if (P.allow_damping) {
          const float dc = 2.f * zeta * sqrtf(Kn * rho) * sqrtf(nvol);
          for (int c = 0; c < D; ++c) f[c] = fmaf(-dc * rvp, u[c], f[c]);
        }
        if (P.allow_friction) {
          float tg[D];
          for (int c = 0; c < D; ++c) tg[c] = fmaf(-rvp, u[c], rv[c]);
          const float tn = sqrtf(dotf<D>(tg, tg));
          if (tn > 0.f) {
            float sfr = -mu * cfn;
            fr = (D == 2 && (tg[1] * u[0] - tg[0] * u[1]) < 0.f) ? FR_SLIDE_NEG : FR_SLIDE;
            if (tn < mu * cfn * dtf / rho) {
              sfr = -tn / rho / dtf;
              fr = FR_STICK;
            }
            const float it = sfr / tn;
            for (int c = 0; c < D; ++c) f[c] = fmaf(it, tg[c], f[c]);
          }
        }
      }
      if constexpr (REC) rent[nrec++] = q | (fr << 30);
    }
  }

  if (mov && other && p_bdry && in.allow_wall) {
    double bmn[D], bmx[D];
    grain_box<D>(P, g, bmn, bmx);
    if (!within_interior<D>(bmn, bmx, in.wall, in.contact_rad)) {
      double xc[D];
      ldv<D>(P.cur, d, xc);
      const double vol_i = (double)P.vol_f[d];
      const float R = (float)in.contact_rad;
      const float Kn = (float)(GC ? gr.kn : in.normal_stiffness);
      const float mu = (float)(GC ? gr.mu : in.friction_coefficient);
      const float zeta = (float)(GC ? gr.zeta : in.damping_ratio);
      const float rho = (float)gr.rho, dtf = (float)P.dt;
      constexpr int NS = 2 * D;
      const int order2[4][2] = {{3, 1}, {0, 0}, {1, 0}, {2, 1}};
      const int order3[6][2] = {{0, 0}, {3, 0}, {1, 1}, {4, 1}, {2, 2}, {5, 2}};
      for (int k = 0; k < NS; ++k) {
        const int side = (D == 2) ? order2[k][0] : order3[k][0];
        const int dir = (D == 2) ? order2[k][1] : order3[k][1];
        const float dist = (float)(xc[dir] - in.wall[side]);
        if (!(fabsf(dist) <= R)) continue;
        wbits |= 1u << (4 * k);
        const float dd = fabsf(dist);
        float Area, I;
        if constexpr (D == 2) {
          Area = 0.5f * (float)M_PI * R * R - R * R * asinf(dd / R) - sqrtf(fmaxf(R * R - dd * dd, 0.f)) * dd;
          I = 0.f;
        } else {
          const float a = R - dd, b = R * R - dd * dd;
          Area = ((float)M_PI / 3.f) * a * a * (2.f * R - dd);
          I = ((float)M_PI / 4.f) * b * b;
        }
        const float centroid = I / Area;
        const float crc = R - centroid;
        const float F = Kn * (crc > 0.f ? crc : 0.f) * Area;
        const float c_sign = dist > 0.f ? 1.f : -1.f;
        f[dir] += c_sign * F;
        WallRec rec;
        rec.a_normal = vol_i * (double)(c_sign * F);
        rec.a_t1 = 0;
        rec.a_t2 = 0;
        rec.a_damp = 0;
        rec.gid = P.nl_bdry_only ? (gr.node_begin + P.bdry_rank[d]) : input_index<PERM>(P, d);
        rec.side = (uint16_t)side;
        rec.has_fric = 0;
        rec.has_damp = 0;
        float rv[D];
        for (int c = 0; c < D; ++c) rv[c] = (float)vpd[c];
        rv[dir] -= (float)in.wall_speed[side];
        if (P.allow_friction) {
          if constexpr (D == 2) {
            const int tg = (dir + 1) % 2;
            if (fabsf(rv[tg]) > 0.f) {
              float ff = -mu * fabsf(F) * (rv[tg] > 0.f ? 1.f : -1.f);
              wbits |= (rv[tg] > 0.f ? 2u : 10u) << (4 * k);
              if (fabsf(rv[tg]) < mu * fabsf(F) * dtf / rho) {
                ff = -rv[tg] * rho / dtf;
                wbits |= 4u << (4 * k);
              }
              f[tg] += ff;
              rec.a_t1 = vol_i * (double)ff;
              rec.has_fric = 1;
            }
          } else {
            const int t1 = (dir + 1) % 3, t2 = (dir + 2) % 3;
            const float vn = sqrtf(rv[t1] * rv[t1] + rv[t2] * rv[t2]);
            if (vn > 0.f) {
              const float u1 = rv[t1] / vn, u2 = rv[t2] / vn;
              float sfr = -mu * fabsf(F);
              wbits |= 2u << (4 * k);
              if (vn < mu * fabsf(F) * dtf / rho) {
                sfr = -vn / rho / dtf;
                wbits |= 4u << (4 * k);
              }
              f[t1] += sfr * u1;
              f[t2] += sfr * u2;
              rec.a_t1 = vol_i * (double)(sfr * u1);
              rec.a_t2 = vol_i * (double)(sfr * u2);
              rec.has_fric = 1;
            }
          }
        }
        if (P.allow_damping) {
          const float df = -(2.f * zeta * sqrtf(Kn * rho) * sqrtf(fabsf(Area))) * rv[dir];
          f[dir] += df;
          rec.a_damp = vol_i * (double)df;
          rec.has_damp = 1;
        }
        const uint32_t slot = atomicAdd(P.wrec_count, 1u);
        if (slot < P.wrec_cap) {
          P.wrec[slot] = rec;
        } else {
          set_status(P.status, PG_ECAPACITY);
        }
      }
    }
  }

  if (mov && P.worm) {
    float ef[D];
    if constexpr (D == 2) {
      for (int c = 0; c < D; ++c) ef[c] = ef_in[c];
    } else {
      ldvf<D>(P.extf_f, d, ef);
    }
    const float gate = (float)((worm_phase(t) + 1u) % 2u);
    for (int c = 0; c < D; ++c) f[c] = fmaf(gate, ef[c], f[c]);
  } else if (mov) {
    float ef[D];
    if constexpr (D == 2) {
      for (int c = 0; c < D; ++c) ef[c] = ef_in[c];
    } else {
      ldvf<D>(P.extf_f, d, ef);
    }
    float sc = 1.f;
    if (P.gradient_extforce) {
      double scd = (double)t / (double)P.extforce_maxstep;
      sc = (float)(scd > 1 ? 1.0 : scd);
    }
    for (int c = 0; c < D; ++c) f[c] = fmaf(sc, ef[c], f[c]);
    if (P.enable_torque) {
      double xc[D];
      ldv<D>(P.cur, d, xc);
      const uint32_t ta = gr.torque_axis;
      float r[3] = {0, 0, 0}, rp[3] = {0, 0, 0};
      for (int c = 0; c < D; ++c) r[c] = (float)(xc[c] - P.torque_c[(size_t)g * 3 + c]);
      if (D == 3) r[ta] = 0;
      rp[(ta + 1) % 3] = -r[(ta + 2) % 3];
      rp[(ta + 2) % 3] = r[(ta + 1) % 3];
      float pn = 0.f;
      for (int c = 0; c < D; ++c) pn = fmaf(rp[c], rp[c], pn);
      pn = sqrtf(pn);
      const float tv = (float)gr.torque_val;
      if (pn > 0.f) {
        for (int c = 0; c < D; ++c) f[c] = fmaf(tv, rp[c] / pn, f[c]);
      }
    }
  }

  // velocity update (timeloop.h:834-863); with P.fuse the next step's position update too
  double cu[D], dp[D];
  for (int c = 0; c < D; ++c) cu[c] = 0.0;
  if (act) {
    if (P.fuse) ldv<D>(P.disp, d, dp);
    if (mov) {
      float ao[D], a[D];
      double v[D];
      if constexpr (D == 2) {
        for (int c = 0; c < D; ++c) ao[c] = ao_in[c];
      } else {
        ldvf<D>(P.acc_f, d, ao);
      }
      const float orho = gr.one_over_rho_f, hdt = P.half_dt_f;
      for (int c = 0; c < D; ++c) {
        a[c] = orho * f[c];
        v[c] = vpd[c] + widen((ao[c] + a[c]) * hdt);  // FP64 accumulation of an FP32 increment
      }
      if ((D == 2) ? clamped_in : (P.clamped[d] != 0)) {
        for (int c = 0; c < D; ++c) {
          a[c] = 0.f;
          v[c] = 0.0;
        }
        if (P.fuse) {
          for (int c = 0; c < D; ++c) dp[c] = 0.0;
        } else {
          P.clamp_pending[d] = 1;
        }
      }
      if (P.worm) worm_clamp<D>(input_index<PERM>(P, d) - gr.node_begin, worm_phase(t), a, v);
      stvf<D>(P.acc_f, d, a);
      stv<D>(P.vel_out, d, v);
      if (P.fuse) {
        advance_mx<D>(P, v, a, dp);
        stv<D>(P.disp, d, dp);
      }
    } else {
      stv<D>(P.vel_out, d, vpd);
    }
    if (P.fuse) {
      double ps[D];
      float db[D];
      ldv<D>(P.pos, d, ps);
      ldf<D>(P.disp_b, d, db);
      place_node_mx<D>(P, d, in, dp, ps, db, P.cur_n, P.curf_n, P.dref_n, P.rebuild_n, cu);
    } else {
      stvf<D>(P.force_f, d, f);
    }
  }
  if (P.fuse) grow_box<D>(P.bbox_n, g, act, cu);

  if constexpr (REC) {
    record_masks(P, d, act, lane, rent, nrec, wbits);
    if (P.rec_x) {
      double xr[D];
      if (act) ldv<D>(P.cur, d, xr);
      record_tape<D>(P, d, act, t, xr, vpd);
    }
  }

  if (P.record_pairs) {
    for (int off = 16; off > 0; off >>= 1) {
      my_pairs += __shfl_down_sync(0xffffffffu, my_pairs, off);
      my_hash += __shfl_down_sync(0xffffffffu, my_hash, off);
    }
    if (lane == 0 && my_pairs) {
      atomicAdd(&P.pair_acc[0], my_pairs);
      atomicAdd(&P.pair_acc[1], my_hash);
    }
  }
  if (my_close) atomicAdd(P.too_close, my_close);
}

// The force kernel's variants: mask recording (REC), per-grain contact parameters (GC), a node
// layout other than the input order (PERM) and candidate lists or the grid search (LIST) are compiled
// in only where used, so the plain kernel keeps its register budget; the plain kernel with lists
// also for BPS = 5, 6 or 7 blocks of 128 threads per SM (96, 80 or 72 registers), see force_bps().
template <int D>
static const void* force_mx_ptr(bool rec, bool gc, bool perm, bool list, int bps) {
#define PG_F(r, g, p, l, b) (const void*)k_force_mx<D, r, g, p, l, b>
  static const void* const plain[2][3] = {{PG_F(0, 0, 0, 1, 5), PG_F(0, 0, 0, 1, 6), PG_F(0, 0, 0, 1, 7)},
                                          {PG_F(0, 0, 1, 1, 5), PG_F(0, 0, 1, 1, 6), PG_F(0, 0, 1, 1, 7)}};
  static const void* const others[14] = {
      PG_F(0, 0, 0, 0, 6), PG_F(0, 0, 1, 0, 6), PG_F(0, 1, 0, 0, 5), PG_F(0, 1, 0, 1, 5), PG_F(0, 1, 1, 0, 5),
      PG_F(0, 1, 1, 1, 5), PG_F(1, 0, 0, 0, 5), PG_F(1, 0, 0, 1, 5), PG_F(1, 0, 1, 0, 5), PG_F(1, 0, 1, 1, 5),
      PG_F(1, 1, 0, 0, 5), PG_F(1, 1, 0, 1, 5), PG_F(1, 1, 1, 0, 5), PG_F(1, 1, 1, 1, 5)};
#undef PG_F
  if (!rec && !gc) return list ? plain[perm ? 1 : 0][bps - 5] : others[perm ? 1 : 0];
  return others[2 + (rec ? (gc ? 8 : 4) : 0) + (perm ? 2 : 0) + (list ? 1 : 0)];
}
template <int D>
static void launch_force_mx(const Dev& P, dim3 grid, dim3 block, cudaStream_t s, bool pdl, bool rec) {
  using K = void (*)(const Dev);
  launch_k((K)force_mx_ptr<D>(rec, P.grain_contact, P.node_orig, P.cand_q, force_bps(P.n_chunks, P.n_sms)), grid, block,
           0, s, pdl, P);
}

cudaError_t kernels_mixed_init() {
  cudaError_t e = cudaFuncSetAttribute(k_finalize<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, FINAL_SMEM);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_finalize<3>, cudaFuncAttributeMaxDynamicSharedMemorySize, FINAL_SMEM);
  if (e != cudaSuccess) return e;
  // the recording variants of the force kernel have local frames of about 1.1 KB
  const void* fs[2 * 48];
  int n = 0;
  for (int k = 0; k < 16; ++k)
    for (int b = 5; b <= 7; ++b) {
      fs[n++] = force_mx_ptr<2>(k & 8, k & 4, k & 2, k & 1, b);
      fs[n++] = force_mx_ptr<3>(k & 8, k & 4, k & 2, k & 1, b);
    }
  size_t need = 0;
  e = max_local_bytes(fs, n, &need);
  return e == cudaSuccess ? ensure_local_bytes(need) : e;
}

template <int D>
static void predict_t(const Dev& P, cudaStream_t s, uint64_t* launches, bool pdl) {
  launch_k(k_predict_mx<D>, cdiv(P.N, 256), 256, 0, s, pdl, P);
  *launches += 1;
}
template <int D>
static void body_t(const Dev& P, const LaunchCfg& L, cudaStream_t s, uint64_t* launches, bool pdl, bool rec,
                   cudaEvent_t e0, cudaEvent_t e1) {
  launch_grid_build<D>(P, s, launches, pdl);
  if (P.enable_torque) {
    launch_k(k_torque_center<D>, cdiv(P.G, 128), 128, 0, s, pdl, P);
    *launches += 1;
  }
  if (e0) cudaEventRecord(e0, s);
  const dim3 grid(cdiv(P.n_chunks * 32, L.force_block)), block(L.force_block);
  launch_force_mx<D>(P, grid, block, s, pdl, rec);
  *launches += 1;
  if (e1) cudaEventRecord(e1, s);
}
template <int D>
static void finalize_t(const Dev& P, cudaStream_t s, uint64_t* launches, bool pdl) {
  launch_k(k_finalize<D>, finalize_blocks(P.I), FINAL_THREADS, P.wrec_smem ? FINAL_SMEM : 0, s, pdl, P);
  *launches += 1;
}

void launch_mixed_predict(const Dev& P, cudaStream_t s, uint64_t* launches, bool pdl) {
  P.dim == 2 ? predict_t<2>(P, s, launches, pdl) : predict_t<3>(P, s, launches, pdl);
}
void launch_mixed_body(const Dev& P, const LaunchCfg& L, cudaStream_t s, uint64_t* launches, bool pdl, bool rec,
                       cudaEvent_t e0, cudaEvent_t e1) {
  P.dim == 2 ? body_t<2>(P, L, s, launches, pdl, rec, e0, e1) : body_t<3>(P, L, s, launches, pdl, rec, e0, e1);
}
void launch_mixed_finalize(const Dev& P, cudaStream_t s, uint64_t* launches, bool pdl) {
  P.dim == 2 ? finalize_t<2>(P, s, launches, pdl) : finalize_t<3>(P, s, launches, pdl);
}

}  // namespace pg
