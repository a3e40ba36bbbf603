// GB300 (sm_103a) kernels of the PeriDEM time step, FP64 parity path.
//
// One step (reference src/particle/timeloop.h:608-879) is these launches on one stream:
//   k_predict      position update (timeloop.h:661-669) + grid key or list-rebuild check + per-grain
//                  bounding box
//   k_grid_coop    candidate lists: grid refit, cell chains and lists on rebuild steps, or
//   k_scan_reduce  \ the grid search: exclusive scan of the per-bucket counts = cell-start table
//   k_scan_final   /
//   k_scatter      nodes -> bucket order (counting sort, one digit spanning all buckets)
//   k_bonds        bond force addends + break (particle2.h:102-232), one bond per thread
//   k_force        sum of the bond forces, self/inter-grain contact (contact.h:668-812), wall
//                  (contact.h:900-964, :314-431, :16-41), external force and torque
//                  (timeloop.h:774-824), velocity update (timeloop.h:834-863) -- fused, one node per
//                  thread
//   k_finalize     ordered wall-reaction sums, pair log, wall move (timeloop.h:866-878)
// With lists the steps of one call run fused: k_force also makes the next step's position update and
// k_grid_coop first ends the step before, so k_predict runs once ahead of the call's first step and
// k_finalize once behind its last.
//
// This file is compiled with --fmad=false: every FP64 operation is the IEEE operation the
// reference performs, in the reference's order, so the non-wall path is bit-exact.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "pg_common.cuh"
#include "pg_device.cuh"
#include "pg_ieee64.cuh"
#include "pg_kernels.h"

namespace pg {

// CurrPos of node d from its displacement, the FP32 image, and either the list-rebuild check (with
// candidate lists: once any node has moved 0.45 skin since the last build) or the node's grid key.
template <int D>
__device__ __forceinline__ void place_node(const Dev& P, uint32_t d, const InstDev& in, const double (&dp)[D],
                                           double* cur, float* curf, uint32_t* rebuild, double (&cu)[D]) {
  double ps[D];
  ldv<D>(P.pos, d, ps);
  for (int c = 0; c < D; ++c) cu[c] = ps[c] + dp[c];
  stv<D>(cur, d, cu);
  // the FP32 offset to the grid origin
  float rf[D];
  bool ok = true;
  for (int c = 0; c < D; ++c) {
    if (!isfinite(cu[c])) ok = false;
    rf[c] = (float)(cu[c] - in.origin[c]);
  }
  if (!ok) set_status(P.status, PG_ENAN);
  stf<D>(curf, d, rf);
  if (P.cand_q) {
    constexpr uint32_t SF = (D == 2) ? 2 : 4;
    float m2 = 0.f;
    for (int c = 0; c < D; ++c) {
      const float dd = (float)dp[c] - P.disp_b[(size_t)d * SF + c];
      m2 += dd * dd;
    }
    if (m2 > in.skin_lim2) *rebuild = 1;
  } else {
    int32_t ci[3] = {0, 0, 0};
    for (int c = 0; c < D; ++c) ci[c] = cell_coord(rf[c] + in.frame_off_f[c], in.inv_cell_f, in.dims[c]);
    const uint32_t key = in.table_off + ((uint32_t)ci[2] * in.dims[1] + (uint32_t)ci[1]) * in.dims[0] + (uint32_t)ci[0];
    P.cell_key[d] = key;
    P.cell_rank[d] = atomicAdd(&P.cell_count[key], 1u);
  }
}

// ---------------------------------------------------------------------------------------------
// k_predict: disp += dt*vel + (dt*dt*0.5)*acc for movable grains; CurrPos = pos + disp.
// ---------------------------------------------------------------------------------------------
template <int D>
__global__ void __launch_bounds__(256) k_predict(const Dev P) {
  pdl_enter();
  const uint32_t d = blockIdx.x * blockDim.x + threadIdx.x;
  const bool act = d < P.N;
  uint32_t g = 0;
  double cu[D];
  for (int c = 0; c < D; ++c) cu[c] = 0.0;
  if (act) {
    g = P.node_grain[d];
    const GrainDev& gr = P.grain[g];
    double dp[D];
    ldv<D>(P.disp, d, dp);
    bool wrote = false;
    if (P.clamp_pending[d]) {
      // a clamped node zeroed at the end of the previous step (timeloop.h:854-860)
      for (int c = 0; c < D; ++c) dp[c] = 0.0;
      P.clamp_pending[d] = 0;
      wrote = true;
    }
    if (gr.flags & GF_MOVABLE) {
      double v[D], a[D];
      ldv<D>(P.vel_in, d, v);
      ldv<D>(P.acc, d, a);
      for (int c = 0; c < D; ++c) dp[c] = dp[c] + ((P.dt * v[c]) + (P.hdt2 * a[c]));
      wrote = true;
    }
    if (wrote) stv<D>(P.disp, d, dp);
    place_node<D>(P, d, P.inst[gr.inst], dp, P.cur, P.curf, P.rebuild, cu);
  }
  grow_box<D>(P.bbox, g, act, cu);
}

// Addend of one bond of a node, the reference's operations in its order, for any operands: the
// stretch in *str.
template <int D>
__device__ __noinline__ void bond_addend_any(const double* e, double xin, double cnot, double vol, double* g,
                                             double* str) {
  double n2 = e[0] * e[0];
  for (int c = 1; c < D; ++c) n2 = n2 + e[c] * e[c];
  const double en = sqrt(n2);
  *str = (en - xin) / xin;
  const double sc = (cnot * *str) * vol;
  for (int c = 0; c < D; ++c) g[c] = sc * (e[c] / en);
}

// Addend of a bond stored for the force kernel, and read back.
template <int D>
__device__ __forceinline__ void st_addend(const Dev& P, uint32_t s, const double (&g)[D]) {
  reinterpret_cast<double2*>(P.addend)[s] = make_double2(g[0], g[1]);
  if constexpr (D == 3) P.addend_z[s] = g[2];
}
template <int D>
__device__ __forceinline__ void ld_addend(const Dev& P, uint32_t s, double (&g)[D]) {
  const double2 q = reinterpret_cast<const double2*>(P.addend)[s];
  g[0] = q.x;
  g[1] = q.y;
  if constexpr (D == 3) g[2] = P.addend_z[s];
}

// Bond forces and bond breaking (particle2.h:102-150, :191-232), one thread per bond of the edge
// list (Dev::edge_ij): the two directions of a bond differ in the sign of the bond vector and in
// the neighbour's volume only, so its length, stretch and unit vector are formed once and the
// addends of both nodes written to their slots of the bond slab, where the force kernel sums each
// node's in bond order. Squares, square root and divisions run on the integer pipe, bit-identical
// to the IEEE operations (pg_ieee64.cuh); a bond with an operand or a result outside their range is
// redone in hardware.
//
// Bound by the FP64 pipe (one warp instruction per 16 cycles and SM) beside the integer ALU: 15
// FP64 instructions per bond in 2D, 21 in 3D, against twice 14 and twice 20 when each node
// computed its own bonds. Collision ensemble (10.0M directed bonds): k_bonds 158 us + k_force 73 us
// (which also updates the next positions) against 364 us fused; 3D spheres (10.8M): 245 + 116 against 804 us; two disks (65k): 4.8 + 8.0
// against 56 us, the work spread over 1,019 warps instead of 79. More of it on the integer pipe
// (the extension en - xin, the scale and force products, the sum of the squares) was slower: the
// ensemble step 250 us as it stands, 263 with the extension moved, 323 with all of them moved.
template <int D>
__global__ void __launch_bounds__(256) k_bonds(const Dev P) {
  pdl_enter();
  const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
  const bool in_list = b < P.n_edges;
  const uint32_t be = in_list ? b : P.n_edges - 1u;
  const uint2 ij = P.edge_ij[be], sl = P.edge_slot[be];
  const double xin = P.edge_xin[be];
  const GrainDev& gr = P.grain[P.node_grain[ij.x]];
  const bool mov = gr.flags & GF_MOVABLE;
  const bool two = sl.y != NONE;
  const uint32_t wi = P.alive[sl.x >> 5], wj = two ? P.alive[sl.y >> 5] : 0u;
  const bool ai = mov && ((wi >> (sl.x & 31)) & 1u), aj = mov && ((wj >> (sl.y & 31)) & 1u);
  const bool use = in_list && (ai || aj);
  double di[D], dj[D], xi[D], xj[D];
  ldv<D>(P.disp, ij.x, di);
  ldv<D>(P.disp, ij.y, dj);
  ldv<D>(P.xpos, ij.x, xi);
  ldv<D>(P.xpos, ij.y, xj);
  const double vi = P.vol[ij.x], vj = P.vol[ij.y], cnot = gr.cnot;
  double e[D];
  uint64_t eb[D];
  for (int c = 0; c < D; ++c) {
    e[c] = (dj[c] - di[c]) + (xj[c] - xi[c]);
    eb[c] = ieee64::bits(e[c]);
  }
  bool ok, all;
  double n2d = ieee64::from_bits(ieee64::mul_bits(eb[0], eb[0], &all));
  for (int c = 1; c < D; ++c) {
    n2d = n2d + ieee64::from_bits(ieee64::mul_bits(eb[c], eb[c], &ok));
    all &= ok;
  }
  const uint64_t n2 = ieee64::bits(n2d);
  const uint64_t en = ieee64::sqrt_bits(n2, &ok);
  all &= ok;
  const uint64_t ext = ieee64::bits(ieee64::from_bits(en) - xin);
  uint64_t str = ieee64::div_bits(ext, ieee64::make_divisor(xin), &ok);
  all &= ok;
  double gi[D], gj[D];
  for (int c = 0; c < D; ++c) {
    gi[c] = 0.0;
    gj[c] = 0.0;
  }
  // an unstretched bond (str = +-0 and |e[c] / en| <= 1) adds +-0, which leaves a sum's bits
  // unchanged (it starts at +0 and never becomes -0 under round-to-nearest)
  if (__any_sync(0xffffffffu, use && (str << 1) != 0)) {
    const double cs = cnot * ieee64::from_bits(str);
    const double si = cs * vj, sj = cs * vi;
    const ieee64::Divisor den = ieee64::make_divisor(ieee64::from_bits(en));
    for (int c = 0; c < D; ++c) {
      const uint64_t u = ieee64::div_bits(eb[c], den, &ok);
      all &= ok;
      const double ud = ieee64::from_bits(u);
      gi[c] = si * ud;
      gj[c] = sj * -ud;
    }
  }
  if (!in_list) return;
  if (use && !all) {
    double ea[D], ga[D], sa;
    for (int c = 0; c < D; ++c) ea[c] = -e[c];
    bond_addend_any<D>(ea, xin, cnot, vi, ga, &sa);
    for (int c = 0; c < D; ++c) {
      gj[c] = ga[c];
      ea[c] = e[c];
    }
    bond_addend_any<D>(ea, xin, cnot, vj, ga, &sa);
    for (int c = 0; c < D; ++c) gi[c] = ga[c];
    str = ieee64::bits(sa);
  }
  for (int c = 0; c < D; ++c) {
    gi[c] = ai ? gi[c] : 0.0;
    gj[c] = aj ? gj[c] : 0.0;
  }
  st_addend<D>(P, sl.x, gi);
  if (two) st_addend<D>(P, sl.y, gj);
  if (use && P.enable_fracture && (gr.flags & GF_BREAKABLE) && (gr.flags & GF_BREAK_BONDS)) {
    // the break test str > snot on the integer pipe when snot is +0 or more and not NaN
    const uint64_t snot_bits = ieee64::bits(gr.snot);
    const double s = ieee64::from_bits(str);
    if (ieee64::gt_nonneg_ok(snot_bits) ? ieee64::gt_nonneg(s, snot_bits) : s > gr.snot) {
      const uint32_t t = *P.step;
      if (ai) {
        atomicAnd(&P.alive[sl.x >> 5], ~(1u << (sl.x & 31)));
        P.break_step[sl.x] = t;
      }
      if (aj) {
        atomicAnd(&P.alive[sl.y >> 5], ~(1u << (sl.y & 31)));
        P.break_step[sl.y] = t;
      }
    }
  }
}

template <int D, bool REC, bool GC, bool LIST, int BPS>
__global__ void __launch_bounds__(128, BPS) k_force(const Dev P) {
  pdl_enter();
  pdl_release();
  const uint32_t d = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t chunk = d >> 5;
  if (chunk >= P.n_chunks) return;  // uniform per warp
  const bool act = d < P.N;
  const uint32_t t = *P.step;
  const uint32_t g = act ? P.node_grain[d] : 0;
  const GrainDev gr = P.grain[g];
  const bool mov = act && (gr.flags & GF_MOVABLE);
  const uint32_t slot0 = P.chunk_slot[chunk] + lane;
  const uint32_t w0 = P.chunk_word[chunk];

  double f[D];
  for (int c = 0; c < D; ++c) f[c] = 0.0;
  double vp[D];
  if (act) ldv<D>(P.vel_in, d, vp);

  // ---- bond forces: the node's addends (k_bonds) in bond order ----
  {
    const uint32_t cdeg = P.chunk_deg[chunk];
#pragma unroll 4
    for (uint32_t k = 0; k < cdeg; ++k) {
      double q[D];
      ld_addend<D>(P, slot0 + 32u * k, q);
      for (int c = 0; c < D; ++c) f[c] = f[c] + q[c];
    }
  }

  unsigned long long my_pairs = 0, my_hash = 0, my_close = 0;
  uint32_t rent[REC ? MAX_CAND : 1];  // recorded contact entries of this node (REC only)
  uint32_t nrec = 0, wbits = 0;
  const InstDev& in = P.inst[gr.inst];
  const bool p_bdry = !P.nl_bdry_only || (act && P.bdry_rank[d] != NONE);
  const bool selfc = mov && P.enable_fracture && (gr.flags & GF_BREAKABLE) && P.self_contact;
  // contact with other grains and walls only for stoppable grains (timeloop.h:719), for every
  // movable grain in the worm loop (timeloop.h:1146-1168)
  const bool other = mov && (P.worm || (gr.flags & GF_STOPPABLE));
  double xpc[D];
  if (act) ldv<D>(P.cur, d, xpc);

  // ---- node-node contact: self-contact first, then grains j ascending (timeloop.h:709-747) ----
  // with candidate lists a node whose list is empty has no contact this step
  const uint32_t ncl = (LIST && act) ? (uint32_t)P.cand_n[d] : 0u;
  if ((selfc || other) && p_bdry && (!LIST || ncl > 0)) {
    double bmn[D], bmx[D];
    grain_box<D>(P, g, bmn, bmx);
    float pf[D];
    ldf<D>(P.curf, d, pf);
    const float thr2 = in.pre_f * in.pre_f;
    // is candidate q beyond the FP32 prefilter; is it within the contact rules and the grain-box test?
    // (the box test of the grain asked about last is kept: a list is sorted by grain)
    uint32_t box_g = NONE;
    bool box_ok = false;
    auto far = [&](const float (&qf)[D]) {
      float d2 = 0.f;
      for (int c = 0; c < D; ++c) {
        float dd = qf[c] - pf[c];
        d2 += dd * dd;
      }
      return d2 > thr2;
    };
    auto allowed = [&](uint32_t q, uint32_t gq) {
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
    unsigned long long keys[LIST ? 1 : MAX_CAND];
    int nc = 0;
    if constexpr (LIST) {
      uint32_t qn = P.cand_q[cbase];  // the next entry is loaded one candidate ahead
      for (uint32_t k = 0; k < ncl; ++k) {
        const uint32_t q = qn;
        if (k + 1 < ncl) qn = P.cand_q[cbase + (size_t)(k + 1) * 32];
        float qf[D];
        ldf<D>(P.curf, q, qf);
        const uint32_t gq = P.node_grain[q];  // issued with the position, used after the prefilter
        if (far(qf) || !allowed(q, gq)) continue;
        if (nc >= (int)P.max_cand) {
          set_status(P.status, PG_ECAPACITY);
          break;
        }
        hits |= 1u << k;
        ++nc;
      }
    } else {
      int32_t cc[3] = {0, 0, 0};
      for (int c = 0; c < D; ++c) cc[c] = cell_coord(pf[c] + in.frame_off_f[c], in.inv_cell_f, in.dims[c]);
      const int z0 = (D == 3) ? max(cc[2] - 1, 0) : 0, z1 = (D == 3) ? min(cc[2] + 1, (int)in.dims[2] - 1) : 0;
      const int y0 = max(cc[1] - 1, 0), y1 = min(cc[1] + 1, (int)in.dims[1] - 1);
      const int x0 = max(cc[0] - 1, 0), x1 = min(cc[0] + 1, (int)in.dims[0] - 1);
      for (int z = z0; z <= z1; ++z)
        for (int y = y0; y <= y1; ++y) {
          const uint32_t row = in.table_off + ((uint32_t)z * in.dims[1] + (uint32_t)y) * in.dims[0];
          const uint32_t b0 = P.cell_start[row + x0], b1 = P.cell_start[row + x1 + 1];
          for (uint32_t b = b0; b < b1; b += CELL_BATCH) {
            uint32_t qs[CELL_BATCH];
            float qf[CELL_BATCH][D];
#pragma unroll
            for (uint32_t k = 0; k < CELL_BATCH; ++k) qs[k] = b + k < b1 ? P.sorted[b + k] : d;
#pragma unroll
            for (uint32_t k = 0; k < CELL_BATCH; ++k) ldf<D>(P.curf, qs[k], qf[k]);
#pragma unroll
            for (uint32_t k = 0; k < CELL_BATCH; ++k) {
              const uint32_t q = qs[k];
              if (q == d || far(qf[k])) continue;
              const uint32_t gq = P.node_grain[q];
              if (!allowed(q, gq)) continue;
              const unsigned long long key =
                  ((unsigned long long)(gq == g ? 0u : 1u) << 63) | ((unsigned long long)gq << 32) | P.node_sub[q];
              insert_cand<D>(keys, idx, nc, key, q, P);
            }
          }
        }
    }
    const uint32_t mydeg = P.node_deg[d];
    for (int ci = 0; ci < nc; ++ci) {
      uint32_t q;
      if constexpr (LIST) {
        q = P.cand_q[cbase + (size_t)(__ffs(hits) - 1) * 32];
        hits &= hits - 1;
      } else {
        q = idx[ci];
      }
      const uint32_t gqi = LIST ? P.node_grain[q] : (uint32_t)(keys[ci] >> 32) & 0x7fffffffu;
      const bool same = gqi == g;
      double xq[D], dir[D];
      ldv<D>(P.cur, q, xq);
      for (int c = 0; c < D; ++c) dir[c] = xq[c] - xpc[c];
      double n2 = dir[0] * dir[0];
      for (int c = 1; c < D; ++c) n2 = n2 + dir[c] * dir[c];
      // dn <= R_c <= contact_rad needs n2 <= contact_s_max (the same outcome as the sqrt test):
      // candidates beyond it skip the square root and the bonded-neighbour scan
      if (!(n2 <= in.contact_s_max)) continue;
      const double dn = ieee64::sqrt_rn(n2);
      double Rc = in.contact_rad, Kn = in.normal_stiffness;
      double zeta = in.damping_ratio, mu = in.friction_coefficient;
      if constexpr (GC) {
        const GrainDev& gq = P.grain[gqi];
        Kn = (gr.kn + gq.kn) * 0.5;
        zeta = (gr.zeta + gq.zeta) * 0.5;
        mu = (gr.mu + gq.mu) * 0.5;
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
        const double ref = ieee64::sqrt_rn(r2);
        Rc = ref < in.contact_rad ? ref : in.contact_rad;
        Kn = ieee64::div_rn(gr.cnot, Rc);
      }
      if (!(dn <= Rc)) continue;
      if (P.record_pairs) {
        my_pairs += 1;
        my_hash += splitmix64(((unsigned long long)orig_of(P, d) << 32) | orig_of(P, q));
      }
      if (dn == 0.0) my_close += 1;
      double u[D];
      {
        const ieee64::Divisor ddn = ieee64::make_divisor(dn);
        for (int c = 0; c < D; ++c) u[c] = ieee64::div_rn(dir[c], ddn);
      }
      const double crc = Rc - dn;
      const double nvol = P.vol[q];
      const double s1 = ((-Kn) * crc) * nvol;
      double fc[D];
      for (int c = 0; c < D; ++c) fc[c] = s1 * u[c];
      double cf2 = fc[0] * fc[0];
      for (int c = 1; c < D; ++c) cf2 = cf2 + fc[c] * fc[c];
      const double cfn = ieee64::sqrt_rn(cf2);
      for (int c = 0; c < D; ++c) f[c] = f[c] + fc[c];
      uint32_t fr = 0;
      if (P.allow_damping || P.allow_friction) {
        double vq[D], rv[D];
        ldv<D>(P.vel_in, q, vq);
        for (int c = 0; c < D; ++c) rv[c] = vp[c] - vq[c];
        double rvp = rv[0] * u[0];
        for (int c = 1; c < D; ++c) rvp = rvp + rv[c] * u[c];
        if (P.allow_damping) {
          const double dc = ((2.0 * zeta) * ieee64::sqrt_rn(Kn * gr.rho)) * ieee64::sqrt_rn(nvol);
          for (int c = 0; c < D; ++c) f[c] = f[c] + ((-dc) * (rvp * u[c]));
        }
        if (P.allow_friction) {
          double tg[D];
          for (int c = 0; c < D; ++c) tg[c] = rv[c] - (rvp * u[c]);
          double t2 = tg[0] * tg[0];
          for (int c = 1; c < D; ++c) t2 = t2 + tg[c] * tg[c];
          const double tn = ieee64::sqrt_rn(t2);
          if (tn > 0) {
            double sfr = (-mu) * cfn;
            fr = (D == 2 && (tg[1] * u[0] - tg[0] * u[1]) < 0) ? FR_SLIDE_NEG : FR_SLIDE;
            if (tn < ieee64::div_rn((mu * cfn) * P.dt, gr.rho)) {
              sfr = ieee64::div_rn(ieee64::div_rn(-tn, gr.rho), P.dt);
              fr = FR_STICK;
            }
            const ieee64::Divisor dtn = ieee64::make_divisor(tn);
            for (int c = 0; c < D; ++c) f[c] = f[c] + sfr * ieee64::div_rn(tg[c], dtn);
          }
        }
      }
      if constexpr (REC) rent[nrec++] = q | (fr << 30);
    }
  }

  // ---- analytic wall (timeloop.h:753-769 -> contact.h:900-964) ----
  if (mov && other && p_bdry && in.allow_wall) {
    double bmn[D], bmx[D];
    grain_box<D>(P, g, bmn, bmx);
    if (!within_interior<D>(bmn, bmx, in.wall, in.contact_rad)) {
      const double vol_i = P.vol[d];
      const double Knw = GC ? gr.kn : in.normal_stiffness;
      const double zetaw = GC ? gr.zeta : in.damping_ratio;
      const double muw = GC ? gr.mu : in.friction_coefficient;
      constexpr int NS = 2 * D;
      // (side, dir) in the reference's call order
      const int order2[4][2] = {{3, 1}, {0, 0}, {1, 0}, {2, 1}};
      const int order3[6][2] = {{0, 0}, {3, 0}, {1, 1}, {4, 1}, {2, 2}, {5, 2}};
      for (int k = 0; k < NS; ++k) {
        const int side = (D == 2) ? order2[k][0] : order3[k][0];
        const int dir = (D == 2) ? order2[k][1] : order3[k][1];
        const double dist = xpc[dir] - in.wall[side];
        const double R = in.contact_rad;
        if (!(fabs(dist) <= R)) continue;
        wbits |= 1u << (4 * k);
        const double dd = fabs(dist);
        // segment_mass<dim>(R, d) (contact.h:16-41)
        double Area, I;
        if constexpr (D == 2) {
          // The reference's pow(x, 2.0) as products (the correctly rounded square): pow takes 6100
          // cycles in a chain, and a node at a wall called it three times. Roots and quotients on the
          // integer pipe. A chunk at a wall: 24000 -> 12000 cycles, the 500-grain compaction's step
          // 41.9 -> 33.9 us.
          const double R2 = R * R, h2 = R2 - dd * dd;
          Area = M_PI * R2 / 2 - R2 * asin(ieee64::div_rn(dd, R)) - ieee64::sqrt_rn(h2) * dd;
          I = 0.0 * h2;  // 0 * pow(h2, 1.5): 2 / 3 is integer division in the reference
        } else {
          const double a = R - dd, h2 = R * R - dd * dd;
          Area = M_PI / 3 * (a * a) * (2 * R - dd);
          I = M_PI / 4 * (h2 * h2);
        }
        const double centroid = ieee64::div_rn(I, Area);
        const double crc = R - centroid;
        const double pcrc = crc > 0 ? crc : 0;
        const double F = (Knw * pcrc) * Area;
        const double c_sign = dist > 0 ? 1 : -1;
        f[dir] = f[dir] + (c_sign * F);
        WallRec rec;
        rec.a_normal = (vol_i * c_sign) * F;
        rec.a_t1 = 0;
        rec.a_t2 = 0;
        rec.a_damp = 0;
        // replay key: the reference sums reactions grain by grain in its node-loop order
        rec.gid = P.nl_bdry_only ? (gr.node_begin + P.bdry_rank[d]) : orig_of(P, d);
        rec.side = (uint16_t)side;
        rec.has_fric = 0;
        rec.has_damp = 0;
        double rv[D];
        for (int c = 0; c < D; ++c) rv[c] = vp[c];
        rv[dir] = rv[dir] - in.wall_speed[side];
        if (P.allow_friction) {
          const double mu = muw;
          if constexpr (D == 2) {
            const int tg = (dir + 1) % 2;
            if (fabs(rv[tg]) > 0) {
              const double vts = rv[tg] > 0 ? 1 : -1;
              double ff = ((-mu) * fabs(F)) * vts;
              wbits |= (rv[tg] > 0 ? 2u : 10u) << (4 * k);
              if (fabs(rv[tg]) < ieee64::div_rn((mu * fabs(F)) * P.dt, gr.rho)) {
                ff = ieee64::div_rn((-rv[tg]) * gr.rho, P.dt);
                wbits |= 4u << (4 * k);
              }
              f[tg] = f[tg] + ff;
              rec.a_t1 = vol_i * ff;
              rec.has_fric = 1;
            }
          } else {
            const int t1 = (dir + 1) % 3, t2 = (dir + 2) % 3;
            const double v1 = rv[t1], v2 = rv[t2];
            const double vn = ieee64::sqrt_rn(v1 * v1 + v2 * v2);
            if (vn > 0) {
              const double u1 = v1 / vn, u2 = v2 / vn;
              double ff1 = ((-mu) * fabs(F)) * u1;
              double ff2 = ((-mu) * fabs(F)) * u2;
              wbits |= 2u << (4 * k);
              if (vn < (((mu * fabs(F)) * P.dt) / gr.rho)) {
                ff1 = (((-vn) / gr.rho) / P.dt) * u1;
                ff2 = (((-vn) / gr.rho) / P.dt) * u2;
                wbits |= 4u << (4 * k);
              }
              f[t1] = f[t1] + ff1;
              f[t2] = f[t2] + ff2;
              rec.a_t1 = vol_i * ff1;
              rec.a_t2 = vol_i * ff2;
              rec.has_fric = 1;
            }
          }
        }
        if (P.allow_damping) {
          const double dc = ((2.0 * zetaw) * ieee64::sqrt_rn(Knw * gr.rho)) * ieee64::sqrt_rn(fabs(Area));
          const double df = (-dc) * rv[dir];
          f[dir] = f[dir] + df;
          rec.a_damp = vol_i * df;
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

  // ---- external force and torque (timeloop.h:774-824) ----
  if (mov && P.worm) {
    // ft_i += ((t_num + 1) % 2) * extforce (timeloop.h:1171)
    double ef[D];
    ldv<D>(P.extf, d, ef);
    const double gate = (double)((worm_phase(t) + 1u) % 2u);
    for (int c = 0; c < D; ++c) f[c] = f[c] + gate * ef[c];
  } else if (mov) {
    double ef[D];
    ldv<D>(P.extf, d, ef);
    if (P.gradient_extforce) {
      double sc = (double)t / (double)P.extforce_maxstep;
      if (sc > 1) sc = 1;
      for (int c = 0; c < D; ++c) f[c] = f[c] + sc * ef[c];
    } else {
      for (int c = 0; c < D; ++c) f[c] = f[c] + ef[c];
    }
    if (P.enable_torque) {
      const uint32_t ta = gr.torque_axis;
      double r[3] = {0, 0, 0}, rp[3] = {0, 0, 0};
      for (int c = 0; c < D; ++c) r[c] = xpc[c] - P.torque_c[(size_t)g * 3 + c];
      if (D == 3) r[ta] = 0;
      if (D == 3) rp[ta] = 0;
      rp[(ta + 1) % 3] = -r[(ta + 2) % 3];
      rp[(ta + 2) % 3] = r[(ta + 1) % 3];
      double pn2 = rp[0] * rp[0];
      for (int c = 1; c < D; ++c) pn2 = pn2 + rp[c] * rp[c];
      const double pn = sqrt(pn2);
      if (pn > 0) {
        for (int c = 0; c < D; ++c) rp[c] = rp[c] / pn;
      } else {
        rp[(ta + 1) % 3] = 0;
        rp[(ta + 2) % 3] = 0;
      }
      for (int c = 0; c < D; ++c) f[c] = f[c] + (gr.torque_val * rp[c]);
    }
  }

  // ---- velocity update (timeloop.h:834-863); with P.fuse the next step's position update too ----
  double cu[D], dp[D];
  for (int c = 0; c < D; ++c) cu[c] = 0.0;
  if (act) {
    if (P.fuse) ldv<D>(P.disp, d, dp);
    if (mov) {
      double ao[D], a[D], v[D];
      ldv<D>(P.acc, d, ao);
      for (int c = 0; c < D; ++c) {
        a[c] = gr.one_over_rho * f[c];
        double tmp = ao[c] + a[c];
        tmp = tmp * P.half_dt;
        v[c] = vp[c] + tmp;
      }
      if (P.clamped[d]) {
        for (int c = 0; c < D; ++c) {
          a[c] = 0.0;
          v[c] = 0.0;
        }
        if (P.fuse) {
          for (int c = 0; c < D; ++c) dp[c] = 0.0;
        } else {
          P.clamp_pending[d] = 1;
        }
      }
      if (P.worm) worm_clamp<D>(orig_of(P, d) - gr.node_begin, worm_phase(t), a, v);
      stv<D>(P.acc, d, a);
      stv<D>(P.vel_out, d, v);
      if (P.fuse) {
        for (int c = 0; c < D; ++c) dp[c] = dp[c] + ((P.dt * v[c]) + (P.hdt2 * a[c]));
        stv<D>(P.disp, d, dp);
      }
    } else {
      stv<D>(P.vel_out, d, vp);
    }
    if (P.fuse) {
      place_node<D>(P, d, in, dp, P.cur_n, P.curf_n, P.rebuild_n, cu);
    } else {
      stv<D>(P.force, d, f);  // zero for grains that are not movable
    }
  }
  if (P.fuse) grow_box<D>(P.bbox_n, g, act, cu);

  if constexpr (REC) {
    record_masks(P, d, act, lane, rent, nrec, wbits);
    if (P.rec_x) record_tape<D>(P, d, act, t, xpc, vp);
  }

  // ---- diagnostics: warp-aggregated counters ----
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

// ---------------------------------------------------------------------------------------------
// host-side launchers
// ---------------------------------------------------------------------------------------------
// The force kernel's variants: mask recording (REC), per-grain contact parameters (GC), candidate
// lists or the grid search (LIST); the plain kernel with lists for 5 or 7 blocks (force_bps(): 6 takes
// 7) of 128 threads per
// SM (96 or 72 registers): the latency of its own chain counts where the chunks do not fill the GPU
// (two disks: 20.5 us a step at 5 blocks, 21.1 at 7), occupancy where they do (3D spheres 366 and 359).
template <int D>
static const void* force_ptr(bool rec, bool gc, bool list, int bps) {
  static const void* const fs[8] = {
      (const void*)k_force<D, false, false, false, 6>, (const void*)k_force<D, false, false, true, 5>,
      (const void*)k_force<D, false, true, false, 5>,  (const void*)k_force<D, false, true, true, 5>,
      (const void*)k_force<D, true, false, false, 5>,  (const void*)k_force<D, true, false, true, 5>,
      (const void*)k_force<D, true, true, false, 5>,   (const void*)k_force<D, true, true, true, 5>};
  if (!rec && !gc && list && bps > 5) return (const void*)k_force<D, false, false, true, 7>;
  return fs[(rec ? 4 : 0) | (gc ? 2 : 0) | (list ? 1 : 0)];
}

template <int D>
static void predict_t(const Dev& P, cudaStream_t s, uint64_t* launches, bool pdl) {
  launch_k(k_predict<D>, cdiv(P.N, 256), 256, 0, s, pdl, P);
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
  if (P.n_edges) {
    launch_k(k_bonds<D>, (P.n_edges - 1u) / 256u + 1u, 256, 0, s, pdl, P);  // up to 2^32 - 1 entries
    *launches += 1;
  }
  const dim3 grid(cdiv(P.n_chunks * 32, L.force_block)), block(L.force_block);
  using K = void (*)(const Dev);
  launch_k((K)force_ptr<D>(rec, P.grain_contact, P.cand_q, force_bps(P.n_chunks, P.n_sms)), grid, block, 0, s, pdl, P);
  *launches += 1;
  if (e1) cudaEventRecord(e1, s);
}
template <int D>
static void finalize_t(const Dev& P, cudaStream_t s, uint64_t* launches, bool pdl) {
  launch_k(k_finalize<D>, finalize_blocks(P.I), FINAL_THREADS, P.wrec_smem ? FINAL_SMEM : 0, s, pdl, P);
  *launches += 1;
}

cudaError_t kernels_init() {
  cudaError_t e = cudaFuncSetAttribute(k_finalize<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, FINAL_SMEM);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_finalize<3>, cudaFuncAttributeMaxDynamicSharedMemorySize, FINAL_SMEM);
  if (e != cudaSuccess) return e;
  // the recording variants of the force kernel have local frames of about 1.1 KB
  const void* fs[32];
  int n = 0;
  for (int k = 0; k < 8; ++k)
    for (int b = 5; b <= 7; b += 2) {
      fs[n++] = force_ptr<2>(k & 4, k & 2, k & 1, b);
      fs[n++] = force_ptr<3>(k & 4, k & 2, k & 1, b);
    }
  size_t need = 0;
  static std::atomic<size_t> known{0};
  e = max_local_bytes(fs, n, &known, &need);
  return e == cudaSuccess ? ensure_local_bytes(need) : e;
}

void launch_predict(const Dev& P, cudaStream_t s, uint64_t* launches, bool pdl) {
  P.dim == 2 ? predict_t<2>(P, s, launches, pdl) : predict_t<3>(P, s, launches, pdl);
}
void launch_body(const Dev& P, const LaunchCfg& L, cudaStream_t s, uint64_t* launches, bool pdl, bool rec,
                 cudaEvent_t e0, cudaEvent_t e1) {
  P.dim == 2 ? body_t<2>(P, L, s, launches, pdl, rec, e0, e1) : body_t<3>(P, L, s, launches, pdl, rec, e0, e1);
}
void launch_finalize(const Dev& P, cudaStream_t s, uint64_t* launches, bool pdl) {
  P.dim == 2 ? finalize_t<2>(P, s, launches, pdl) : finalize_t<3>(P, s, launches, pdl);
}

uint32_t grid_coop_blocks(const Dev& P, int device) {
  int per_sm = 0, sms = 0, coop = 0;
  const void* k = P.dim == 2 ? (const void*)k_grid_coop<2> : (const void*)k_grid_coop<3>;
  if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device) != cudaSuccess || !coop) return 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, COOP_THREADS, 0) != cudaSuccess || per_sm < 1) return 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || sms < 1) return 0;
  const uint32_t want = cdiv(P.N, COOP_THREADS);
  // three blocks per SM: threads enough for the candidate-list phase, few blocks to schedule on
  // the (common) steps without a rebuild and to meet at the grid barriers (same box, collision
  // ensemble: 2 -> 3 blocks 0.0793 -> 0.0780 ms/step at skin 0.25; 4 and 5 blocks were slower
  // than 3, other workloads unchanged)
  return std::max(1u, std::min((uint32_t)(std::min(per_sm, 3) * sms), want));
}

// ---------------------------------------------------------------------------------------------
// Check kernel of the integer FP64 arithmetic (pg_ieee64.cuh): out[i] = op(a[i], b[i]), the
// division through a prepared divisor.
// ---------------------------------------------------------------------------------------------
__global__ void k_ieee64_check(int32_t op, const double* a, const double* b, int64_t n, double* out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double x = a[i], y = b[i];
  double r;
  switch (op) {
    case PG_IEEE_DIV: r = ieee64::div_rn(x, ieee64::make_divisor(y)); break;
    case PG_IEEE_SQRT: r = ieee64::sqrt_rn(fabs(x)); break;
    case PG_IEEE_ADD: r = ieee64::add_rn(x, y); break;
    case PG_IEEE_SUB: r = ieee64::sub_rn(x, y); break;
    case PG_IEEE_MUL: r = ieee64::mul_rn(x, y); break;
    default: r = ieee64::widen_f32((float)x); break;
  }
  out[i] = r;
}

cudaError_t launch_ieee64_check(int32_t op, const double* a, const double* b, int64_t n, double* out,
                                cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  const int64_t blocks = (n + 255) / 256;
  k_ieee64_check<<<(unsigned)blocks, 256, 0, s>>>(op, a, b, n, out);
  return cudaGetLastError();
}

}  // namespace pg
