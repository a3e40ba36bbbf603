// GB300 (sm_103a) kernels of the gradient path, reverse side: the hand-written adjoint of one
// frozen-mask time step (the forward map is spelled out in pg_adjoint.cu) and the per-grain
// parameter reduction.
//
// With cotangents (db, vb, ab) of the state (disp', vel', acc') after step t:
//   Fb   = (ab + 0.5*dt*vb) / rho                         cotangent of the force density
//   Xb   = (dF/dX)^T Fb  (+ wall-reaction cotangent at the objective's step)
//   Vf   = (dF/dvel)^T Fb
//   db_o = db + Xb ;  vb_o = vb + dt*(db + Xb) + Vf ;  ab_o = 0.5*dt*vb + (dt*dt*0.5)*(db + Xb)
// and the step's parameter cotangents are added per node. Every pair term is gathered at both of
// its nodes (a node reads its own contact list and finds itself in each partner's list), so the
// step is atomic-free and deterministic.
//
// One kernel per reverse step, two blocks per 32-node SELL chunk. Bonds: SUB warps per block, warp w
// taking the node's bond slots k = w, w+SUB, ... (one coalesced access per warp and
// slot, as in the force kernels), partial sums added in shared memory in a fixed order; its bond
// products run in FP32 for mixed-precision handles (GB300 runs FP64 at a small fraction of its
// FP32 rate) and in FP64 for FP64 handles and frozen replays (the FP64 reference gradient).
// Contacts and walls: tasks over the block's threads, FP64. The later of the two blocks runs the
// integrator; the cotangent state is FP64 throughout.
#include <cuda_runtime.h>

#include <cmath>

#include "pg_adjoint.cuh"
#include "pg_adjoint.h"
#include "pg_common.cuh"
#include "pg_device.cuh"
#include "pg_hilo.cuh"

namespace pg {

constexpr int SUB = 4;
// Cotangents a chunk's contact block adds up per node: xb[D], vfb[D], pc[NPARAM].
template <int D>
constexpr int ADJ_NV = 2 * D + NPARAM;

// Adjoint of one node-node contact force phi(y, r) received by a node of density rho from a
// partner of volume vq; y = x_partner - x_node, r = v_node - v_partner, g = cotangent of phi.
// Adds the cotangents of y and r to yb, rb and of (K_n, zeta, mu) to pb.
template <int D>
__device__ void pair_vjp(const double* y, const double* r, const double* g, double Kn, double Rc, double zeta,
                         double mu, double vq, double rho, uint32_t fr, bool damp, bool fric, double dt, double* yb,
                         double* rb, double* pb) {
  double n2 = 0.0;
  for (int c = 0; c < D; ++c) n2 += y[c] * y[c];
  const double dn = sqrt(n2);
  if (!(dn > 0.0)) return;
  const double idn = 1.0 / dn;
  double u[D];
  for (int c = 0; c < D; ++c) u[c] = y[c] * idn;
  double gu = 0.0;
  for (int c = 0; c < D; ++c) gu += g[c] * u[c];
  // elastic: phi1 = s1*u, s1 = -K_n (R_c - |y|) vol_q
  const double s1 = -Kn * (Rc - dn) * vq;
  for (int c = 0; c < D; ++c) yb[c] += Kn * vq * gu * u[c] + (s1 * idn) * (g[c] - gu * u[c]);
  pb[0] += -(Rc - dn) * vq * gu;
  if (!(damp || (fric && fr))) return;
  double ru = 0.0;
  for (int c = 0; c < D; ++c) ru += r[c] * u[c];
  if (damp) {
    // phi2 = -dc (r.u) u, dc = 2 zeta sqrt(K_n rho) sqrt(vol_q)
    const double sq = sqrt(Kn * rho) * sqrt(vq);
    const double dc = 2.0 * zeta * sq;
    for (int c = 0; c < D; ++c) {
      rb[c] += -dc * gu * u[c];
      yb[c] += -dc * (gu * (r[c] - ru * u[c]) + ru * (g[c] - gu * u[c])) * idn;
    }
    const double dcb = -ru * gu;
    pb[1] += dcb * 2.0 * sq;
    if (Kn != 0.0) pb[0] += dcb * dc / (2.0 * Kn);
  }
  if (!(fric && fr)) return;
  double z[D];
  if (fr == FR_STICK) {
    // phi3 = -tg / (rho dt), tg = r - (r.u) u
    for (int c = 0; c < D; ++c) z[c] = -g[c] / (rho * dt);
  } else {
    // phi3 = -mu cfn th, th = tg/|tg| (2D: the recorded direction +-perp(u)); cfn = |s1| = -s1
    // on the recorded run, continued as -s1 (the replay's smooth extension)
    const double cfn = -s1;
    const double sgn = -1.0;
    if constexpr (D == 2) {
      const double sg = (fr == FR_SLIDE_NEG) ? -1.0 : 1.0;
      const double th[2] = {-sg * u[1], sg * u[0]};
      const double a = g[0] * th[0] + g[1] * th[1];
      for (int c = 0; c < D; ++c) yb[c] += -mu * a * sgn * Kn * vq * u[c] + mu * cfn * gu * th[c] * idn;
      pb[2] += -cfn * a;
      pb[0] += -mu * a * vq * (Rc - dn);
      return;
    } else {
      double tg[D], t2 = 0.0;
      for (int c = 0; c < D; ++c) {
        tg[c] = r[c] - ru * u[c];
        t2 += tg[c] * tg[c];
      }
      const double tn = sqrt(t2);
      if (!(tn > 0.0)) return;
      double a = 0.0;
      for (int c = 0; c < D; ++c) a += g[c] * tg[c] / tn;
      for (int c = 0; c < D; ++c) {
        z[c] = -mu * cfn * (g[c] - a * tg[c] / tn) / tn;
        yb[c] += -mu * a * sgn * Kn * vq * u[c];
      }
      pb[2] += -cfn * a;
      pb[0] += -mu * a * vq * (Rc - dn);
    }
  }
  // through tg = r - (r.u) u
  double zu = 0.0;
  for (int c = 0; c < D; ++c) zu += z[c] * u[c];
  for (int c = 0; c < D; ++c) {
    rb[c] += z[c] - zu * u[c];
    yb[c] += -(zu * (r[c] - ru * u[c]) + ru * (z[c] - zu * u[c])) * idn;
  }
}

// Wall geometry of one side at distance dd <= R (segment_mass, contact.h:16-41): F = K_n*FK with
// FK = max(R - centroid, 0) * Area, and the derivatives d(Area)/d(dd), d(FK)/d(dd).
template <int D>
__device__ __forceinline__ void wall_geom(double R, double dd, double* A, double* Ap, double* FK, double* FKp) {
  if constexpr (D == 2) {
    const double s = sqrt(fmax(R * R - dd * dd, 0.0));
    *A = M_PI * R * R / 2 - R * R * asin(dd / R) - s * dd;
    *Ap = -2.0 * s;
    // the centroid is 0 (integer 2/3 in the reference), so FK = R * Area
    *FK = R * *A;
    *FKp = R * *Ap;
  } else {
    const double a = R - dd, b = R * R - dd * dd;
    *A = M_PI / 3 * a * a * (2 * R - dd);
    *Ap = -M_PI / 3 * a * (5 * R - 3 * dd);
    const double I = M_PI / 4 * b * b;
    const double Ip = -M_PI * dd * b;
    const double crc = R - I / *A;
    if (crc > 0) {
      *FK = R * *A - I;
      *FKp = R * *Ap - Ip;
    } else {
      *FK = 0.0;
      *FKp = 0.0;
    }
  }
}

// cotangent of the force on node j: Fb = (ab + 0.5 dt vb) / rho; zero where the force does not
// reach the state (grains that are not movable, clamped nodes)
template <int D>
__device__ __forceinline__ bool force_bar(const Dev& P, const AdjStep& A, uint32_t j, double* Fb) {
  double ab[D], vb[D];
  ldv<D>(A.ab, j, ab);
  ldv<D>(A.vb, j, vb);
  const GrainDev& gj = P.grain[P.node_grain[j]];
  if (!(gj.flags & GF_MOVABLE) || P.clamped[j]) {
    for (int c = 0; c < D; ++c) Fb[c] = 0.0;
    return false;
  }
  for (int c = 0; c < D; ++c) Fb[c] = gj.one_over_rho * (ab[c] + P.half_dt * vb[c]);
  return true;
}

template <int D>
__device__ __forceinline__ void ldfv(const float* a, uint32_t i, float (&v)[D]) {
  if constexpr (D == 2) {
    const float2 t = reinterpret_cast<const float2*>(a)[i];
    v[0] = t.x;
    v[1] = t.y;
  } else {
    const float4 t = reinterpret_cast<const float4*>(a)[i];
    v[0] = t.x;
    v[1] = t.y;
    v[2] = t.z;
  }
}
template <int D>
__device__ __forceinline__ void stfv(float* a, uint32_t i, const float (&v)[D]) {
  if constexpr (D == 2) {
    reinterpret_cast<float2*>(a)[i] = make_float2(v[0], v[1]);
  } else {
    reinterpret_cast<float4*>(a)[i] = make_float4(v[0], v[1], v[2], 0.f);
  }
}

// Bond part of the reverse step: f_p = sum_j cnot vol_j s(eta) e(eta), eta = X_j - X_p; H =
// d(s e)/d(eta) is symmetric, so Xb_p = cnot sum_j H (vol_p Fb_j - vol_j Fb_p), and
// dF_p/dcnot = f_p / cnot. Writes the node's bond share of Xb (xbb) and of the cnot cotangent
// (pcb). F32: the mixed engine's form -- xi from the hi/lo reference positions,
// the displacement difference from the tape's hi/lo pairs, the cancellation-free stretch
// s = (2 xi.et + et.et) / (|xi| (|xi + et| + |xi|)), force cotangents from the FP32 array fbf.
template <int D, bool F32>
__device__ __forceinline__ void adj_bonds(const Dev& P, const AdjStep& A, uint32_t chunk, double (*red)[D + 1][32]) {
  const uint32_t lane = threadIdx.x & 31, sub = threadIdx.x >> 5;
  const uint32_t d = chunk * 32 + lane;
  const bool act = d < P.N;
  double part[D + 1];
  for (int v = 0; v <= D; ++v) part[v] = 0.0;
  const uint32_t g = act ? P.node_grain[d] : 0;
  const GrainDev& gr = P.grain[g];
  const bool mov = act && (gr.flags & GF_MOVABLE);
  if (mov) {
    const uint32_t t = *A.tstep;
    const uint32_t cdeg = P.chunk_deg[chunk];
    const uint32_t slot0 = P.chunk_slot[chunk] + lane;
    const uint32_t w0 = P.chunk_word[chunk];
    if constexpr (F32) {
      float dh[D], dl[D], xh[D], xl[D], Fb[D], xb[D], pc = 0.f;
      ld_hl<D>(A.df, P.np, d, dh, dl);
      ld_hl<D>(P.xref, P.np, d, xh, xl);
      ldfv<D>(A.fbf, d, Fb);
      for (int c = 0; c < D; ++c) xb[c] = 0.f;
      const float volp = P.vol_f[d];
      for (uint32_t k = sub; k < cdeg; k += SUB) {
        const uint32_t s = slot0 + 32u * k;
        if (!bond_used(A.end_alive, A.break_step, w0 + k, lane, s, t)) continue;
        const uint32_t j = P.bcol[s];
        float jdh[D], jdl[D], jxh[D], jxl[D], Fj[D];
        ld_hl<D>(A.df, P.np, j, jdh, jdl);
        ld_hl<D>(P.xref, P.np, j, jxh, jxl);
        ldfv<D>(A.fbf, j, Fj);
        const float volj = P.vol_f[j];
        float xi[D], et[D], y[D];
        for (int c = 0; c < D; ++c) {
          xi[c] = (jxh[c] - xh[c]) + (jxl[c] - xl[c]);
          et[c] = (jdh[c] - dh[c]) + (jdl[c] - dl[c]);
          y[c] = xi[c] + et[c];
        }
        float xx = 0.f, yy = 0.f, xe = 0.f, ee = 0.f;
        for (int c = 0; c < D; ++c) {
          xx = fmaf(xi[c], xi[c], xx);
          yy = fmaf(y[c], y[c], yy);
          xe = fmaf(xi[c], et[c], xe);
          ee = fmaf(et[c], et[c], ee);
        }
        const float ixn = rsqrtf(xx), iyn = rsqrtf(yy);
        const float str = __fdividef(fmaf(2.f, xe, ee) * ixn, fmaf(yy, iyn, xx * ixn));
        float e[D], w[D], ew = 0.f, eF = 0.f;
        for (int c = 0; c < D; ++c) {
          e[c] = y[c] * iyn;
          w[c] = volp * Fj[c] - volj * Fb[c];
          ew = fmaf(e[c], w[c], ew);
          eF = fmaf(e[c], Fb[c], eF);
        }
        for (int c = 0; c < D; ++c) xb[c] += e[c] * ew * ixn + str * (w[c] - e[c] * ew) * iyn;
        pc = fmaf(volj * str, eF, pc);
      }
      for (int c = 0; c < D; ++c) part[c] = gr.cnot * (double)xb[c];
      part[D] = (double)pc;
    } else {
      double Fb[D], xp[D];
      force_bar<D>(P, A, d, Fb);
      ldv<D>(A.X, d, xp);
      const double volp = P.vol[d];
      for (uint32_t k = sub; k < cdeg; k += SUB) {
        const uint32_t s = slot0 + 32u * k;
        if (!bond_used(A.end_alive, A.break_step, w0 + k, lane, s, t)) continue;
        const uint32_t j = P.bcol[s];
        const double xin = P.bxin[s];
        double xj[D], Fj[D], e[D];
        ldv<D>(A.X, j, xj);
        force_bar<D>(P, A, j, Fj);
        double n2 = 0.0;
        for (int c = 0; c < D; ++c) {
          e[c] = xj[c] - xp[c];
          n2 += e[c] * e[c];
        }
        const double en = sqrt(n2);
        const double ien = 1.0 / en, ixin = 1.0 / xin;
        for (int c = 0; c < D; ++c) e[c] *= ien;
        const double str = (en - xin) * ixin;
        const double volj = P.vol[j];
        double w[D], ew = 0.0, eF = 0.0;
        for (int c = 0; c < D; ++c) {
          w[c] = volp * Fj[c] - volj * Fb[c];
          ew += e[c] * w[c];
          eF += e[c] * Fb[c];
        }
        for (int c = 0; c < D; ++c) part[c] += gr.cnot * (e[c] * ew * ixin + str * (w[c] - e[c] * ew) * ien);
        part[D] += volj * str * eF;
      }
    }
  }
  // fixed-order sum of the SUB partial cotangents
  for (int v = 0; v <= D; ++v) red[sub][v][lane] = part[v];
  __syncthreads();
  if (sub != 0) return;
  double out[D];
  for (int c = 0; c < D; ++c) {
    double s = red[0][c][lane];
    for (int w = 1; w < SUB; ++w) s += red[w][c][lane];
    out[c] = s;
  }
  double pcs = red[0][D][lane];
  for (int w = 1; w < SUB; ++w) pcs += red[w][D][lane];
  if (act) {
    stv<D>(A.xbb, d, out);
    A.pcb[d] = pcs;
  }
}

// Contact and wall part of the reverse step, one block per 32-node chunk. A contact of a
// pair acts on the node through two forces, its own and its partner's, and each is a task of a few
// hundred dependent FP64 operations. The chunk's tasks are laid out over the block's threads, 64
// entries of the nodes' lists a round with the own forces on warps 0 and 1 and the partners' on 2 and
// 3, so a chunk with contacts takes one such chain where a lane a node took two for every SUB
// entries of its node. The walls are a chain of their own, on a warp that mostly has no task. The
// node lanes add the results in a fixed order, warp w the entries i = w, w+SUB, ..., then warp 0 the
// warps' sums. Bound by that latency: 592 chunks are one wave of one or two active warps a block;
// 20k nodes in 50 grains, us, with the integrator and as a kernel of its own: 21.6 -> 13.7 (about 5
// with neither contacts nor walls).
constexpr uint32_t ADJ_ENTRIES = 16 * SUB;  // entries of a round

// The contact tasks of entry e of node p (grain g, force cotangent Fb): its own force, or the
// partner's. r[0..D): position share, r[D..2D): velocity share, then the parameters'.
template <int D>
__device__ __forceinline__ void contact_task(const Dev& P, const AdjStep& A, uint32_t p, uint32_t g, const double* Fb,
                                             uint32_t entry, bool partner, double* out) {
  const uint32_t q = entry & ENT_NODE;
  const uint32_t gqi = P.node_grain[q], oq = A.off[q], nq = A.cnt[q];
  double xp[D], xq[D], vp[D], vq[D], F[D], y[D], r[D], yb[D], rb[D], pb[3] = {0.0, 0.0, 0.0};
  ldv<D>(A.X, p, xp);
  ldv<D>(A.X, q, xq);
  ldv<D>(A.V, p, vp);
  ldv<D>(A.V, q, vq);
  const double vol = P.vol[partner ? p : q];
  const GrainDev &gr = P.grain[g], &gq = P.grain[gqi];
  uint32_t fr = entry >> 30;
  if (partner) {
    // the partner's force from this node, if the partner recorded it
    if (!force_bar<D>(P, A, q, F)) return;
    fr = 4u;
#pragma unroll 4
    for (uint32_t k = 0; k < nq; ++k) {
      const uint32_t eq = A.ent[oq + k];
      if ((eq & ENT_NODE) == p) fr = eq >> 30;
    }
    if (fr == 4u) return;
  }
  const bool same = gqi == g;
  double Kn, Rc, zeta, mu;
  pair_params<D>(P, P.inst[gr.inst], gr, gq, same, p, q, &Kn, &Rc, &zeta, &mu);
  const double sg = partner ? -1.0 : 1.0;
#pragma unroll
  for (int c = 0; c < D; ++c) {
    if (!partner) F[c] = Fb[c];
    y[c] = sg * (xq[c] - xp[c]);
    r[c] = sg * (vp[c] - vq[c]);
    yb[c] = 0.0;
    rb[c] = 0.0;
  }
  pair_vjp<D>(y, r, F, Kn, Rc, zeta, mu, vol, partner ? gq.rho : gr.rho, fr, P.allow_damping, P.allow_friction, P.dt,
              yb, rb, pb);
#pragma unroll
  for (int c = 0; c < D; ++c) {
    out[c] = -sg * yb[c];
    out[D + c] = sg * rb[c];
  }
  double* pc = out + 2 * D;
  if (!same) {
    pc[1] = 0.5 * pb[0];
    pc[2] = 0.5 * pb[1];
    pc[3] = 0.5 * pb[2];
  } else if (!partner) {
    pc[0] = pb[0] / Rc;  // K_n' = cnot / R_c'
    pc[2] = pb[1];
    pc[3] = pb[2];
  }
}

template <int D>
__device__ __forceinline__ void adj_contacts(const Dev& P, const AdjStep& A, uint32_t chunk,
                                             double (*red)[ADJ_NV<D>][32], double (*res)[32 * SUB]) {
  constexpr int NS = 2 * D, NV = ADJ_NV<D>;
  const uint32_t lane = threadIdx.x & 31, sub = threadIdx.x >> 5;
  const uint32_t d = chunk * 32 + lane;
  const bool act = d < P.N;
  double acc[NV];
  for (int v = 0; v < NV; ++v) acc[v] = 0.0;
  double* xb = acc;
  double* vfb = acc + D;
  double* pc = acc + 2 * D;
  double Fb[D] = {};
  uint32_t g = 0, o = 0, n = 0, wbits = 0;
  bool live = false;
  if (act) {
    g = P.node_grain[d];
    o = A.off[d];
    n = A.cnt[d];
    wbits = A.wall[d];
    live = force_bar<D>(P, A, d, Fb);
    if (!live) n = wbits = 0;
  }
  uint32_t incl = n;
#pragma unroll
  for (int s = 1; s < 32; s <<= 1) {
    const uint32_t v = __shfl_up_sync(0xffffffffu, incl, s);
    if (lane >= (uint32_t)s) incl += v;
  }
  const uint32_t first = incl - n, total = __shfl_sync(0xffffffffu, incl, 31);
  const bool pairs = total || __any_sync(0xffffffffu, wbits);  // the same in every warp
  if (!pairs && sub != 0) return;

  // walls: the node's force and, at the objective's step, its share of the wall reactions
  if (sub == SUB - 1 && wbits) {
    const GrainDev& gr = P.grain[g];
    const InstDev& in = P.inst[gr.inst];
    double xp[D], vp[D];
    ldv<D>(A.X, d, xp);
    ldv<D>(A.V, d, vp);
    const double volp = P.vol[d];
    const bool damp = P.allow_damping, fric = P.allow_friction;
    const double R = in.contact_rad, Kn = gr.kn, rho = gr.rho;
    for (int k = 0; k < NS; ++k) {
      if (!wb_contact(wbits, k)) continue;
      int side, dir;
      wall_side<D>(k, &side, &dir);
      double gv[D];
      for (int c = 0; c < D; ++c) gv[c] = Fb[c];
      if (A.rbar) {
        // reaction[side] -= vol_p * (the node's wall force of this side)
        for (int c = 0; c < D; ++c) gv[c] -= volp * A.rbar[((size_t)gr.inst * NS + side) * D + c];
      }
      const double dist = xp[dir] - A.W[(size_t)gr.inst * NS + side];
      const double dd = fmin(fabs(dist), R);  // the replay's extension beyond R
      const double cs = dist > 0 ? 1.0 : -1.0;
      double Ar, Ap, FK, FKp;
      wall_geom<D>(R, dd, &Ar, &Ap, &FK, &FKp);
      const double F = Kn * FK, Fp = Kn * FKp;  // dF/d(dd); d(dd)/dX = cs
      // normal: f[dir] += cs F
      xb[dir] += gv[dir] * Fp;
      pc[1] += gv[dir] * cs * FK;
      double rv[D];
      for (int c = 0; c < D; ++c) rv[c] = vp[c];
      rv[dir] -= in.wall_speed[side];
      if (fric && wb_fric(wbits, k)) {
        const bool stick = wb_stick(wbits, k);
        const double sF = F > 0 ? 1.0 : (F < 0 ? -1.0 : 0.0);
        if constexpr (D == 2) {
          const int tg = (dir + 1) % 2;
          if (stick) {
            vfb[tg] += gv[tg] * (-rho / P.dt);
          } else {
            const double vts = wb_neg(wbits, k) ? -1.0 : 1.0;
            xb[dir] += gv[tg] * (-gr.mu * vts * sF * Fp * cs);
            pc[3] += gv[tg] * (-fabs(F) * vts);
            pc[1] += gv[tg] * (-gr.mu * vts * sF * FK);
          }
        } else {
          const int t1 = (dir + 1) % 3, t2 = (dir + 2) % 3;
          if (stick) {
            vfb[t1] += gv[t1] * (-1.0 / (rho * P.dt));
            vfb[t2] += gv[t2] * (-1.0 / (rho * P.dt));
          } else {
            const double v1 = rv[t1], v2 = rv[t2];
            const double vn = sqrt(v1 * v1 + v2 * v2);
            if (vn > 0) {
              const double u1 = v1 / vn, u2 = v2 / vn;
              const double a = gv[t1] * u1 + gv[t2] * u2;
              xb[dir] += -gr.mu * a * sF * Fp * cs;
              pc[3] += -fabs(F) * a;
              pc[1] += -gr.mu * a * sF * FK;
              vfb[t1] += -gr.mu * fabs(F) * (gv[t1] - a * u1) / vn;
              vfb[t2] += -gr.mu * fabs(F) * (gv[t2] - a * u2) / vn;
            }
          }
        }
      }
      if (damp) {
        // df = -dc rv[dir], dc = 2 zeta sqrt(K_n rho) sqrt(|Area|)
        const double sq = sqrt(Kn * rho);
        const double sa = sqrt(fabs(Ar));
        const double dc = 2.0 * gr.zeta * sq * sa;
        vfb[dir] += gv[dir] * (-dc);
        if (sa > 0) xb[dir] += gv[dir] * (-rv[dir]) * gr.zeta * sq * (Ap / sa) * cs;
        pc[2] += gv[dir] * (-rv[dir]) * 2.0 * sq * sa;
        if (Kn != 0.0) pc[1] += gv[dir] * (-rv[dir]) * dc / (2.0 * Kn);
      }
    }
  }

  // contacts: the node's own forces (its list) and the partners' forces from it (their lists)
  for (uint32_t e0 = 0; e0 < total; e0 += ADJ_ENTRIES) {
    const uint32_t m = min(total - e0, ADJ_ENTRIES);
    const bool partner = threadIdx.x >= m;
    const uint32_t e = e0 + (partner ? threadIdx.x - m : threadIdx.x);
    uint32_t pl = 0;  // the lane of entry e: as many lanes' lists end at or before it
#pragma unroll
    for (uint32_t s = 16; s; s >>= 1)
      if (__shfl_sync(0xffffffffu, incl, pl + s - 1) <= e) pl += s;
    const uint32_t gp = __shfl_sync(0xffffffffu, g, pl);
    const uint32_t at = __shfl_sync(0xffffffffu, o - first, pl) + e;
    double Fp[D];
#pragma unroll
    for (int c = 0; c < D; ++c) Fp[c] = __shfl_sync(0xffffffffu, Fb[c], pl);
    if (threadIdx.x < 2 * m) {
      double out[NV];
#pragma unroll
      for (int v = 0; v < NV; ++v) out[v] = 0.0;
      contact_task<D>(P, A, chunk * 32 + pl, gp, Fp, A.ent[at], partner, out);
#pragma unroll
      for (int v = 0; v < NV; ++v) res[v][threadIdx.x] = out[v];
    }
    __syncthreads();
    // entries of this round: [e0, e0 + ADJ_ENTRIES)
    const uint32_t i1 = min(n, e0 + ADJ_ENTRIES > first ? e0 + ADJ_ENTRIES - first : 0u);
    uint32_t i = sub;
    if (e0 > first + sub) i += (e0 - first - sub + SUB - 1) / SUB * SUB;
    for (; i < i1; i += SUB) {
      const uint32_t k = first + i - e0;
#pragma unroll
      for (int v = 0; v < NV; ++v) acc[v] = (acc[v] + res[v][k]) + res[v][m + k];
    }
    __syncthreads();
  }

  // fixed-order sum of the SUB partial cotangents (warp 0)
  if (pairs) {
    for (int v = 0; v < NV; ++v) red[sub][v][lane] = acc[v];
    __syncthreads();
  }
  if (sub != 0) return;
  if (pairs)
    for (int v = 0; v < NV; ++v) {
      double sm = red[0][v][lane];
      for (int w = 1; w < SUB; ++w) sm += red[w][v][lane];
      acc[v] = sm;
    }
  double* rs = A.rest + (size_t)chunk * NV * 32 + lane;
  for (int v = 0; v < NV; ++v) rs[32 * v] = acc[v];
}

// The end of a reverse step for a chunk (one warp): both shares are there.
template <int D>
__device__ __forceinline__ void adj_finish(const Dev& P, const AdjStep& A, uint32_t chunk) {
  constexpr int NV = ADJ_NV<D>;
  const uint32_t lane = threadIdx.x & 31, d = chunk * 32 + lane;
  if (d >= P.N) return;
  const GrainDev& gr = P.grain[P.node_grain[d]];
  if (!(gr.flags & GF_MOVABLE) || P.clamped[d]) {
    // the state of this node does not depend on the parameters
    double zero[D];
    for (int c = 0; c < D; ++c) zero[c] = 0.0;
    stv<D>(A.db_o, d, zero);
    stv<D>(A.vb_o, d, zero);
    stv<D>(A.ab_o, d, zero);
    if (A.fbf_o) {
      float zf[D];
      for (int c = 0; c < D; ++c) zf[c] = 0.f;
      stfv<D>(A.fbf_o, d, zf);
    }
    return;
  }
  const double* rs = A.rest + (size_t)chunk * NV * 32 + lane;
  double acc[NV];
  for (int v = 0; v < NV; ++v) acc[v] = __ldcg(rs + 32 * v);
  double* xb = acc;
  double* vfb = acc + D;
  double* pc = acc + 2 * D;
  const double* xbond = A.xbb + (size_t)d * (D == 2 ? 2 : 4);
  for (int c = 0; c < D; ++c) xb[c] += __ldcg(xbond + c);
  pc[0] += __ldcg(A.pcb + d);

  // integrator
  double db[D], vb[D], o1[D], o2[D], o3[D];
  ldv<D>(A.db, d, db);
  ldv<D>(A.vb, d, vb);
  for (int c = 0; c < D; ++c) {
    const double dtot = db[c] + xb[c];
    o1[c] = dtot;
    o2[c] = vb[c] + P.dt * dtot + vfb[c];
    o3[c] = P.half_dt * vb[c] + P.hdt2 * dtot;
  }
  stv<D>(A.db_o, d, o1);
  stv<D>(A.vb_o, d, o2);
  stv<D>(A.ab_o, d, o3);
  if (A.fbf_o) {
    // force cotangent of the previous step, for the FP32 bond products of the next reverse step
    float nf[D];
    for (int c = 0; c < D; ++c) nf[c] = (float)(gr.one_over_rho * (o3[c] + P.half_dt * o2[c]));
    stfv<D>(A.fbf_o, d, nf);
  }
  double* pa = A.pacc + (size_t)d * NPARAM;
  for (int k = 0; k < NPARAM; ++k) pa[k] += pc[k];
}

// A reverse step: two blocks a chunk, the contacts and walls of all chunks first (the longer chains),
// then the bonds, which run beside them. Each writes its share; the one that comes second (a ticket a
// chunk, back at 0 when the step ends) runs the integrator. Nothing waits. In 2D 5 blocks per SM (96
// registers), so that bond blocks are resident beside a wave of contact blocks. 592 chunks, 300 steps
// forward, recomputed and reversed, ms: two kernels 15.8; one, at 4 / 5 / 6 / 8 blocks per SM
// 15.1 / 14.0 / 14.2 / 14.5.
template <int D, bool F32>
__global__ void __launch_bounds__(32 * SUB, D == 2 ? 5 : 3) k_adj_step(const Dev P, const AdjStep A) {
  pdl_enter();
  constexpr int NV = ADJ_NV<D>;
  __shared__ double red[SUB][NV][32];
  __shared__ double res[NV][32 * SUB];
  const bool bonds = blockIdx.x >= P.n_chunks;
  const uint32_t chunk = bonds ? blockIdx.x - P.n_chunks : blockIdx.x;
  if (bonds) {
    adj_bonds<D, F32>(P, A, chunk, reinterpret_cast<double(*)[D + 1][32]>(&red[0][0][0]));
  } else {
    adj_contacts<D>(P, A, chunk, red, res);
  }
  if (threadIdx.x >= 32) return;
  __threadfence();
  __syncwarp();
  uint32_t other = 0;
  if (threadIdx.x == 0) other = atomicAdd(&A.ticket[chunk], 1u);
  if (!__shfl_sync(0xffffffffu, other, 0)) return;
  if (threadIdx.x == 0) A.ticket[chunk] = 0;
  __threadfence();
  adj_finish<D>(P, A, chunk);
}

// force cotangents of the first reverse step from the seed cotangent (FP32 bond path)
template <int D>
__global__ void k_fb_init(const Dev P, const AdjStep A) {
  pdl_enter();
  const uint32_t d = blockIdx.x * blockDim.x + threadIdx.x;
  if (d >= P.N) return;
  double Fb[D];
  force_bar<D>(P, A, d, Fb);
  float f[D];
  for (int c = 0; c < D; ++c) f[c] = (float)Fb[c];
  stfv<D>(A.fbf_o, d, f);
}

// per-grain sums of the per-node parameter cotangents, one block per grain, fixed order
__global__ void __launch_bounds__(256) k_grad_reduce(const Dev P, const double* pacc, double* grad) {
  __shared__ double sm[NPARAM][256];
  const uint32_t g = blockIdx.x;
  const GrainDev& gr = P.grain[g];
  double s[NPARAM] = {0.0, 0.0, 0.0, 0.0};
  for (uint32_t o = gr.node_begin + threadIdx.x; o < gr.node_end; o += blockDim.x) {  // input order
    const uint32_t i = at_of(P, o);
    for (int k = 0; k < NPARAM; ++k) s[k] += pacc[(size_t)i * NPARAM + k];
  }
  for (int k = 0; k < NPARAM; ++k) sm[k][threadIdx.x] = s[k];
  __syncthreads();
  for (uint32_t w = blockDim.x / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w)
      for (int k = 0; k < NPARAM; ++k) sm[k][threadIdx.x] += sm[k][threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x < NPARAM) grad[(size_t)g * NPARAM + threadIdx.x] = sm[threadIdx.x][0];
}

void launch_adjoint_step(const Dev& P, const AdjStep& A, cudaStream_t s, uint64_t* launches) {
  // programmatic dependent launch: each kernel waits on its predecessor in pdl_enter()
  const dim3 g(2 * P.n_chunks), b(32 * SUB);
  if (P.dim == 2) {
    launch_k(A.fbf ? k_adj_step<2, true> : k_adj_step<2, false>, g, b, 0, s, true, P, A);
  } else {
    launch_k(A.fbf ? k_adj_step<3, true> : k_adj_step<3, false>, g, b, 0, s, true, P, A);
  }
  *launches += 1;
}

void launch_fb_init(const Dev& P, const AdjStep& A, cudaStream_t s, uint64_t* launches) {
  const uint32_t nb = (P.N + 127) / 128;
  if (P.dim == 2) {
    launch_k(k_fb_init<2>, nb, 128, 0, s, true, P, A);
  } else {
    launch_k(k_fb_init<3>, nb, 128, 0, s, true, P, A);
  }
  *launches += 1;
}

void launch_grad_reduce(const Dev& P, const double* pacc, double* grad, cudaStream_t s, uint64_t* launches) {
  if (P.G == 0) return;
  k_grad_reduce<<<P.G, 256, 0, s>>>(P, pacc, grad);
  *launches += 1;
}

}  // namespace pg
