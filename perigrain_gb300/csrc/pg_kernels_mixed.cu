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
#include "pg_sqrt_float.cuh"

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

// |v|^2 in FP64, fused, with the products' order written out so that every variant of the force kernel
// takes the same contact decisions to the last bit.
template <int D>
__device__ __forceinline__ double sum_sq64(const double (&v)[D]) {
  double s = fma(v[0], v[0], __dmul_rn(v[1], v[1]));
  if constexpr (D == 3) s = fma(v[2], v[2], s);
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
__device__ __forceinline__ float bond_term(const float (&dh)[D], const float (&dl)[D], const float (&xh)[D],
                                          const float (&xl)[D], const float (&jdh)[D], const float (&jdl)[D],
                                          const float (&jxh)[D], const float (&jxl)[D], float cv, bool use,
                                          float (&y)[D], float* str_out) {
  float xi[D], et[D];
  for (int c = 0; c < D; ++c) {
    xi[c] = (jxh[c] - xh[c]) + (jxl[c] - xl[c]);
    et[c] = (jdh[c] - dh[c]) + (jdl[c] - dl[c]);
    y[c] = xi[c] + et[c];
  }
  const float xx = dotf<D>(xi, xi), yy = dotf<D>(y, y);
  const float ixn = rsqrtf(xx), iyn = rsqrtf(yy);
  const float num = fmaf(2.f, dotf<D>(xi, et), dotf<D>(et, et));
  const float str = __fdividef(num * ixn, fmaf(yy, iyn, xx * ixn));
  *str_out = str;
  return use ? cv * str * iyn : 0.f;
}

// What a contact reads of its partner q; loaded before anything is known of it, so that one latency
// is waited for instead of one a test.
template <int D>
struct Partner {
  double x[D], v[D];
  float vol;
  __device__ __forceinline__ Partner(const Dev& P, uint32_t q) {
    ldv<D>(P.cur, q, x);
    ldv<D>(P.vel_in, q, v);
    vol = P.vol_f[q];
  }
  // The same for a team, whose tests follow one another on an idle SM: volatile loads stay where they
  // are written (the compiler moves plain ones behind the tests that precede their use), so that all
  // are in flight at once. gq: the partner's grain.
  __device__ __forceinline__ Partner(const Dev& P, uint32_t q, uint32_t& gq, float (&qf)[D]) {
    gq = *(const volatile uint32_t*)(P.node_grain + q);
    constexpr uint32_t SF = D == 2 ? 2 : 4, S = D == 2 ? 2 : 4;
    if constexpr (D == 2)
      asm volatile("ld.volatile.global.v2.f32 {%0, %1}, [%2];" : "=f"(qf[0]), "=f"(qf[1]) : "l"(P.curf + (size_t)q * SF));
    else
      for (int c = 0; c < D; ++c) qf[c] = *(const volatile float*)(P.curf + (size_t)q * SF + c);
    const double *px = P.cur + (size_t)q * S, *pv = P.vel_in + (size_t)q * S;
    asm volatile("ld.volatile.global.v2.f64 {%0, %1}, [%2];" : "=d"(x[0]), "=d"(x[1]) : "l"(px));
    if constexpr (D == 3) x[2] = *(const volatile double*)(px + 2);
    asm volatile("ld.volatile.global.v2.f64 {%0, %1}, [%2];" : "=d"(v[0]), "=d"(v[1]) : "l"(pv));
    if constexpr (D == 3) v[2] = *(const volatile double*)(pv + 2);
    vol = *(const volatile float*)(P.vol_f + q);
  }
};

// What a contact needs of the node itself: its state, its row of the bond slab and the contact
// parameters of its grain and instance in FP32.
template <int D>
struct Side {
  double x[D], v[D], rad, s_max;
  float Kn, zeta, mu, rho, Rc, pre2, pf[D];
  uint32_t g, deg, w0, slot0, lane;
  uint32_t rules;  // SIDE_*
  __device__ __forceinline__ void of(const Dev& P, const InstDev& in, const GrainDev& gr) {
    rad = in.contact_rad;
    s_max = in.contact_s_max;
    Kn = (float)in.normal_stiffness;
    zeta = (float)in.damping_ratio;
    mu = (float)in.friction_coefficient;
    rho = (float)gr.rho;
    Rc = (float)in.contact_rad;
  }
};

// Node q's contact with node d (s): false if there is none, else what the force receives, to be added in this order:
// s1 u, sd u where damp, sf tg where fr. None of it depends on the force so far, so a team of warps
// can form it for all contacts of a chunk at once.
template <int D>
struct ContactTerm {
  float s1, sd, sf, u[D], tg[D];
  float far;       // the largest component of x_q - x_p
  uint32_t close;  // the two nodes are at the same place
  uint32_t fr;     // FR_* of the friction branch taken, 0: none
};
template <int D, bool GC>
__device__ __forceinline__ bool contact_term(const Dev& P, const Side<D>& s, uint32_t gqi, uint32_t d, uint32_t q,
                                             const Partner<D>& pq, ContactTerm<D>& o) {
  const bool same = gqi == s.g;
  // The contact decision |x_q - x_p| <= R_c' is made in FP64 (the squares summed with fused products):
  // contact damping switches on at full strength at that boundary, so a decision flipped by
  // FP32 rounding would kick a node by metres per second.
  double dir64[D];
  for (int c = 0; c < D; ++c) dir64[c] = pq.x[c] - s.x[c];
  const double n2 = sum_sq64<D>(dir64);
  // |x_q - x_p| <= contact_rad as n2 <= contact_s_max, the same outcome without the square root
  if (!(n2 <= s.s_max)) return false;
  float Kn = s.Kn, zeta = s.zeta, mu = s.mu;
  if constexpr (GC) {
    const GrainDev &gr = P.grain[s.g], &gq = P.grain[gqi];
    Kn = (float)((gr.kn + gq.kn) * 0.5);
    zeta = (float)((gr.zeta + gq.zeta) * 0.5);
    mu = (float)((gr.mu + gq.mu) * 0.5);
  }
  float Rc = s.Rc;
  if (same) {
    double pp[D], ps[D], r[D];
    ldv<D>(P.pos, d, pp);
    ldv<D>(P.pos, q, ps);
    for (int c = 0; c < D; ++c) r[c] = pp[c] - ps[c];
    const double r2 = sum_sq64<D>(r);
    // |x_q - x_p| <= R_c' = min(ref, contact_rad), ref = sqrt(r2): the roots compare as n2 and r2 do
    // unless these are within a few units in the last place (1 + 2^-50: roots two such units apart)
    if (n2 > r2 * 1.0000000000000009) return false;
    bool bonded = false;
    for (uint32_t k = 0; k < s.deg && !bonded; k += 8)  // eight at a time: independent loads
#pragma unroll
      for (uint32_t j = 0; j < 8; ++j) {
        const uint32_t kk = min(k + j, s.deg - 1);
        bonded |= ((P.alive[s.w0 + kk] >> s.lane) & 1u) && P.bcol[s.slot0 + 32u * kk] == q;
      }
    if (bonded) return false;
    const double ref = sqrt(r2);
    const double Rc64 = ref < s.rad ? ref : s.rad;
    if (!(n2 <= r2) && !(sqrt(n2) <= Rc64)) return false;
    Kn = (float)(P.grain[s.g].cnot / Rc64);
    Rc = (float)Rc64;
  }
  const float dn = sqrt_to_float(n2);
  float dir[D];
  for (int c = 0; c < D; ++c) dir[c] = (float)dir64[c];
  o.far = 0.f;
  for (int c = 0; c < D; ++c) o.far = fmaxf(o.far, fabsf(dir[c]));
  o.close = dn == 0.f;
  const float inv = 1.f / dn;
  float(&u)[D] = o.u;
  for (int c = 0; c < D; ++c) u[c] = dir[c] * inv;
  const float nvol = pq.vol;
  const float s1 = -Kn * (Rc - dn) * nvol;
  o.s1 = s1;
  const float cfn = fabsf(s1);
  const float rho = s.rho, dtf = (float)P.dt;
  o.sd = o.sf = 0.f;
  for (int c = 0; c < D; ++c) o.tg[c] = 0.f;
  uint32_t fr = 0;
  if (P.allow_damping || P.allow_friction) {
    float rv[D];
    for (int c = 0; c < D; ++c) rv[c] = (float)(s.v[c] - pq.v[c]);
    const float rvp = dotf<D>(rv, u);
    if (P.allow_damping) {
      const float dc = 2.f * zeta * sqrtf(Kn * rho) * sqrtf(nvol);
      o.sd = -dc * rvp;
    }
    if (P.allow_friction) {
      float(&tg)[D] = o.tg;
      for (int c = 0; c < D; ++c) tg[c] = fmaf(-rvp, u[c], rv[c]);
      const float tn = sqrtf(dotf<D>(tg, tg));
      if (tn > 0.f) {
        float sfr = -mu * cfn;
        fr = (D == 2 && (tg[1] * u[0] - tg[0] * u[1]) < 0.f) ? FR_SLIDE_NEG : FR_SLIDE;
        if (tn < mu * cfn * dtf / rho) {
          sfr = -tn / rho / dtf;
          fr = FR_STICK;
        }
        o.sf = sfr / tn;
      }
    }
  }
  o.fr = fr;
  return true;
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
// ---------------------------------------------------------------------------------------------
// Teams: a chunk worked on by a block of four warps, where the chunks alone leave the GPU nearly idle
// and a step's time is one warp's chain (force_team()). Each warp forms a quarter of the bond terms
// and warp 0 adds them in the order of the bonds; the entries of the candidate lists are tasks for
// all threads, and warp 0 adds the contacts in the order of the lists: the force is the same to the
// bit. Bound by latency: an FP64 operation takes 63 cycles, a load that misses L1 250 to 500. Cycles
// of a chunk with contacts, two disks, a warp / a team: bonds 7200 / 2800, contacts 8000-10900 /
// 3300, the rest (start, walls, position update) 5200 / 4700.
constexpr uint32_t TEAM_WARPS = 4;
constexpr uint32_t TEAM_BONDS = 32;  // bonds between two barriers

// The contacts a node may have; whether its list can overflow max_cand; whether its coordinates are
// below 1e9 contact radii.
constexpr uint32_t SIDE_SELF = 1u, SIDE_OTHER = 2u, SIDE_COUNT = 4u, SIDE_NEAR = 8u;

template <int D, bool ON>
struct TeamMem {
  float sc[2][TEAM_BONDS][32], y[2][TEAM_BONDS][D][32];
  uint32_t what[32 * TEAM_WARPS], node[32 * TEAM_WARPS];
  ContactTerm<D> term[32 * TEAM_WARPS];
  Side<D> side[32];
  __device__ __forceinline__ void put(uint32_t k, uint32_t lane, float s, const float (&v)[D]) {
    const uint32_t b = k / TEAM_BONDS % 2, i = k % TEAM_BONDS;
    sc[b][i][lane] = s;
    for (int c = 0; c < D; ++c) y[b][i][c][lane] = v[c];
  }
};
template <int D>
struct TeamMem<D, false> {};

// All warps have put the bonds [k0, k1), at most TEAM_BONDS, into their buffer; warp 0 adds them. The
// other buffer may be filled meanwhile: this one is not written again before the next barrier.
template <int D>
__device__ __forceinline__ void team_add(TeamMem<D, true>& tm, uint32_t k0, uint32_t k1, uint32_t lane, uint32_t sub,
                                         float (&f)[D]) {
  __syncthreads();
  if (sub != 0) return;
  const uint32_t b = k0 / TEAM_BONDS % 2;
#pragma unroll 8
  for (uint32_t i = 0; i < k1 - k0; ++i)
    for (int c = 0; c < D; ++c) f[c] = fmaf(tm.sc[b][i][lane], tm.y[b][i][c][lane], f[c]);
}

// A team's bonds: of each TEAM_BONDS the warp forms eight in a row, their indices and (GB at a time)
// their neighbours loaded before any is used, so a warp waits for two latencies, not two a pair.
template <int D>
__device__ __forceinline__ void team_bonds(const Dev& P, TeamMem<D, true>& tm, uint32_t d, uint32_t lane, uint32_t sub,
                                           uint32_t cdeg, uint32_t w0, uint32_t slot0, bool mov, const float (&dh)[D],
                                           const float (&dl)[D], const float (&xh)[D], const float (&xl)[D], float cnot,
                                           float snot, uint32_t t, float (&f)[D]) {
  constexpr uint32_t W = TEAM_BONDS / TEAM_WARPS, GB = D == 2 ? 8 : 4;
  const uint32_t full = (cdeg + 1) & ~1u;  // a row without a last bond ends on an unused one, as in the pairs of a lone warp
  for (uint32_t kb = 0; kb < cdeg; kb += TEAM_BONDS) {
    const uint32_t k0 = kb + W * sub;
    uint32_t word[W], col[W];
#pragma unroll
    for (uint32_t i = 0; i < W; ++i) {
      word[i] = 0u;
      col[i] = d;
      if (k0 + i < cdeg) {
        word[i] = P.alive[w0 + k0 + i];
        col[i] = P.bcol[slot0 + 32u * (k0 + i)];
      }
    }
#pragma unroll
    for (uint32_t h = 0; h < W; h += GB) {
      if (k0 + h >= full) continue;
      float jdh[GB][D], jdl[GB][D], jxh[GB][D], jxl[GB][D], vol[GB];
#pragma unroll
      for (uint32_t i = 0; i < GB; ++i) {
        const uint32_t j = mov && ((word[h + i] >> lane) & 1u) ? col[h + i] : d;
        ld_hl<D>(P.dref, P.np, j, jdh[i], jdl[i]);
        ld_hl<D>(P.xref, P.np, j, jxh[i], jxl[i]);
        vol[i] = P.vol_f[j];
      }
      uint32_t broken = 0;
      float s[GB], y[GB][D];
#pragma unroll
      for (uint32_t i = 0; i < GB; ++i) {
        const bool use = mov && ((word[h + i] >> lane) & 1u);
        float str;
        s[i] = bond_term<D>(dh, dl, xh, xl, jdh[i], jdl[i], jxh[i], jxl[i], cnot * vol[i], use, y[i], &str);
        broken |= (uint32_t)(use && str > snot) << i;
      }
#pragma unroll
      for (uint32_t i = 0; i < GB; ++i) tm.put(k0 + h + i, lane, s[i], y[i]);
      if (!__any_sync(0xffffffffu, broken)) continue;
#pragma unroll
      for (uint32_t i = 0; i < GB; ++i) {
        const uint32_t k = k0 + h + i;
        if (broken >> i & 1u) P.break_step[slot0 + 32u * k] = t;
        const uint32_t now = word[h + i] & ~__ballot_sync(0xffffffffu, broken >> i & 1u);
        if (lane == 0 && now != word[h + i]) P.alive[w0 + k] = now;
      }
    }
    team_add<D>(tm, kb, min(kb + TEAM_BONDS, full), lane, sub, f);
  }
  if (!cdeg) __syncthreads();  // the Side records
}

// Entry q of node p's list: 0 = not within the prefilter or the rules, 1 = passed, 2 = a contact (o).
// The box test of the grains is left out where it cannot matter: a contact well within the radius
// lies in both boxes (0.999998 leaves room for the test's two roundings, SIDE_NEAR), and an entry without contact only counts where the list could overflow.
template <int D, bool GC>
__device__ __forceinline__ uint32_t team_contact(const Dev& P, const Side<D>& s, uint32_t p, uint32_t q,
                                                 ContactTerm<D>& o) {
  float qf[D];
  uint32_t gq;
  const Partner<D> pq(P, q, gq, qf);
  float d2 = 0.f;
  for (int c = 0; c < D; ++c) {
    float dd = qf[c] - s.pf[c];
    d2 = fmaf(dd, dd, d2);
  }
  if (d2 > s.pre2) return 0;
  const bool same = gq == s.g;
  if (!(s.rules & (same ? SIDE_SELF : SIDE_OTHER))) return 0;
  if (P.nl_bdry_only && P.bdry_rank[q] == NONE) return 0;
  const bool hit = contact_term<D, GC>(P, s, gq, p, q, pq, o);
  if (same) return hit ? 2 : 1;
  const bool sure = hit ? (s.rules & SIDE_NEAR) && o.far < 0.999998f * s.Rc : !(s.rules & SIDE_COUNT);
  if (!sure) {
    double bmn[D], bmx[D], qmn[D], qmx[D];
    grain_box<D>(P, s.g, bmn, bmx);
    grain_box<D>(P, gq, qmn, qmx);
    if (!boxes_touch<D>(bmn, bmx, qmn, qmx, s.rad)) return 0;
  }
  return hit ? 2 : 1;
}

template <int D, bool REC, bool GC, bool PERM, bool LIST, int BPS, bool TEAM>
__global__ void __launch_bounds__(128, BPS) k_force_mx(const Dev P) {
  static_assert(LIST || !TEAM, "a team works on candidate lists");
  pdl_enter();
  pdl_release();
  // a warp a chunk, or (TEAM) a block of four warps, of which warp 0 holds the force and ends the step
  const uint32_t lane = threadIdx.x & 31, sub = TEAM ? threadIdx.x >> 5 : 0u;
  const uint32_t d = TEAM ? blockIdx.x * 32 + lane : blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t chunk = d >> 5;
  if (chunk >= P.n_chunks) return;
  __shared__ TeamMem<D, TEAM> tm;
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
  // (a team's warp 0 has registers to spare and loads the position update's inputs here as well)
  double dp[D], ps[D];
  float db[D];
  if constexpr (TEAM) {
    if (act && sub == 0 && P.fuse) {
      ldv<D>(P.disp, d, dp);
      ldv<D>(P.pos, d, ps);
      ldf<D>(P.disp_b, d, db);
    }
  }
  constexpr int DE = (D == 2) ? D : 1;
  float ef_in[DE], ao_in[DE];
  bool clamped_in = false;
  if constexpr (D == 2) {
    if (mov && sub == 0) {
      ldvf<D>(P.extf_f, d, ef_in);
      ldvf<D>(P.acc_f, d, ao_in);
      clamped_in = P.clamped[d] != 0;
    }
  }

  const InstDev& in = P.inst[gr.inst];
  // which contacts the node may have; a team looks before its bonds, a lone warp after them (its
  // registers are full until then: 1.5 % of a step of the collision ensemble)
  bool p_bdry, selfc, other;
  uint32_t ncl;
  auto rules = [&] {
    p_bdry = !P.nl_bdry_only || (act && P.bdry_rank[d] != NONE);
    selfc = mov && P.enable_fracture && (gr.flags & GF_BREAKABLE) && P.self_contact;
    other = mov && (P.worm || (gr.flags & GF_STOPPABLE));
    // with candidate lists a node whose list is empty has no contact this step
    ncl = (LIST && act) ? (uint32_t)P.cand_n[d] : 0u;
  };
  if constexpr (TEAM) rules();
  // a team's last warp notes each node's side of its contacts; its loads overlap the others' bonds
  [[maybe_unused]] auto team_side = [&] {
    if constexpr (TEAM) {
      if (sub != TEAM_WARPS - 1 || !act) return;
      Side<D>& s = tm.side[lane];
      s.of(P, in, gr);
      ldv<D>(P.cur, d, s.x);
      for (int c = 0; c < D; ++c) s.v[c] = vpd[c];
      ldf<D>(P.curf, d, s.pf);
      s.pre2 = in.pre_f * in.pre_f;
      s.g = g;
      s.deg = P.node_deg[d];
      s.w0 = P.chunk_word[chunk];
      s.slot0 = P.chunk_slot[chunk] + lane;
      s.lane = lane;
      s.rules = (selfc ? SIDE_SELF : 0u) | (other ? SIDE_OTHER : 0u) | (ncl > P.max_cand ? SIDE_COUNT : 0u) | SIDE_NEAR;
      for (int c = 0; c < D; ++c)
        if (!(fabs(s.x[c]) < 1e9 * s.rad)) s.rules &= ~SIDE_NEAR;
    }
  };

  // a team's contacts: every list entry of the chunk is a task, the entries of the 32 lists, end to
  // end, over the block's threads; a thread's first entry q (of lane pl's list) is loaded ahead
  uint32_t total = 0, incl = 0, first = 0, pl = 0, q = 0;
  auto entry = [&](uint32_t e) {
    pl = 0;  // as many lanes' lists end at or before e
#pragma unroll
    for (uint32_t s = 16; s; s >>= 1)
      if (__shfl_sync(0xffffffffu, incl, pl + s - 1) <= e) pl += s;
    const uint32_t at = e - __shfl_sync(0xffffffffu, first, pl);
    if (e < total) q = P.cand_q[((size_t)chunk * P.cand_cap + at) * 32 + pl];
  };
  if constexpr (TEAM) {
    const uint32_t n = (selfc || other) && p_bdry ? ncl : 0u;
    if (__any_sync(0xffffffffu, n)) {
      incl = n;
#pragma unroll
      for (int s = 1; s < 32; s <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, incl, s);
        if (lane >= (uint32_t)s) incl += v;
      }
      first = incl - n;
      total = __shfl_sync(0xffffffffu, incl, 31);
      entry(threadIdx.x);
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
    // (loaded for lanes without bonds in use too: those add 0 times a vector, which must be finite)
    float dh[D], dl[D], xh[D], xl[D];
    ld_hl<D>(P.dref, P.np, d, dh, dl);
    ld_hl<D>(P.xref, P.np, d, xh, xl);
    if constexpr (REC) {
      if (mov && sub == 0 && P.rec_df) st_hl<D>(P.rec_df, P.np, d, dh, dl);
    }
    if constexpr (TEAM) {
      team_side();
      team_bonds<D>(P, tm, d, lane, sub, cdeg, w0, slot0, mov, dh, dl, xh, xl, cnot, snot, t, f);
    } else {
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
      float stra, strb, ya[D], yb[D];
      const float fa = bond_term<D>(dh, dl, xh, xl, adh, adl, axh, axl, cnot * va, ua, ya, &stra);
      const float fb = bond_term<D>(dh, dl, xh, xl, bdh, bdl, bxh, bxl, cnot * vb, ub, yb, &strb);
      for (int c = 0; c < D; ++c) f[c] = fmaf(fb, yb[c], fmaf(fa, ya[c], f[c]));
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
  }
  __syncwarp();

  unsigned long long my_pairs = 0, my_hash = 0, my_close = 0;
  uint32_t rent[REC ? MAX_CAND : 1];  // recorded contact entries of this node (REC only)
  uint32_t nrec = 0, wbits = 0;
  if constexpr (!TEAM) rules();
  // the contact of node q (o) as it acts on the force
  auto apply = [&](uint32_t q, const ContactTerm<D>& o) {
    if (P.record_pairs) {  // the pair log hashes input indices
      my_pairs += 1;
      my_hash += splitmix64(((unsigned long long)input_index<PERM>(P, d) << 32) | input_index<PERM>(P, q));
    }
    if (o.close) my_close += 1;
    for (int c = 0; c < D; ++c) f[c] = fmaf(o.s1, o.u[c], f[c]);
    if (P.allow_damping)
      for (int c = 0; c < D; ++c) f[c] = fmaf(o.sd, o.u[c], f[c]);
    if (o.fr)
      for (int c = 0; c < D; ++c) f[c] = fmaf(o.sf, o.tg[c], f[c]);
    if constexpr (REC) rent[nrec++] = q | (o.fr << 30);
  };
  if constexpr (TEAM) {
    uint32_t passed = 0;
    bool over = false;
    for (uint32_t e0 = 0; e0 < total; e0 += 32 * TEAM_WARPS) {
      if (e0) entry(e0 + threadIdx.x);
      if (e0 + threadIdx.x < total) {
        tm.what[threadIdx.x] = team_contact<D, GC>(P, tm.side[pl], chunk * 32 + pl, q, tm.term[threadIdx.x]);
        tm.node[threadIdx.x] = q;
      }
      __syncthreads();
      if (sub == 0) {
        const uint32_t b = max(first, e0), e1 = min(incl, e0 + 32 * TEAM_WARPS);
        for (uint32_t x = b; x < e1; ++x) {
          const uint32_t w = tm.what[x - e0];
          if (w == 0 || over) continue;
          if (passed++ >= P.max_cand) {
            set_status(P.status, PG_ECAPACITY);
            over = true;
          } else if (w == 2) {
            apply(tm.node[x - e0], tm.term[x - e0]);
          }
        }
      }
      __syncthreads();
    }
    if (sub != 0) return;
  } else if ((selfc || other) && p_bdry && (!LIST || ncl > 0)) {
    double bmn[D], bmx[D];
    grain_box<D>(P, g, bmn, bmx);
    float ph[D];
    ldf<D>(P.curf, d, ph);
    const float thr2 = in.pre_f * in.pre_f;
    // is candidate q beyond the FP32 prefilter; is it within the contact rules and the grain-box test?
    // (the box test of the grain asked about last is kept: a list is sorted by grain)
    uint32_t box_g = NONE;
    bool box_ok = false;
    auto far = [&](const float (&qf)[D]) {
      float d2 = 0.f;
      for (int c = 0; c < D; ++c) {
        float dd = qf[c] - ph[c];
        d2 = fmaf(dd, dd, d2);
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
      for (int c = 0; c < D; ++c) cc[c] = cell_coord(ph[c] + in.frame_off_f[c], in.inv_cell_f, in.dims[c]);
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
    Side<D> s;
    if (nc) {
      s.of(P, in, gr);
      ldv<D>(P.cur, d, s.x);
      for (int c = 0; c < D; ++c) s.v[c] = vpd[c];
      s.g = g;
      s.deg = P.node_deg[d];
      s.w0 = w0;
      s.slot0 = slot0;
      s.lane = lane;
    }
    for (int ci = 0; ci < nc; ++ci) {
      if constexpr (LIST) {
        q = P.cand_q[cbase + (size_t)(__ffs(hits) - 1) * 32];
        hits &= hits - 1;
      } else {
        q = idx[ci];
      }
      const uint32_t gqi = LIST ? P.node_grain[q] : (uint32_t)(keys[ci] >> 32) & 0x7fffffffu;
      ContactTerm<D> o;
      if (!contact_term<D, GC>(P, s, gqi, d, q, Partner<D>(P, q), o)) continue;
      apply(q, o);
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
        // products and sums written out where the compiler may fuse either product or none: it chose
        // differently for the variant of seven blocks an SM, whose wall forces were an ulp off the others'
        const float dd = fabsf(dist), R2 = __fmul_rn(R, R), h2 = fmaf(-dd, dd, R2);
        float Area, I;
        if constexpr (D == 2) {
          const float half = __fmul_rn(__fmul_rn(0.5f * (float)M_PI, R), R);
          Area = fmaf(-sqrtf(fmaxf(h2, 0.f)), dd, fmaf(-R2, asinf(dd / R), half));
          I = 0.f;
        } else {
          const float a = R - dd, b = h2;
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
              f[tg] = __fadd_rn(f[tg], ff);
              rec.a_t1 = vol_i * (double)ff;
              rec.has_fric = 1;
            }
          } else {
            const int t1 = (dir + 1) % 3, t2 = (dir + 2) % 3;
            const float vn = sqrtf(fmaf(rv[t1], rv[t1], __fmul_rn(rv[t2], rv[t2])));
            if (vn > 0.f) {
              const float u1 = rv[t1] / vn, u2 = rv[t2] / vn;
              float sfr = -mu * fabsf(F);
              wbits |= 2u << (4 * k);
              if (vn < mu * fabsf(F) * dtf / rho) {
                sfr = -vn / rho / dtf;
                wbits |= 4u << (4 * k);
              }
              f[t1] = __fadd_rn(f[t1], __fmul_rn(sfr, u1));
              f[t2] = __fadd_rn(f[t2], __fmul_rn(sfr, u2));
              rec.a_t1 = vol_i * (double)(sfr * u1);
              rec.a_t2 = vol_i * (double)(sfr * u2);
              rec.has_fric = 1;
            }
          }
        }
        if (P.allow_damping) {
          const float df = -(2.f * zeta * sqrtf(Kn * rho) * sqrtf(fabsf(Area))) * rv[dir];
          f[dir] = __fadd_rn(f[dir], df);
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
  double cu[D];
  for (int c = 0; c < D; ++c) cu[c] = 0.0;
  if (act) {
    if (!TEAM && P.fuse) ldv<D>(P.disp, d, dp);
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
        a[c] = __fmul_rn(orho, f[c]);
        v[c] = vpd[c] + widen(__fmul_rn(__fadd_rn(ao[c], a[c]), hdt));  // FP64 accumulation of an FP32 increment
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
      if constexpr (!TEAM) {
        ldv<D>(P.pos, d, ps);
        ldf<D>(P.disp_b, d, db);
      }
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
// in only where used, so the plain kernel keeps its register budget; the plain kernel with lists also
// for BPS = 5, 6 or 7 blocks of 128 threads per SM (96, 80 or 72 registers), without lists for 5 or 6, see
// force_bps(), and each with lists also for teams of warps (TEAM).
template <int D>
static const void* force_mx_ptr(bool rec, bool gc, bool perm, bool list, int bps, bool team) {
#define PG_F(r, g, p, l, b) (const void*)k_force_mx<D, r, g, p, l, b, false>
#define PG_T(r, g, p) (const void*)k_force_mx<D, r, g, p, true, 4, true>
  static const void* const teams[8] = {PG_T(0, 0, 0), PG_T(0, 0, 1), PG_T(0, 1, 0), PG_T(0, 1, 1),
                                       PG_T(1, 0, 0), PG_T(1, 0, 1), PG_T(1, 1, 0), PG_T(1, 1, 1)};
  if (team) return teams[(rec ? 4 : 0) + (gc ? 2 : 0) + (perm ? 1 : 0)];
#undef PG_T
  static const void* const plain[2][3] = {{PG_F(0, 0, 0, 1, 5), PG_F(0, 0, 0, 1, 6), PG_F(0, 0, 0, 1, 7)},
                                          {PG_F(0, 0, 1, 1, 5), PG_F(0, 0, 1, 1, 6), PG_F(0, 0, 1, 1, 7)}};
  static const void* const search[2] = {PG_F(0, 0, 0, 0, 6), PG_F(0, 0, 1, 0, 6)};
  static const void* const others[14] = {
      PG_F(0, 0, 0, 0, 5), PG_F(0, 0, 1, 0, 5), PG_F(0, 1, 0, 0, 5), PG_F(0, 1, 0, 1, 5), PG_F(0, 1, 1, 0, 5),
      PG_F(0, 1, 1, 1, 5), PG_F(1, 0, 0, 0, 5), PG_F(1, 0, 0, 1, 5), PG_F(1, 0, 1, 0, 5), PG_F(1, 0, 1, 1, 5),
      PG_F(1, 1, 0, 0, 5), PG_F(1, 1, 0, 1, 5), PG_F(1, 1, 1, 0, 5), PG_F(1, 1, 1, 1, 5)};
#undef PG_F
  if (!rec && !gc && list) return plain[perm ? 1 : 0][bps - 5];
  if (!rec && !gc) return bps > 5 ? search[perm ? 1 : 0] : others[perm ? 1 : 0];
  return others[2 + (rec ? (gc ? 8 : 4) : 0) + (perm ? 2 : 0) + (list ? 1 : 0)];
}
template <int D>
static void launch_force_mx(const Dev& P, uint32_t block, cudaStream_t s, bool pdl, bool rec) {
  using K = void (*)(const Dev);
  const bool team = force_team(P, block);
  launch_k((K)force_mx_ptr<D>(rec, P.grain_contact, P.node_orig, P.cand_q, force_bps(P.n_chunks, P.n_sms), team),
           team ? P.n_chunks : cdiv(P.n_chunks * 32, block), block, 0, s, pdl, P);
}

cudaError_t kernels_mixed_init() {
  cudaError_t e = cudaFuncSetAttribute(k_finalize<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, FINAL_SMEM);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_finalize<3>, cudaFuncAttributeMaxDynamicSharedMemorySize, FINAL_SMEM);
  if (e != cudaSuccess) return e;
  // the recording variants of the force kernel have local frames of about 1.1 KB
  const void* fs[2 * 48 + 2 * 8];
  int n = 0;
  for (int k = 0; k < 16; ++k)
    for (int b = 5; b <= 7; ++b) {
      fs[n++] = force_mx_ptr<2>(k & 8, k & 4, k & 2, k & 1, b, false);
      fs[n++] = force_mx_ptr<3>(k & 8, k & 4, k & 2, k & 1, b, false);
    }
  for (int k = 0; k < 8; ++k) {
    fs[n++] = force_mx_ptr<2>(k & 4, k & 2, k & 1, true, 5, true);
    fs[n++] = force_mx_ptr<3>(k & 4, k & 2, k & 1, true, 5, true);
  }
  size_t need = 0;
  static std::atomic<size_t> known{0};
  e = max_local_bytes(fs, n, &known, &need);
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
  launch_force_mx<D>(P, L.force_block, s, pdl, rec);
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
