// Incircle packing of a simplex mesh on the GPU (C ABI pg_pack_incenters of include/perigrain.h):
// the reference's get_incenter_mesh_loc (exp_dict.py:1072-1313) from the mesh its mesher returns.
//
//   element pass  incenter and inradius of every triangle (exp_dict.py:1087-1125: side lengths,
//                 length-weighted vertex mean, Heron's area, r = 2A / perimeter) or tetrahedron
//                 (:1127-1172: |det| / 6 volume, face-area weighted vertex mean, r = 6V / sum of
//                 doubled face areas), the same IEEE operations in the same order (this file is
//                 compiled with --fmad=false), so the element circles are bit-identical to numpy's.
//   adjacency     the elements of every node (get_nbd_vertex_elem, exp_dict.py:71-86) by a counting
//                 sort: per-node counts, exclusive scan, fill.
//   nodal pass    one circle per mesh node, appended after the element circles in node order:
//       plain     (:1280-1296, modify_nodal_circles = False) interior nodes only; centre = node,
//                 radius = min over its elements of |incenter - node| - inradius.
//       maximin   (:1186-1278, modify_nodal_circles = True, 2D) the problem the reference hands to
//                 GEKKO per interior node (and per boundary node with gen_bdry): maximise Z subject to
//                 Z <= |x - c_k| - r_k for the node's element circles, Z <= distance from x to the
//                 line of each boundary edge holding the node (boundary nodes), x in the bounding box
//                 of the circle centres (plus the node, for boundary nodes), started from the node
//                 (interior) or the mean of the centres and the node (boundary). Solved per node by an
//                 ascent from that initial guess to its local maximum (steepest ascent of the
//                 minimum over the eps-active constraints) followed by an exact solve of the three
//                 constraints tight there (two linear equations and one quadratic).
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <string>

#include "../../include/perigrain.h"
#include "pg_bonds.h"
#include "pg_ieee64.cuh"

namespace pg {

namespace {

constexpr int PT = 128;       // threads per block
constexpr int PK_MAX = 16;    // element circles around one node in the maximin pass
constexpr int PL_MAX = 4;     // boundary-edge lines through one node
constexpr int PS_MAX = 12;    // constraints tight at the ascent's end considered by the exact solve

// error codes raised by the kernels (first one wins)
constexpr int32_t PE_INDEX = 1;     // element vertex or boundary index out of range
constexpr int32_t PE_ISOLATED = 2;  // a node that needs a circle belongs to no element
constexpr int32_t PE_CIRCLES = 3;   // more than PK_MAX elements around a node (maximin)
constexpr int32_t PE_LINES = 4;     // more than PL_MAX boundary edges through a node

__device__ __forceinline__ void set_err(int32_t* err, int32_t code) { atomicCAS(err, 0, code); }

// ---------------------------------------------------------------------------------------------
// element circles
// ---------------------------------------------------------------------------------------------
__global__ void k_pack_tri(const double* pos, const uint32_t* T, uint32_t ne, uint32_t nn, double* cen, double* rad,
                           uint32_t* cnt, int32_t* err) {
  const uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= ne) return;
  const uint32_t ia = T[3 * (size_t)e], ib = T[3 * (size_t)e + 1], ic = T[3 * (size_t)e + 2];
  if (ia >= nn || ib >= nn || ic >= nn) {
    set_err(err, PE_INDEX);
    return;
  }
  atomicAdd(&cnt[ia], 1u);
  atomicAdd(&cnt[ib], 1u);
  atomicAdd(&cnt[ic], 1u);
  const double ax = pos[2 * (size_t)ia], ay = pos[2 * (size_t)ia + 1];
  const double bx = pos[2 * (size_t)ib], by = pos[2 * (size_t)ib + 1];
  const double cx = pos[2 * (size_t)ic], cy = pos[2 * (size_t)ic + 1];
  const double abx = bx - ax, aby = by - ay;
  const double acx = cx - ax, acy = cy - ay;
  const double bcx = cx - bx, bcy = cy - by;
  // roots and quotients on the integer pipe, the same bits (800 x 500 cells: 143 -> 63 us)
  const double la = ieee64::sqrt_rn(bcx * bcx + bcy * bcy);  // side opposite a
  const double lb = ieee64::sqrt_rn(acx * acx + acy * acy);
  const double lc = ieee64::sqrt_rn(abx * abx + aby * aby);
  const double sl = la + lb + lc;
  const ieee64::Divisor dsl = ieee64::make_divisor(sl);
  cen[2 * (size_t)e] = ieee64::div_rn(la * ax + lb * bx + lc * cx, dsl);
  cen[2 * (size_t)e + 1] = ieee64::div_rn(la * ay + lb * by + lc * cy, dsl);
  const double area = 0.25 * ieee64::sqrt_rn(sl * (la - lb + lc) * (lb - lc + la) * (lc - la + lb));
  rad[e] = ieee64::div_rn(2.0 * area, dsl);
}

// doubled area of the face (p, q, s): the norm of the three 2x2 minors, in the order the
// reference writes them
__device__ __forceinline__ double face2(const double* p, const double* q, const double* s) {
  const double A = (p[0] - s[0]) * (p[1] - q[1]) - (p[0] - q[0]) * (p[1] - s[1]);
  const double B = (p[0] - s[0]) * (p[2] - q[2]) - (p[0] - q[0]) * (p[2] - s[2]);
  const double C = (p[1] - s[1]) * (p[2] - q[2]) - (p[1] - q[1]) * (p[2] - s[2]);
  return sqrt(A * A + B * B + C * C);
}

__global__ void k_pack_tet(const double* pos, const uint32_t* T, uint32_t ne, uint32_t nn, double* cen, double* rad,
                           uint32_t* cnt, int32_t* err) {
  const uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= ne) return;
  uint32_t v[4];
  for (int k = 0; k < 4; ++k) {
    v[k] = T[4 * (size_t)e + k];
    if (v[k] >= nn) {
      set_err(err, PE_INDEX);
      return;
    }
  }
  for (int k = 0; k < 4; ++k) atomicAdd(&cnt[v[k]], 1u);
  double p1[3], p2[3], p3[3], p4[3];
  for (int c = 0; c < 3; ++c) {
    p1[c] = pos[3 * (size_t)v[0] + c];
    p2[c] = pos[3 * (size_t)v[1] + c];
    p3[c] = pos[3 * (size_t)v[2] + c];
    p4[c] = pos[3 * (size_t)v[3] + c];
  }
  const double x1 = p1[0], y1 = p1[1], z1 = p1[2], x2 = p2[0], y2 = p2[1], z2 = p2[2];
  const double x3 = p3[0], y3 = p3[1], z3 = p3[2], x4 = p4[0], y4 = p4[1], z4 = p4[2];
  const double det = (x4 - x1) * ((y2 - y1) * (z3 - z1) - (z2 - z1) * (y3 - y1)) +
                     (y4 - y1) * ((z2 - z1) * (x3 - x1) - (x2 - x1) * (z3 - z1)) +
                     (z4 - z1) * ((x2 - x1) * (y3 - y1) - (y2 - y1) * (x3 - x1));
  const double vol = fabs((1.0 / 6.0) * det);
  const double alpha = vol * 6.0;
  const double s123 = face2(p1, p2, p3), s124 = face2(p1, p2, p4), s134 = face2(p1, p3, p4);
  const double s234 = face2(p2, p3, p4);
  const double den = s123 + s124 + s134 + s234;
  for (int c = 0; c < 3; ++c)
    cen[3 * (size_t)e + c] = (s234 * p1[c] + s134 * p2[c] + s124 * p3[c] + s123 * p4[c]) / den;
  rad[e] = alpha / den;
}

// ---------------------------------------------------------------------------------------------
// adjacency and node classes
// ---------------------------------------------------------------------------------------------
__global__ void k_pack_fill(const uint32_t* T, uint32_t ne, uint32_t nv, uint32_t nn, const uint32_t* off,
                            uint32_t* fill, uint32_t* adj) {
  const uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= ne) return;
  // an element with a vertex out of range was not counted (and has raised PE_INDEX)
  for (uint32_t k = 0; k < nv; ++k)
    if (T[(size_t)e * nv + k] >= nn) return;
  for (uint32_t k = 0; k < nv; ++k) {
    const uint32_t v = T[(size_t)e * nv + k];
    adj[off[v] + atomicAdd(&fill[v], 1u)] = e;
  }
}

__global__ void k_pack_bdry(const uint32_t* bn, uint32_t nb, uint32_t nn, uint32_t* mask, int32_t* err) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nb) return;
  if (bn[k] >= nn) {
    set_err(err, PE_INDEX);
    return;
  }
  mask[bn[k]] = 1;
}

__global__ void k_pack_bedges(const uint32_t* be, uint32_t nbe, uint32_t nn, uint32_t* bcnt, uint32_t* bedge,
                              int32_t* err) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nbe) return;
  for (int s = 0; s < 2; ++s) {
    const uint32_t v = be[2 * (size_t)k + s];
    if (v >= nn) {
      set_err(err, PE_INDEX);
      return;
    }
    const uint32_t j = atomicAdd(&bcnt[v], 1u);
    if (j < (uint32_t)PL_MAX) bedge[(size_t)v * PL_MAX + j] = k;
    else set_err(err, PE_LINES);
  }
}

// The maximin pass handles its nodes by classes of how much shared memory their problem takes:
// interior nodes (no lines) with up to 4, 6, 8, 12 and 16 circles, boundary nodes with up to 8 circles
// and 2 lines, all others (those that are refused among them). With one class for all, a mesh whose
// largest node has 9 elements would run six warps an SM instead of 12 to 20.
constexpr int MM_CLASSES = 7;
__device__ __forceinline__ int mm_class(bool bdry, uint32_t nc, uint32_t nl) {
  if (nc == 0 || nc > (uint32_t)PK_MAX) return 6;
  if (bdry) return nc <= 8 && nl <= 2 ? 5 : 6;
  return nc <= 4 ? 0 : nc <= 6 ? 1 : nc <= 8 ? 2 : nc <= 12 ? 3 : 4;
}

// which nodes get a circle: interior nodes, plus boundary nodes when `all_bdry`; with `classes` also
// how many there are of each class
__global__ void k_pack_flags(uint32_t nn, const uint32_t* mask, int all_bdry, const uint32_t* cnt,
                             const uint32_t* bcnt, uint32_t* flag, uint32_t* classes) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool f = i < nn && (!mask[i] || all_bdry);
  if (i < nn) flag[i] = f ? 1u : 0u;
  if (!classes) return;
  const int c = f ? mm_class(mask[i] != 0, cnt[i], bcnt[i]) : -1;
  for (int k = 0; k < MM_CLASSES; ++k) {
    const uint32_t b = __ballot_sync(0xffffffffu, c == k);
    if (b && (threadIdx.x & 31) == 0) atomicAdd(&classes[k], (uint32_t)__popc(b));
  }
}
struct ClassStart {
  uint32_t at[MM_CLASSES];
};
// The nodes of each class, at its start in `list` (in no particular order: a node's circle does not
// depend on the lanes beside it); fill: zeroed cursors.
__global__ void k_pack_classes(uint32_t nn, const uint32_t* mask, const uint32_t* flag, const uint32_t* cnt,
                               const uint32_t* bcnt, ClassStart start, uint32_t* fill, uint32_t* list) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t lane = threadIdx.x & 31;
  const int c = i < nn && flag[i] ? mm_class(mask[i] != 0, cnt[i], bcnt[i]) : -1;
  for (int k = 0; k < MM_CLASSES; ++k) {
    const uint32_t b = __ballot_sync(0xffffffffu, c == k);
    if (!b) continue;
    uint32_t base = 0;
    if (lane == 0) base = atomicAdd(&fill[k], (uint32_t)__popc(b));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (c == k) list[start.at[k] + base + __popc(b & ((1u << lane) - 1u))] = i;
  }
}

// ---------------------------------------------------------------------------------------------
// plain nodal circles
// ---------------------------------------------------------------------------------------------
template <int D>
__global__ void k_pack_plain(const double* pos, uint32_t nn, uint32_t ne, const double* cen, const double* rad,
                             const uint32_t* off, const uint32_t* adj, const uint32_t* flag, const uint32_t* rank,
                             double* ocen, double* orad, int32_t* err) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nn || !flag[i]) return;
  const uint32_t b = off[i], e = off[i + 1];
  if (b == e) {
    set_err(err, PE_ISOLATED);
    return;
  }
  double x[D];
  for (int c = 0; c < D; ++c) x[c] = pos[(size_t)i * D + c];
  double m = 0.0;
  bool nan = false;
  for (uint32_t k = b; k < e; ++k) {
    const uint32_t t = adj[k];
    double s = 0.0;
    for (int c = 0; c < D; ++c) {
      const double d = cen[(size_t)t * D + c] - x[c];
      s = (c == 0) ? d * d : s + d * d;
    }
    const double v = sqrt(s) - rad[t];
    if (v != v) nan = true;
    if (k == b || v < m) m = v;
  }
  const uint32_t o = ne + rank[i];
  for (int c = 0; c < D; ++c) ocen[(size_t)o * D + c] = x[c];
  orad[o] = nan ? (double)NAN : m;
}

// ---------------------------------------------------------------------------------------------
// maximin nodal circles (2D)
// ---------------------------------------------------------------------------------------------
// One thread per node, MM_T threads per block. A thread's problem -- its circles, lines, constraint
// values and the gradients of the ascent -- lives in its own column of the block's shared memory, so
// the kernel keeps almost nothing in local memory. Coordinates are shifted to the initial guess and
// scaled by the box extent L, so the solve works on numbers of order one. PK, PL: the most
// circles and lines of a node the launch provides for (rows of shared memory).
constexpr int MM_T = 32;
// Nodes a warp takes on: 32, or 12 for meshes of up to MM_FEW nodes, whose warps do not fill the GPU:
// their rounds are shorter. ms a call at 12 / 32 nodes a warp: 20 x 28 cells (609 nodes) 1.26 / 1.94,
// 200 x 150 (30k) 3.0 / 3.7, 300 x 250 (76k) 4.3 / 5.3, 400 x 300 (121k) 6.3 / 5.8; a lane a node
// throughout: 2.09, 3.06, 5.08, 8.87.
constexpr int MM_FEW_W = 12;
constexpr uint32_t MM_FEW = 100000;
template <int PK, int PL>
struct Rows {
  static constexpr int CX = 0, CY = CX + PK, CR = CY + PK;         // circles
  static constexpr int AX = CR + PK, AY = AX + PL, AB = AY + PL;   // lines |ax x + ay y + ab|
  static constexpr int V = AB + PL;            // ordered keys of the constraint values, two sets in turn
  static constexpr int GY = V + 2 * (PK + PL);  // ascent gradients: y here, x in the idle set of V
  static constexpr int N = GY + PK + PL;
};

// What the lanes of a warp tell one another during the ascent, an entry per lane (node).
struct Shared {
  double px[MM_T], py[MM_T];               // the point, then the hull point
  unsigned long long rk[MM_T];             // results of a batch of tasks: key and point
  double rx[MM_T], ry[MM_T];
  uint32_t rm[MM_T];                       // and the constraints it comes from
  uint32_t first[MM_T], mask[MM_T], bad[MM_T];  // first task; active constraints; those flagged by tasks
  int32_t nc[MM_T], n[MM_T], set[MM_T];    // circles, gradients, the set of keys in use
};

template <int PK, int PL, int NW>  // NW: nodes of the warp
struct MaxiMin {
  double (*sm)[NW];  // shared rows, column t
  Shared* sh;
  int t, nc, nl;
  double lo[2], hi[2];  // box
  __device__ __forceinline__ double& at(int row, int k) const { return sm[row + k][t]; }
  __device__ __forceinline__ double& of(int o, int row, int k) const { return sm[row + k][o]; }  // node o's
  __device__ __forceinline__ unsigned long long& key(int o, int set, int k) const {
    return reinterpret_cast<unsigned long long&>(sm[Rows<PK, PL>::V + set * (PK + PL) + k][o]);
  }
  // gradient k of node o, whose keys in use are those of `set`
  __device__ __forceinline__ double& gx(int o, int set, int k) const {
    return sm[Rows<PK, PL>::V + (set ^ 1) * (PK + PL) + k][o];
  }
};

// Comparisons on the integer pipe (the FP64 pipe, which bounds the kernel, runs compares, minima and
// maxima too): the ordered keys of numbers order as the numbers do; a NaN's is the largest, so a
// minimum passes over it as fmin does. No value compared here is -0 but through a clamp, where the
// keys put it below +0 as the hardware's minimum and maximum do.
__device__ __forceinline__ unsigned long long okey(double x) {
  const unsigned long long b = ieee64::bits(x);
  return (b << 1) > 0xffe0000000000000ull ? ~0ull : ((b >> 63) ? ~b : (b | 0x8000000000000000ull));
}
__device__ __forceinline__ double from_okey(unsigned long long k) {
  return ieee64::from_bits((k >> 63) ? (k & 0x7fffffffffffffffull) : ~k);
}
__device__ __forceinline__ double clampd(double v, double lo, double hi) {
  const unsigned long long kv = okey(v);
  if (kv == ~0ull || kv < okey(lo)) v = lo;  // fmax(NaN, lo) = lo
  return okey(v) > okey(hi) ? hi : v;
}
__device__ __forceinline__ bool positive(double x) {  // x > 0
  const unsigned long long b = ieee64::bits(x);
  return b - 1 < 0x7ff0000000000000ull;
}
__device__ __forceinline__ bool negative(double x) {  // x < 0
  return positive(ieee64::from_bits(ieee64::bits(x) ^ ieee64::kSign));
}

// The ascent's square roots and quotients as calls: inlined at six places they overran the
// instruction cache (15.7 ms against 13.3).
__device__ __noinline__ double sqrt_call(double x) { return ieee64::sqrt_rn(x); }
__device__ __noinline__ double div_call(double a, double b) { return ieee64::div_rn(a, b); }

// Index of the q-th set bit.
__device__ __forceinline__ int nth_bit(uint32_t mask, int q) {
  for (; q > 0; --q) mask &= mask - 1;
  return __ffs(mask) - 1;
}

// Constraint k of node o at (x, y), as an ordered key.
template <int PK, int PL, int NW>
__device__ __forceinline__ unsigned long long mm_key(const MaxiMin<PK, PL, NW>& M, int o, int k, int nc, double x, double y) {
  using R = Rows<PK, PL>;
  if (k < nc) {
    const double dx = x - M.of(o, R::CX, k), dy = y - M.of(o, R::CY, k);
    return okey(sqrt_call(dx * dx + dy * dy) - M.of(o, R::CR, k));
  }
  const int l = k - nc;
  return okey(fabs(M.of(o, R::AX, l) * x + M.of(o, R::AY, l) * y + M.of(o, R::AB, l)));
}
// Minimum over the constraints of the lane's node at (x, y).
template <int PK, int PL, int NW>
__device__ __forceinline__ double mm_value(const MaxiMin<PK, PL, NW>& M, double x, double y) {
  unsigned long long m = okey(INFINITY);
  for (int k = 0; k < M.nc + M.nl; ++k) {
    const unsigned long long v = mm_key<PK, PL, NW>(M, M.t, k, M.nc, x, y);
    m = v < m ? v : m;
  }
  return from_okey(m);
}

// The lanes of a warp share out the tasks of its nodes: node o has `mine` tasks (its lane's argument);
// f(o, q, task) runs task q of node o on some lane, 32 tasks at a time, and after(b) on every lane
// when the tasks b .. b + 31 are done. All 32 lanes call; shared memory is synchronised around both.
template <class F, class A>
__device__ __forceinline__ void share_tasks(Shared* sh, int mine, F f, A after) {
  const uint32_t full = 0xffffffffu;
  const int lane = (int)threadIdx.x;
  int incl = mine;
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(full, incl, o);
    if (lane >= o) incl += v;
  }
  const int total = __shfl_sync(full, incl, 31);
  sh->first[lane] = (uint32_t)(incl - mine);
  __syncwarp();
  for (int b = 0; b < total; b += 32) {
    const int task = b + lane;
    if (task < total) {
      int o = 0;  // the last node whose first task is at or before this one: it has tasks
      for (int s = 16; s > 0; s >>= 1)
        if (sh->first[o + s] <= (uint32_t)task) o += s;
      f(o, task - (int)sh->first[o]);
    }
    __syncwarp();
    after(b, incl - mine, incl);
    __syncwarp();
  }
}

// Ascent from the origin (the initial guess) to a local maximum of the minimum over the
// constraints; returns the value, the point in (*px, *py) and the final step in *step_out.
//
// Of the 67 iterations of a node 57 % find no direction and only halve the step, and half of the
// trial points are rejected: the point is the same, and unless the smaller step drops a constraint
// from the active set so is the direction. So the constraint values are kept with the point (the
// trial point's in the other set of keys) and the direction is formed anew only when the point or
// the active set has changed. The nodes of a warp stand at different places of this and have
// different numbers of constraints (4 to 8) and of active ones (1 to 8), so the warp alternates
// between forming directions, halving steps and trying points, and the lanes share out the
// constraints, gradients and pairs of all nodes that take part. Every number is the one the plain
// loop forms, and minima keep its order.
//
// Bound by the latency of its integer and FP64 chains at 13 to 20 warps an SM (issue 35 % of cycles,
// FP64 pipe 53 %). 800 x 500 cells, 401k nodes, ms a call: 23.4 with a lane a node throughout (12 of 32
// lanes active, FP64 pipe 67 %), 15.4 with the kept values, 12.1 shared out.
template <int PK, int PL, int NW>
__device__ __forceinline__ double mm_ascent(const MaxiMin<PK, PL, NW>& M, bool node, double* px, double* py,
                                            double* step_out) {
  using R = Rows<PK, PL>;
  const uint32_t full = 0xffffffffu;
  Shared* sh = M.sh;
  const int me = M.t, ni = node ? M.nc + M.nl : 0;
  double x = 0.0, y = 0.0, fx = 0.0, step = 0.25, dx = 0.0, dy = 0.0, nd = 0.0;
  if (node) {
    x = clampd(0.0, M.lo[0], M.hi[0]);
    y = clampd(0.0, M.lo[1], M.hi[1]);
  }
  int set = 1, it = 0;
  unsigned long long kfx = 0, last = 0;  // the point's value; the largest key in the active set
  bool zero = true, turn = false, start = true;  // turn: the direction is to be formed
  // what holds while the point stays: constraints without a gradient, the hull's closest point, the
  // constraints it comes from, and those that show the hull to hold the origin
  uint32_t flat = 0u, pair = 0u, inside = 0u;
  double bx = 0.0, by = 0.0;
  bool moved = true;
  const uint64_t stop = ieee64::bits(1e-7);
  sh->nc[me] = node ? M.nc : 0;
  auto threshold = [&]() {  // constraints with a key up to it are active
    const double top = fx + step;
    return top != top ? 0ull : okey(top);
  };
  // the ascent only has to bring the point within reach of the exact solve, which takes the
  // constraints within max(1e-6, 8 step) of the minimum; stopping at step 1e-7 (instead of running
  // to 1e-13) halves the iterations and leaves every solved circle unchanged on the test meshes
  for (;;) {
    // ---- a trial point (at first the initial guess): its constraint values and their minimum
    const bool trial = node && (start || (!zero && !turn && it < 6000 && ieee64::bits(step) > stop));
    double nx = x, ny = y;
    if (trial && !start) {
      const double s = div_call(0.5 * step, nd);
      nx = clampd(x + s * dx, M.lo[0], M.hi[0]);
      ny = clampd(y + s * dy, M.lo[1], M.hi[1]);
    }
    sh->px[me] = nx;
    sh->py[me] = ny;
    sh->set[me] = set ^ 1;
    share_tasks(
        sh, trial ? ni : 0,
        [&](int o, int q) { M.key(o, sh->set[o], q) = mm_key<PK, PL, NW>(M, o, q, sh->nc[o], sh->px[o], sh->py[o]); },
        [](int, int, int) {});
    if (trial) {
      unsigned long long kfn = okey(INFINITY);
      for (int k = 0; k < ni; ++k) {
        const unsigned long long v = M.key(me, set ^ 1, k);
        kfn = v < kfn ? v : kfn;
      }
      if (!start) ++it;
      if (start || kfn > kfx) {
        x = nx;
        y = ny;
        kfx = kfn;
        fx = from_okey(kfn);
        set ^= 1;
        turn = true;
        moved = true;
        if (!start) {
          step = step * 1.5;
          if (ieee64::bits(step) > ieee64::bits(0.25)) step = 0.25;
        }
        start = false;
      } else {
        step *= 0.5;
        turn = threshold() < last;
      }
    }
    // ---- directions: gradients of the constraints within `step` of the minimum; moving by step / 2
    // along the min-norm point of their hull raises all of them, and no other one can drop below fx
    const bool go = node && it < 6000 && ieee64::bits(step) > stop;
    if (!__any_sync(full, go)) break;
    const bool form = go && turn;
    uint32_t active = 0u;
    if (form) {
      turn = false;
      const unsigned long long thr = threshold();
      last = 0;
      for (int k = 0; k < ni; ++k) {
        const unsigned long long v = M.key(me, set, k);
        const bool a = v <= thr;
        active |= (a ? 1u : 0u) << k;
        last = a && v > last ? v : last;
      }
    }
    __syncwarp();
    sh->px[me] = x;
    sh->py[me] = y;
    sh->set[me] = set;
    sh->mask[me] = active;
    sh->bad[me] = 0u;
    // At the same point a smaller active set with the constraints of the closest point has the same
    // closest point, and all that is known about it: nothing to compute.
    const bool need = form && (moved || (active & ~flat & pair) != pair || pair == 0u);
    share_tasks(
        sh, need ? __popc(active) : 0,
        [&](int o, int q) {
          const int k = nth_bit(sh->mask[o], q);
          const double ox = sh->px[o], oy = sh->py[o];
          if (k < sh->nc[o]) {
            const double ex = ox - M.of(o, R::CX, k), ey = oy - M.of(o, R::CY, k);
            const double d = sqrt_call(ex * ex + ey * ey);
            if (!positive(d)) atomicOr(&sh->bad[o], 1u << k);  // centred on the point: no gradient
            M.gx(o, sh->set[o], k) = div_call(ex, d);
            M.of(o, R::GY, k) = div_call(ey, d);
          } else {
            const int l = k - sh->nc[o];
            const double ax = M.of(o, R::AX, l), ay = M.of(o, R::AY, l);
            const double s = ax * ox + ay * oy + M.of(o, R::AB, l);
            const double sg = negative(s) ? -1.0 : 1.0;
            M.gx(o, sh->set[o], k) = sg * ax;
            M.of(o, R::GY, k) = sg * ay;
          }
        },
        [](int, int, int) {});
    if (need) flat = sh->bad[me];
    active &= ~flat;
    const int n = need ? __popc(active) : 0;
    __syncwarp();
    sh->mask[me] = active;
    // minimum-norm point of the convex hull of the n gradients (0 when the hull holds the origin):
    // the gradients and the closest points of their segments in the order (i), (i, i + 1), (i, i + 2)...,
    // the first of the smallest wins
    sh->n[me] = n;
    unsigned long long bn = okey(INFINITY);
    if (need) {
      moved = false;
      bx = 0.0;
      by = 0.0;
      pair = 0u;
    }
    share_tasks(
        sh, n * (n + 1) / 2,
        [&](int o, int q) {
          int i = 0;
          for (int w = sh->n[o]; q >= w; --w) {
            q -= w;
            ++i;
          }
          const uint32_t mask = sh->mask[o];
          const int set_o = sh->set[o], ki = nth_bit(mask, i), kj = nth_bit(mask, i + q);
          const double gix = M.gx(o, set_o, ki), giy = M.of(o, R::GY, ki);
          double qx = gix, qy = giy;
          unsigned long long k = 0;
          if (q > 0) {
            const double ex = M.gx(o, set_o, kj) - gix, ey = M.of(o, R::GY, kj) - giy;
            const double dd = ex * ex + ey * ey;
            if ((ieee64::bits(dd) << 1) == 0) k = ~0ull;  // dd <= 0: a sum of squares
            const double t = clampd(div_call(-(gix * ex + giy * ey), dd), 0.0, 1.0);
            qx = gix + t * ex;
            qy = giy + t * ey;
          }
          if (k == 0) k = okey(qx * qx + qy * qy);
          sh->rk[me] = k;
          sh->rx[me] = qx;
          sh->ry[me] = qy;
          sh->rm[me] = (1u << ki) | (1u << kj);
        },
        [&](int b, int lo, int hi) {
          for (int q = max(lo, b); q < min(hi, b + 32); ++q)
            if (sh->rk[q - b] < bn) {
              bn = sh->rk[q - b];
              bx = sh->rx[q - b];
              by = sh->ry[q - b];
              pair = sh->rm[q - b];
            }
        });
    // p is the hull's closest point to the origin iff p . (g - p) >= 0 for every g
    sh->px[me] = bx;
    sh->py[me] = by;
    sh->bad[me] = 0u;
    share_tasks(
        sh, n,
        [&](int o, int q) {
          const double ox = sh->px[o], oy = sh->py[o];
          const int k = nth_bit(sh->mask[o], q);
          if (ox * (M.gx(o, sh->set[o], k) - ox) + oy * (M.of(o, R::GY, k) - oy) < -1e-12)
            atomicOr(&sh->bad[o], 1u << k);
        },
        [](int, int, int) {});
    if (need) inside = sh->bad[me];
    if (form) {
      dx = (inside & active) ? 0.0 : bx;
      dy = (inside & active) ? 0.0 : by;
      // box faces: no motion through a face the point sits on
      const unsigned long long kx = okey(x), ky = okey(y);
      if ((kx <= okey(M.lo[0]) && negative(dx)) || (kx >= okey(M.hi[0]) && positive(dx))) dx = 0.0;
      if ((ky <= okey(M.lo[1]) && negative(dy)) || (ky >= okey(M.hi[1]) && positive(dy))) dy = 0.0;
      nd = sqrt_call(dx * dx + dy * dy);
      zero = nd < 1e-12;
    }
    // ---- no direction: halve the step until a constraint leaves the active set
    while (node && zero && !turn && it < 6000 && ieee64::bits(step) > stop) {
      step *= 0.5;
      ++it;
      turn = threshold() < last;
    }
    __syncwarp();
  }
  *px = x;
  *py = y;
  *step_out = step;
  return fx;
}

// One constraint of the exact solve, packed in 32 bits: kind << 8 | idx, plus bit 16 = negative
// side (lines) or upper face (box). kind 0 circle, 1 line, 2 box face (idx = axis).
constexpr uint32_t PC_CIRCLE = 0, PC_LINE = 1, PC_BOX = 2, PC_NEG = 1u << 16;
__device__ __forceinline__ uint32_t pc_kind(uint32_t p) { return (p >> 8) & 0xffu; }
__device__ __forceinline__ int pc_idx(uint32_t p) { return (int)(p & 0xffu); }

// linear row r . (x, y, Z) = rhs of a line or box piece
template <int PK, int PL, int NW>
__device__ __forceinline__ void piece_row(const MaxiMin<PK, PL, NW>& M, uint32_t p, double* r, double* rhs) {
  if (pc_kind(p) == PC_LINE) {
    const double sg = (p & PC_NEG) ? -1.0 : 1.0;
    const int l = pc_idx(p);
    r[0] = sg * M.at(Rows<PK, PL>::AX, l);
    r[1] = sg * M.at(Rows<PK, PL>::AY, l);
    r[2] = -1.0;
    *rhs = -sg * M.at(Rows<PK, PL>::AB, l);
  } else {
    const int a = pc_idx(p);
    r[0] = a == 0 ? 1.0 : 0.0;
    r[1] = a == 1 ? 1.0 : 0.0;
    r[2] = 0.0;
    *rhs = (p & PC_NEG) ? M.hi[a] : M.lo[a];
  }
}

__device__ __forceinline__ double det3(const double (&A)[3][3]) {
  return A[0][0] * (A[1][1] * A[2][2] - A[1][2] * A[2][1]) - A[0][1] * (A[1][0] * A[2][2] - A[1][2] * A[2][0]) +
         A[0][2] * (A[1][0] * A[2][1] - A[1][1] * A[2][0]);
}

// points where the three pieces are tight; returns how many (0..2) were written to (qx, qy, qz)
template <int PK, int PL, int NW>
__device__ __forceinline__ int solve_triple(const MaxiMin<PK, PL, NW>& M, const uint32_t (&P)[3], double (&qx)[2],
                                            double (&qy)[2], double (&qz)[2]) {
  int circ[3] = {0, 0, 0}, nc = 0;
  double R[3][3], rhs[3];
  int nr = 0;
  for (int k = 0; k < 3; ++k)
    if (pc_kind(P[k]) == PC_CIRCLE) circ[nc++] = pc_idx(P[k]);
  for (int k = 0; k < 3; ++k)
    if (pc_kind(P[k]) != PC_CIRCLE) {
      piece_row(M, P[k], R[nr], &rhs[nr]);
      ++nr;
    }
  if (nc == 0) {
    const double det = det3(R);
    if (fabs(det) < 1e-14) return 0;
    double sol[3];
    for (int c = 0; c < 3; ++c) {
      double A[3][3];
      for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) A[i][j] = (j == c) ? rhs[i] : R[i][j];
      sol[c] = det3(A) / det;
    }
    qx[0] = sol[0];
    qy[0] = sol[1];
    qz[0] = sol[2];
    return 1;
  }
  // differences of the circle equations against the first circle are linear in (x, y, Z)
  const int c1 = circ[0];
  const double p1x = M.at(Rows<PK, PL>::CX, c1), p1y = M.at(Rows<PK, PL>::CY, c1), r1 = M.at(Rows<PK, PL>::CR, c1);
  for (int k = 1; k < nc; ++k) {
    const int cj = circ[k];
    const double pjx = M.at(Rows<PK, PL>::CX, cj), pjy = M.at(Rows<PK, PL>::CY, cj), rj = M.at(Rows<PK, PL>::CR, cj);
    R[nr][0] = 2.0 * (pjx - p1x);
    R[nr][1] = 2.0 * (pjy - p1y);
    R[nr][2] = 2.0 * (rj - r1);
    rhs[nr] = (pjx * pjx + pjy * pjy - rj * rj) - (p1x * p1x + p1y * p1y - r1 * r1);
    ++nr;
  }
  // nr == 2: solutions Q0 + t * Dir, Dir = R0 x R1, Q0 the least-norm solution
  const double Dx = R[0][1] * R[1][2] - R[0][2] * R[1][1];
  const double Dy = R[0][2] * R[1][0] - R[0][0] * R[1][2];
  const double Dz = R[0][0] * R[1][1] - R[0][1] * R[1][0];
  const double g00 = R[0][0] * R[0][0] + R[0][1] * R[0][1] + R[0][2] * R[0][2];
  const double g01 = R[0][0] * R[1][0] + R[0][1] * R[1][1] + R[0][2] * R[1][2];
  const double g11 = R[1][0] * R[1][0] + R[1][1] * R[1][1] + R[1][2] * R[1][2];
  const double gd = g00 * g11 - g01 * g01;
  if (Dx * Dx + Dy * Dy + Dz * Dz < 1e-24 || fabs(gd) < 1e-24) return 0;
  const double u0 = (g11 * rhs[0] - g01 * rhs[1]) / gd, u1 = (g00 * rhs[1] - g01 * rhs[0]) / gd;
  const double q0x = u0 * R[0][0] + u1 * R[1][0], q0y = u0 * R[0][1] + u1 * R[1][1], q0z = u0 * R[0][2] + u1 * R[1][2];
  const double ex = q0x - p1x, ey = q0y - p1y, ez = q0z + r1;
  const double a = Dx * Dx + Dy * Dy - Dz * Dz, b = 2.0 * (ex * Dx + ey * Dy - ez * Dz), c = ex * ex + ey * ey - ez * ez;
  double t[2] = {0.0, 0.0};
  int nt = 0;
  if (fabs(a) < 1e-14) {
    if (fabs(b) < 1e-300) return 0;
    t[nt++] = -c / b;
  } else {
    double disc = b * b - 4.0 * a * c;
    if (disc < 0.0) {
      if (disc < -1e-12 * (b * b + fabs(4.0 * a * c))) return 0;
      disc = 0.0;
    }
    const double q = -0.5 * (b + copysign(sqrt(disc), b));
    t[nt++] = q / a;
    if (q != 0.0) t[nt++] = c / q;
  }
  int w = 0;
  for (int k = 0; k < nt; ++k) {
    const double zx = q0x + t[k] * Dx, zy = q0y + t[k] * Dy, zz = q0z + t[k] * Dz;
    bool ok = true;
    for (int j = 0; j < nc; ++j) ok = ok && (zz + M.at(Rows<PK, PL>::CR, circ[j]) >= -1e-12);  // external tangency
    if (!ok) continue;
    qx[w] = zx;
    qy[w] = zy;
    qz[w] = zz;
    ++w;
  }
  return w;
}

// Node i's problem: circles, lines and box in the shifted and scaled coordinates; (x0, y0) and L map
// them back.
struct PackMeshDev {
  const double *pos, *cen, *rad;
  const uint32_t *off, *adj, *mask, *bcnt, *bedge, *be;
};
template <int PK, int PL, int NW>
__device__ __forceinline__ void load_problem(const PackMeshDev& P, uint32_t i, MaxiMin<PK, PL, NW>& M, double* x0_out,
                                             double* y0_out, double* L_out) {
  using R = Rows<PK, PL>;
  const double *pos = P.pos, *cen = P.cen, *rad = P.rad;
  const uint32_t b = P.off[i], e = P.off[i + 1];
  const bool bdry = P.mask[i] != 0;
  double x0, y0;
  const double nx = pos[2 * (size_t)i], ny = pos[2 * (size_t)i + 1];
  // the node's elements in ascending order (the fill order is not deterministic), kept in the
  // circle rows as doubles until the coordinates replace them
  const int ncir = (int)(e - b);
  for (int k = 0; k < ncir; ++k) {
    const double t = (double)P.adj[b + k];
    int j = k;
    while (j > 0 && M.at(R::CR, j - 1) > t) {
      M.at(R::CR, j) = M.at(R::CR, j - 1);
      --j;
    }
    M.at(R::CR, j) = t;
  }
  // box and initial guess in the reference's terms (exp_dict.py:1196-1199 interior, :1250-1260
  // boundary)
  double lo[2] = {INFINITY, INFINITY}, hi[2] = {-INFINITY, -INFINITY}, sx = 0.0, sy = 0.0;
  for (int k = 0; k < ncir; ++k) {
    const uint32_t t = (uint32_t)M.at(R::CR, k);
    const double px = cen[2 * (size_t)t], py = cen[2 * (size_t)t + 1];
    lo[0] = fmin(lo[0], px);
    hi[0] = fmax(hi[0], px);
    lo[1] = fmin(lo[1], py);
    hi[1] = fmax(hi[1], py);
    sx += px;
    sy += py;
  }
  x0 = nx;
  y0 = ny;
  if (bdry) {
    lo[0] = fmin(lo[0], nx);
    hi[0] = fmax(hi[0], nx);
    lo[1] = fmin(lo[1], ny);
    hi[1] = fmax(hi[1], ny);
    x0 = (sx + nx) / (double)(e - b + 1);
    y0 = (sy + ny) / (double)(e - b + 1);
  }
  const double L = fmax(fmax(hi[0] - lo[0], hi[1] - lo[1]), 1e-300);
  const double iL = 1.0 / L;
  M.nc = ncir;
  for (int k = 0; k < ncir; ++k) {
    const uint32_t t = (uint32_t)M.at(R::CR, k);
    M.at(R::CX, k) = (cen[2 * (size_t)t] - x0) * iL;
    M.at(R::CY, k) = (cen[2 * (size_t)t + 1] - y0) * iL;
    M.at(R::CR, k) = rad[t] * iL;
  }
  M.nl = 0;
  if constexpr (PL > 0) if (bdry) {
    // boundary edges through the node in ascending order
    const uint32_t nb = min(P.bcnt[i], (uint32_t)PL);
    uint32_t eds[PL] = {0};
    for (uint32_t k = 0; k < nb; ++k) {
      const uint32_t t = P.bedge[(size_t)i * PL_MAX + k];
      uint32_t j = k;
      while (j > 0 && eds[j - 1] > t) {
        eds[j] = eds[j - 1];
        --j;
      }
      eds[j] = t;
    }
    for (uint32_t k = 0; k < nb; ++k) {
      const uint32_t ed = eds[k];
      const uint32_t v1 = P.be[2 * (size_t)ed], v2 = P.be[2 * (size_t)ed + 1];
      const double e1x = pos[2 * (size_t)v1], e1y = pos[2 * (size_t)v1 + 1];
      const double ux = pos[2 * (size_t)v2] - e1x, uy = pos[2 * (size_t)v2 + 1] - e1y;
      const double un = sqrt(ux * ux + uy * uy);
      if (!(un > 0.0)) continue;
      // |u x (p - e1)| / |u| (exp_dict.py:1240-1247) = |n . (p - e1)|, n = (-uy, ux) / |u|
      const double ax = -uy / un, ay = ux / un;
      M.at(R::AX, M.nl) = ax;
      M.at(R::AY, M.nl) = ay;
      M.at(R::AB, M.nl) = (ax * (x0 - e1x) + ay * (y0 - e1y)) * iL;
      ++M.nl;
    }
  }
  M.lo[0] = (lo[0] - x0) * iL;
  M.hi[0] = (hi[0] - x0) * iL;
  M.lo[1] = (lo[1] - y0) * iL;
  M.hi[1] = (hi[1] - y0) * iL;
  *x0_out = x0;
  *y0_out = y0;
  *L_out = L;
}

// Ascent of the nodes of a list, NW a warp, in its first lanes: its end, value and last step to asc[4 rank + 0..3].
template <int PK, int PL, int NW>
__global__ void __launch_bounds__(MM_T) k_pack_ascent(const PackMeshDev P, const uint32_t* list, uint32_t count,
                                                      const uint32_t* rank, double* asc, int32_t* err) {
  asm volatile("griddepcontrol.launch_dependents;");
  __shared__ double sm[Rows<PK, PL>::N][NW];
  __shared__ Shared sh;
  const uint32_t at = blockIdx.x * NW + threadIdx.x;
  bool node = threadIdx.x < (uint32_t)NW && at < count;  // every lane stays for its warp's ascent
  const uint32_t i = node ? list[at] : 0u;
  const uint32_t n = P.off[i + 1] - P.off[i];
  if (node && n == 0) {
    set_err(err, PE_ISOLATED);
    node = false;
  }
  if (node && n > (uint32_t)PK) {
    set_err(err, PE_CIRCLES);
    node = false;
  }
  MaxiMin<PK, PL, NW> M;
  M.sm = sm;
  M.sh = &sh;
  M.t = (int)threadIdx.x;
  M.nc = 0;
  M.nl = 0;
  double x0, y0, L, x, y, step;
  if (node) load_problem<PK, PL, NW>(P, i, M, &x0, &y0, &L);
  __syncwarp();
  const double fx = mm_ascent<PK, PL, NW>(M, node, &x, &y, &step);
  // Launched programmatically, this grid may end before the classes launched ahead of it. What follows
  // the last class on the stream needs all of them, so a grid does not complete before its predecessor
  // has: one block waits for it (all of them would hold their places on the SMs meanwhile).
  if (blockIdx.x == 0) asm volatile("griddepcontrol.wait;" ::: "memory");
  if (!node) return;
  double2* o = reinterpret_cast<double2*>(asc) + 2 * (size_t)rank[i];
  o[0] = make_double2(x, y);
  o[1] = make_double2(fx, step);
}

// The exact solve behind the ascent, a thread a node (a kernel of its own: the ascent then fits more
// warps in an SM's registers), and the circle in the mesh's coordinates.
template <int PK, int PL>
__global__ void __launch_bounds__(MM_T) k_pack_solve(const PackMeshDev P, uint32_t nn, uint32_t ne,
                                                     const uint32_t* flag, const uint32_t* rank, const double* asc,
                                                     double* ocen, double* orad, uint32_t* unpolished) {
  using R = Rows<PK, PL>;
  constexpr int NW = MM_T;
  __shared__ double sm[R::V][NW];  // circles and lines only
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nn || !flag[i]) return;
  const uint32_t n = P.off[i + 1] - P.off[i];
  if (n == 0 || n > (uint32_t)PK) return;  // reported by the ascent
  MaxiMin<PK, PL, NW> M;
  M.sm = sm;
  M.sh = nullptr;
  M.t = (int)threadIdx.x;
  double x0, y0, L;
  load_problem<PK, PL, NW>(P, i, M, &x0, &y0, &L);
  const double2* a = reinterpret_cast<const double2*>(asc) + 2 * (size_t)rank[i];
  const double x = a[0].x, y = a[0].y, fx = a[1].x, step = a[1].y;
  // exact solve: constraints within `near` of the minimum (and box faces within `near`) at the
  // ascent's end; the tight point with value >= fx closest to the ascent's end is the maximum
  const double near = fmax(1e-6, 8.0 * step);
  uint32_t S[PS_MAX];
  int ns = 0;
  for (int k = 0; k < M.nc && ns < PS_MAX; ++k) {
    const double dx = x - M.at(R::CX, k), dy = y - M.at(R::CY, k);
    const double v = sqrt(dx * dx + dy * dy) - M.at(R::CR, k);
    if (v <= fx + near) S[ns++] = (PC_CIRCLE << 8) | (uint32_t)k;
  }
  for (int l = 0; l < M.nl && ns < PS_MAX; ++l) {
    const double s = M.at(R::AX, l) * x + M.at(R::AY, l) * y + M.at(R::AB, l);
    if (fabs(s) <= fx + near) S[ns++] = (PC_LINE << 8) | (uint32_t)l | (s < 0.0 ? PC_NEG : 0u);
  }
  for (int a = 0; a < 2 && ns < PS_MAX; ++a) {
    const double w = a == 0 ? x : y;
    if (w - M.lo[a] <= near && ns < PS_MAX) S[ns++] = (PC_BOX << 8) | (uint32_t)a;
    if (M.hi[a] - w <= near && ns < PS_MAX) S[ns++] = (PC_BOX << 8) | (uint32_t)a | PC_NEG;
  }
  double bx = x, by = y, bf = fx, bd = INFINITY;
  for (int p = 0; p < ns; ++p)
    for (int q = p + 1; q < ns; ++q)
      for (int r = q + 1; r < ns; ++r) {
        const uint32_t T3[3] = {S[p], S[q], S[r]};
        int boxes = 0, axes = 0;
        for (int k = 0; k < 3; ++k)
          if (pc_kind(T3[k]) == PC_BOX) {
            ++boxes;
            axes |= 1 << pc_idx(T3[k]);
          }
        if (boxes == 3 || (boxes == 2 && axes != 3)) continue;
        double qx[2], qy[2], qz[2];
        const int nq = solve_triple<PK, PL, NW>(M, T3, qx, qy, qz);
        for (int k = 0; k < nq; ++k) {
          const double tol = 1e-11;
          if (qx[k] < M.lo[0] - tol || qx[k] > M.hi[0] + tol || qy[k] < M.lo[1] - tol || qy[k] > M.hi[1] + tol) continue;
          const double cxk = clampd(qx[k], M.lo[0], M.hi[0]), cyk = clampd(qy[k], M.lo[1], M.hi[1]);
          const double v = mm_value<PK, PL, NW>(M, cxk, cyk);
          if (boxes < 2 && fabs(v - qz[k]) > 1e-9) continue;  // another constraint is lower there
          if (v < fx - 1e-12) continue;
          const double d = (cxk - x) * (cxk - x) + (cyk - y) * (cyk - y);
          if (d < bd) {
            bd = d;
            bx = cxk;
            by = cyk;
            bf = v;
          }
        }
      }
  if (bd == INFINITY) atomicAdd(unpolished, 1u);
  const uint32_t o = ne + rank[i];
  ocen[2 * (size_t)o] = x0 + bx * L;
  ocen[2 * (size_t)o + 1] = y0 + by * L;
  orad[o] = bf * L;
}

inline uint32_t cdivp(uint64_t a, uint32_t b) { return (uint32_t)((a + b - 1) / b); }

}  // namespace

}  // namespace pg

// ---------------------------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------------------------
namespace {
thread_local std::string g_pack_err;

int pack_fail(int code, const std::string& msg) {
  g_pack_err = msg;
  return code;
}
}  // namespace

extern "C" const char* pg_pack_last_error(void) { return g_pack_err.c_str(); }

extern "C" int pg_pack_incenters(const pg_pack_mesh* m, int32_t modify_nodal_circles, int32_t gen_bdry,
                                 double* centers, double* radii, uint32_t* n_out, uint32_t* n_unpolished,
                                 void* stream) {
  using namespace pg;
  if (!m || !n_out || !centers || !radii) return pack_fail(PG_EINVAL, "null argument");
  *n_out = 0;
  if (n_unpolished) *n_unpolished = 0;
  const uint32_t D = m->dim, nn = m->n_nodes, ne = m->n_elems, nv = D + 1;
  if (D != 2 && D != 3) return pack_fail(PG_EINVAL, "dim must be 2 or 3");
  if (modify_nodal_circles && D != 2) return pack_fail(PG_EINVAL, "modified nodal circles are defined for 2D meshes");
  if ((nn && !m->pos) || (ne && !m->elems) || (m->n_bdry_nodes && !m->bdry_nodes) ||
      (m->n_bdry_edges && !m->bdry_edges))
    return pack_fail(PG_EINVAL, "null mesh array");
  if (ne == 0) return PG_OK;
  if (nn == 0) return pack_fail(PG_EINVAL, "elements without nodes");
  cudaStream_t st = (cudaStream_t)stream;
  const uint32_t tiles = bond_scan_tiles(nn);
  // scratch (u32 words): cnt, off[nn+1], fill, mask, bcnt, bedge[nn*PL_MAX], flag, rank[nn+1],
  // adj[ne*nv], tile_sum, done, err, unpolished, classes and their cursors; in
  // front, for the maximin circles, the ascents' ends (4 doubles a node) and the class lists
  const size_t front = modify_nodal_circles ? (size_t)nn * 9 + (nn & 1) : 0;
  const size_t words = front + (size_t)nn * (7 + PL_MAX) + 2 + (size_t)ne * nv + tiles + 3 + 2 * MM_CLASSES;
  void* block = nullptr;
  cudaError_t e = cudaMalloc(&block, words * 4);
  if (e != cudaSuccess) return pack_fail(PG_ENOMEM, cudaGetErrorString(e));
  double* asc = (double*)block;
  uint32_t* w = (uint32_t*)block + front;
  uint32_t *cnt = w, *off = cnt + nn, *fill = off + nn + 1, *mask = fill + nn, *bcnt = mask + nn;
  uint32_t *bedge = bcnt + nn, *flag = bedge + (size_t)nn * PL_MAX, *rank = flag + nn;
  uint32_t *adj = rank + nn + 1, *tsum = adj + (size_t)ne * nv, *done = tsum + tiles;
  int32_t* err = (int32_t*)(done + 1);
  uint32_t *unpol = done + 2, *d_classes = done + 3, *list = (uint32_t*)block + (size_t)nn * 8;
  int rc = PG_OK;
  int32_t derr = 0;
  uint32_t unp = 0, classes[MM_CLASSES] = {0};
  e = cudaMemsetAsync(w, 0, (words - front) * 4, st);
  if (e == cudaSuccess) {
    if (D == 2) {
      k_pack_tri<<<cdivp(ne, PT), PT, 0, st>>>(m->pos, m->elems, ne, nn, centers, radii, cnt, err);
    } else {
      k_pack_tet<<<cdivp(ne, PT), PT, 0, st>>>(m->pos, m->elems, ne, nn, centers, radii, cnt, err);
    }
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = scan_u32_dev(cnt, nn, off, tsum, done, st);
  if (e == cudaSuccess) {
    k_pack_fill<<<cdivp(ne, PT), PT, 0, st>>>(m->elems, ne, nv, nn, off, fill, adj);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess && m->n_bdry_nodes) {
    k_pack_bdry<<<cdivp(m->n_bdry_nodes, PT), PT, 0, st>>>(m->bdry_nodes, m->n_bdry_nodes, nn, mask, err);
    e = cudaGetLastError();
  }
  const bool maximin = modify_nodal_circles != 0;
  const bool all_bdry = maximin && gen_bdry;
  if (e == cudaSuccess && all_bdry && m->n_bdry_edges) {
    k_pack_bedges<<<cdivp(m->n_bdry_edges, PT), PT, 0, st>>>(m->bdry_edges, m->n_bdry_edges, nn, bcnt, bedge, err);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) {
    k_pack_flags<<<cdivp(nn, PT), PT, 0, st>>>(nn, mask, all_bdry ? 1 : 0, cnt, bcnt, flag,
                                              maximin ? d_classes : nullptr);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = scan_u32_dev(flag, nn, rank, tsum, done, st);
  // the element pass must be error-free before the nodal pass reads the adjacency
  if (e == cudaSuccess) e = cudaMemcpyAsync(&derr, err, 4, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess && maximin)
    e = cudaMemcpyAsync(classes, d_classes, sizeof classes, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e == cudaSuccess && derr == 0) {
    if (maximin) {
      ClassStart start;
      uint32_t nodes = 0;
      for (int k = 0; k < MM_CLASSES; ++k) {
        start.at[k] = nodes;
        nodes += classes[k];
      }
      k_pack_classes<<<cdivp(nn, PT), PT, 0, st>>>(nn, mask, flag, cnt, bcnt, start, d_classes + MM_CLASSES, list);
      const PackMeshDev Q = {m->pos, centers, radii, off, adj, mask, bcnt, bedge, m->bdry_edges};
      // A warp of the ascent runs for about two milliseconds, so the classes run into one another: each
      // launch lets the next one's blocks in as its last ones start (the classes share no data; they
      // all read what was complete before the first began) and completes after it (k_pack_ascent):
      // 13.4 -> 12.1 ms for 800 x 500 cells
      const bool few = nodes <= MM_FEW;
      bool first = true;
      auto ascent = [&](int k, auto* many_kernel, auto* few_kernel) {
        if (!classes[k]) return;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(cdivp(classes[k], few ? MM_FEW_W : MM_T));
        cfg.blockDim = dim3(MM_T);
        cfg.stream = st;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = at;
        cfg.numAttrs = first ? 0 : 1;
        first = false;
        if (e == cudaSuccess)
          e = cudaLaunchKernelEx(&cfg, few ? few_kernel : many_kernel, Q, (const uint32_t*)(list + start.at[k]),
                                 classes[k], (const uint32_t*)rank, asc, err);
      };
#define PG_ASCENT(k, pk, pl) ascent(k, k_pack_ascent<pk, pl, MM_T>, k_pack_ascent<pk, pl, MM_FEW_W>)
      PG_ASCENT(4, 16, 0);
      PG_ASCENT(3, 12, 0);
      PG_ASCENT(6, PK_MAX, PL_MAX);
      PG_ASCENT(5, 8, 2);
      PG_ASCENT(2, 8, 0);
      PG_ASCENT(1, 6, 0);
      PG_ASCENT(0, 4, 0);
#undef PG_ASCENT
      auto* solve = classes[3] + classes[4] + classes[6] ? k_pack_solve<PK_MAX, PL_MAX> : k_pack_solve<8, 2>;
      solve<<<cdivp(nn, MM_T), MM_T, 0, st>>>(Q, nn, ne, flag, rank, asc, centers, radii, unpol);
    } else if (D == 2) {
      k_pack_plain<2><<<cdivp(nn, PT), PT, 0, st>>>(m->pos, nn, ne, centers, radii, off, adj, flag, rank, centers,
                                                     radii, err);
    } else {
      k_pack_plain<3><<<cdivp(nn, PT), PT, 0, st>>>(m->pos, nn, ne, centers, radii, off, adj, flag, rank, centers,
                                                     radii, err);
    }
    if (e == cudaSuccess) e = cudaGetLastError();
  }
  uint32_t total = 0;
  if (e == cudaSuccess) e = cudaMemcpyAsync(&total, rank + nn, 4, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(&derr, err, 4, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(&unp, unpol, 4, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) {
    rc = pack_fail(PG_ECUDA, cudaGetErrorString(e));
  } else if (derr == PE_INDEX) {
    rc = pack_fail(PG_EINVAL, "node index out of range in elems, bdry_nodes or bdry_edges");
  } else if (derr == PE_ISOLATED) {
    rc = pack_fail(PG_EINVAL, "a node that needs a circle belongs to no element");
  } else if (derr == PE_CIRCLES) {
    rc = pack_fail(PG_ECAPACITY, "more than 16 elements around one node");
  } else if (derr == PE_LINES) {
    rc = pack_fail(PG_ECAPACITY, "more than 4 boundary edges through one node");
  } else {
    *n_out = ne + total;
    if (n_unpolished) *n_unpolished = unp;
  }
  cudaFree(block);
  return rc;
}
