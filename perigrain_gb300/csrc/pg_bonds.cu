// GPU bond-list builder: the Connectivity of one grain -- all node pairs (i, j), i < j, with
// sqrt(sum((p_j - p_i)^2)) <= delta, in lexicographic order. The reference builds it in Python
// over all n(n-1)/2 pairs (exp_dict.py:171-222: itertools.combinations + single_bond); here a
// uniform grid of cell >= delta / 2 restricts each node to the 5^dim surrounding cells.
//
// Passes, all on the caller's stream with one host wait at the end: bounding box and grid -> cell
// key and count -> scan of the counts -> scatter into cell order -> count of partners j > i per
// node -> scan of the counts -> write of each node's partners in ascending j. Compiled with
// --fmad=false so the distance is the same IEEE computation numpy performs, and the pair set is
// identical to the reference's.
//
// Bound by launch and memory latency: 200k nodes in 2D are 21 MB of pairs, a few us of bandwidth.
// 200k nodes, 3 spacings, us a call: 545 with the grid fitted on the host (a wait in the middle),
// FP64 distances in both pair passes (164 + 162) and rows sorted in global memory; 244 now, 23 + 43 in
// the pair passes; 115 with the scratch kept (pg_bond_scratch.cu).
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <string>

#include "../../include/perigrain.h"
#include "pg_bonds.h"
#include "pg_sqrt_threshold.h"
#include "pg_device.cuh"

namespace pg {

constexpr int BT = 256;               // threads per block
constexpr int SCAN_T = 1024;          // scan block
constexpr int SCAN_TILE_B = SCAN_T * 4;
static_assert(SCAN_TILE_B == (int)BOND_SCAN_TILE, "scan tile of the bond builder and its declared size differ");
constexpr int MAX_PARTNERS = 4096;    // partners j > i of one node
constexpr int ROW_T = 128;            // threads of a block of the pair passes
// Candidates come from the cells up to REACH away. Half the horizon a cell: 56 candidates a node in 2D
// and 425 in 3D at three spacings, against 81 and 729 with cells of a horizon; a third of it has more
// rows than it saves. us a call, REACH 1 / 2 / 3: 200k nodes in 2D 293 / 282 / 293, 180k in 3D
// 723 / 698 / 847.
constexpr uint32_t REACH = 2, ROWS = 2 * REACH + 1;
// Lanes a node in the pair passes, by the length of a row of candidates (11 in 2D, 17 in 3D): fewer
// lanes waste less of a row's last round, more walk a row in fewer rounds. us a call: 200k nodes in
// 2D, lanes 1 / 2 / 4 / 8: 279 / 290 / 282 / 308; 4.4k nodes 234 / 244 / 219 / 219; 3D, lanes
// 1 / 4 / 8 / 16: 180k nodes 2385 / 663 / 698 / 856, 2k nodes 606 / 283 / 244 / 246.
constexpr int BOND_LANES_2D = 4, BOND_LANES_3D = 8;
constexpr int32_t ERR_NONFINITE = 1, ERR_GRID = 2, ERR_PARTNERS = 4;  // BondHead::error

// Programmatic dependent launch: a pass may be placed on the GPU while the one before it drains,
// and waits here until that one is complete (which waited for its own predecessor).
__device__ __forceinline__ void kb_enter() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// The grid over the box (cells >= delta (1 + 1e-6) / REACH, at most max_cells of them) and the
// thresholds of the FP32 pair test. One warp, a lane an axis.
//
// A pair passes when the FP64 sum s of squared differences is <= s_max. Positions are also kept in
// 32-bit fixed point, 2^30 units over the longest side of the box, so a difference is off by at most
// 1 unit an axis (two roundings of half a unit) and a length by at most sqrt(3) < 2 units; FP32
// arithmetic on the exact integer differences is off by less than 5 x 2^-24 of its sum. A sum of at
// most s_lo therefore passes and one above s_hi fails; only between them does FP64 decide. The
// bounds hold where no FP64 square underflows or overflows: outside 1e-140..1e140 every pair is
// left to FP64.
__device__ void fit_grid(BondHead* H, uint32_t dim, double delta, uint32_t max_cells) {
  const uint32_t full = 0xffffffffu, c = threadIdx.x & 31;
  const double lo = c < dim ? ordered_to_dbl(~__ldcg(&H->box[c])) : 0.0;
  const double hi = c < dim ? ordered_to_dbl(__ldcg(&H->box[3 + c])) : 0.0;
  if (__any_sync(full, !isfinite(lo) || !isfinite(hi))) {
    if (c == 0) H->error = ERR_NONFINITE;
    return;  // H->grid.cells stays 0
  }
  double ext = hi - lo;
  ext = fmax(ext, fmax(__shfl_sync(full, ext, 1), __shfl_sync(full, ext, 2)));
  ext = __shfl_sync(full, ext, 0);
  double cell = delta > 0 ? delta * (1 + 1e-6) : fmax(ext, 1e-300) / 64;
  double count = 1, cells = 1;
  const auto fits = [&] {
    count = floor((hi - lo) / cell) + 1;
    cells = __shfl_sync(full, count, 0) * __shfl_sync(full, count, 1) * __shfl_sync(full, count, 2);
    return cells <= (double)max_cells;
  };
  bool ok = fits();
  for (int it = 0; it < 200 && !ok; ++it) {
    cell *= 1.25;
    ok = fits();
  }
  if (!ok) {
    if (c == 0) H->error = ERR_GRID;
    return;
  }
  const double whole = cell;
  cell /= REACH;
  ok = cell > 0 && fits();
  for (int it = 0; it < 4 && !ok; ++it) {
    cell *= 1.25;
    ok = cell > 0 && fits();
  }
  if (!ok) {
    cell = whole;
    fits();
  }
  BondGrid* g = &H->grid;
  if (c < 3) {
    g->origin[c] = lo;
    g->dims[c] = (uint32_t)count;
  }
  if (c != 0) return;
  float s_lo = -1.0f, s_hi = INFINITY;
  double unit = 0;
  if (delta >= 1e-140 && delta <= 1e140 && ext >= 1e-140 && ext <= 1e140) {
    unit = 1073741824.0 / ext;
    const double in = delta * unit - 2.0, out = delta * unit + 2.0;
    if (in > 0) s_lo = __double2float_rd(in * in * (1 - 1e-6));
    s_hi = __double2float_ru(out * out * (1 + 1e-6));
  }
  g->inv_cell = 1.0 / cell;
  g->unit = unit;
  g->s_lo = s_lo;
  g->s_hi = s_hi;
  g->cells = (uint32_t)cells;
}

// Bounding box of the positions as ordered keys (minima inverted, so that both start at zero): each
// block folds its nodes with warp reductions and shared memory, then one atomic per block and bound
// (a per-thread atomic on the same six words serialised in L2: 54 us for 20k nodes). The last block
// to finish fits the grid.
__global__ void __launch_bounds__(BT) kb_box(const double* pos, uint32_t n, uint32_t dim, double delta, BondScratch S) {
  __shared__ unsigned long long red[6][BT / 32];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned long long mn[3] = {0, 0, 0}, mx[3] = {0, 0, 0};
  for (uint32_t i = blockIdx.x * BT + threadIdx.x; i < n; i += gridDim.x * BT)
#pragma unroll
    for (uint32_t c = 0; c < 3; ++c)
      if (c < dim) {
        const unsigned long long k = dbl_to_ordered(pos[(size_t)i * dim + c]);
        mn[c] = max(mn[c], ~k);
        mx[c] = max(mx[c], k);
      }
  for (uint32_t c = 0; c < 3; ++c) {
    mn[c] = warp_max_u64(mn[c]);
    mx[c] = warp_max_u64(mx[c]);
    if (lane == 0) {
      red[c][warp] = mn[c];
      red[3 + c][warp] = mx[c];
    }
  }
  __syncthreads();
  if (warp != 0) return;
  for (uint32_t c = 0; c < 6; ++c) {
    const unsigned long long v = warp_max_u64(lane < BT / 32 ? red[c][lane] : 0ull);
    if (lane == 0) atomicMax(&S.head->box[c], v);
  }
  uint32_t ticket = 0;
  if (lane == 0) {
    __threadfence();
    ticket = atomicAdd(&S.head->done[0], 1u);
  }
  if (__shfl_sync(0xffffffffu, ticket, 0) != gridDim.x - 1) return;
  __threadfence();
  fit_grid(S.head, dim, delta, S.cells);
}

__global__ void kb_key(const double* pos, uint32_t n, uint32_t dim, BondScratch S) {
  kb_enter();
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  const BondGrid g = S.head->grid;
  if (i >= n || !g.cells) return;
  uint32_t cc[3] = {0, 0, 0};
#pragma unroll
  for (uint32_t c = 0; c < 3; ++c)
    if (c < dim) {
      const double f = floor((pos[(size_t)i * dim + c] - g.origin[c]) * g.inv_cell);
      cc[c] = f < 0 ? 0 : (f >= (double)(g.dims[c] - 1) ? g.dims[c] - 1 : (uint32_t)f);
    }
  const uint32_t k = (cc[2] * g.dims[1] + cc[1]) * g.dims[0] + cc[0];
  S.key[i] = k;
  S.rank[i] = atomicAdd(&S.cell[k], 1u);
}

__device__ __forceinline__ uint32_t blk_excl(uint32_t v, uint32_t* ws, uint32_t* total) {
  const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  uint32_t x = v;
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= (uint32_t)o) x += y;
  }
  if (lane == 31) ws[wid] = x;
  __syncthreads();
  if (wid == 0) {
    const uint32_t nw = blockDim.x >> 5;
    uint32_t s = lane < nw ? ws[lane] : 0;
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t y = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= (uint32_t)o) s += y;
    }
    if (lane < nw) ws[lane] = s;
  }
  __syncthreads();
  const uint32_t base = wid ? ws[wid - 1] : 0;
  if (total) *total = ws[(blockDim.x >> 5) - 1];
  __syncthreads();
  return base + x - v;
}

// Exclusive scan in place, in two levels: a[i] becomes the sum over its tile's entries before i, and
// tsum[t] the sum of the tiles before t (the last block to finish scans the tile sums), so the prefix
// of i is a[i] + tsum[i / SCAN_TILE_B] (prefix()): one pass less than writing it out. len entries, or
// the grid's cells + 1 for len = 0. The total goes to *total.
__global__ void __launch_bounds__(SCAN_T)
    kb_scan(uint32_t* a, uint32_t len, uint32_t* tsum, uint32_t* done, uint32_t* total, const BondHead* head) {
  __shared__ uint32_t ws[32];
  __shared__ bool last;
  kb_enter();
  if (!head->grid.cells) return;
  if (!len) len = head->grid.cells + 1;
  const uint32_t base = blockIdx.x * SCAN_TILE_B + threadIdx.x * 4;
  uint32_t v[4], s = 0, tot = 0;
  if (blockIdx.x * SCAN_TILE_B < len) {
    for (int k = 0; k < 4; ++k) {
      v[k] = base + k < len ? a[base + k] : 0;
      s += v[k];
    }
    uint32_t ex = blk_excl(s, ws, &tot);
    for (int k = 0; k < 4; ++k) {
      if (base + k < len) a[base + k] = ex;
      ex += v[k];
    }
  }
  if (threadIdx.x == 0) {
    tsum[blockIdx.x] = tot;
    __threadfence();
    last = atomicAdd(done, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  uint32_t carry = 0;
  for (uint32_t b0 = 0; b0 < gridDim.x; b0 += SCAN_T) {
    const uint32_t i = b0 + threadIdx.x;
    const uint32_t w = i < gridDim.x ? __ldcg(tsum + i) : 0;
    uint32_t t2;
    const uint32_t ex = blk_excl(w, ws, &t2);
    if (i < gridDim.x) tsum[i] = carry + ex;
    carry += t2;
  }
  if (threadIdx.x == 0) *total = carry;
}

__device__ __forceinline__ uint32_t prefix(const uint32_t* a, const uint32_t* tsum, uint32_t i) {
  return a[i] + tsum[i / SCAN_TILE_B];
}

// exclusive scan of in[0..len) into out[0..len], out[len] = total; tile sums in tsum, done flag
__global__ void kb_scan_tiles(const uint32_t* in, uint32_t len, uint32_t* tsum, uint32_t* done) {
  __shared__ uint32_t ws[32];
  __shared__ bool last;
  const uint32_t base = blockIdx.x * SCAN_TILE_B + threadIdx.x * 4;
  uint32_t s = 0;
  for (int k = 0; k < 4; ++k)
    if (base + k < len) s += in[base + k];
  uint32_t tot;
  blk_excl(s, ws, &tot);
  if (threadIdx.x == 0) {
    tsum[blockIdx.x] = tot;
    __threadfence();
    last = (atomicAdd(done, 1u) == gridDim.x - 1);
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  uint32_t carry = 0;
  for (uint32_t b0 = 0; b0 < gridDim.x; b0 += SCAN_T) {
    const uint32_t i = b0 + threadIdx.x;
    const uint32_t v = i < gridDim.x ? ((volatile uint32_t*)tsum)[i] : 0;
    uint32_t t2;
    const uint32_t ex = blk_excl(v, ws, &t2);
    if (i < gridDim.x) tsum[i] = carry + ex;
    carry += t2;
  }
  if (threadIdx.x == 0) *done = 0;
}

__global__ void kb_scan_final(const uint32_t* in, uint32_t len, const uint32_t* tsum, uint32_t* out) {
  __shared__ uint32_t ws[32];
  const uint32_t base = blockIdx.x * SCAN_TILE_B + threadIdx.x * 4;
  uint32_t v[4], s = 0;
  for (int k = 0; k < 4; ++k) {
    v[k] = base + k < len ? in[base + k] : 0;
    s += v[k];
  }
  uint32_t ex = blk_excl(s, ws, nullptr) + tsum[blockIdx.x];
  for (int k = 0; k < 4; ++k) {
    if (base + k < len) out[base + k] = ex;
    ex += v[k];
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == blockDim.x - 1) out[len] = ex;
}

// Cell order: fixed-point position and node index, 16 bytes a node in 2D and 3D.
__global__ void kb_scatter(const double* pos, uint32_t n, uint32_t dim, BondScratch S) {
  kb_enter();
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  const BondGrid g = S.head->grid;
  if (i >= n || !g.cells) return;
  const double* p = pos + (size_t)i * dim;
  uint4 q;
  q.x = (uint32_t)__double2int_rn((p[0] - g.origin[0]) * g.unit);
  q.y = (uint32_t)__double2int_rn((p[1] - g.origin[1]) * g.unit);
  q.z = dim == 3 ? (uint32_t)__double2int_rn((p[2] - g.origin[2]) * g.unit) : 0u;
  q.w = i;
  S.sorted[prefix(S.cell, S.cell_tile, S.key[i]) + S.rank[i]] = q;
}

// The test of a candidate pair (fit_grid): in FP32 from the fixed-point positions, in FP64 where
// that leaves it open.
template <int D>
__device__ __forceinline__ bool bonded(const double* pos, const uint4& a, const uint4& b, const BondGrid& g,
                                       double s_max) {
  const float dx = (float)(int32_t)(b.x - a.x), dy = (float)(int32_t)(b.y - a.y);
  float f = __fmaf_rn(dx, dx, dy * dy);
  if (D == 3) {
    const float dz = (float)(int32_t)(b.z - a.z);
    f = __fmaf_rn(dz, dz, f);
  }
  if (f <= g.s_lo) return true;
  if (f > g.s_hi) return false;
  const double *pi = pos + (size_t)a.w * D, *pj = pos + (size_t)b.w * D;
  double s = (pj[0] - pi[0]) * (pj[0] - pi[0]);
#pragma unroll
  for (int c = 1; c < D; ++c) s = s + (pj[c] - pi[c]) * (pj[c] - pi[c]);
  return s <= s_max;
}

// Row r of a node's cells: those up to REACH away on x, consecutive in cell order. Candidates [b, e).
template <int D>
__device__ __forceinline__ void cand_row(const BondGrid& g, const BondScratch& S, uint32_t key, int r, uint32_t& b,
                                         uint32_t& e) {
  const uint32_t yz = key / g.dims[0], x = key - yz * g.dims[0];
  const uint32_t z = D == 3 ? yz / g.dims[1] : 0, y = yz - z * g.dims[1];
  const uint32_t yy = y + (uint32_t)(r % ROWS) - REACH, zz = D == 3 ? z + (uint32_t)(r / ROWS) - REACH : 0u;
  b = e = 0;
  if (yy >= g.dims[1] || zz >= g.dims[2]) return;
  const uint32_t row = (zz * g.dims[1] + yy) * g.dims[0];
  b = prefix(S.cell, S.cell_tile, row + (x > REACH ? x - REACH : 0));
  e = prefix(S.cell, S.cell_tile, row + min(x + REACH, g.dims[0] - 1) + 1);
}

// One thread's walk over the partners j > i of a node: f(j).
template <int D, class F>
__device__ void each_partner(const double* pos, const uint4& me, uint32_t key, const BondGrid& g,
                             const BondScratch& S, double s_max, F f) {
#pragma unroll 1
  for (int r = 0; r < (D == 2 ? (int)ROWS : (int)(ROWS * ROWS)); ++r) {
    uint32_t b, e;
    cand_row<D>(g, S, key, r, b, e);
    for (; b < e; ++b) {
      const uint4 q = S.sorted[b];
      if (q.w > me.w && bonded<D>(pos, me, q, g, s_max)) f(q.w);
    }
  }
}

// The pair passes, G lanes a node, nodes in cell order so that the lanes of a warp walk the same
// cells. WRITE = false: count node i's partners j > i. WRITE = true: write row i, pairs (i, j) with
// j ascending, at its offset. The partners are collected in shared memory and each goes straight to
// its place in the row, the number of smaller ones. A row of more than CAP partners is put down
// unsorted in the row's own i column and ranked from there; the one row that crosses `capacity` gets
// its smallest partners that fit.
template <int D, int G, bool WRITE>
__global__ void __launch_bounds__(ROW_T) kb_rows(const double* pos, uint32_t n, double s_max, BondScratch S,
                                                 uint32_t* pairs, uint64_t capacity) {
  constexpr uint32_t NG = ROW_T / G, CAP = 32 * G, GMASK = G == 32 ? 0xffffffffu : (1u << (G & 31)) - 1u;
  __shared__ uint32_t lists[WRITE ? NG * (CAP + 1) : 1];  // + 1: the groups' entries k on different banks
  kb_enter();
  const BondGrid g = S.head->grid;
  if (!g.cells) return;
  const uint32_t grp = threadIdx.x / G, gl = threadIdx.x % G, slot = blockIdx.x * NG + grp;
  const uint32_t gbase = (threadIdx.x & 31) - gl;  // the group's first lane
  uint4 me = make_uint4(0, 0, 0, 0);
  const bool act = slot < n;
  if (act) me = S.sorted[slot];
  const uint32_t i = me.w;
  const uint32_t key = S.key[i];
  constexpr int R = D == 2 ? ROWS : ROWS * ROWS;
  uint32_t* list = lists + (WRITE ? grp * (CAP + 1) : 0);
  uint32_t cnt = 0;
  uint32_t nb, ne;
  cand_row<D>(g, S, key, 0, nb, ne);
#pragma unroll 1
  for (int r = 0; r < R; ++r) {
    const uint32_t b0 = nb, b1 = act ? ne : b0;
    if (r + 1 < R) cand_row<D>(g, S, key, r + 1, nb, ne);  // ahead of its use
    const uint32_t its = __reduce_max_sync(0xffffffffu, (b1 - b0 + G - 1) / G);
    for (uint32_t it = 0; it < its; ++it) {
      const uint32_t b = b0 + it * G + gl;
      uint4 q = make_uint4(0, 0, 0, 0);
      bool hit = false;
      if (b < b1) {
        q = S.sorted[b];
        hit = q.w > i && bonded<D>(pos, me, q, g, s_max);
      }
      const uint32_t m = (__ballot_sync(0xffffffffu, hit) >> gbase) & GMASK;
      if (WRITE && hit) {
        const uint32_t at = cnt + __popc(m & ((1u << gl) - 1u));
        if (at < CAP) list[at] = q.w;
      }
      cnt += __popc(m);
    }
  }
  if (!WRITE) {
    if (act && gl == 0) {
      S.poff[i] = cnt;
      if (cnt > (uint32_t)MAX_PARTNERS) atomicOr(&S.head->error, ERR_PARTNERS);
      if (slot == 0) S.poff[n] = 0;
    }
    return;
  }
  __syncwarp();
  if (!act || !cnt) return;
  const uint64_t off = prefix(S.poff, S.poff_tile, i);
  if (off >= capacity) return;
  if (cnt <= CAP) {
    for (uint32_t a = gl; a < cnt; a += G) {
      const uint32_t v = list[a];
      uint64_t at = off;
#pragma unroll 4
      for (uint32_t k = 0; k < cnt; ++k) at += list[k] < v;
      if (at < capacity) {
        pairs[2 * at] = i;
        pairs[2 * at + 1] = v;
      }
    }
    return;
  }
  const uint32_t gm = GMASK << gbase;
  if (off + cnt <= capacity) {
    uint32_t* row = pairs + 2 * off;
    if (gl == 0) {
      uint32_t k = 0;
      each_partner<D>(pos, me, key, g, S, s_max, [&](uint32_t j) { row[2 * (size_t)k++] = j; });
    }
    __syncwarp(gm);
    for (uint32_t a = gl; a < cnt; a += G) {
      const uint32_t v = row[2 * (size_t)a];
      uint32_t at = 0;
      for (uint32_t k = 0; k < cnt; ++k) at += row[2 * (size_t)k] < v;
      row[2 * (size_t)at + 1] = v;
    }
    __syncwarp(gm);
    for (uint32_t a = gl; a < cnt; a += G) row[2 * (size_t)a] = i;
  } else if (gl == 0) {
    uint32_t prev = i;
    for (uint64_t k = off; k < capacity; ++k) {
      uint32_t best = 0xffffffffu;
      each_partner<D>(pos, me, key, g, S, s_max, [&](uint32_t j) {
        if (j > prev && j < best) best = j;
      });
      pairs[2 * k] = i;
      pairs[2 * k + 1] = best;
      prev = best;
    }
  }
}

static inline uint32_t cdivb(uint64_t a, uint32_t b) { return (uint32_t)((a + b - 1) / b); }

cudaError_t scan_u32_dev(const uint32_t* in, uint32_t len, uint32_t* out, uint32_t* tile_sum, uint32_t* done,
                         cudaStream_t st) {
  const uint32_t tiles = cdivb(len ? len : 1, SCAN_TILE_B);
  kb_scan_tiles<<<tiles, SCAN_T, 0, st>>>(in, len, tile_sum, done);
  kb_scan_final<<<tiles, SCAN_T, 0, st>>>(in, len, tile_sum, out);
  return cudaGetLastError();
}

uint32_t bond_scan_tiles(uint32_t len) { return bond_scan_tiles_c(len); }

template <class... KArgs, class... Args>
static cudaError_t launch_next(void (*k)(KArgs...), uint32_t grid, uint32_t block, cudaStream_t st, Args... args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k, KArgs(args)...);
}

BondScratch bond_scratch(uint32_t* base, uint32_t n) {
  BondScratch S;
  S.cells = bond_grid_cells_c(n);
  S.sorted = (uint4*)base;
  S.head = (BondHead*)(base + (size_t)n * 4);
  S.cell = base + (size_t)n * 4 + BOND_HEAD_WORDS;
  S.cell_tile = S.cell + S.cells + 1;
  S.poff = S.cell_tile + bond_scan_tiles_c(S.cells + 1);
  S.poff_tile = S.poff + n + 1;
  S.key = S.poff_tile + bond_scan_tiles_c(n + 1);
  S.rank = S.key + n;
  return S;
}

template <int D, int G>
static cudaError_t run_passes(const double* pos, uint32_t n, double delta, uint32_t* pairs, uint64_t capacity,
                              cudaStream_t st, const BondScratch& S, BondHead* out) {
  BondHead* H = S.head;
  const double s_max = sqrt_le_max(delta);
  const uint32_t nb = cdivb(n, BT), nr = cdivb(n, ROW_T / G);
  // the head and the cell counts follow one another
  cudaError_t e = cudaMemsetAsync(H, 0, (BOND_HEAD_WORDS + (size_t)S.cells + 1) * 4, st);
  if (e != cudaSuccess) return e;
  kb_box<<<nb < 304 ? nb : 304, BT, 0, st>>>(pos, n, D, delta, S);
  e = cudaGetLastError();
  if (e == cudaSuccess) e = launch_next(kb_key, nb, BT, st, pos, n, (uint32_t)D, S);
  if (e == cudaSuccess)
    e = launch_next(kb_scan, bond_scan_tiles_c(S.cells + 1), SCAN_T, st, S.cell, 0u, S.cell_tile, H->done + 1,
                    &H->nodes, H);
  if (e == cudaSuccess) e = launch_next(kb_scatter, nb, BT, st, pos, n, (uint32_t)D, S);
  if (e == cudaSuccess) e = launch_next(kb_rows<D, G, false>, nr, ROW_T, st, pos, n, s_max, S, pairs, capacity);
  if (e == cudaSuccess)
    e = launch_next(kb_scan, bond_scan_tiles_c(n + 1), SCAN_T, st, S.poff, n + 1, S.poff_tile, H->done + 2,
                    &H->total, H);
  if (e == cudaSuccess) e = launch_next(kb_rows<D, G, true>, nr, ROW_T, st, pos, n, s_max, S, pairs, capacity);
  if (e == cudaSuccess) e = cudaMemcpyAsync(out, H, sizeof *out, cudaMemcpyDeviceToHost, st);
  const cudaError_t w = cudaStreamSynchronize(st);  // also after a failed launch: the scratch is still in use
  return e != cudaSuccess ? e : w;
}

int run_bond_build(const double* pos, uint32_t n, uint32_t dim, double delta, uint32_t* pairs, uint64_t capacity,
                   uint64_t* n_pairs, cudaStream_t st, const BondScratch& S, std::string* err) {
  *n_pairs = 0;
  if (n < 2) return PG_OK;
  BondHead h;
  const cudaError_t e = dim == 2 ? run_passes<2, BOND_LANES_2D>(pos, n, delta, pairs, capacity, st, S, &h)
                                 : run_passes<3, BOND_LANES_3D>(pos, n, delta, pairs, capacity, st, S, &h);
  if (e != cudaSuccess) {
    *err = cudaGetErrorString(e);
    return PG_ECUDA;
  }
  if (h.error & ERR_NONFINITE) {
    *err = "non-finite node position";
    return PG_EINVAL;
  }
  if (h.error & ERR_GRID) {
    *err = "bond grid does not fit its scratch";
    return PG_ECAPACITY;
  }
  *n_pairs = h.total;
  if (h.error) {
    *err = "a node has more than 4096 partners j > i within delta";
    return PG_ECAPACITY;
  }
  if (h.total > capacity) {
    *err = "pair buffer too small: " + std::to_string(h.total) + " pairs";
    return PG_ECAPACITY;
  }
  return PG_OK;
}

}  // namespace pg

// ---------------------------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------------------------
namespace {
thread_local std::string g_bond_err;
}

extern "C" const char* pg_bond_last_error(void) { return g_bond_err.c_str(); }

extern "C" int pg_build_bonds(const double* pos, uint32_t n, uint32_t dim, double delta, uint32_t* pairs,
                              uint64_t capacity, uint64_t* n_pairs, void* stream) {
  using namespace pg;
  if (!n_pairs || (n && !pos) || (dim != 2 && dim != 3) || (capacity && !pairs)) {
    g_bond_err = "bad arguments";
    return PG_EINVAL;
  }
  *n_pairs = 0;
  if (n < 2) return PG_OK;
  cudaStream_t st = (cudaStream_t)stream;
  const KeptBondScratch kept(n);  // released after run_bond_build, which waits for the stream
  void* block = nullptr;
  if (!kept.base) {
    const cudaError_t e = cudaMalloc(&block, bond_scratch_words(n) * 4);
    if (e != cudaSuccess) {
      g_bond_err = cudaGetErrorString(e);
      return PG_ENOMEM;
    }
  }
  const BondScratch S = bond_scratch(kept.base ? kept.base : (uint32_t*)block, n);
  std::string err;
  int rc = run_bond_build(pos, n, dim, delta, pairs, capacity, n_pairs, st, S, &err);
  cudaFree(block);
  if (rc) g_bond_err = err;
  return rc;
}
