// Internal interface of the GPU bond-list builder (pg_bonds.cu).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <string>

namespace pg {

// Grid of one bond build (cells = 0: none, the build has failed), the fixed-point unit of its
// cell-ordered positions and the FP32 thresholds of the pair test.
struct BondGrid {
  double origin[3];
  double inv_cell, unit;
  uint32_t dims[3];
  uint32_t cells;
  float s_lo, s_hi;
};

// What the passes hand on, and the host reads back at the end.
struct BondHead {
  unsigned long long box[6];  // ordered-key bounding box, minima inverted
  uint32_t done[3];           // tickets: box, cell scan, row scan
  int32_t error;
  uint32_t nodes, total;      // totals of the cell and row scans
  BondGrid grid;
};

// Device scratch of one bond build: one block of bond_scratch_words(n) words.
struct BondScratch {
  uint4* sorted;        // [n] in cell order: fixed-point position, node
  BondHead* head;
  uint32_t* cell;       // [cells + 1] nodes per cell, then their scan
  uint32_t* cell_tile;  // its tile sums
  uint32_t* poff;       // [n + 1] partners per node, then their scan
  uint32_t* poff_tile;
  uint32_t* key;        // [n] cell
  uint32_t* rank;       // [n] place in the cell
  uint32_t cells;       // capacity of the cell array
};

// Entries per tile of the bond builder's exclusive scan (1024 threads x 4 entries).
constexpr uint32_t BOND_SCAN_TILE = 4096;
// Grid cells of a bond build over n nodes, and scan tiles of a scan over len entries (both also
// usable where a scratch size must be known at compile time).
constexpr uint32_t bond_grid_cells_c(uint32_t n) { return 4u * n + 64u; }
constexpr uint32_t bond_scan_tiles_c(uint32_t len) { return ((len ? len : 1u) + BOND_SCAN_TILE - 1u) / BOND_SCAN_TILE; }

constexpr size_t BOND_HEAD_WORDS = 64;
static_assert(sizeof(BondHead) <= BOND_HEAD_WORDS * 4, "bond head");
constexpr size_t bond_scratch_words(uint32_t n) {
  return (size_t)n * 7 + BOND_HEAD_WORDS + bond_grid_cells_c(n) + 2 + bond_scan_tiles_c(bond_grid_cells_c(n) + 1) +
         bond_scan_tiles_c(n + 1);
}
// The arrays of a build over n nodes in a block of bond_scratch_words(n) words on a 16-byte boundary.
BondScratch bond_scratch(uint32_t* base, uint32_t n);
// Exclusive scan of in[0..len) into out[0..len], out[len] = total, on stream st. tile_sum holds
// bond_scan_tiles(len) words; *done must be 0 (and is 0 again when the scan ends).
cudaError_t scan_u32_dev(const uint32_t* in, uint32_t len, uint32_t* out, uint32_t* tile_sum, uint32_t* done,
                         cudaStream_t st);
uint32_t bond_scan_tiles(uint32_t len);
// The kept scratch, held while the object lives: base is null if n is too large for it, another call
// has it, or it cannot be had on this device.
struct KeptBondScratch {
  uint32_t* base = nullptr;
  explicit KeptBondScratch(uint32_t n);
  ~KeptBondScratch();
  KeptBondScratch(const KeptBondScratch&) = delete;
  KeptBondScratch& operator=(const KeptBondScratch&) = delete;
};
int run_bond_build(const double* pos, uint32_t n, uint32_t dim, double delta, uint32_t* pairs, uint64_t capacity,
                   uint64_t* n_pairs, cudaStream_t st, const BondScratch& S, std::string* err);

}  // namespace pg
