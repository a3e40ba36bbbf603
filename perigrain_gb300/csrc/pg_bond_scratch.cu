// Scratch that pg_build_bonds keeps: one device array, big enough for a grain of KEPT_NODES nodes
// (11.6 MB, taken when the first build on a GPU loads this file's module, given back with the
// context). Allocating and freeing the scratch on each call costs 105 us in a process that also runs
// torch, and about 130 us with the wait that the free implies: 100 nodes 220 -> 63 us a call, 200k
// nodes 244 -> 115 us. Above KEPT_NODES a build takes its own memory: there the passes are most of
// the call.
//
// One call at a time holds the array, from before its first pass until its stream has completed; a
// call that finds it taken (another host thread, any device) allocates as a larger one does, so
// calls on several threads and streams run side by side. Each call clears what it needs zeroed. The
// address is asked for on each call and not kept: it is the current device's, and after a reset of
// the device the reloaded module's.
#include <cuda_runtime.h>

#include <mutex>

#include "pg_bonds.h"

namespace pg {

namespace {
constexpr uint32_t KEPT_NODES = 1u << 18;
constexpr size_t KEPT_WORDS = bond_scratch_words(KEPT_NODES);
__device__ __align__(256) uint32_t g_kept[KEPT_WORDS];
std::mutex g_kept_lock;
}  // namespace

KeptBondScratch::KeptBondScratch(uint32_t n) {
  if (n > KEPT_NODES || !g_kept_lock.try_lock()) return;
  if (cudaGetSymbolAddress((void**)&base, g_kept) != cudaSuccess) {
    cudaGetLastError();  // the caller allocates instead
    base = nullptr;
    g_kept_lock.unlock();
  }
}

KeptBondScratch::~KeptBondScratch() {
  if (base) g_kept_lock.unlock();
}

}  // namespace pg
