// cell_sort.cuh -- stable counting sort of particles by hash cell, and the
// cell table: the B200 replacement of thrust::stable_sort_by_key and
// Kernel_SpatialDecomp_BinData in the reference
// (Collision_Detection_BroadPhase.cuh:110-117, 126-325).  A stable sort has
// one result, so the order equals the reference's bit for bit.
//
// Four passes over the particles' keys, between the caller's own kernels:
//   count   (in the caller's key kernel, cell_count): every particle's
//           arrival number in its cell, the members per cell and per tile of
//           kTileCells cells
//   scan    (k_cell_scan) a block per tile (or some): the members of the tiles
//           before it, then the exclusive scan of its own cells -> start[]; the
//           counts are zeroed for the next sort as they are read
//   place   (k_cell_place) member[start[cell] + arrival] = particle: the
//           cells' members together, in arrival order
//   move    (in the caller's gather kernel, cell_dest): a particle's rank is
//           the number of members of its cell with a lower index
// The rank makes the order independent of the order in which the atomics
// arrived.  It costs a cell's population squared, a 27th of what the
// neighbour search over the same cells costs.  Particles without a cell
// (outside the grid, or parked) go behind the others in index order by a
// scan of the blocks' counts, since they can be any number.
//
// start[] is defined for empty cells too (a lower bound), so the particles of
// consecutive cells [a, b] are [start[a], start[b + 1]): the neighbour search
// reads a row of three cells with two loads.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace blaze {

constexpr int kSortThreads = 256;          // threads per block of the count and move kernels
constexpr int kScanThreads = 512;
constexpr int kScanItems = 8;
constexpr int kTileCells = kScanThreads * kScanItems;
constexpr uint32_t kScanBlocks = 2048;

struct CellSort {
  uint32_t* key;      // per particle: its cell; ncell: outside the grid, ncell + 1: parked
  uint32_t* slot;     // per particle: arrival number in its cell
  int32_t* member;    // the cells' members, cell by cell, in arrival order
  int32_t* perm;      // sorted position -> particle before the sort (null: not wanted)
  uint32_t* cnt;      // cell_tiles(ncell) * kTileCells, zero between sorts
  uint32_t* start;    // the same size; entries 0 .. ncell are the cell table
  uint32_t* tile;     // cell_tiles(ncell) + 1, zero between sorts; the last: any particle without a cell
  uint32_t* spec;     // 2 per block of kSortThreads particles: outside, parked
  uint32_t ncell;
};

// the tiles that hold entries 0 .. ncell
__host__ __device__ constexpr uint32_t cell_tiles(uint32_t ncell) { return ncell / kTileCells + 1u; }
__host__ __device__ constexpr int sort_blocks(int n) { return (n + kSortThreads - 1) / kSortThreads; }

// Count pass of particle i (block of kSortThreads threads, every thread
// calls it; valid: i < n).
__device__ __forceinline__ void cell_count(const CellSort& c, int i, bool valid, uint32_t key) {
  const bool in = valid && key < c.ncell;
  if (valid) c.key[i] = key;
  if (in) c.slot[i] = atomicAdd(c.cnt + key, 1u);
  // neighbours in memory are neighbours in space: mostly one tile per warp
  const uint32_t t = in ? key / (uint32_t)kTileCells : 0xffffffffu;
  const unsigned peers = __match_any_sync(0xffffffffu, t);
  if (in && (int)(threadIdx.x & 31) == __ffs(peers) - 1)
    atomicAdd(c.tile + t, (uint32_t)__popc(peers));
  const int outside = __syncthreads_count(valid && key == c.ncell);
  const int parked = __syncthreads_count(valid && key > c.ncell);
  if (threadIdx.x == 0) {
    c.spec[2 * blockIdx.x] = (uint32_t)outside;
    c.spec[2 * blockIdx.x + 1] = (uint32_t)parked;
    if (outside | parked) c.tile[cell_tiles(c.ncell)] = 1u;
  }
}

// The sorted position of particle i (every thread of the block calls it,
// blocks as in the count pass).
__device__ __forceinline__ int cell_dest(const CellSort& c, int i, bool valid) {
  const uint32_t key = valid ? c.key[i] : 0u;
  const bool in = valid && key < c.ncell;
  int dst = 0;
  if (in) {
    const uint32_t s = c.start[key], e = c.start[key + 1];
    uint32_t rank = 0;
    for (uint32_t q = s; q < e; ++q) rank += c.member[q] < i ? 1u : 0u;
    dst = (int)(s + rank);
  }
  if (__syncthreads_or(valid && !in)) {
    // behind the cells, by block and then by thread
    __shared__ uint32_t s_out[kSortThreads / 32], s_park[kSortThreads / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const bool park = valid && key > c.ncell;
    const unsigned mo = __ballot_sync(0xffffffffu, valid && key == c.ncell);
    const unsigned mp = __ballot_sync(0xffffffffu, park);
    if (lane == 0) {
      s_out[w] = (uint32_t)__popc(mo);
      s_park[w] = (uint32_t)__popc(mp);
    }
    __syncthreads();
    if (valid && !in) {
      uint32_t r = c.spec[2 * blockIdx.x + (park ? 1 : 0)] +
                   (uint32_t)__popc((park ? mp : mo) & ((1u << lane) - 1u));
      for (int q = 0; q < w; ++q) r += park ? s_park[q] : s_out[q];
      dst = (int)r;
    }
  }
  if (valid && c.perm) c.perm[dst] = i;
  return dst;
}

// The scan and place passes over n particles; *epoch (may be null) is
// incremented and *clear (may be null) set to 0.  `gate` (may be null): when
// non-null and *gate == 0 every kernel returns at once, so the launch
// sequence can stay fixed while the work is skipped.
void cell_scan_place(const CellSort& c, int n, int* epoch, int* clear, const int* gate,
                     cudaStream_t stream);
constexpr int kCellSortKernels = 2;

}  // namespace blaze
