// cell_sort.cu -- see cell_sort.cuh.
#include "cell_sort.cuh"

namespace blaze {

namespace {

// Exclusive scan of v over the block; the block's sum in total.
__device__ __forceinline__ uint32_t block_scan(uint32_t v, uint32_t* sh, uint32_t& total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) sh[w] = x;
  __syncthreads();
  uint32_t before = 0, sum = 0;
#pragma unroll
  for (int q = 0; q < kScanThreads / 32; ++q) {
    const uint32_t t = sh[q];
    if (q < w) before += t;
    sum += t;
  }
  __syncthreads();
  total = sum;
  return before + x - v;
}

// Members of the tiles [0, t).
__device__ __forceinline__ uint32_t tiles_before(const uint32_t* tile, uint32_t t, uint32_t* sh) {
  uint32_t s = 0;
  for (uint32_t q = threadIdx.x; q < t; q += kScanThreads) s += tile[q];
  uint32_t total;
  block_scan(s, sh, total);
  return total;
}

// A block per `chunk` tiles of cells, and a last one for the particles without a
// cell: their blocks' counts become positions.
__global__ void __launch_bounds__(kScanThreads)
k_cell_scan(CellSort c, int nblocks, uint32_t chunk, int* clear, const int* gate) {
  if (gate != nullptr && *gate == 0) return;
  if (clear && blockIdx.x == 0 && threadIdx.x == 0) *clear = 0;
  __shared__ uint32_t sh[kScanThreads / 32];
  const uint32_t tiles = cell_tiles(c.ncell);
  const uint32_t first = blockIdx.x * chunk;
  if (first < tiles) {
    uint32_t run = tiles_before(c.tile, first, sh);
    for (uint32_t t = first; t < min(first + chunk, tiles); ++t) {
      uint4* cnt = reinterpret_cast<uint4*>(c.cnt + (size_t)t * kTileCells) + 2 * threadIdx.x;
      uint4* start = reinterpret_cast<uint4*>(c.start + (size_t)t * kTileCells);
      if (c.tile[t] == 0u) {   // no members: no counts to read or zero
        start[threadIdx.x] = make_uint4(run, run, run, run);
        start[threadIdx.x + kScanThreads] = make_uint4(run, run, run, run);
        continue;
      }
      start += 2 * threadIdx.x;
      const uint4 a = cnt[0], b = cnt[1];
      const uint32_t sum = a.x + a.y + a.z + a.w + b.x + b.y + b.z + b.w;
      uint32_t total;
      const uint32_t at = run + block_scan(sum, sh, total);
      run += total;
      uint4 sa, sb;
      sa.x = at;
      sa.y = sa.x + a.x;
      sa.z = sa.y + a.y;
      sa.w = sa.z + a.z;
      sb.x = sa.w + a.w;
      sb.y = sb.x + b.x;
      sb.z = sb.y + b.y;
      sb.w = sb.z + b.z;
      start[0] = sa;
      start[1] = sb;
      if (sum) {
        const uint4 z = make_uint4(0u, 0u, 0u, 0u);
        cnt[0] = z;
        cnt[1] = z;
      }
    }
    return;
  }
  if (c.tile[tiles] == 0u) return;
  uint32_t run = tiles_before(c.tile, tiles, sh);
  for (int kind = 0; kind < 2; ++kind)
    for (int b0 = 0; b0 < nblocks; b0 += kScanThreads) {
      const int b = b0 + (int)threadIdx.x;
      const uint32_t v = b < nblocks ? c.spec[2 * b + kind] : 0u;
      uint32_t total;
      const uint32_t x = block_scan(v, sh, total);
      if (b < nblocks) c.spec[2 * b + kind] = run + x;
      run += total;
    }
}

__global__ void __launch_bounds__(kSortThreads)
k_cell_place(CellSort c, int n, int* epoch, const int* gate) {
  if (gate != nullptr && *gate == 0) return;
  const int i = blockIdx.x * kSortThreads + threadIdx.x;
  if (i == 0 && epoch) *epoch += 1;
  // the scan has read the tiles' counts: zero for the next sort
  const uint32_t words = cell_tiles(c.ncell) + 1u;
  for (uint32_t q = (uint32_t)i; q < words; q += gridDim.x * kSortThreads) c.tile[q] = 0u;
  if (i >= n) return;
  const uint32_t key = c.key[i];
  if (key < c.ncell) c.member[c.start[key] + c.slot[i]] = i;
}

}  // namespace

void cell_scan_place(const CellSort& c, int n, int* epoch, int* clear, const int* gate,
                     cudaStream_t stream) {
  const int nb = sort_blocks(n);
  // Up to kScanBlocks tiles a block each; a larger grid's blocks take several in
  // a row, which saves adding up the tiles before each and the blocks themselves:
  // a step of 10,000 particles in 104 million cells 227 -> 91 us, in 343 million
  // 1001 -> 231.
  const uint32_t tiles = cell_tiles(c.ncell), chunk = (tiles + kScanBlocks - 1u) / kScanBlocks;
  k_cell_scan<<<(tiles + chunk - 1u) / chunk + 1u, kScanThreads, 0, stream>>>(c, nb, chunk, clear,
                                                                           gate);
  k_cell_place<<<nb, kSortThreads, 0, stream>>>(c, n, epoch, gate);
}

}  // namespace blaze
