// pd_tile.cu -- the arrays of the tiled bond kernel (k_bond32t, pd_fp32c.cu), built on the device
// from the SELL column entries: per tile of kTileNodes nodes the ascending list of the distinct
// node records its bonds read, and every bond's place in that list. Integer work only, once per
// handle: a tile's partners are collected in a hash table in shared memory, its entries sorted, and
// every column entry looked up in the sorted list.
#include <cuda_runtime.h>

#include "pd_engine.h"

namespace pdg {

namespace {

constexpr uint32_t kHash = 8192;  // table slots (at most kTileRecords + kTileNodes are taken)
constexpr uint32_t kList = 4096;  // kTileRecords rounded up to a power of two
constexpr int kThreads = 256;
constexpr uint32_t kEmpty = 0xFFFFFFFFu;
static_assert(kTileRecords <= kList && kTileRecords * 16 <= 65536, "places are 12 bits");

// One block per tile. Shared: the hash table, then the list.
__global__ void __launch_bounds__(kThreads) k_tile_build(const __grid_constant__ DevView v, uint32_t *tile_rec,
                                                         uint32_t *tile_n, uint16_t *tcol) {
  extern __shared__ uint32_t sh[];
  uint32_t *table = sh, *list = sh + kHash;
  __shared__ uint32_t distinct, filled;
  const uint64_t s0 = (uint64_t)blockIdx.x * (kTileNodes / 32);
  const uint64_t s1 = min(s0 + kTileNodes / 32, (v.N + 31) / 32);
  const uint64_t e0 = v.slice_ptr[s0], e1 = v.slice_ptr[s1];
  for (uint32_t i = threadIdx.x; i < kHash; i += kThreads) table[i] = kEmpty;
  for (uint32_t i = threadIdx.x; i < kList; i += kThreads) list[i] = kEmpty;
  if (threadIdx.x == 0) distinct = filled = 0;
  __syncthreads();
  for (uint64_t e = e0 + threadIdx.x; e < e1; e += kThreads) {
    const uint32_t c = v.col[e];
    if (c == kNoCol) continue;
    const uint32_t q = c & kColIndex;
    uint32_t at = (q * 0x9E3779B1u) >> 19;  // 13 bits
    while (*(volatile uint32_t *)&distinct <= kTileRecords) {  // the table cannot fill up
      const uint32_t was = atomicCAS(&table[at], kEmpty, q);
      if (was == kEmpty) atomicAdd(&distinct, 1u);
      if (was == kEmpty || was == q) break;
      at = (at + 1) & (kHash - 1);
    }
  }
  __syncthreads();
  const uint32_t cnt = distinct;
  if (cnt == 0 || cnt > kTileRecords) {  // no bonds, or too many records: the tile gathers globally
    if (threadIdx.x == 0) tile_n[blockIdx.x] = 0;
    for (uint64_t e = e0 + threadIdx.x; e < e1; e += kThreads) tcol[e] = kTileBroken;
    return;
  }
  for (uint32_t i = threadIdx.x; i < kHash; i += kThreads)
    if (table[i] != kEmpty) list[atomicAdd(&filled, 1u)] = table[i];
  __syncthreads();
  uint32_t n2 = 2;
  while (n2 < cnt) n2 <<= 1;
  for (uint32_t len = 2; len <= n2; len <<= 1)  // bitonic sort, ascending
    for (uint32_t d = len >> 1; d > 0; d >>= 1) {
      for (uint32_t i = threadIdx.x; i < n2 / 2; i += kThreads) {
        const uint32_t a = 2 * i - (i & (d - 1)), b = a + d;
        const uint32_t x = list[a], y = list[b];
        if ((x > y) == ((a & len) == 0)) {
          list[a] = y;
          list[b] = x;
        }
      }
      __syncthreads();
    }
  for (uint32_t i = threadIdx.x; i < cnt; i += kThreads) tile_rec[(uint64_t)blockIdx.x * kTileRecords + i] = list[i];
  if (threadIdx.x == 0) tile_n[blockIdx.x] = cnt;
  for (uint64_t s = s0; s < s1; ++s) {
    const uint64_t b = v.slice_ptr[s], w = v.slice_ptr[s + 1] - b;
    for (uint64_t i = threadIdx.x; i < w; i += kThreads) {
      const uint32_t c = v.col[b + i], lane = (uint32_t)(i & 31), j = (uint32_t)(i >> 5);
      uint16_t t = kTileBroken;
      if (c != kNoCol) {
        const uint32_t q = c & kColIndex;
        uint32_t lo = 0, hi = cnt;
        while (hi - lo > 1) {
          const uint32_t mid = (lo + hi) >> 1;
          if (list[mid] <= q) lo = mid;
          else hi = mid;
        }
        t = (uint16_t)((lo << 4) | ((c & kColBroken) ? kTileBroken : 0));
      }
      tcol[b + 128ull * (j >> 2) + 4ull * lane + (j & 3u)] = t;
    }
  }
}

}  // namespace

cudaError_t launch_tile_build(const DevView &v, uint32_t *tile_rec, uint32_t *tile_n, uint16_t *tcol, cudaStream_t s) {
  constexpr int bytes = (kHash + kList) * 4;
  const cudaError_t e = cudaFuncSetAttribute(k_tile_build, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e != cudaSuccess) return e;
  const uint64_t nt = (v.N + kTileNodes - 1) / kTileNodes;
  if (nt) k_tile_build<<<(unsigned)nt, kThreads, bytes, s>>>(v, tile_rec, tile_n, tcol);
  return cudaGetLastError();
}

}  // namespace pdg
