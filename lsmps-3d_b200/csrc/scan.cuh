// scan.cuh - block-level pieces of the exclusive scans (scan.cu: counts to
// offsets; cells.cu: cell counts to cell ranges).  Sums are carried in 64 bits.
#pragma once

#include "common.cuh"

namespace lsmps {

constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;
// A set of at most this many values is scanned by one block of 1,024 threads.
constexpr int kSmallScan = 8192;
constexpr int kSmallScanThreads = 1024;
// Up to this many tiles every block of the second kernel adds the tiles before
// its own itself; above, a kernel between the two scans them.
constexpr int kDirectTiles = 4096;

__device__ __forceinline__ long long warp_inclusive(long long x) {
  const int lane = threadIdx.x & (kWarp - 1);
#pragma unroll
  for (int o = 1; o < kWarp; o <<= 1) {
    const long long y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  return x;
}

// Sum over a block of up to 1,024 threads, in every thread.
__device__ __forceinline__ long long block_total(long long v) {
  __shared__ long long warp_sum[kWarp];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & (kWarp - 1)) == 0) warp_sum[threadIdx.x / kWarp] = v;
  __syncthreads();
  long long t = 0;
  for (int w = 0; w < static_cast<int>(blockDim.x) / kWarp; ++w) t += warp_sum[w];
  return t;
}

// One block of kSmallScanThreads: store(i, sum of load(0 .. i - 1), load(i)) for
// i < n (n <= kSmallScan); returns the grand total in every thread.  Each warp
// takes a contiguous stretch, 32 values a round.
template <typename Load, typename Store>
__device__ __forceinline__ long long scan_small(int n, Load load, Store store) {
  constexpr int kRounds = kSmallScan / kSmallScanThreads;
  __shared__ long long warp_sum[kWarp];
  const int lane = threadIdx.x & (kWarp - 1), warp = threadIdx.x / kWarp;
  const int rounds = (n + kSmallScanThreads - 1) / kSmallScanThreads;
  const int first = warp * rounds * kWarp + lane;
  index_t v[kRounds];
  long long sum = 0;
#pragma unroll
  for (int r = 0; r < kRounds; ++r) {
    const int i = first + r * kWarp;
    v[r] = r < rounds && i < n ? load(i) : 0;
    sum += v[r];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if (lane == 0) warp_sum[warp] = sum;
  __syncthreads();
  const long long mine = warp_sum[lane];
  const long long upto = warp_inclusive(mine);
  long long before = __shfl_sync(0xffffffffu, upto - mine, warp);
  const long long total = __shfl_sync(0xffffffffu, upto, kWarp - 1);
#pragma unroll
  for (int r = 0; r < kRounds; ++r) {
    if (r >= rounds) break;
    const int i = first + r * kWarp;
    const long long x = warp_inclusive(v[r]);
    if (i < n) store(i, before + x - v[r], v[r]);
    before += __shfl_sync(0xffffffffu, x, kWarp - 1);
  }
  return total;
}

// Tile blockIdx.x's sum of load(i) (kScanThreads threads), in thread 0.
template <typename Load>
__device__ __forceinline__ long long tile_sum(size_t n, Load load) {
  const size_t base = static_cast<size_t>(blockIdx.x) * kScanTile;
  long long sum = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    const size_t i = base + static_cast<size_t>(k) * kScanThreads + threadIdx.x;
    if (i < n) sum += load(i);
  }
  return block_total(sum);
}

// The sum of the tiles before tile blockIdx.x: of their totals, or (scanned)
// as the kernel between left it.
__device__ __forceinline__ long long before_tile(const long long* __restrict__ partials, bool scanned) {
  if (scanned) return partials[blockIdx.x];
  long long sum = 0;
  for (int b = threadIdx.x; b < static_cast<int>(blockIdx.x); b += kScanThreads) sum += partials[b];
  return block_total(sum);
}

// store(i, sum of all values before i, load(i)) for tile blockIdx.x, given the
// sum before the tile; returns that sum plus the tile's.
template <typename Load, typename Store>
__device__ __forceinline__ long long scan_tile(size_t n, long long before, Load load, Store store) {
  __shared__ long long warp_sum[kScanThreads / kWarp];
  const size_t base = static_cast<size_t>(blockIdx.x) * kScanTile + static_cast<size_t>(threadIdx.x) * kScanItems;
  long long v[kScanItems];
  long long local = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    v[k] = base + k < n ? load(base + k) : 0;
    local += v[k];
  }
  const int lane = threadIdx.x & (kWarp - 1), warp = threadIdx.x / kWarp;
  const long long x = warp_inclusive(local);
  if (lane == kWarp - 1) warp_sum[warp] = x;
  __syncthreads();
  long long at = before + x - local, total = before;
  for (int w = 0; w < kScanThreads / kWarp; ++w) {
    if (w < warp) at += warp_sum[w];
    total += warp_sum[w];
  }
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    if (base + k < n) store(base + k, at, static_cast<index_t>(v[k]));
    at += v[k];
  }
  return total;
}

// Scans the tile totals in place (one block), for sets of more than
// kDirectTiles tiles.
__global__ void __launch_bounds__(1024) scan_partials_kernel(long long* __restrict__ partials, int count);

}  // namespace lsmps
