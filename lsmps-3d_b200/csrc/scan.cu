// scan.cu - device-wide exclusive scan of int32 counts (no inter-block
// waiting).  One block scans a small set in one launch; otherwise one kernel
// adds up the tiles and a second one scans them, each of its blocks first adding
// the tiles before its own (with a kernel between the two for very large sets).
// Sums are carried in 64 bits so an overflow of the 32-bit index type is detected
// instead of wrapping.
#include <climits>

#include "scan.cuh"

namespace lsmps {

__global__ void __launch_bounds__(1024) scan_partials_kernel(long long* __restrict__ partials, int count) {
  wait_for_previous();
  __shared__ long long warp_sum[32];
  __shared__ long long carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int base = 0; base < count; base += blockDim.x) {
    const int i = base + threadIdx.x;
    const long long v = i < count ? partials[i] : 0;
    const long long x = warp_inclusive(v);
    if (lane == 31) warp_sum[warp] = x;
    __syncthreads();
    if (warp == 0) warp_sum[lane] = warp_inclusive(warp_sum[lane]);
    __syncthreads();
    const long long before = carry + (warp > 0 ? warp_sum[warp - 1] : 0) + x - v;
    if (i < count) partials[i] = before;
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) carry = before + v;
    __syncthreads();
  }
}

namespace {

// out[i] clamped to the index range, flagging an overflow.
__device__ __forceinline__ void store_offset(index_t* out, size_t i, long long v, DeviceStatus* status) {
  if (v > INT_MAX) raise_flag(status, kFlagIndexOverflow);
  out[i] = static_cast<index_t>(v > INT_MAX ? INT_MAX : v);
}

__device__ __forceinline__ void store_total(long long v, unsigned long long* total, index_t* total_i32,
                                            DeviceStatus* status) {
  if (total) *total = static_cast<unsigned long long>(v);
  if (total_i32) store_offset(total_i32, 0, v, status);
}

// Up to two sets of the same length, blockIdx.y the set (in may be out).
struct ScanSets {
  ScanSet t[2];
};

__global__ void __launch_bounds__(kSmallScanThreads) scan_small_kernel(const __grid_constant__ ScanSets sets, int n,
                                                                       DeviceStatus* status) {
  wait_for_previous();
  const ScanSet& a = sets.t[blockIdx.y];
  const long long sum =
      scan_small(n, [&](int i) { return a.in[i]; },
                 [&](int i, long long before, index_t) { store_offset(a.out, i, before, status); });
  if (threadIdx.x == 0) store_total(sum, a.total, a.total_i32, status);
}

__global__ void __launch_bounds__(kScanThreads) scan_reduce_kernel(const __grid_constant__ ScanSets sets, size_t n,
                                                                   long long* __restrict__ partials) {
  wait_for_previous();
  const ScanSet& a = sets.t[blockIdx.y];
  const long long t = tile_sum(n, [&](size_t i) { return a.in[i]; });
  if (threadIdx.x == 0) partials[static_cast<size_t>(blockIdx.y) * gridDim.x + blockIdx.x] = t;
}

__global__ void __launch_bounds__(kScanThreads) scan_down_kernel(const __grid_constant__ ScanSets sets, size_t n,
                                                                 const long long* __restrict__ partials, int scanned,
                                                                 DeviceStatus* status) {
  wait_for_previous();
  const ScanSet& a = sets.t[blockIdx.y];
  const long long end =
      scan_tile(n, before_tile(partials + static_cast<size_t>(blockIdx.y) * gridDim.x, scanned != 0),
                [&](size_t i) { return a.in[i]; },
                [&](size_t i, long long before, index_t) { store_offset(a.out, i, before, status); });
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) store_total(end, a.total, a.total_i32, status);
}

}  // namespace

size_t scan_scratch_bytes(size_t n) {
  const size_t tiles = (n + kScanTile - 1) / kScanTile + 1;
  return tiles * sizeof(long long) + 512;
}

// One block takes 13 us for 21,793 counts and 4 for 1,000, two kernels 2 x 3; three kernels,
// the middle one scanning the tiles' totals, took 3 x 3.5 for any size.
lsmps_status exclusive_scans_i32(lsmps_ctx* ctx, Scratch& scratch, const ScanSet* sets, int count, size_t n) {
  ScanSets a{};
  for (int k = 0; k < count; ++k) a.t[k] = sets[k];
  if (n <= static_cast<size_t>(kSmallScan)) {
    launch(ctx, scan_small_kernel, dim3(1, count), dim3(kSmallScanThreads), 0, a, static_cast<int>(n), ctx->d_status);
    return check_launch(ctx, "exclusive scan");
  }
  const int tiles = div_up(static_cast<long long>(n), kScanTile);
  long long* partials = scratch.take<long long>(static_cast<size_t>(count) * tiles);
  if (!partials) return fail(ctx, LSMPS_CUDA_ERROR, "scan scratch exhausted");
  launch(ctx, scan_reduce_kernel, dim3(tiles, count), dim3(kScanThreads), 0, a, n, partials);
  const bool between = tiles > kDirectTiles;
  for (int k = 0; between && k < count; ++k)
    launch(ctx, scan_partials_kernel, dim3(1), dim3(1024), 0, partials + static_cast<size_t>(k) * tiles, tiles);
  launch(ctx, scan_down_kernel, dim3(tiles, count), dim3(kScanThreads), 0, a, n,
         static_cast<const long long*>(partials), between ? 1 : 0, ctx->d_status);
  return check_launch(ctx, "exclusive scan");
}

lsmps_status exclusive_scan_i32(lsmps_ctx* ctx, Scratch& scratch, const index_t* in, index_t* out, size_t n,
                                unsigned long long* total, index_t* total_i32) {
  const ScanSet set{in, out, total, total_i32};
  return exclusive_scans_i32(ctx, scratch, &set, 1, n);
}

}  // namespace lsmps
