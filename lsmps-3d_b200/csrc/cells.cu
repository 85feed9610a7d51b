// cells.cu - cell lists of one or two particle sets: each set's particles by
// cell, ascending index inside a cell, and every cell's range.  Replaces
// build_cell_list_impl of src/neighbor/neighbor_search.cu:255-292, whose Thrust
// sort_by_key of (cell id, particle index) is stable, so that cell_ids /
// sorted_indices / cell_begin / cell_end are identical to the reference's.
//
// A counting sort, both sets in the same launches: every particle takes a
// number in its cell (in no particular order), the cells' counts are scanned
// into ranges, the particles are put there by number, and each cell's few
// particles are then ordered by index.  No block waits on another.  The
// radix-sort kernels at the end of the kernels' list are those of the
// allocation-free entry point (cells_noalloc.cu).
#include <climits>
#include <cmath>

#include "cells.cuh"
#include "scan.cuh"

namespace lsmps {
namespace {

// clamp_cell_index, neighbor_search.cu:36-46, with the float-to-int
// conversion of an out-of-range or NaN value made explicit.
__device__ __forceinline__ index_t cell_coord(double coordinate, double origin, double cell_size, index_t dim,
                                              bool& bad) {
  const double scaled = (coordinate - origin) / cell_size;
  if (!(scaled == scaled) || isinf(scaled)) {
    bad = true;
    return 0;
  }
  const double f = floor(scaled);
  if (f < 0.0) return 0;
  if (f >= static_cast<double>(dim)) return dim - 1;
  return static_cast<index_t>(f);
}

}  // namespace

// assign_cells_kernel (neighbor_search.cu:61-73) fused with the cell-range
// reset of reset_cell_ranges_kernel (:75-83).
__global__ void hash_kernel(const double* __restrict__ x, const double* __restrict__ y,
                            const double* __restrict__ z, index_t n, lsmps_grid grid,
                            index_t* __restrict__ keys, index_t* __restrict__ vals,
                            index_t* __restrict__ cell_begin, index_t* __restrict__ cell_end, index_t ncell,
                            DeviceStatus* __restrict__ status) {
  wait_for_previous();
  const index_t total = n > ncell ? n : ncell;
  for (index_t t = blockIdx.x * blockDim.x + threadIdx.x; t < total; t += gridDim.x * blockDim.x) {
    if (t < ncell) {
      cell_begin[t] = -1;
      cell_end[t] = -1;
    }
    if (t < n) {
      bool bad = false;
      const index_t ix = cell_coord(x[t], grid.origin[0], grid.cell_size, grid.dims[0], bad);
      const index_t iy = cell_coord(y[t], grid.origin[1], grid.cell_size, grid.dims[1], bad);
      const index_t iz = cell_coord(z[t], grid.origin[2], grid.cell_size, grid.dims[2], bad);
      if (bad) raise_flag(status, kFlagNonFinite);
      keys[t] = (iz * grid.dims[1] + iy) * grid.dims[0] + ix;  // flatten_cell, :32-34
      vals[t] = t;
    }
  }
}

// Per-tile histogram of one digit, stored digit-major: hist[d * tiles + tile].
__global__ void __launch_bounds__(kSortThreads) radix_hist_kernel(const index_t* __restrict__ keys, index_t n,
                                                                  int shift, index_t* __restrict__ hist,
                                                                  int tiles) {
  wait_for_previous();
  __shared__ unsigned int bins[kRadixBins];
  bins[threadIdx.x] = 0;
  __syncthreads();
  const size_t base = static_cast<size_t>(blockIdx.x) * kSortTile;
#pragma unroll 4
  for (int k = 0; k < kSortItems; ++k) {
    const size_t i = base + static_cast<size_t>(k) * kSortThreads + threadIdx.x;
    if (i < static_cast<size_t>(n)) atomicAdd(&bins[(keys[i] >> shift) & (kRadixBins - 1)], 1u);
  }
  __syncthreads();
  hist[static_cast<size_t>(threadIdx.x) * tiles + blockIdx.x] = static_cast<index_t>(bins[threadIdx.x]);
}

// Stable scatter of one digit.  The tile is walked in rounds of kSortThreads
// consecutive keys; inside a round, keys are ordered by warp then lane, so
// rank = tile base of the digit + keys of that digit in earlier rounds +
// keys in earlier warps of this round + lower lanes of this warp.
__global__ void __launch_bounds__(kSortThreads) radix_scatter_kernel(
    const index_t* __restrict__ keys_in, const index_t* __restrict__ vals_in, index_t* __restrict__ keys_out,
    index_t* __restrict__ vals_out, index_t n, int shift, const index_t* __restrict__ hist_scanned, int tiles) {
  wait_for_previous();
  __shared__ unsigned int base[kRadixBins];
  __shared__ unsigned int warp_count[kSortWarps][kRadixBins];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  base[threadIdx.x] = static_cast<unsigned int>(hist_scanned[static_cast<size_t>(threadIdx.x) * tiles + blockIdx.x]);
  const unsigned lanemask_lt = (1u << lane) - 1u;
  const size_t tile_base = static_cast<size_t>(blockIdx.x) * kSortTile;
  for (int r = 0; r < kSortItems; ++r) {
    // Each warp clears its own counters for this round.
#pragma unroll
    for (int b = lane; b < kRadixBins; b += kWarp) warp_count[warp][b] = 0;
    __syncwarp();
    const size_t i = tile_base + static_cast<size_t>(r) * kSortThreads + threadIdx.x;
    const bool valid = i < static_cast<size_t>(n);
    index_t key = 0, val = 0;
    int digit = kRadixBins;  // invalid lanes form their own group
    if (valid) {
      key = keys_in[i];
      val = vals_in[i];
      digit = (key >> shift) & (kRadixBins - 1);
    }
    const unsigned peers = __match_any_sync(0xffffffffu, digit);
    const unsigned rank_in_warp = __popc(peers & lanemask_lt);
    if (valid && rank_in_warp == 0) warp_count[warp][digit] = __popc(peers);
    __syncthreads();
    {
      // Thread t owns digit t: exclusive prefix over the warps of this round.
      unsigned running = base[threadIdx.x];
#pragma unroll
      for (int w = 0; w < kSortWarps; ++w) {
        const unsigned c = warp_count[w][threadIdx.x];
        warp_count[w][threadIdx.x] = running;
        running += c;
      }
      base[threadIdx.x] = running;
    }
    __syncthreads();
    if (valid) {
      const unsigned pos = warp_count[warp][digit] + rank_in_warp;
      keys_out[pos] = key;
      vals_out[pos] = val;
    }
    __syncthreads();
  }
}

// build_cell_ranges_kernel, neighbor_search.cu:85-98.
__global__ void ranges_kernel(const index_t* __restrict__ keys, index_t n, index_t* __restrict__ cell_begin,
                              index_t* __restrict__ cell_end) {
  wait_for_previous();
  for (index_t p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
    const index_t c = keys[p];
    if (p == 0 || keys[p - 1] != c) cell_begin[c] = p;
    if (p + 1 == n || keys[p + 1] != c) cell_end[c] = p + 1;
  }
}

namespace {

constexpr int kCellThreads = 256;

// One or two sets as one index range: set s's particles at first[s] .., its
// cells' counts at s * ncell ...
struct CellArgs {
  CellSet set[2];
  int sets;
  index_t first1;  // particles of set 0
  index_t total;   // of both
  lsmps_grid grid;
  index_t ncell;
  const BoxGrid* boxes;
  int nbox;
  index_t* key;     // [total] cell of each particle
  index_t* number;  // [total] its number in the cell
  index_t* count;   // [sets * ncell] particles per cell, then the cells' first positions
  index_t* placed;  // [total] particles by cell, unordered inside a cell
  DeviceStatus* status;
};

// assign_cells_kernel (neighbor_search.cu:61-73) of both sets, with the count
// of every cell.  In a merged batch a particle is hashed on the grid of the box
// whose range of its set holds it.
__global__ void __launch_bounds__(kCellThreads) cell_count_kernel(CellArgs a) {
  wait_for_previous();
  for (index_t p = blockIdx.x * kCellThreads + threadIdx.x; p < a.total; p += gridDim.x * kCellThreads) {
    const int s = p >= a.first1 ? 1 : 0;
    const CellSet& set = a.set[s];
    const index_t t = p - (s ? a.first1 : 0);
    double o[3] = {a.grid.origin[0], a.grid.origin[1], a.grid.origin[2]};
    index_t d[3] = {a.grid.dims[0], a.grid.dims[1], a.grid.dims[2]}, base = 0;
    if (a.boxes) {
      const BoxGrid& g = a.boxes[box_of(a.boxes, a.nbox, t, set.box_field)];
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        o[k] = g.origin[k];
        d[k] = g.dims[k];
      }
      base = g.cell_base;
    }
    bool bad = false;
    const index_t ix = cell_coord(set.x[t], o[0], a.grid.cell_size, d[0], bad);
    const index_t iy = cell_coord(set.y[t], o[1], a.grid.cell_size, d[1], bad);
    const index_t iz = cell_coord(set.z[t], o[2], a.grid.cell_size, d[2], bad);
    if (bad) raise_flag(a.status, kFlagNonFinite);
    const index_t key = base + (iz * d[1] + iy) * d[0] + ix;  // flatten_cell, :32-34
    a.key[p] = key;
    a.number[p] = atomicAdd(&a.count[static_cast<size_t>(s) * a.ncell + key], 1);
  }
}

// Cell c's range from its count and the sum of the counts before it (both
// sets' cells in one scan; set 1's positions start at 0 again).
__device__ __forceinline__ void store_range(const CellArgs& a, size_t c, long long before, index_t count) {
  const int s = c >= static_cast<size_t>(a.ncell) ? 1 : 0;
  const index_t first = static_cast<index_t>(before - (s ? a.first1 : 0));
  const size_t at = c - (s ? static_cast<size_t>(a.ncell) : 0);
  a.count[c] = first;
  a.set[s].begin[at] = count ? first : -1;
  a.set[s].end[at] = count ? first + count : -1;
}

__global__ void __launch_bounds__(kSmallScanThreads) cell_ranges_small_kernel(CellArgs a) {
  wait_for_previous();
  scan_small(
      a.sets * a.ncell, [&](int i) { return a.count[i]; },
      [&](int i, long long before, index_t v) { store_range(a, i, before, v); });
}

__global__ void __launch_bounds__(kScanThreads) cell_totals_kernel(CellArgs a, long long* __restrict__ partials) {
  wait_for_previous();
  const long long t = tile_sum(static_cast<size_t>(a.sets) * a.ncell, [&](size_t i) { return a.count[i]; });
  if (threadIdx.x == 0) partials[blockIdx.x] = t;
}

__global__ void __launch_bounds__(kScanThreads) cell_ranges_kernel(CellArgs a, const long long* __restrict__ partials,
                                                                  int scanned) {
  wait_for_previous();
  scan_tile(
      static_cast<size_t>(a.sets) * a.ncell, before_tile(partials, scanned != 0), [&](size_t i) { return a.count[i]; },
      [&](size_t i, long long before, index_t v) { store_range(a, i, before, v); });
}

__global__ void __launch_bounds__(kCellThreads) cell_place_kernel(CellArgs a) {
  wait_for_previous();
  for (index_t p = blockIdx.x * kCellThreads + threadIdx.x; p < a.total; p += gridDim.x * kCellThreads) {
    const int s = p >= a.first1 ? 1 : 0;
    const index_t first = s ? a.first1 : 0;
    a.placed[first + a.count[static_cast<size_t>(s) * a.ncell + a.key[p]] + a.number[p]] = p - first;
  }
}

// A cell of more particles than this is ordered by a walk over the whole set
// instead of by comparing its particles with one another.
constexpr index_t kManyInCell = 1024;

// Orders the particles of cell c of set s by index (one warp), writes its
// stretch of the sorted list and, where asked for, the sorted positions.
__device__ __forceinline__ void order_cell(const CellArgs& a, const CellSet& set, index_t first, index_t n, index_t c,
                                           index_t b, index_t e) {
  const int lane = threadIdx.x & (kWarp - 1);
  const index_t* __restrict__ placed = a.placed + first;
  const auto put = [&](index_t at, index_t i) {
    set.sorted[at] = i;
    set.ids[at] = c;
    if (set.pos) set.pos[at] = make_double4(set.x[i], set.y[i], set.z[i], 0.0);
  };
  const index_t many = e - b;
  if (many <= kWarp) {
    const index_t v = lane < many ? placed[b + lane] : INT_MAX;
    index_t rank = 0;
    for (index_t k = 0; k < many; ++k) rank += __shfl_sync(0xffffffffu, v, k) < v ? 1 : 0;
    if (lane < many) put(b + rank, v);
  } else if (many <= kManyInCell) {
    for (index_t k = b + lane; k < e; k += kWarp) {
      const index_t v = placed[k];
      index_t rank = 0;
      for (index_t q = b; q < e; ++q) rank += placed[q] < v ? 1 : 0;
      put(b + rank, v);
    }
  } else {
    index_t at = b;
    for (index_t k = 0; k < n; k += kWarp) {
      const bool mine = k + lane < n && a.key[first + k + lane] == c;
      const unsigned in = __ballot_sync(0xffffffffu, mine);
      if (mine) put(at + __popc(in & ((1u << lane) - 1u)), k + lane);
      at += __popc(in);
    }
  }
}

// Each warp orders the non-empty ones of `span` (1 .. 32) consecutive cells.
__global__ void __launch_bounds__(kCellThreads) cell_order_kernel(CellArgs a, int span) {
  wait_for_previous();
  const int lane = threadIdx.x & (kWarp - 1);
  const long long cells = static_cast<long long>(a.sets) * a.ncell;
  const long long warps = static_cast<long long>(gridDim.x) * (kCellThreads / kWarp);
  for (long long g = static_cast<long long>(blockIdx.x) * (kCellThreads / kWarp) + threadIdx.x / kWarp;
       g * span < cells; g += warps) {
    const long long c = g * span + lane;
    const bool mine = lane < span && c < cells;
    const int s = c >= a.ncell ? 1 : 0;
    const index_t at = static_cast<index_t>(c - (s ? a.ncell : 0));
    const index_t b = mine ? a.set[s].begin[at] : -1, e = mine ? a.set[s].end[at] : -1;
    for (unsigned rem = __ballot_sync(0xffffffffu, b >= 0); rem; rem &= rem - 1) {
      const int k = __ffs(rem) - 1;
      const int sk = __shfl_sync(0xffffffffu, s, k);
      const index_t ck = __shfl_sync(0xffffffffu, at, k), bk = __shfl_sync(0xffffffffu, b, k),
                    ek = __shfl_sync(0xffffffffu, e, k);
      order_cell(a, a.set[sk], sk ? a.first1 : 0, sk ? a.total - a.first1 : a.first1, ck, bk, ek);
    }
  }
}

}  // namespace

int key_bits(long long ncell) {
  int bits = 0;
  while ((1LL << bits) < ncell) ++bits;
  return bits;
}

lsmps_status validate_grid(lsmps_ctx* ctx, const lsmps_grid& grid) {
  if (!(grid.cell_size > 0.0) || grid.dims[0] <= 0 || grid.dims[1] <= 0 || grid.dims[2] <= 0)
    return fail(ctx, LSMPS_INVALID_ARGUMENT, "Invalid cell grid configuration");
  const long long ncell = static_cast<long long>(grid.dims[0]) * grid.dims[1] * grid.dims[2];
  if (ncell > INT_MAX) return fail(ctx, LSMPS_INDEX_OVERFLOW, "cell count exceeds the 32-bit index range");
  return LSMPS_OK;
}

size_t cell_list_scratch_bytes(size_t n, size_t ncell) {
  // keys, numbers and placed particles; the cells' counts; their scan
  return 3 * (n * sizeof(index_t) + 256) + ncell * sizeof(index_t) + scan_scratch_bytes(ncell) + 4096;
}

lsmps_status check_cell_set(lsmps_ctx* ctx, const CellSet& set, size_t count, const lsmps_grid& grid,
                            const lsmps_cells& cells) {
  const long long ncell = static_cast<long long>(grid.dims[0]) * grid.dims[1] * grid.dims[2];
  if (static_cast<size_t>(ncell) != cells.cell_count)
    return fail(ctx, LSMPS_INVALID_ARGUMENT, "Cell list capacity does not match grid cell count");
  if (count > cells.particle_count)
    return fail(ctx, LSMPS_INVALID_ARGUMENT, "Cell list particle capacity is smaller than particle count");
  if (count > static_cast<size_t>(INT_MAX))
    return fail(ctx, LSMPS_INDEX_OVERFLOW, "Particle count exceeds 32-bit index capacity");
  if (!cells.cell_begin || !cells.cell_end ||
      (count && (!cells.cell_ids || !cells.sorted_indices || !set.x || !set.y || !set.z)))
    return fail(ctx, LSMPS_INVALID_ARGUMENT, "cell list buffers missing");
  return LSMPS_OK;
}

lsmps_status build_cell_lists_impl(lsmps_ctx* ctx, Scratch& scratch, CellSet* sets, const size_t* counts,
                                   const lsmps_cells* const* cells, int many, const lsmps_grid& grid,
                                   const BoxGrid* boxes) {
  lsmps_status st = validate_grid(ctx, grid);
  for (int s = 0; s < many && !st; ++s) st = check_cell_set(ctx, sets[s], counts[s], grid, *cells[s]);
  if (st) return st;
  // both sets' particles in one index range: one after the other where that
  // would pass 32 bits
  if (many == 2 && counts[0] + counts[1] > static_cast<size_t>(INT_MAX)) {
    for (int s = 0; s < 2 && !st; ++s)
      st = build_cell_lists_impl(ctx, scratch, sets + s, counts + s, cells + s, 1, grid, boxes);
    return st;
  }
  CellArgs a{};
  a.sets = many;
  a.grid = grid;
  a.ncell = static_cast<index_t>(static_cast<long long>(grid.dims[0]) * grid.dims[1] * grid.dims[2]);
  a.boxes = boxes;
  a.nbox = ctx->nbox;
  a.first1 = static_cast<index_t>(counts[0]);
  a.total = a.first1 + (many == 2 ? static_cast<index_t>(counts[1]) : 0);
  a.status = ctx->d_status;
  for (int s = 0; s < many; ++s) {
    a.set[s] = sets[s];
    a.set[s].ids = cells[s]->cell_ids;
    a.set[s].sorted = cells[s]->sorted_indices;
    a.set[s].begin = cells[s]->cell_begin;
    a.set[s].end = cells[s]->cell_end;
  }
  const size_t m = static_cast<size_t>(many) * a.ncell;
  a.key = scratch.take<index_t>(static_cast<size_t>(a.total) + 1);
  a.number = scratch.take<index_t>(static_cast<size_t>(a.total) + 1);
  a.placed = scratch.take<index_t>(static_cast<size_t>(a.total) + 1);
  a.count = scratch.take<index_t>(m + 1);
  const int tiles = div_up(static_cast<long long>(m), kScanTile);
  long long* partials = scratch.take<long long>(tiles + 1);
  if (!a.key || !a.number || !a.placed || !a.count || !partials)
    return fail(ctx, LSMPS_CUDA_ERROR, "cell list scratch exhausted");
  if (cudaMemsetAsync(a.count, 0, m * sizeof(index_t), ctx->stream) != cudaSuccess)
    return check_launch(ctx, "cell counts");
  const int blocks = static_cast<int>(
      std::min<long long>(div_up(static_cast<long long>(a.total), kCellThreads), ctx->sm_count * 8LL));
  if (a.total) launch(ctx, cell_count_kernel, dim3(blocks), dim3(kCellThreads), 0, a);
  if (m <= static_cast<size_t>(kSmallScan)) {
    launch(ctx, cell_ranges_small_kernel, dim3(1), dim3(kSmallScanThreads), 0, a);
  } else {
    launch(ctx, cell_totals_kernel, dim3(tiles), dim3(kScanThreads), 0, a, partials);
    if (tiles > kDirectTiles) launch(ctx, scan_partials_kernel, dim3(1), dim3(1024), 0, partials, tiles);
    launch(ctx, cell_ranges_kernel, dim3(tiles), dim3(kScanThreads), 0, a, static_cast<const long long*>(partials),
           tiles > kDirectTiles ? 1 : 0);
  }
  if (a.total == 0) return check_launch(ctx, "cell lists");
  launch(ctx, cell_place_kernel, dim3(blocks), dim3(kCellThreads), 0, a);
  // cells per warp: few enough to give every SM 32 warps, up to 32
  const long long span = std::min<long long>(
      32, std::max<long long>(1, static_cast<long long>(m) / (ctx->sm_count * 32LL)));
  const int order_blocks = static_cast<int>(std::min<long long>(
      div_up(div_up(static_cast<long long>(m), static_cast<int>(span)), kCellThreads / kWarp), ctx->sm_count * 32LL));
  launch(ctx, cell_order_kernel, dim3(order_blocks), dim3(kCellThreads), 0, a, static_cast<int>(span));
  return check_launch(ctx, "cell lists");
}

}  // namespace lsmps

using namespace lsmps;

extern "C" lsmps_status lsmps_build_cell_list(lsmps_ctx* ctx, const double* x, const double* y, const double* z,
                                              size_t count, const lsmps_grid* grid, const lsmps_cells* cells) {
  if (!ctx || !grid || !cells) return LSMPS_INVALID_ARGUMENT;
  lsmps_status st = begin_call(ctx);
  if (st) return st;
  Scratch scratch(ctx);
  if (!scratch.reserve(cell_list_scratch_bytes(count, cells->cell_count)))
    return fail(ctx, LSMPS_CUDA_ERROR, "scratch allocation failed");
  CellSet set{};
  set.x = x;
  set.y = y;
  set.z = z;
  st = build_cell_lists_impl(ctx, scratch, &set, &count, &cells, 1, *grid, nullptr);
  return end_call(ctx, st);
}
