// cells.cu - cell lists of one or two particle sets: each set's particles by
// cell, ascending index inside a cell, and every cell's range.  Replaces
// build_cell_list_impl of src/neighbor/neighbor_search.cu:255-292, whose Thrust
// sort_by_key of (cell id, particle index) is stable, so that cell_ids /
// sorted_indices / cell_begin / cell_end are identical to the reference's.
//
// A counting sort, both sets in the same launches: every particle takes a
// number in its cell (in no particular order), the cells' counts are scanned
// into ranges, the particles are put there by number, and each cell's
// particles are then ordered by index.  No block waits on another.  A set with
// many particles a cell is sorted by a stable radix sort instead, whose kernels
// the allocation-free entry point (cells_noalloc.cu) uses too.
#include <climits>
#include <cmath>

#include "cells.cuh"
#include "packed.cuh"
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

// A cell of more particles than this and than a 32nd of its set (so at most 32 of
// them) is ordered by a walk over the set's keys, the places of the others by
// comparison.  Comparing takes 14 ns a particle of the cell, for the chain of one
// thread's loads (more once the threads fill the GPU), and the walk 0.6 ns a particle
// of the set: a cell of 9,000 among 20,000 costs 127 us compared and 10 walked; among
// 2,000,000, 106 us compared and 1,100 walked; of 100,000 there, 2,400 and 1,100.
constexpr index_t kComparedCell = 1024;
constexpr int kOrderThreads = 256;
constexpr int kOrderWarps = kOrderThreads / kWarp;

// The cell's list entry `at` is particle i; its position where asked for.
__device__ __forceinline__ void put_in_cell(const CellSet& set, index_t c, index_t at, index_t i) {
  set.sorted[at] = i;
  set.ids[at] = c;
  if (set.pos) set.pos[at] = make_double4(set.x[i], set.y[i], set.z[i], 0.0);
}

// One block finds cell c's particles among the keys first .. last - 1 of its set, in
// index order: each warp counts those of its stretch, then lists them.
__device__ __forceinline__ void order_by_walk(const CellSet& set, const index_t* __restrict__ key, index_t first,
                                              index_t last, index_t c) {
  __shared__ index_t s_found[kOrderWarps];
  constexpr int kLoads = 4;  // of four keys, in flight per lane
  constexpr int kRound = kLoads * 4 * kWarp;
  const int lane = threadIdx.x & (kWarp - 1), warp = threadIdx.x / kWarp;
  const unsigned below = (1u << lane) - 1u;
  const long long start = first & ~3;
  const long long share = (last - start + kRound * kOrderWarps - 1) / (kRound * kOrderWarps) * kRound;  // of a warp
  const long long k0 = start + warp * share, k1 = min(static_cast<long long>(last), k0 + share);
  // visit(index of the lane's four keys, which of them are the cell's)
  const auto walk = [&](auto visit) {
    for (long long k = k0 + 4 * lane; k - 4 * lane < k1; k += kRound) {
      int4 v[kLoads];
#pragma unroll
      for (int u = 0; u < kLoads; ++u) {
        const long long at = k + u * 4 * kWarp;
        v[u] = at < k1 ? *reinterpret_cast<const int4*>(key + at) : make_int4(-1, -1, -1, -1);
      }
#pragma unroll
      for (int u = 0; u < kLoads; ++u) {
        const long long at = k + u * 4 * kWarp;
        const auto mine = [&](int w, int x) { return x == c && at + w >= first && at + w < k1; };
        const bool in[4] = {mine(0, v[u].x), mine(1, v[u].y), mine(2, v[u].z), mine(3, v[u].w)};
        visit(at, in);
      }
    }
  };
  index_t found = 0;
  walk([&](long long, const bool(&in)[4]) { found += in[0] + in[1] + in[2] + in[3]; });
  found = __reduce_add_sync(0xffffffffu, found);
  if (lane == 0) s_found[warp] = found;
  __syncthreads();
  index_t at = set.begin[c];
  for (int w = 0; w < warp; ++w) at += s_found[w];
  walk([&](long long k, const bool(&in)[4]) {
    index_t before = 0, many = 0;  // of the lanes below, of the warp
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      const unsigned all = __ballot_sync(0xffffffffu, in[w]);
      before += __popc(all & below);
      many += __popc(all);
    }
#pragma unroll
    for (int w = 0; w < 4; ++w)
      if (in[w]) put_in_cell(set, c, at + before++, static_cast<index_t>(k + w - first));
    at += many;
  });
}

// Orders each cell's particles by index: a thread takes one of the unordered list's
// places, finds how many of its cell come before its particle and writes the
// particle to its own place of the sorted list.  The comparisons of a warp are with
// one or two cells' particles, four a load, and those of a crowded cell are spread
// over as many threads as it has particles.  Bound by latency: 20 us for 500,000
// particles and 186,225 walls (72 with one warp per cell), 2,000,000 with theirs 64
// (112).  A list of 2,000,000 particles, 27 a cell, takes 91 us in all (93 with one
// warp per cell, which took 15,100 with 1,025 of them in one cell; 92 here); 300,000:
// 34 (34; 2,340; 41).
__global__ void __launch_bounds__(kOrderThreads) cell_order_kernel(const __grid_constant__ CellArgs a) {
  wait_for_previous();
  __shared__ index_t s_huge;
  __shared__ int s_set;
  const long long place = static_cast<long long>(blockIdx.x) * kOrderThreads + threadIdx.x;
  const index_t p = static_cast<index_t>(place);
  bool huge = false;
  if (place < a.total) {
    const int s = p >= a.first1 ? 1 : 0;
    const CellSet& set = a.set[s];
    const index_t first = s ? a.first1 : 0;
    const index_t i = a.placed[p], c = a.key[first + i];
    const index_t b = set.begin[c], e = set.end[c];
    const index_t many = s ? a.total - a.first1 : a.first1;
    if (e - b > max(kComparedCell, many / 32)) {
      huge = p == first + b;  // (one such place in a block's stretch, at most)
      if (huge) {
        s_huge = c;
        s_set = s;
      }
    } else {
      index_t at = b, q = first + b;
      const index_t end = first + e;
      for (; q < end && (q & 3) != 0; ++q) at += a.placed[q] < i ? 1 : 0;
#pragma unroll 8
      for (; q + 4 <= end; q += 4) {
        const int4 v = *reinterpret_cast<const int4*>(a.placed + q);
        at += (v.x < i) + (v.y < i) + (v.z < i) + (v.w < i);
      }
      for (; q < end; ++q) at += a.placed[q] < i ? 1 : 0;
      put_in_cell(set, c, at, i);
    }
  }
  if (__syncthreads_or(huge))
    order_by_walk(a.set[s_set], a.key, s_set ? a.first1 : 0, s_set ? a.total : a.first1, s_huge);
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

// A set of more particles than this per cell on average is sorted by cell id
// instead of counted, as the comparisons grow with the number per cell and the sort
// does not: 2,000,000 particles 116 us counted at 128 a cell and 152 at 250, sorted
// 104; 300,000: 38, 49 and 55 (and 84 counted at 585 a cell); 20,000: 24 at 160, 34
// at 740, and 28.
constexpr size_t kCrowdedMean = 128;

size_t cell_list_scratch_bytes(size_t n, size_t ncell) {
  // keys, numbers and placed particles; the cells' counts; their scan (the sort of a
  // crowded set takes less: keys and particles once more, its table of digits)
  return 3 * (n * sizeof(index_t) + 256) + ncell * sizeof(index_t) + scan_scratch_bytes(ncell) + 8192;
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

namespace {

// The cell list of one set by a stable radix sort of (cell id, particle index),
// whose time does not depend on how many particles a cell has.
lsmps_status sort_cell_list(lsmps_ctx* ctx, Scratch& scratch, const CellSet& set, index_t n, const lsmps_grid& grid) {
  const long long ncell = static_cast<long long>(grid.dims[0]) * grid.dims[1] * grid.dims[2];
  const int passes = (key_bits(ncell) + kRadixBits - 1) / kRadixBits;
  const int tiles = div_up(n, kSortTile);
  index_t* other[2] = {scratch.take<index_t>(static_cast<size_t>(n) + 1), scratch.take<index_t>(static_cast<size_t>(n) + 1)};
  index_t* hist = scratch.take<index_t>(static_cast<size_t>(tiles) * kRadixBins + 1);
  if (!other[0] || !other[1] || !hist) return fail(ctx, LSMPS_CUDA_ERROR, "cell list scratch exhausted");
  // back and forth so that the last pass ends in the caller's arrays
  index_t* from[2] = {passes % 2 ? other[0] : set.ids, passes % 2 ? other[1] : set.sorted};
  index_t* to[2] = {passes % 2 ? set.ids : other[0], passes % 2 ? set.sorted : other[1]};
  const auto blocks = [&](long long work) {
    return dim3(static_cast<int>(std::min<long long>(div_up(work, kCellThreads), ctx->sm_count * 8LL)));
  };
  launch(ctx, hash_kernel, blocks(std::max<long long>(n, ncell)), dim3(kCellThreads), 0, set.x, set.y, set.z, n, grid,
         from[0], from[1], set.begin, set.end, static_cast<index_t>(ncell), ctx->d_status);
  for (int p = 0; p < passes; ++p) {
    launch(ctx, radix_hist_kernel, dim3(tiles), dim3(kSortThreads), 0, static_cast<const index_t*>(from[0]), n,
           p * kRadixBits, hist, tiles);
    if (const lsmps_status st =
            exclusive_scan_i32(ctx, scratch, hist, hist, static_cast<size_t>(tiles) * kRadixBins, nullptr, nullptr))
      return st;
    launch(ctx, radix_scatter_kernel, dim3(tiles), dim3(kSortThreads), 0, static_cast<const index_t*>(from[0]),
           static_cast<const index_t*>(from[1]), to[0], to[1], n, p * kRadixBits, static_cast<const index_t*>(hist), tiles);
    std::swap(from[0], to[0]);
    std::swap(from[1], to[1]);
  }
  launch(ctx, ranges_kernel, blocks(n), dim3(kCellThreads), 0, static_cast<const index_t*>(set.ids), n, set.begin, set.end);
  if (set.pos) pack4(ctx, set.x, set.y, set.z, nullptr, static_cast<size_t>(n), set.pos, set.sorted);
  return check_launch(ctx, "cell list");
}

}  // namespace

lsmps_status build_cell_lists_impl(lsmps_ctx* ctx, Scratch& scratch, CellSet* sets, const size_t* counts,
                                   const lsmps_cells* const* cells, int many, const lsmps_grid& grid,
                                   const BoxGrid* boxes) {
  lsmps_status st = validate_grid(ctx, grid);
  for (int s = 0; s < many && !st; ++s) st = check_cell_set(ctx, sets[s], counts[s], grid, *cells[s]);
  if (st) return st;
  for (int s = 0; s < many; ++s) {
    sets[s].ids = cells[s]->cell_ids;
    sets[s].sorted = cells[s]->sorted_indices;
    sets[s].begin = cells[s]->cell_begin;
    sets[s].end = cells[s]->cell_end;
  }
  const size_t ncell = cells[0]->cell_count;
  const auto coarse = [&](int s) { return !boxes && counts[s] > kCrowdedMean * ncell; };
  // both sets' particles in one index range: one after the other where that
  // would pass 32 bits
  if (many == 2 && (counts[0] + counts[1] > static_cast<size_t>(INT_MAX) || coarse(0) || coarse(1))) {
    for (int s = 0; s < 2 && !st; ++s)
      st = build_cell_lists_impl(ctx, scratch, sets + s, counts + s, cells + s, 1, grid, boxes);
    return st;
  }
  if (coarse(0)) return sort_cell_list(ctx, scratch, sets[0], static_cast<index_t>(counts[0]), grid);
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
  launch(ctx, cell_order_kernel, dim3(div_up(static_cast<long long>(a.total), kOrderThreads)), dim3(kOrderThreads), 0, a);
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
