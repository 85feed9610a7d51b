// neighbors.cu - fluid-fluid and fluid-wall CSR neighbour tables.
// Replaces build_neighbor_lists / build_one_neighbor_list of
// src/neighbor/neighbor_search.cu:294-367 (count kernel :221-236, Thrust
// exclusive scan :319-320, host capacity check :323-328, write kernel
// :238-253).
//
// Layout of the work.  A home cell's candidates are the particles of the 27
// surrounding source cells in the reference's dz -> dy -> dx order, ascending
// sorted position inside a cell (its "sequence"): nine runs of three cells that
// are neighbours in x and so follow one another in the sorted list.  Both passes
// give a home cell a block.  The count pass stages the sequence in shared memory
// as cell-relative FP32 coordinates, one lane per home particle and a quarter of
// the sequence per warp: every lane tests its particle against the candidates
// through broadcast loads, keeping one 32-bit accept mask per 32 candidates.
// After the scan of the counts, the write pass stages the candidate indices and
// replays the masks, again one lane per home particle: set bits are listed in
// shared memory and leave it as whole rows, in exactly the reference's traversal
// order; the distance tests run once per table.  Both tables go through the same
// launches (blockIdx.y).
//
// Both passes are bound by instruction issue once the cells fill the GPU, and by
// the chain of one block's loads and barriers before that.  500,000 particles
// (18,513 occupied cells of 55,062, 27 particles and 730 candidates a cell), both
// tables: count 290 us (371 with one warp per cell and a launch per table), write
// 331 us (411 with one warp per row that looked each entry's bit up by rank);
// 21,793 particles 29 and 33 us (61 and 60); 1,000 particles 13 and 17 (39 and
// 39).  Two warps a block: count 278, 38, 19, write 570, 59, 31; eight: 383, 37,
// 13 and 594, 47, 19 (with an earlier staging, whose four warps took 349, 35, 15
// and 405, 39, 21).  Threads in (particle, part) pairs, so that a cell of 33 does
// not take a second round: no change (287 and 334).
//
// Exactness: the FP32 distance is only a screen.  With coordinates scaled by
// 1/h and re-centred on the home cell, every component is at most 2 in
// magnitude for particles inside the grid, and the FP32 value of
// e = d^2 - lo2 (lo2 = (r/h)^2 - kScreenMargin, formed by three fused
// multiply-adds on the FP32 differences) is within a few hundred 2^-24 of the
// exact one, far inside kScreenMargin = 1e-4.  A candidate is accepted from
// FP32 when e < 0 and rejected when e >= 2 kScreenMargin; everything between,
// and every particle outside the +-2 window (clamped into an edge cell), is
// decided by the reference's own FP64 test dx*dx + dy*dy + dz*dz <= r^2
// (neighbor_search.cu:48-59).  The neighbour sets are therefore the FP64 ones.
#include <algorithm>
#include <climits>
#include <cmath>

#include "f32x2.cuh"
#include "impl.cuh"
#include "packed.cuh"

namespace lsmps {
namespace {

constexpr int kCsrThreads = 128;
constexpr int kCsrWarps = kCsrThreads / kWarp;
constexpr int kStageCap = 1024;
constexpr float kScreenMargin = 1.0e-4f;
constexpr float kFarLimit = 2.0f;
constexpr int kMaskWords = kStageCap / 32;
constexpr int kCellBlocks = 32;              // blocks per SM and table, at most
constexpr int kCountThreads = 128;
constexpr int kCountWarps = kCountThreads / kWarp;
constexpr float kSentinel = 1.0e18f;         // far enough that d^2 stays finite and rejected
constexpr int kStageBatch = 4;               // candidate loads in flight per lane while staging
constexpr int kStoreBatch = 4;                // row entries a lane stores at a time
constexpr int kRowStage = 162;               // row entries listed at a time (an odd number of words)

struct CsrArgs {
  const double* fx;
  const double* fy;
  const double* fz;
  const double* sx;
  const double* sy;
  const double* sz;
  const index_t* home_begin;
  const index_t* home_end;
  const index_t* home_sorted;
  const index_t* src_begin;
  const index_t* src_end;
  const index_t* src_sorted;
  lsmps_grid grid;
  double r2;
  double inv_h;
  float lo2;   // (r/h)^2 - kScreenMargin
  float band;  // a little over 2 kScreenMargin: FP32 rejects only e >= band
  index_t ncell;
  int exclude_self;
  index_t* offsets;  // count pass: per-particle counts; write pass: row offsets
  index_t* indices;
  // write pass, or NULL: each entry's sorted position (the position of the
  // neighbour in the source cell list) beside its index
  index_t* spos;
  unsigned long long capacity;
  const index_t* total;  // write pass: offsets[N]
  // Per home particle, one 32-bit accept mask per 32 staged candidates
  // (bits[i * kMaskWords + chunk]); written by the count pass, replayed by the
  // write pass.
  unsigned* bits;
  // Source positions in cell-sorted order (src_pos[k] = position of
  // src_sorted[k]), so that staging a cell reads one contiguous range.
  const double4* src_pos;
  const double4* home_pos;  // the home list's, in its sorted order
  DeviceStatus* status;
  // merged batch (batch.cu): every box's cells and grid, or NULL for one box
  // on a.grid; the cell size (a.grid.cell_size) is shared by all boxes
  const BoxGrid* boxes;
  int nbox;
};

// The fluid and the wall table, built by the same launches: blockIdx.y is the
// table.
struct CsrTables {
  CsrArgs t[2];
};

// A home cell's place in its grid: its coordinates, the grid's dims and
// origin, and the box's first global cell (0 for one box).
struct CellFrame {
  int dims[3];
  int cx, cy, cz;
  index_t base;
  double origin[3];
};

__device__ __forceinline__ CellFrame frame_of(const CsrArgs& a, index_t c) {
  CellFrame f;
  if (a.boxes) {
    const BoxGrid& g = a.boxes[box_of(a.boxes, a.nbox, c, 0)];
    f.base = g.cell_base;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      f.dims[k] = g.dims[k];
      f.origin[k] = g.origin[k];
    }
  } else {
    f.base = 0;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      f.dims[k] = a.grid.dims[k];
      f.origin[k] = a.grid.origin[k];
    }
  }
  const index_t lc = c - f.base;
  f.cx = lc % f.dims[0];
  f.cy = (lc / f.dims[0]) % f.dims[1];
  f.cz = lc / (f.dims[0] * f.dims[1]);
  return f;
}

__device__ __forceinline__ bool within_radius(double ax, double ay, double az, double bx, double by, double bz,
                                              double r2) {
  const double dx = ax - bx;
  const double dy = ay - by;
  const double dz = az - bz;
  return dx * dx + dy * dy + dz * dz <= r2;
}

__device__ __forceinline__ float to_rel(double v, double centre, double inv_h) {
  const float r = static_cast<float>((v - centre) * inv_h);
  return fabsf(r) <= kFarLimit ? r : __int_as_float(0x7fc00000);  // NaN forces the exact test
}

// (acc << 1) | sign bit of the FP32 value in v's low (kHigh: high) half.
template <bool kHigh>
__device__ __forceinline__ unsigned shift_in_sign(unsigned acc, unsigned long long v) {
  return __funnelshift_l(static_cast<unsigned>(kHigh ? v >> 32 : v), acc, 1);
}

__device__ __forceinline__ index_t warp_sum(index_t v) {
  for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
  return v;
}

// The block's cells are c = blockIdx.x + k gridDim.x.  Most cells of a tank may
// hold no fluid: thirty-two starts are read at a time and the occupied ones
// visited.  visit(cell, first home position) runs block-wide.
template <typename Visit>
__device__ __forceinline__ void for_home_cells(const CsrArgs& a, Visit visit) {
  const int lane = threadIdx.x & 31;
  for (long long c0 = blockIdx.x; c0 < a.ncell; c0 += static_cast<long long>(kWarp) * gridDim.x) {
    const long long cl = c0 + static_cast<long long>(lane) * gridDim.x;
    const index_t mine = cl < a.ncell ? a.home_begin[cl] : -1;
    for (unsigned todo = __ballot_sync(0xffffffffu, mine >= 0); todo; todo &= todo - 1) {
      const int k = __ffs(todo) - 1;
      visit(static_cast<index_t>(c0 + static_cast<long long>(k) * gridDim.x), __shfl_sync(0xffffffffu, mine, k));
    }
  }
}

// The 27 source cells of a home cell are nine runs of three cells that follow
// one another in x, so in the sorted list too: run r is sorted positions
// first[r] .. first[r] + (pre[r + 1] - pre[r]), the sequence positions from
// pre[r]; pre[9] is the number of candidates.
struct SourceRuns {
  index_t first[9];
  index_t pre[10];
};

// One warp finds a home cell's runs.
__device__ __forceinline__ void source_runs(const CsrArgs& a, const CellFrame& fr, SourceRuns& runs) {
  const int lane = threadIdx.x & 31;
  index_t b = INT_MAX, n = 0;
  if (lane < 27) {
    const int nz = fr.cz + lane / 9 - 1, ny = fr.cy + (lane / 3) % 3 - 1, nx = fr.cx + lane % 3 - 1;
    if (nz >= 0 && nz < fr.dims[2] && ny >= 0 && ny < fr.dims[1] && nx >= 0 && nx < fr.dims[0]) {
      const index_t cell = fr.base + (nz * fr.dims[1] + ny) * fr.dims[0] + nx;
      const index_t cb = a.src_begin[cell], ce = a.src_end[cell];
      if (cb >= 0 && ce >= 0) {
        b = cb;
        n = ce - cb;
      }
    }
  }
  // lane 3r: the run's first position and length
  b = min(b, min(__shfl_down_sync(0xffffffffu, b, 1), __shfl_down_sync(0xffffffffu, b, 2)));
  n += __shfl_down_sync(0xffffffffu, n, 1) + __shfl_down_sync(0xffffffffu, n, 2);
  b = __shfl_sync(0xffffffffu, b, 3 * lane);
  n = __shfl_sync(0xffffffffu, n, 3 * lane);
  if (lane >= 9) n = 0;
  index_t incl = n;
#pragma unroll
  for (int d = 1; d < 16; d <<= 1) {
    const index_t t = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += t;
  }
  if (lane < 9) {
    runs.first[lane] = b;
    runs.pre[lane] = incl - n;
  }
  if (lane == 8) runs.pre[9] = incl;
}

// The sorted position of candidate k of the sequence.
__device__ __forceinline__ index_t sorted_position(const SourceRuns& runs, index_t k) {
  int r = 0;
  while (runs.pre[r + 1] <= k) ++r;
  return runs.first[r] + (k - runs.pre[r]);
}

// Every candidate of the sequence by the block's warps: load(sorted position)
// and store(sequence position, value, sorted position).  A warp takes whole runs
// and has kStageBatch loads in flight per lane (a chain of L2 round trips
// otherwise).
template <int Warps, typename Load, typename Store>
__device__ __forceinline__ void stage_runs(const SourceRuns& runs, Load load, Store store) {
  const int lane = threadIdx.x & 31;
  for (int r = threadIdx.x / kWarp; r < 9; r += Warps) {
    const index_t first = runs.first[r], at = runs.pre[r];
    const int n = runs.pre[r + 1] - at;
    for (int k0 = lane; k0 < n; k0 += kStageBatch * kWarp) {
      decltype(load(index_t(0))) v[kStageBatch];
#pragma unroll
      for (int u = 0; u < kStageBatch; ++u)
        if (k0 + u * kWarp < n) v[u] = load(first + k0 + u * kWarp);
#pragma unroll
      for (int u = 0; u < kStageBatch; ++u)
        if (k0 + u * kWarp < n) store(at + k0 + u * kWarp, v[u], first + k0 + u * kWarp);
    }
  }
}

// Count pass: one block per home cell of a table, one lane per home particle.
// The block stages the 27-cell candidate sequence (cell-relative FP32
// coordinates) in shared memory, padded to whole 32-candidate chunks with far
// sentinels and laid out by candidate pairs ({x0, x1, y0, y1} and {z0, z1}: 12
// bytes per candidate; the rare FP64 test finds a candidate's sorted position
// from the cell starts).  Each warp then takes every fourth chunk for all home
// particles: every lane walks the chunk with broadcast loads and tests two
// candidates per packed FP32 instruction; the sign of e = d^2 - lo2 is shifted
// straight into the mask.  Bit b of chunk c of a particle's mask is the candidate
// at sequence position 32c + b, the numbering the write pass replays.  In the
// fluid table the home cell is the centre source cell, so a particle's own bit
// sits at sequence position (start of the centre cell) + (its sorted position in
// the home cell) and is cleared after the tests (the reference skips j == i).
// The masks meet in shared memory and leave it as whole lines.
__global__ void __launch_bounds__(kCountThreads) csr_count_kernel(const __grid_constant__ CsrTables tables) {
  wait_for_previous();
  __shared__ float4 sxy[kStageCap / 2];  // pair p: {x_2p, x_2p+1, y_2p, y_2p+1}
  __shared__ float2 sz[kStageCap / 2];   // pair p: {z_2p, z_2p+1}
  __shared__ unsigned far[kMaskWords];   // per chunk: candidates outside the window
  __shared__ unsigned s_mask[kWarp][kMaskWords + 1];
  __shared__ SourceRuns runs;
  __shared__ double s_centre[3];
  const CsrArgs& a = tables.t[blockIdx.y];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for_home_cells(a, [&](index_t c, index_t hb) {
    const index_t he = a.home_end[c];
    if (w == 0) {
      const CellFrame fr = frame_of(a, c);
      if (lane == 0) {
        s_centre[0] = fr.origin[0] + (fr.cx + 0.5) * a.grid.cell_size;
        s_centre[1] = fr.origin[1] + (fr.cy + 0.5) * a.grid.cell_size;
        s_centre[2] = fr.origin[2] + (fr.cz + 0.5) * a.grid.cell_size;
      }
      source_runs(a, fr, runs);
    }
    __syncthreads();
    const index_t nc = runs.pre[9];
    if (nc == 0) {
      // no candidates (most home cells of the wall table): empty rows
      for (index_t h = hb + threadIdx.x; h < he; h += kCountThreads) a.offsets[a.home_sorted[h]] = 0;
      __syncthreads();
      return;
    }
    if (nc > kStageCap) {
      // More candidates than the stage holds (overloaded edge cells): exact
      // tests straight from global memory; only the count is needed here.
      for (index_t h = hb + w; h < he; h += kCountWarps) {
        const index_t i = a.home_sorted[h];
        const double xi = a.fx[i], yi = a.fy[i], zi = a.fz[i];
        index_t count = 0;
        for (int r = 0; r < 9; ++r) {
          const index_t b0 = runs.first[r], cnt = runs.pre[r + 1] - runs.pre[r];
          for (index_t k = lane; k < cnt; k += kWarp) {
            const index_t j = a.src_sorted[b0 + k];
            if (!(a.exclude_self && j == i) && within_radius(xi, yi, zi, a.sx[j], a.sy[j], a.sz[j], a.r2)) ++count;
          }
        }
        count = warp_sum(count);
        if (lane == 0) a.offsets[i] = count;
      }
      __syncthreads();
      return;
    }
    const double ccx = s_centre[0], ccy = s_centre[1], ccz = s_centre[2];
    const int chunks = static_cast<int>((nc + kWarp - 1) / kWarp);
    if (threadIdx.x < kMaskWords) far[threadIdx.x] = 0u;
    const auto place = [&](index_t k, float x, float y, float z) {
      float* xy = reinterpret_cast<float*>(sxy + (k >> 1)) + (k & 1);
      xy[0] = x;
      xy[2] = y;
      reinterpret_cast<float*>(sz + (k >> 1))[k & 1] = z;
    };
    if (nc + static_cast<index_t>(threadIdx.x) < chunks * kWarp)  // (at most 31)
      place(nc + threadIdx.x, kSentinel, kSentinel, kSentinel);
    __syncthreads();
    stage_runs<kCountWarps>(
        runs, [&](index_t pos) { return ld4(a.src_pos, pos); },
        [&](index_t k, const double4& q, index_t) {
          const float x = to_rel(q.x, ccx, a.inv_h), y = to_rel(q.y, ccy, a.inv_h), z = to_rel(q.z, ccz, a.inv_h);
          place(k, x, y, z);
          if (isnan(x) || isnan(y) || isnan(z)) atomicOr(&far[k >> 5], 1u << (k & 31));
        });
    __syncthreads();
    for (index_t h0 = hb; h0 < he; h0 += kWarp) {
      const index_t h = h0 + lane;
      const bool live = h < he;
      double4 home = make_double4(0.0, 0.0, 0.0, 0.0);
      // idle lanes sit far from every candidate and from the sentinels
      float rx = -kSentinel, ry = -kSentinel, rz = -kSentinel;
      int self_chunk = -1;
      unsigned self_bit = 0u;
      bool home_far = false;
      if (live) {
        home = ld4(a.home_pos, h);
        rx = to_rel(home.x, ccx, a.inv_h);
        ry = to_rel(home.y, ccy, a.inv_h);
        rz = to_rel(home.z, ccz, a.inv_h);
        home_far = isnan(rx) || isnan(ry) || isnan(rz);
        if (a.exclude_self) {
          const index_t k = runs.pre[4] + (h - runs.first[4]);
          self_chunk = static_cast<int>(k >> 5);
          self_bit = 1u << (k & 31);
        }
      }
      const unsigned long long rxx = pack2(rx, rx), ryy = pack2(ry, ry), rzz = pack2(rz, rz);
      const unsigned long long nlo = pack2(-a.lo2, -a.lo2);
      for (int ch = w; ch < chunks; ch += kCountWarps) {
        const ulonglong2* qxy = reinterpret_cast<const ulonglong2*>(sxy + ch * (kWarp / 2));
        const unsigned long long* qz = reinterpret_cast<const unsigned long long*>(sz + ch * (kWarp / 2));
        // bit 31 - b: candidate b accepted from FP32 (e < 0).  The least e that is
        // not negative, as an unsigned number, tells whether any lies below band.
        unsigned lo = 0u, least = ~0u;
#pragma unroll
        for (int pr = 0; pr < kWarp / 2; ++pr) {
          const ulonglong2 xy = qxy[pr];
          const unsigned long long dx = sub2(rxx, xy.x), dy = sub2(ryy, xy.y), dz = sub2(rzz, qz[pr]);
          unsigned long long e = fma2(dx, dx, nlo);
          e = fma2(dy, dy, e);
          e = fma2(dz, dz, e);
          lo = shift_in_sign<true>(shift_in_sign<false>(lo, e), e);
          least = min(least, min(static_cast<unsigned>(e), static_cast<unsigned>(e >> 32)));
        }
        lo = __brev(lo);
        // between the thresholds, or a coordinate outside the window: FP64
        unsigned amb = far[ch];
        if (least < __float_as_uint(a.band)) {
          for (int b = 0; b < kWarp; ++b) {
            const float2 xy = make_float2(reinterpret_cast<const float*>(sxy + ch * (kWarp / 2) + (b >> 1))[b & 1],
                                          reinterpret_cast<const float*>(sxy + ch * (kWarp / 2) + (b >> 1))[2 + (b & 1)]);
            const float dx = rx - xy.x, dy = ry - xy.y;
            const float dz = rz - reinterpret_cast<const float*>(sz + ch * (kWarp / 2) + (b >> 1))[b & 1];
            const float e = __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmaf_rn(dx, dx, -a.lo2)));
            if (!(e < 0.0f) && e < a.band) amb |= 1u << b;
          }
        }
        if (home_far) amb = ~0u;
        for (; amb; amb &= amb - 1) {
          const int bit = __ffs(amb) - 1;
          const index_t k = static_cast<index_t>(ch) * kWarp + bit;
          const index_t pos = k < nc ? sorted_position(runs, k) : -1;
          bool in = false;
          if (pos >= 0) {
            const double4 sp = ld4(a.src_pos, pos);
            in = within_radius(home.x, home.y, home.z, sp.x, sp.y, sp.z, a.r2);
          }
          lo = in ? (lo | (1u << bit)) : (lo & ~(1u << bit));
        }
        if (ch == self_chunk) lo &= ~self_bit;
        s_mask[lane][ch] = lo;
      }
      __syncthreads();
      const int rows = static_cast<int>(min(static_cast<index_t>(kWarp), he - h0));
      for (int r = w; r < rows; r += kCountWarps) {
        const index_t i = a.home_sorted[h0 + r];
        const unsigned word = lane < chunks ? s_mask[r][lane] : 0u;
        if (lane < chunks) a.bits[static_cast<size_t>(i) * kMaskWords + lane] = word;
        const index_t count = __reduce_add_sync(0xffffffffu, __popc(word));
        if (lane == 0) a.offsets[i] = count;
      }
      __syncthreads();
    }
  });
}

// Write pass: one block per home cell of a table; the block stages the candidate
// indices of the 27-cell sequence and its home particles' masks.  One lane per
// home particle, each warp a run of mask words: a lane lists the set bits of its
// particle's run in shared memory (from where the runs before end), then each
// warp stores whole rows, 32 consecutive entries at a time.  Rows come out in the
// reference's order.
__global__ void __launch_bounds__(kCsrThreads) csr_write_kernel(const __grid_constant__ CsrTables tables) {
  wait_for_previous();
  __shared__ index_t s_idx[kStageCap];
  __shared__ index_t s_sp[kStageCap];  // the candidates' sorted positions
  __shared__ SourceRuns runs;
  __shared__ unsigned s_word[kWarp][kMaskWords + 1];
  __shared__ int s_count[kCsrWarps][kWarp];
  __shared__ unsigned short s_row[kWarp][kRowStage];
  const CsrArgs& a = tables.t[blockIdx.y];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned lanemask_lt = (1u << lane) - 1u;
  if (blockIdx.x == 0 && threadIdx.x == 0 && static_cast<unsigned long long>(*a.total) > a.capacity)
    record_required(a.status, static_cast<unsigned long long>(*a.total));
  for_home_cells(a, [&](index_t c, index_t hb) {
    const index_t he = a.home_end[c];
    if (warp == 0) source_runs(a, frame_of(a, c), runs);
    __syncthreads();
    const index_t nc = runs.pre[9];
    if (nc == 0) {
      // no candidates, so no rows to write (every thread has read nc before
      // warp 0 moves on to the next cell)
      __syncthreads();
      return;
    }
    if (nc > kStageCap) {
      // More candidates than the stage holds (overloaded edge cells): exact
      // tests straight from global memory, same order.
      for (index_t h = hb + warp; h < he; h += kCsrWarps) {
        const index_t i = a.home_sorted[h];
        index_t out = a.offsets[i];
        const double xi = a.fx[i], yi = a.fy[i], zi = a.fz[i];
        for (int r = 0; r < 9; ++r) {
          const index_t cnt = runs.pre[r + 1] - runs.pre[r];
          const index_t b = runs.first[r];
          for (index_t base = 0; base < cnt; base += kWarp) {
            const index_t k = base + lane;
            bool pass = false;
            index_t j = 0;
            if (k < cnt) {
              j = a.src_sorted[b + k];
              if (!(a.exclude_self && j == i)) pass = within_radius(xi, yi, zi, a.sx[j], a.sy[j], a.sz[j], a.r2);
            }
            const unsigned m = __ballot_sync(0xffffffffu, pass);
            if (pass) {
              const unsigned long long pos = static_cast<unsigned long long>(out) + __popc(m & lanemask_lt);
              if (pos < a.capacity) {
                a.indices[pos] = j;
                if (a.spos) a.spos[pos] = b + k;
              }
            }
            out += __popc(m);
          }
        }
      }
      __syncthreads();
      return;
    }
    stage_runs<kCsrWarps>(
        runs, [&](index_t pos) { return a.src_sorted[pos]; },
        [&](index_t k, index_t j, index_t pos) {
          s_idx[k] = j;
          s_sp[k] = pos;
        });
    const int chunks = static_cast<int>((nc + kWarp - 1) / kWarp);
    const int run = (chunks + kCsrWarps - 1) / kCsrWarps;  // a warp's words
    const int v0 = min(warp * run, chunks), v1 = min(v0 + run, chunks);
    for (index_t h0 = hb; h0 < he; h0 += kWarp) {
      const int rows = static_cast<int>(min(static_cast<index_t>(kWarp), he - h0));
      const index_t mine = lane < rows ? a.home_sorted[h0 + lane] : 0;
      const index_t start = lane < rows ? a.offsets[mine] : 0;
#pragma unroll 4
      for (int r = warp; r < rows; r += kCsrWarps) {
        const index_t i = __shfl_sync(0xffffffffu, mine, r);
        if (lane < chunks) s_word[r][lane] = a.bits[static_cast<size_t>(i) * kMaskWords + lane];
      }
      __syncthreads();
      const unsigned* word = s_word[lane];
      int count = 0;
      if (lane < rows)
        for (int v = v0; v < v1; ++v) count += __popc(word[v]);
      s_count[warp][lane] = count;
      __syncthreads();
      int first = 0, total = 0;
#pragma unroll
      for (int w = 0; w < kCsrWarps; ++w) {
        if (w < warp) first += s_count[w][lane];
        total += s_count[w][lane];
      }
      const int longest = __reduce_max_sync(0xffffffffu, total);  // the same in every warp
      for (int r0 = 0; r0 < longest; r0 += kRowStage) {
        if (count > 0) {
          int at = first - r0, v = v0;
          unsigned m = word[v], next = word[min(v + 1, v1 - 1)];
          // every step lists one bit and moves on to the next word when the
          // present one is done, without a branch: the lanes stay together
          do {
            const bool any = m != 0u;
            if (any && static_cast<unsigned>(at) < static_cast<unsigned>(kRowStage))
              s_row[lane][at] = static_cast<unsigned short>(v * kWarp + __ffs(m) - 1);
            at += any ? 1 : 0;
            m &= m - 1u;
            const bool done = m == 0u;
            v += done ? 1 : 0;
            m = done ? next : m;
            next = word[min(v + 1, v1 - 1)];
          } while (v < v1);
        }
        __syncthreads();
        for (int r = warp; r < rows; r += kCsrWarps) {
          const unsigned long long out = static_cast<unsigned long long>(__shfl_sync(0xffffffffu, start, r)) + r0;
          const unsigned long long room = out < a.capacity ? a.capacity - out : 0ull;
          int n = max(min(__shfl_sync(0xffffffffu, total, r) - r0, kRowStage), 0);
          if (static_cast<unsigned long long>(n) > room) n = static_cast<int>(room);
          index_t* indices = a.indices + out;
          index_t* spos = a.spos + out;
          for (int e0 = lane; e0 < n; e0 += kStoreBatch * kWarp) {
            int k[kStoreBatch];
#pragma unroll
            for (int u = 0; u < kStoreBatch; ++u) k[u] = e0 + u * kWarp < n ? s_row[r][e0 + u * kWarp] : 0;
#pragma unroll
            for (int u = 0; u < kStoreBatch; ++u)
              if (e0 + u * kWarp < n) indices[e0 + u * kWarp] = s_idx[k[u]];
            if (a.spos) {
#pragma unroll
              for (int u = 0; u < kStoreBatch; ++u)
                if (e0 + u * kWarp < n) spos[e0 + u * kWarp] = s_sp[k[u]];
            }
          }
        }
        __syncthreads();
      }
    }
    __syncthreads();
  });
}

lsmps_status table_args(lsmps_ctx* ctx, const lsmps_fluid& fluid, const double* sx, const double* sy,
                        const double* sz, const lsmps_cells& home, const lsmps_cells& src, const lsmps_grid& grid,
                        double radius, bool exclude_self, const lsmps_csr& out, size_t n_src, unsigned* bits,
                        const double4* src_pos, const double4* home_pos, index_t* spos,
                        CsrArgs& a) {
  if (fluid.count > out.particle_count || !out.offsets)
    return fail(ctx, LSMPS_INVALID_ARGUMENT, "Neighbor list particle capacity is smaller than fluid count");
  a.fx = fluid.x;
  a.fy = fluid.y;
  a.fz = fluid.z;
  a.sx = sx;
  a.sy = sy;
  a.sz = sz;
  a.home_begin = home.cell_begin;
  a.home_end = home.cell_end;
  a.home_sorted = home.sorted_indices;
  a.src_begin = src.cell_begin;
  a.src_end = src.cell_end;
  a.src_sorted = src.sorted_indices;
  a.grid = grid;
  a.r2 = radius * radius;
  a.inv_h = 1.0 / grid.cell_size;
  const double r2n = a.r2 * a.inv_h * a.inv_h;
  a.lo2 = static_cast<float>(r2n) - kScreenMargin;
  a.band = 2.0f * kScreenMargin * 1.001f;
  a.ncell = static_cast<index_t>(static_cast<long long>(grid.dims[0]) * grid.dims[1] * grid.dims[2]);
  a.boxes = ctx->boxes;
  a.nbox = ctx->nbox;
  a.exclude_self = exclude_self ? 1 : 0;
  // the count pass finds a particle's own bit through the home cell's place
  // in the source list, so the self-excluding table must use one cell list
  if (exclude_self && (home.sorted_indices != src.sorted_indices || home.cell_begin != src.cell_begin))
    return fail(ctx, LSMPS_INVALID_ARGUMENT, "self-excluding neighbour table needs one cell list");
  a.offsets = out.offsets;
  a.indices = out.indices;
  a.spos = spos;
  a.capacity = out.neighbor_count;
  a.total = out.offsets + fluid.count;
  a.bits = bits;
  a.src_pos = src_pos;
  a.home_pos = home_pos;
  a.status = ctx->d_status;
  // n_src is the source set's particle count (the cell list holds that many
  // sorted entries; its particle_count is only a capacity)
  if (n_src > src.particle_count)
    return fail(ctx, LSMPS_INVALID_ARGUMENT, "Cell list particle capacity is smaller than particle count");
  return LSMPS_OK;
}

// Both tables: counts, row offsets, rows.
lsmps_status build_tables(lsmps_ctx* ctx, Scratch& scratch, const CsrTables& tables, size_t n) {
  const long long ncell = tables.t[0].ncell;
  const dim3 grid(static_cast<int>(std::min<long long>(ncell, static_cast<long long>(ctx->sm_count) * kCellBlocks)), 2);
  if (n) launch(ctx, csr_count_kernel, grid, dim3(kCountThreads), 0, tables);
  ScanSet sets[2]{};
  for (int k = 0; k < 2; ++k) sets[k] = ScanSet{tables.t[k].offsets, tables.t[k].offsets, nullptr, tables.t[k].offsets + n};
  if (const lsmps_status st = exclusive_scans_i32(ctx, scratch, sets, 2, n)) return st;
  if (n) launch(ctx, csr_write_kernel, grid, dim3(kCsrThreads), 0, tables);
  return check_launch(ctx, "neighbour list");
}

}  // namespace

size_t neighbor_scratch_bytes(size_t n_fluid, size_t n_wall, size_t ncell) {
  return cell_list_scratch_bytes(n_fluid, ncell) + cell_list_scratch_bytes(n_wall, ncell) + scan_scratch_bytes(ncell) +
         2 * scan_scratch_bytes(n_fluid + 1) + 2 * n_fluid * kMaskWords * sizeof(unsigned) +
         (n_fluid + n_wall) * sizeof(double4) + 8192;
}

lsmps_status build_neighbor_lists_impl(lsmps_ctx* ctx, Scratch& scratch, const lsmps_fluid& fluid,
                                       const lsmps_walls& walls, const lsmps_params& p, const lsmps_cells& fc,
                                       const lsmps_cells& wc, const lsmps_csr& fn, const lsmps_csr& wn) {
  const double radius = p.support_radius;
  if (!(radius > 0.0)) return fail(ctx, LSMPS_INVALID_ARGUMENT, "Neighbor search radius must be positive");
  if (radius > p.grid.cell_size)
    return fail(ctx, LSMPS_INVALID_ARGUMENT, "Neighbor search currently requires radius <= cell_size");
  unsigned* bits[2] = {scratch.take<unsigned>(fluid.count * kMaskWords + 1),
                       scratch.take<unsigned>(fluid.count * kMaskWords + 1)};
  double4* fluid_pos = scratch.take<double4>(fluid.count + 1);
  double4* wall_pos = scratch.take<double4>(walls.count + 1);
  if (!bits[0] || !bits[1] || !fluid_pos || !wall_pos) return fail(ctx, LSMPS_CUDA_ERROR, "neighbour scratch exhausted");
  ctx->built_order = nullptr;
  CellSet sets[2]{};
  sets[0].x = fluid.x;
  sets[0].y = fluid.y;
  sets[0].z = fluid.z;
  sets[0].pos = fluid_pos;
  sets[0].box_field = 1;
  sets[1].x = walls.x;
  sets[1].y = walls.y;
  sets[1].z = walls.z;
  sets[1].pos = wall_pos;
  sets[1].box_field = 2;
  const size_t counts[2] = {fluid.count, walls.count};
  const lsmps_cells* lists[2] = {&fc, &wc};
  lsmps_status st = build_cell_lists_impl(ctx, scratch, sets, counts, lists, 2, p.grid, ctx->boxes);
  if (!st) {
    ctx->built_order = fc.sorted_indices;
    ctx->built_order_count = fluid.count;
  }
  // The fluid table's cell-sorted rows go to the context's own array, where
  // they stay for the next step's gathers.
  ctx->spos_table = nullptr;
  index_t* spos = nullptr;
  if (ctx->sorted_rows && fluid.count > 0 && ensure_sorted_rows(ctx, fn.neighbor_count, fluid.count))
    spos = ctx->fluid_spos;
  CsrTables tables{};
  if (!st)
    st = table_args(ctx, fluid, fluid.x, fluid.y, fluid.z, fc, fc, p.grid, radius, true, fn, fluid.count, bits[0],
                    fluid_pos, fluid_pos, spos, tables.t[0]);
  if (!st)
    st = table_args(ctx, fluid, walls.x, walls.y, walls.z, fc, wc, p.grid, radius, false, wn, walls.count, bits[1],
                    wall_pos, fluid_pos, nullptr, tables.t[1]);
  if (!st) st = build_tables(ctx, scratch, tables, fluid.count);
  if (!st && spos) {
    ctx->spos_table = fn.offsets;
    ctx->spos_order = fc.sorted_indices;
    ctx->spos_count = fluid.count;
  }
  return st;
}

}  // namespace lsmps

using namespace lsmps;

extern "C" lsmps_status lsmps_build_neighbor_lists(lsmps_ctx* ctx, const lsmps_fluid* fluid,
                                                   const lsmps_walls* walls, const lsmps_params* params,
                                                   const lsmps_cells* fluid_cells, const lsmps_cells* wall_cells,
                                                   const lsmps_csr* fluid_neighbors,
                                                   const lsmps_csr* wall_neighbors) {
  if (!ctx || !fluid || !walls || !params || !fluid_cells || !wall_cells || !fluid_neighbors || !wall_neighbors)
    return LSMPS_INVALID_ARGUMENT;
  lsmps_status st = begin_call(ctx);
  if (st) return st;
  Scratch scratch(ctx);
  if (!scratch.reserve(neighbor_scratch_bytes(fluid->count, walls->count, fluid_cells->cell_count)))
    return fail(ctx, LSMPS_CUDA_ERROR, "scratch allocation failed");
  st = build_neighbor_lists_impl(ctx, scratch, *fluid, *walls, *params, *fluid_cells, *wall_cells, *fluid_neighbors,
                                 *wall_neighbors);
  return end_call(ctx, st);
}
