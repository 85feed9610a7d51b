// solve.cu - the PPE solve on the device: restarted GMRES(m) over the PPE CSR
// rows, replacing AmgxPpeSolver::solve (src/ppe/ppe_matrix.cu:586-679).
//
// The reference hands the system to AMGX (a third-party library, linked only
// when found at configure time; no version is pinned in the tree) with
// AMGX's GMRES sample configuration (ppe_matrix.cu:604-610): GMRES, no
// preconditioner, at most 100 iterations, stop when the L2 norm of the
// residual falls to 1e-6 of the initial one (RELATIVE_INI), initial guess
// zero (:625), and clamps negative pressures to zero afterwards (:662).  AMGX
// copies the CSR to the host and back around every solve (:621-661); here
// the matrix stays where the assembly wrote it.
//
// Algorithm: GMRES(m) of Saad and Schultz (1986) with right preconditioning
// (none, or Jacobi: M = diag(A)).  Arnoldi uses classical Gram-Schmidt with
// one re-orthogonalisation (CGS2), so every projection is a batch of
// independent dot products.  An Arnoldi step is four kernels: the new basis
// vector scaled and multiplied by A; the product projected (h = V^T w; with up to
// 2,048 rows in the kernel before); the projection taken off and the remainder
// projected again; that taken off, and the norm.  Each kernel's last block to
// finish adds the blocks' partial sums in a fixed order, and that of the last
// extends the Hessenberg matrix by its column and rotates it, so a solve is bitwise reproducible, nothing waits for the host
// within a restart cycle, and what is queued of a cycle that has converged returns
// at once.  How far a cycle is the device writes to host memory, so that the host
// queues nothing for a system that starts converged and, where a step is long,
// little that would not be wanted.
#include <algorithm>
#include <cmath>

#include "impl.cuh"

namespace lsmps {
namespace {

constexpr int kSolveThreads = 256;
constexpr int kSolveWarps = kSolveThreads / kWarp;
constexpr int kRowLanes = 8;       // lanes per CSR row in products that end in dot products
constexpr int kProductLanes = 16;  // ... in the products without
constexpr int kMaxRestart = 64;
// Rows up to which a product and its dot products are one kernel (measured at
// product_dots_kernel).
constexpr index_t kFusedRows = 2048;

// A progress past every step's: nothing more of this cycle is wanted.
constexpr int kStopped = 1 << 30;
// Above kFollowRows a step is queued once the last but one has finished: a solve
// that converges in its first step takes 255 us at 500,000 rows, and 500 with up to
// twenty steps queued that then return at once (31,250 blocks each in the product).
// Below, the write to host memory would cost a step 0.8 of its 16 us (8,000 rows)
// and the launches cost less.
constexpr int kAhead = 1;
constexpr index_t kFollowRows = 100000;

// What the host reads after a cycle.
struct SolveHead {
  double beta, beta0, target;
  double scale;  // 1 / norm of the vector that the next product takes
  int iters;
  int steps;      // of this cycle
  int converged;  // the residual has reached the target
  int stop;       // the rest of this cycle's launches return at once
};

// The solve's scalars, in device memory.
struct SolveState : SolveHead {
  unsigned tickets;
  double h[kMaxRestart + 1];                       // first projection of the step
  double h2[kMaxRestart + 1];                      // second projection
  double H[kMaxRestart * (kMaxRestart + 1)];       // rotated Hessenberg columns
  double cs[kMaxRestart], sn[kMaxRestart], g[kMaxRestart + 1];
};

struct SolveArgs {
  index_t n;
  const index_t* ro;
  const index_t* ci;
  const double* va;
  const double* dinv;        // Jacobi: 1 / a_ii, or NULL
  double* V;                 // [restart][ldv]
  size_t ldv;
  double* w[2];  // the vector to be normalised next, and its product
  double* x;
  const double* b;
  double* partial;  // [kMaxRestart + 1][gridDim.x]
  SolveState* st;
  volatile int* progress;  // host memory: 1 + the cycle's finished steps (counted with `follow`), kStopped with st->stop
  int follow;
  int restart;
  int max_iters;
  double tolerance;
  int relative;
};

// Lane l's share of row . (x, or dinv ∘ x): the entries l, l + G, ... of the row,
// so that the lanes' gathers of x fall on neighbouring columns together, four
// rounds of values and columns in flight.  500,000 rows of 109 entries, B200:
// 122 us a product with 16 lanes (5.4 TB/s), 138 with 8, 137 with 32, 179 with 4:
// bound by the load pipe's wavefronts (ncu at 8 lanes: 85%), of which the gathers
// of x take most; rows of one warp that lie next to each other share the lines
// of their values.  Tried: four consecutive entries a lane with 32-byte loads
// (160 us: fewer loads, scattered gathers).
template <int G>
__device__ __forceinline__ double row_product(const SolveArgs& a, index_t row, int l, const double* __restrict__ x) {
  constexpr int kRounds = 4;
  const index_t e = a.ro[row + 1];
  double acc = 0.0;
  for (index_t k = a.ro[row] + l; k < e; k += kRounds * G) {
    index_t c[kRounds];
    double v[kRounds];
#pragma unroll
    for (int r = 0; r < kRounds; ++r) {
      const index_t at = k + r * G;
      c[r] = at < e ? __ldcs(a.ci + at) : -1;
      v[r] = at < e ? __ldcs(a.va + at) : 0.0;
    }
#pragma unroll
    for (int r = 0; r < kRounds; ++r)
      if (c[r] >= 0) acc = fma(v[r], a.dinv ? a.dinv[c[r]] * x[c[r]] : x[c[r]], acc);
  }
  return group_sum<G>(acc, group_mask<G>());
}

// True in every thread of the last block to get here; the blocks' earlier
// global writes are then visible to it.  No block waits for another.
__device__ __forceinline__ bool last_block(SolveState* st) {
  __shared__ bool last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    last = atomicAdd(&st->tickets, 1u) == gridDim.x - 1;
    if (last) st->tickets = 0u;
  }
  __syncthreads();
  if (last) __threadfence();
  return last;
}

// Sum over the block's threads, in thread 0 (and every thread of warp 0).
__device__ __forceinline__ double block_sum(double v) {
  __shared__ double red[kSolveWarps];
  v = group_sum<kWarp>(v, 0xffffffffu);
  __syncthreads();
  if ((threadIdx.x & (kWarp - 1)) == 0) red[threadIdx.x / kWarp] = v;
  __syncthreads();
  double sum = 0.0;
  if (threadIdx.x < kWarp) {
#pragma unroll
    for (int w = 0; w < kSolveWarps; ++w) sum += red[w];
  }
  return sum;
}

// out[k] = the blocks' partials of k < count in order (the whole block).
__device__ __forceinline__ void add_partials(const double* partial, int count, double* out) {
  const int lane = threadIdx.x & (kWarp - 1);
  for (int k = threadIdx.x / kWarp; k < count; k += kSolveWarps) {
    double acc = 0.0;
    for (int b = lane; b < static_cast<int>(gridDim.x); b += kWarp)
      acc += __ldcg(partial + static_cast<size_t>(k) * gridDim.x + b);
    acc = group_sum<kWarp>(acc, 0xffffffffu);
    if (lane == 0) out[k] = acc;
  }
  __syncthreads();
}

// r = b - A x into w[0] and its norm (First: x = 0, so r = b): opens a cycle.
template <bool First>
__global__ void __launch_bounds__(kSolveThreads) residual_kernel(SolveArgs a, int report) {
  wait_for_previous();
  constexpr int G = kProductLanes;
  const int l = threadIdx.x & (G - 1);
  const index_t rows = static_cast<index_t>(gridDim.x * (kSolveThreads / G));
  double acc = 0.0;
  SolveArgs plain = a;
  plain.dinv = nullptr;
  for (index_t row = static_cast<index_t>((blockIdx.x * kSolveThreads + threadIdx.x) / G); row < a.n; row += rows) {
    double r = a.b[row];
    if (First) {
      if (l == 0) a.x[row] = 0.0;
    } else {
      r -= row_product<G>(plain, row, l, a.x);
    }
    if (l == 0) {
      a.w[0][row] = r;
      acc = fma(r, r, acc);
    }
  }
  const double sum = block_sum(acc);
  if (threadIdx.x == 0) a.partial[blockIdx.x] = sum;
  SolveState* st = a.st;
  if (!last_block(st)) return;
  __shared__ double total;
  add_partials(a.partial, 1, &total);
  if (threadIdx.x != 0) return;
  const double beta = sqrt(total);
  if (report) {  // the solve's first residual
    st->beta0 = beta;
    st->target = a.relative ? a.tolerance * beta : a.tolerance;
    st->iters = 0;
  }
  st->beta = beta;
  st->scale = 1.0 / beta;
  st->steps = 0;
  st->g[0] = beta;
  st->converged = beta <= st->target ? 1 : 0;
  st->stop = st->converged || st->iters >= a.max_iters;
  if (report) *a.progress = st->stop ? kStopped : 1;
}

// Step j: v_j = scale w[j & 1] into the basis, w[(j + 1) & 1] = A v_j.
__global__ void __launch_bounds__(kSolveThreads) product_kernel(SolveArgs a, int j) {
  wait_for_previous();
  const SolveState* st = a.st;
  if (st->stop) return;
  const double scale = st->scale;
  const index_t row = static_cast<index_t>((static_cast<long long>(blockIdx.x) * kSolveThreads + threadIdx.x) / kProductLanes);
  const int l = threadIdx.x & (kProductLanes - 1);
  if (row >= a.n) return;  // the whole group
  const double* __restrict__ from = a.w[j & 1];
  const double w = scale * row_product<kProductLanes>(a, row, l, from);
  if (l == 0) {
    a.V[static_cast<size_t>(j) * a.ldv + row] = scale * from[row];
    a.w[(j + 1) & 1][row] = w;
  }
}

// The same with the product's dot products with v_0 .. v_j: a row's eight lanes
// take the basis vectors lane, lane + 8, ..., and the four rows of a warp read whole
// sectors of them.  It saves a launch and costs a wait per row, as the vectors'
// loads hold up the row's.  A solve of 100 iterations, fused and in two kernels: 343
// rows 1,740 and 1,815 us, 1,000 1,968 and 2,018, 3,120 2,038 and 1,966, 8,000 2,180
// and 2,068, 61,250 4,772 and 4,393, 163,840 9,225 and 8,132.
template <int Dots>
__global__ void __launch_bounds__(kSolveThreads) product_dots_kernel(SolveArgs a, int j) {
  wait_for_previous();
  SolveState* st = a.st;
  if (st->stop) return;
  const double scale = st->scale;
  const int l = threadIdx.x & (kRowLanes - 1);
  const double* __restrict__ from = a.w[j & 1];
  double* __restrict__ to = a.w[(j + 1) & 1];
  double* __restrict__ vj = a.V + static_cast<size_t>(j) * a.ldv;
  const index_t rows = static_cast<index_t>(gridDim.x * (kSolveThreads / kRowLanes));
  double acc[Dots];
#pragma unroll
  for (int d = 0; d < Dots; ++d) acc[d] = 0.0;
  for (index_t row = static_cast<index_t>((blockIdx.x * kSolveThreads + threadIdx.x) / kRowLanes); row < a.n;
       row += rows) {
    const double own = scale * from[row];
    double v[Dots];
#pragma unroll
    for (int d = 0; d < Dots; ++d) {
      const int k = d * kRowLanes + l;
      v[d] = k < j ? a.V[static_cast<size_t>(k) * a.ldv + row] : k == j ? own : 0.0;
    }
    const double w = scale * row_product<kRowLanes>(a, row, l, from);
    if (l == 0) {
      vj[row] = own;
      to[row] = w;
    }
#pragma unroll
    for (int d = 0; d < Dots; ++d) acc[d] = fma(v[d], w, acc[d]);
  }
  // over the warp's four rows, then the block's warps
  __shared__ double s_dot[kSolveWarps][kRowLanes * Dots];
#pragma unroll
  for (int d = 0; d < Dots; ++d) {
    acc[d] += __shfl_xor_sync(0xffffffffu, acc[d], 8);
    acc[d] += __shfl_xor_sync(0xffffffffu, acc[d], 16);
    if ((threadIdx.x & (kWarp - 1)) < kRowLanes) s_dot[threadIdx.x / kWarp][d * kRowLanes + l] = acc[d];
  }
  __syncthreads();
  for (int k = threadIdx.x; k <= j; k += kSolveThreads) {
    double sum = 0.0;
#pragma unroll
    for (int w = 0; w < kSolveWarps; ++w) sum += s_dot[w][k];
    a.partial[static_cast<size_t>(k) * gridDim.x + blockIdx.x] = sum;
  }
  if (!last_block(st)) return;
  add_partials(a.partial, j + 1, st->h);
}

// Update: w -= sum_k h[k] v_k, and the remainder's dot products with the same
// vectors (their values are still in registers) into h2, the second projection
// of CGS2; else w's dot products into h, the first.  K: the most vectors this
// instance holds.
template <int K, bool Update>
__global__ void __launch_bounds__(kSolveThreads) project_kernel(SolveArgs a, int j) {
  wait_for_previous();
  SolveState* st = a.st;
  if (st->stop) return;
  __shared__ double sh[K];
  __shared__ double s_dot[kSolveWarps][K];
  if (Update) {
    for (int k = threadIdx.x; k < K; k += kSolveThreads) sh[k] = k <= j ? st->h[k] : 0.0;
    __syncthreads();
  }
  double* __restrict__ w = a.w[(j + 1) & 1];
  double acc[K];
#pragma unroll
  for (int k = 0; k < K; ++k) acc[k] = 0.0;
  for (index_t i = blockIdx.x * kSolveThreads + threadIdx.x; i < a.n; i += gridDim.x * kSolveThreads) {
    double v[K];
    double wi = w[i];
#pragma unroll
    for (int k = 0; k < K; ++k) v[k] = k <= j ? a.V[static_cast<size_t>(k) * a.ldv + i] : 0.0;
    if (Update) {
#pragma unroll
      for (int k = 0; k < K; ++k) wi = fma(-sh[k], v[k], wi);
      w[i] = wi;
    }
#pragma unroll
    for (int k = 0; k < K; ++k) acc[k] = fma(v[k], wi, acc[k]);
  }
  int base = 0, count = K;
  lane_totals<K, 16>(acc, base, count);
#pragma unroll
  for (int k = 0; k < lane_totals_left(K, 16); ++k)
    if (k < count) s_dot[threadIdx.x / kWarp][base + k] = acc[k];
  __syncthreads();
  for (int k = threadIdx.x; k <= j; k += kSolveThreads) {
    double sum = 0.0;
#pragma unroll
    for (int q = 0; q < kSolveWarps; ++q) sum += s_dot[q][k];
    a.partial[static_cast<size_t>(k) * gridDim.x + blockIdx.x] = sum;
  }
  if (!last_block(st)) return;
  add_partials(a.partial, j + 1, Update ? st->h2 : st->h);
}

// w -= sum_k h2[k] v_k and its norm; the last block extends the Hessenberg
// matrix by column j and applies the previous rotations and the one that zeroes
// its subdiagonal.
// (h2 is padded with zeros to K: with the additions under k <= j
// each load waited for the one before it, 83 us at 2,000,000 rows against 49 of
// project_kernel; 500,000 rows: a solve 17.8 -> 17.3 ms)
template <int K>
__global__ void __launch_bounds__(kSolveThreads) extend_kernel(SolveArgs a, int j) {
  wait_for_previous();
  SolveState* st = a.st;
  if (st->stop) return;
  __shared__ double sh[kMaxRestart + 1];
  for (int k = threadIdx.x; k < K; k += kSolveThreads) sh[k] = k <= j ? st->h2[k] : 0.0;
  __syncthreads();
  double* __restrict__ w = a.w[(j + 1) & 1];
  double acc = 0.0;
  for (index_t i = blockIdx.x * kSolveThreads + threadIdx.x; i < a.n; i += gridDim.x * kSolveThreads) {
    double wi = w[i], v[K];
#pragma unroll
    for (int k = 0; k < K; ++k) v[k] = k <= j ? a.V[static_cast<size_t>(k) * a.ldv + i] : 0.0;
#pragma unroll
    for (int k = 0; k < K; ++k) wi = fma(-sh[k], v[k], wi);
    w[i] = wi;
    acc = fma(wi, wi, acc);
  }
  const double sum = block_sum(acc);
  if (threadIdx.x == 0) a.partial[blockIdx.x] = sum;
  if (!last_block(st)) return;
  __shared__ double total, col[kMaxRestart + 1], cs[kMaxRestart], sn[kMaxRestart];
  add_partials(a.partial, 1, &total);
  for (int k = threadIdx.x; k <= j; k += kSolveThreads) {
    col[k] = st->h[k] + sh[k];
    if (k < j) {
      cs[k] = st->cs[k];
      sn[k] = st->sn[k];
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const double hnext = sqrt(total);
    for (int k = 0; k < j; ++k) {
      const double t = cs[k] * col[k] + sn[k] * col[k + 1];
      col[k + 1] = -sn[k] * col[k] + cs[k] * col[k + 1];
      col[k] = t;
    }
    const double den = hypot(col[j], hnext);
    const double c = den > 0.0 ? col[j] / den : 1.0;
    const double s = den > 0.0 ? hnext / den : 0.0;
    col[j] = den;
    st->cs[j] = c;
    st->sn[j] = s;
    const double g = st->g[j];
    st->g[j + 1] = -s * g;
    st->g[j] = c * g;
    st->scale = 1.0 / hnext;
    st->steps = j + 1;
    st->iters += 1;
    // hnext == 0: the Krylov space is invariant (the correction solves the
    // system on it); the cycle stops there.
    const bool stop = fabs(s * g) <= st->target || hnext == 0.0 || st->iters >= a.max_iters;
    if (stop) st->stop = 1;
    if (stop || a.follow) *a.progress = stop ? kStopped : j + 2;
  }
  __syncthreads();
  for (int k = threadIdx.x; k <= j; k += kSolveThreads) st->H[static_cast<size_t>(j) * (kMaxRestart + 1) + k] = col[k];
}

// y = R^-1 g (back substitution on the rotated Hessenberg, by the first warp of
// each block), x += M^-1 V y.
__global__ void __launch_bounds__(kSolveThreads) correct_kernel(SolveArgs a) {
  wait_for_previous();
  const SolveState* st = a.st;
  __shared__ double sy[kMaxRestart];
  const int m = st->steps;
  if (threadIdx.x < kWarp) {
    const int lane = threadIdx.x;
    double t[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) t[q] = lane + q * kWarp < m ? st->g[lane + q * kWarp] : 0.0;
    for (int k = m - 1; k >= 0; --k) {
      const double* __restrict__ col = st->H + static_cast<size_t>(k) * (kMaxRestart + 1);
      const double tk = __shfl_sync(0xffffffffu, k < kWarp ? t[0] : t[1], k & (kWarp - 1));
      const double d = col[k];
      const double y = d != 0.0 ? tk / d : 0.0;
      if (lane == 0) sy[k] = y;
#pragma unroll
      for (int q = 0; q < 2; ++q)
        if (lane + q * kWarp < k) t[q] = fma(-col[lane + q * kWarp], y, t[q]);
    }
  }
  __syncthreads();
  for (index_t i = blockIdx.x * kSolveThreads + threadIdx.x; i < a.n; i += gridDim.x * kSolveThreads) {
    double u = 0.0;
#pragma unroll 8
    for (int k = 0; k < m; ++k) u = fma(sy[k], a.V[static_cast<size_t>(k) * a.ldv + i], u);
    a.x[i] += a.dinv ? a.dinv[i] * u : u;
  }
}

// dinv[i] = 1 / a_ii (1 where the row has no non-zero diagonal entry).
__global__ void __launch_bounds__(kSolveThreads)
    jacobi_kernel(index_t n, const index_t* __restrict__ ro, const index_t* __restrict__ ci,
                  const double* __restrict__ va, double* __restrict__ dinv) {
  wait_for_previous();
  const index_t i = blockIdx.x * kSolveThreads + threadIdx.x;
  if (i >= n) return;
  double d = 0.0;
  for (index_t k = ro[i]; k < ro[i + 1]; ++k)
    if (ci[k] == i) d += va[k];
  dinv[i] = d != 0.0 ? 1.0 / d : 1.0;
}

// clamp_pressure_kernel, ppe_matrix.cu:373-379
__global__ void __launch_bounds__(kSolveThreads) clamp_kernel(index_t n, double* __restrict__ x) {
  wait_for_previous();
  const index_t i = blockIdx.x * kSolveThreads + threadIdx.x;
  if (i < n && x[i] < 0.0) x[i] = 0.0;
}

// Launch shapes: blocks of the streaming passes, of the row passes.
struct SolveShape {
  int stream, rows;
  bool fused;  // the first projection in the product
};

void launch_residual(lsmps_ctx* ctx, const SolveArgs& a, bool zero, bool report, const SolveShape& g) {
  const auto queue = [&](const char* name, auto kernel) {
    launch_named(ctx, name, kernel, dim3(g.rows), dim3(kSolveThreads), 0, a, report ? 1 : 0);
  };
  zero ? queue("residual_kernel<first>", residual_kernel<true>) : queue("residual_kernel", residual_kernel<false>);
}

// Step j's passes over the basis with the smallest instances that hold its
// j + 1 vectors.
template <int K>
void launch_projections(lsmps_ctx* ctx, const SolveArgs& a, int j, const SolveShape& g) {
  const dim3 grid(g.stream), block(kSolveThreads);
  if (!g.fused) launch_named(ctx, "project_kernel<first>", project_kernel<K, false>, grid, block, 0, a, j);
  launch_named(ctx, "project_kernel", project_kernel<K, true>, grid, block, 0, a, j);
  launch_named(ctx, "extend_kernel", extend_kernel<K>, grid, block, 0, a, j);
}

void launch_step(lsmps_ctx* ctx, const SolveArgs& a, int j, const SolveShape& g) {
  const auto product = [&](auto kernel) {
    launch_named(ctx, "product_dots_kernel", kernel, dim3(g.rows), dim3(kSolveThreads), 0, a, j);
  };
  if (!g.fused)
    launch(ctx, product_kernel, dim3(div_up(static_cast<long long>(a.n) * kProductLanes, kSolveThreads)),
           dim3(kSolveThreads), 0, a, j);
  else if (j < 8)
    product(product_dots_kernel<1>);
  else if (j < 24)
    product(product_dots_kernel<3>);
  else
    product(product_dots_kernel<kMaxRestart / kRowLanes>);
  if (j < 8)
    launch_projections<8>(ctx, a, j, g);
  else if (j < 16)
    launch_projections<16>(ctx, a, j, g);
  else if (j < 24)
    launch_projections<24>(ctx, a, j, g);
  else
    launch_projections<kMaxRestart>(ctx, a, j, g);
}

}  // namespace

void solver_options_default(lsmps_solver_options* o) {
  o->max_iters = 100;
  o->restart = 20;
  o->tolerance = 1.0e-6;
  o->convergence = LSMPS_CONVERGENCE_RELATIVE_INITIAL;
  o->preconditioner = LSMPS_PRECONDITIONER_NONE;
  o->clamp_negative = 1;
  o->use_initial_guess = 0;
}

lsmps_status solve_ppe_impl(lsmps_ctx* ctx, const lsmps_csr_matrix& A, const double* b, double* x,
                            const lsmps_solver_options& opt, lsmps_solver_report* report) {
  if (report) *report = lsmps_solver_report{0, 0, 0.0, 0.0};
  if (A.rows == 0) return LSMPS_OK;
  if (const lsmps_status cs = check_table(ctx, A.row_offsets, A.col_indices, A.rows, A.nnz, A.cols,
                                          "PPE matrix: row offset or column index out of range"))
    return cs;
  if (A.rows != A.cols || !A.row_offsets || !A.col_indices || !A.values || !b || !x)
    return fail(ctx, LSMPS_INVALID_ARGUMENT, "AMGX PPE solve requires a square CSR matrix, rhs, and solution buffer");
  if (A.rows > static_cast<size_t>(INT32_MAX)) return fail(ctx, LSMPS_INDEX_OVERFLOW, "PPE rows exceed 32-bit indices");
  if (opt.restart < 1 || opt.restart > kMaxRestart || opt.max_iters < 0 || !(opt.tolerance >= 0.0) ||
      (opt.convergence != LSMPS_CONVERGENCE_RELATIVE_INITIAL && opt.convergence != LSMPS_CONVERGENCE_ABSOLUTE) ||
      (opt.preconditioner != LSMPS_PRECONDITIONER_NONE && opt.preconditioner != LSMPS_PRECONDITIONER_JACOBI))
    return fail(ctx, LSMPS_INVALID_ARGUMENT, "invalid PPE solver options");
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  cudaStreamIsCapturing(ctx->stream, &cap);
  if (cap != cudaStreamCaptureStatusNone)
    return fail(ctx, LSMPS_INVALID_ARGUMENT, "the PPE solve reads residuals back and cannot be captured");

  const index_t n = static_cast<index_t>(A.rows);
  const int m = opt.restart;
  // Streaming passes: up to four blocks per SM; passes over the rows that end
  // in a sum: eight.
  SolveShape g;
  g.stream = static_cast<int>(std::min<long long>(div_up(static_cast<long long>(n), kSolveThreads), 4LL * ctx->sm_count));
  g.rows = static_cast<int>(
      std::min<long long>(div_up(static_cast<long long>(n) * kRowLanes, kSolveThreads), 8LL * ctx->sm_count));
  g.fused = n <= kFusedRows;
  const size_t ldv = (static_cast<size_t>(n) + 31) & ~size_t(31);
  const size_t partials = static_cast<size_t>(kMaxRestart + 1) * std::max(g.stream, g.rows);
  Scratch scratch(ctx);
  const size_t need = (static_cast<size_t>(m) * ldv + 3 * ldv) * sizeof(double) + partials * sizeof(double) +
                      sizeof(SolveState) + 16 * 256;
  if (!scratch.reserve(need)) return fail(ctx, LSMPS_CUDA_ERROR, "scratch allocation failed");
  SolveArgs a{};
  a.n = n;
  a.ro = A.row_offsets;
  a.ci = A.col_indices;
  a.va = A.values;
  a.V = scratch.take<double>(static_cast<size_t>(m) * ldv);
  a.ldv = ldv;
  a.w[0] = scratch.take<double>(ldv);
  a.w[1] = scratch.take<double>(ldv);
  double* dinv = scratch.take<double>(ldv);
  a.partial = scratch.take<double>(partials);
  a.st = scratch.take<SolveState>(1);
  if (!a.V || !a.w[0] || !a.w[1] || !dinv || !a.partial || !a.st)
    return fail(ctx, LSMPS_CUDA_ERROR, "scratch exhausted");
  // pinned: what is read back after a cycle, and how far the cycle is
  struct Pinned {
    SolveHead state;
    volatile int progress;
  };
  static thread_local Pinned* pinned = nullptr;
  if (!pinned && cudaMallocHost(&pinned, sizeof(Pinned)) != cudaSuccess) {
    pinned = nullptr;
    return fail(ctx, LSMPS_CUDA_ERROR, "pinned allocation failed");
  }
  a.progress = &pinned->progress;
  a.follow = n > kFollowRows ? 1 : 0;
  a.x = x;
  a.b = b;
  a.restart = m;
  a.max_iters = opt.max_iters;
  a.tolerance = opt.tolerance;
  a.relative = opt.convergence == LSMPS_CONVERGENCE_RELATIVE_INITIAL;
  if (opt.preconditioner == LSMPS_PRECONDITIONER_JACOBI) {
    launch(ctx, jacobi_kernel, dim3(div_up(n, kSolveThreads)), dim3(kSolveThreads), 0, n, a.ro, a.ci, a.va, dinv);
    a.dinv = dinv;
  }
  cudaMemsetAsync(&a.st->tickets, 0, sizeof(unsigned), ctx->stream);
  const SolveHead& st = pinned->state;
  pinned->progress = 0;
  launch_residual(ctx, a, !opt.use_initial_guess, true, g);
  const auto read = [&]() {
    return cudaMemcpyAsync(&pinned->state, static_cast<SolveHead*>(a.st), sizeof(SolveHead), cudaMemcpyDeviceToHost,
                           ctx->stream) == cudaSuccess &&
           cudaStreamSynchronize(ctx->stream) == cudaSuccess;
  };
  // Waits until the cycle has come to `reached`, or until nothing is queued.
  const auto wait = [&](int reached) {
    for (unsigned spins = 1; pinned->progress < reached; ++spins)
      if (spins % 4096 == 0 && cudaStreamQuery(ctx->stream) != cudaErrorNotReady) break;
    return pinned->progress != kStopped;
  };
  for (bool first = true;; first = false) {
    int j = 0;
    for (; j < m && wait(j > 0 && a.follow ? j + 1 - kAhead : 1); ++j) launch_step(ctx, a, j, g);
    if (j > 0) launch(ctx, correct_kernel, dim3(g.stream), dim3(kSolveThreads), 0, a);
    // (without a step the residual stands, but one of x = 0 has not met A yet,
    // whose NaN would show there)
    if (j > 0 || (first && !opt.use_initial_guess)) launch_residual(ctx, a, false, false, g);
    // (a launch that failed leaves the state as it was, and the cycle would come again)
    if (!read() || cudaPeekAtLastError() != cudaSuccess) return check_launch(ctx, "PPE solve");
    if (st.converged || st.iters >= opt.max_iters) break;
    pinned->progress = 1;
  }
  if (opt.clamp_negative) launch(ctx, clamp_kernel, dim3(div_up(n, kSolveThreads)), dim3(kSolveThreads), 0, n, x);
  if (report) *report = lsmps_solver_report{st.iters, st.converged ? 1 : 0, st.beta0, st.beta};
  return check_launch(ctx, "PPE solve");
}

}  // namespace lsmps

using namespace lsmps;

extern "C" void lsmps_solver_options_default(lsmps_solver_options* options) {
  if (options) solver_options_default(options);
}

extern "C" lsmps_status lsmps_solve_ppe(lsmps_ctx* ctx, const lsmps_csr_matrix* matrix, const double* rhs,
                                        double* pressure, const lsmps_solver_options* options,
                                        lsmps_solver_report* report) {
  if (!ctx || !matrix) return LSMPS_INVALID_ARGUMENT;
  lsmps_solver_options opt;
  solver_options_default(&opt);
  if (options) opt = *options;
  lsmps_status st = begin_call(ctx);
  if (st) return st;
  st = solve_ppe_impl(ctx, *matrix, rhs, pressure, opt, report);
  return end_call(ctx, st);
}
