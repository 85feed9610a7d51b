// operators.cu - kernels of the two differentiable operator pairs
// (adjoint.cu: fluid-only operators; step_adjoint.cu: the step's operators
// with their wall terms).
//
// Both pairs are the same computation over four fields of a particle's row:
// three velocity components on the velocity kind's inverse and one scalar (f,
// or the pressure) on the pressure kind's, plus the PPE row of the pressure
// kind.  The fluid-only pair has one inverse for both kinds, takes the
// Laplacian of the scalar instead of the velocity's, and has no walls.  The
// formulas are in the two files' headers.
//
// Mapping: one warp per particle, the lanes over its row.  A row's
// right-hand sides (nine sums for each of four fields and for the PPE rows'
// cotangent) are added over the warp, the inverses are applied out of shared
// memory, and in the backward the row is walked a second time for the entries'
// own terms.
#include <algorithm>
#include <new>
#include <vector>

#include "adjoint.cuh"
#include "impl.cuh"
#include "packed.cuh"

namespace lsmps {
namespace {

constexpr int kAdjThreads = 128;
constexpr int kAdjWarps = kAdjThreads / kWarp;

// s = d / r_e and the Type-A basis of s (moment_matrix.cu:152-175).
__device__ __forceinline__ void basis_div(double dx, double dy, double dz, double inv_re, double b[9], double s[3]) {
  s[0] = dx * inv_re;
  s[1] = dy * inv_re;
  s[2] = dz * inv_re;
  b[0] = s[0];
  b[1] = s[1];
  b[2] = s[2];
  b[3] = s[0] * s[0];
  b[4] = s[1] * s[1];
  b[5] = s[2] * s[2];
  b[6] = s[0] * s[1];
  b[7] = s[1] * s[2];
  b[8] = s[2] * s[0];
}

// J_b(s)^T beta: the derivative of b . beta with respect to s.
__device__ __forceinline__ void basis_jt(const double s[3], const double beta[9], double out[3]) {
  out[0] = beta[0] + 2.0 * s[0] * beta[3] + s[1] * beta[6] + s[2] * beta[8];
  out[1] = beta[1] + 2.0 * s[1] * beta[4] + s[0] * beta[6] + s[2] * beta[7];
  out[2] = beta[2] + 2.0 * s[2] * beta[5] + s[1] * beta[7] + s[0] * beta[8];
}

__device__ __forceinline__ double opt(const double* p, index_t i) { return p ? p[i] : 0.0; }

__device__ __forceinline__ bool dirichlet_row(const int32_t* label, index_t i) {
  if (!label) return false;
  const int t = label[i];
  return t == LSMPS_SURFACE_SURFACE || t == LSMPS_SURFACE_SPLASH;
}

__device__ __forceinline__ bool splash_row(const int32_t* label, index_t i) {
  return label && label[i] == LSMPS_SURFACE_SPLASH;
}

__device__ __forceinline__ double dot9(const double* a, const double* b) {
  double v = 0.0;
#pragma unroll
  for (int k = 0; k < 9; ++k) v = fma(a[k], b[k], v);
  return v;
}

// Entries of a row that a warp holds in shared memory at a time.
constexpr int kRowEntries = 128, kRowRounds = kRowEntries / kWarp;

// Up to kRowEntries entries of a row as its warp works on them: the offsets
// x_j - x_i, the differences of the four fields and the PPE row's cotangent,
// the reciprocal distance, the weight, the neighbour and its record.
struct StagedRow {
  double d[3][kRowEntries];
  double phi[5][kRowEntries];
  double rdist[kRowEntries];
  double w[kRowEntries];
  index_t j[kRowEntries];
  index_t record[kRowEntries];  // the entry's record at its neighbour, or -1
};

// Entries first .. first + count - 1 (count <= kRowEntries) of particle i's
// row into `row`: all rounds' indices, then all their records, are in flight
// together.  ppe_bar: the cotangents of their matrix slots, or NULL.  claim:
// take each entry's record at its neighbour too (all rounds' atomics in flight;
// claimed one after the other, the round trips were a quarter of the kernel).
__device__ __forceinline__ void stage_row(const OperatorArgs& a, const double4& pi, const double4& ui, index_t first,
                                          int count, const double* __restrict__ ppe_bar, double diag_bar,
                                          bool claim, StagedRow& row) {
  if (count <= 0) return;
  const int lane = threadIdx.x & (kWarp - 1);
  index_t j[kRowRounds];
#pragma unroll
  for (int k = 0; k < kRowRounds; ++k) {
    const int e = k * kWarp + lane;
    j[k] = a.fi[first + (e < count ? e : 0)];
  }
  double4 q[kRowRounds], v[kRowRounds];
  index_t rec[kRowRounds];
#pragma unroll
  for (int k = 0; k < kRowRounds; ++k) {
    q[k] = ld4(a.fp, j[k]);
    v[k] = ld4(a.fv, j[k]);
    const bool wanted = claim && k * kWarp + lane < count && j[k] >= a.j0 && j[k] < a.j1;
    rec[k] = wanted ? atomicAdd(&a.next[j[k]], 1) : -1;
  }
  const index_t rec0 = claim ? a.begin[a.j0] : 0;
#pragma unroll
  for (int k = 0; k < kRowRounds; ++k) {
    const int e = k * kWarp + lane;
    const double dx = q[k].x - pi.x, dy = q[k].y - pi.y, dz = q[k].z - pi.z;
    row.d[0][e] = dx;
    row.d[1][e] = dy;
    row.d[2][e] = dz;
    row.phi[0][e] = v[k].x - ui.x;
    row.phi[1][e] = v[k].y - ui.y;
    row.phi[2][e] = v[k].z - ui.z;
    row.phi[3][e] = q[k].w - pi.w;
    row.phi[4][e] = ppe_bar && e < count ? a.c_ppe * (ppe_bar[e] - diag_bar) : 0.0;
    const double dist = sqrt(dx * dx + dy * dy + dz * dz);
    // an entry at distance 0 has weight 1 in the sums and no terms of its own
    row.rdist[e] = dist <= 0.0 ? 0.0 : 1.0 / dist;
    row.w[e] = lin_weight(dist, a.re);
    row.j[e] = j[k];
    row.record[e] = rec[k] < 0 ? -1 : rec[k] - rec0;
  }
}

// The later stretches of a row longer than kRowEntries (a call, so that their
// records in flight do not share the registers of the sums in progress).
__device__ __noinline__ void stage_row_again(const OperatorArgs& a, const double4& pi, const double4& ui,
                                             index_t first, int count, const double* __restrict__ ppe_bar,
                                             double diag_bar, bool claim, StagedRow& row) {
  __syncwarp();
  stage_row(a, pi, ui, first, count, ppe_bar, diag_bar, claim, row);
  __syncwarp();
}

// Forward: the operators and the PPE row of one particle per warp, entries
// written a warp at a time (consecutive slots).  The rows of the inverses that
// the outputs need are applied to each entry's basis vector, read from shared
// memory by broadcast: 8 sums a lane instead of the 36 right-hand sides, so that
// 20 warps per SM are resident where 8 were, for 72 fused products an entry
// instead of 45.  262,144 particles: 0.67 ms (0.90 with the right-hand sides;
// 0.88 with one thread a particle, which wrote its row slot by slot).
template <bool Walls>
__global__ void __launch_bounds__(kAdjThreads, 5) operators_forward_kernel(OperatorArgs a) {
  wait_for_previous();
  // per warp: the Laplacian row of the scalar's (pressure's) inverse, its rows
  // 0..2, rows 0..2 of the velocity's and, with walls, its Laplacian row
  __shared__ __align__(16) double s_row[kAdjWarps][8][10];
  const int lane = threadIdx.x & (kWarp - 1), warp = threadIdx.x / kWarp;
  const index_t i = blockIdx.x * kAdjWarps + warp;
  if (i >= a.n) return;  // the whole warp
  {
    const size_t at = static_cast<size_t>(i) * 81;
    for (int e = lane; e < (Walls ? 72 : 63); e += kWarp) {
      const int r = e / 9, c = e % 9;
      const double* x = (r < 4 ? a.inv_p : a.inv_v) + at + 9 * c;
      s_row[warp][r][c] = r == 0 || r == 7 ? x[3] + x[4] + x[5] : x[r < 4 ? r - 1 : r - 4];
    }
    __syncwarp();
  }
  const double(*row_of)[10] = s_row[warp];
  const auto row_dot = [&](int r, const double* b) {
    const double2* p = reinterpret_cast<const double2*>(row_of[r]);
    double v = 0.0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const double2 x = p[k];
      v = fma(x.x, b[2 * k], v);
      v = fma(x.y, b[2 * k + 1], v);
    }
    return fma(row_of[r][8], b[8], v);
  };
  const double4 pi = ld4(a.fp, i), ui = ld4(a.fv, i);
  const bool dir = Walls && dirichlet_row(a.label, i);
  const bool ppe = a.values != nullptr;
  const index_t nb = a.fo[i], ne = a.fo[i + 1];
  const index_t slot = i + nb;
  // gradient (0..2), Laplacian (3..5 of the velocity, or 3 of the scalar),
  // divergence (6), diagonal (7), wall source
  double r[8], wall_rhs = 0.0, b[9], s[3];
#pragma unroll
  for (int k = 0; k < 8; ++k) r[k] = 0.0;
  index_t o = nb + lane;
  index_t jn = o < ne ? a.fi[o] : i;
  double4 qn = ld4(a.fp, jn), vn = ld4(a.fv, jn);
  index_t jnn = o + kWarp < ne ? a.fi[o + kWarp] : i;
  for (; o < ne; o += kWarp) {
    // the next entry's records, and the index after that, are loaded while
    // this one is summed
    const index_t j = jn;
    const double4 q = qn, v = vn;
    if (o + kWarp < ne) {
      jn = jnn;
      qn = ld4(a.fp, jn);
      vn = ld4(a.fv, jn);
      if (o + 2 * kWarp < ne) jnn = a.fi[o + 2 * kWarp];
    }
    const double dx = q.x - pi.x, dy = q.y - pi.y, dz = q.z - pi.z;
    const double w = lin_weight(sqrt(dx * dx + dy * dy + dz * dz), a.re);
    double coef = 0.0;
    if (w > 0.0) {
      basis_div(dx, dy, dz, a.inv_re, b, s);
      const double lb = row_dot(0, b);
      const double wx = w * (v.x - ui.x), wy = w * (v.y - ui.y), wz = w * (v.z - ui.z), wf = w * (q.w - pi.w);
#pragma unroll
      for (int c = 0; c < 3; ++c) r[c] = fma(wf, row_dot(1 + c, b), r[c]);
      r[6] = fma(wx, row_dot(4, b), r[6]);
      r[6] = fma(wy, row_dot(5, b), r[6]);
      r[6] = fma(wz, row_dot(6, b), r[6]);
      if (Walls) {
        const double lv = row_dot(7, b);
        r[3] = fma(wx, lv, r[3]);
        r[4] = fma(wy, lv, r[4]);
        r[5] = fma(wz, lv, r[5]);
      } else {
        r[3] = fma(wf, lb, r[3]);
      }
      if (ppe && !dir) {
        coef = a.c_ppe * w * lb;
        r[7] -= coef;
      }
    }
    if (a.columns) a.columns[slot + 1 + o - nb] = j;
    if (ppe) a.values[slot + 1 + o - nb] = coef;
  }
  if (Walls) {
    const index_t we = a.wo[i + 1];
    for (index_t o = a.wo[i] + lane; o < we; o += kWarp) {
      const index_t j = a.wi[o];
      const double4 q = ld4(a.wp, j), v = ld4(a.wv, j), nrm = ld4(a.wn, j);
      const double dx = q.x - pi.x, dy = q.y - pi.y, dz = q.z - pi.z;
      const double w = lin_weight(sqrt(dx * dx + dy * dy + dz * dz), a.re);
      if (w <= 0.0) continue;
      const double om = a.lam_w * w;
      basis_div(dx, dy, dz, a.inv_re, b, s);
      const double wx = om * (v.x - ui.x), wy = om * (v.y - ui.y), wz = om * (v.z - ui.z);
      r[6] = fma(wx, row_dot(4, b), r[6]);
      r[6] = fma(wy, row_dot(5, b), r[6]);
      r[6] = fma(wz, row_dot(6, b), r[6]);
      const double lv = row_dot(7, b);
      r[3] = fma(wx, lv, r[3]);
      r[4] = fma(wy, lv, r[4]);
      r[5] = fma(wz, lv, r[5]);
      neumann_a(dx, dy, dz, nrm.x, nrm.y, nrm.z, a.inv_re, b);
      const double gn = a.gx * nrm.x + a.gy * nrm.y + a.gz * nrm.z;
      const double src = om * (a.re * a.rho * gn);
#pragma unroll
      for (int c = 0; c < 3; ++c) r[c] = fma(src, row_dot(1 + c, b), r[c]);
      wall_rhs += 2.0 * om * gn * row_dot(0, b) * a.inv_re;
    }
    wall_rhs = group_sum<kWarp>(wall_rhs, 0xffffffffu);
  }
  int base = 0, count = 8;
  lane_totals<8, 16>(r, base, count);  // lane 4 k holds total k
  const double t = r[0];
  const double diag = __shfl_sync(0xffffffffu, t, 28);
  if ((lane & 3) != 0) return;
  // (each output by its own pointer: any may be missing)
  if (base < 3) {
    double* grad = base == 0 ? a.grad[0] : base == 1 ? a.grad[1] : a.grad[2];
    if (grad) grad[i] = Walls && splash_row(a.label, i) ? 0.0 : t * a.inv_re;
  } else if (base < (Walls ? 6 : 4)) {
    double* lap = !Walls ? a.lap_f : base == 3 ? a.lap_u[0] : base == 4 ? a.lap_u[1] : a.lap_u[2];
    if (lap) lap[i] = 2.0 * t * a.inv_re * a.inv_re;
  } else if (base == 6) {
    const double div = dir ? 0.0 : t * a.inv_re;
    if (dir) wall_rhs = 0.0;
    if (a.div) a.div[i] = div;
    if (Walls && a.wall_rhs) a.wall_rhs[i] = wall_rhs;
    if (a.rhs) a.rhs[i] = dir ? 0.0 : div * a.inv_dt - wall_rhs;
    if (a.row_offsets) {
      a.row_offsets[i] = slot;
      if (i + 1 == a.n) a.row_offsets[a.n] = a.n + ne;
    }
    if (a.columns) a.columns[slot] = i;
    if (ppe) a.values[slot] = dir ? 1.0 : diag;
  }
}

// Backward, one particle's row per warp: the cotangents of its moment
// systems (Rbar, y of the four fields, hhat and l of the PPE row, in shared
// memory) and from them the terms of each of its entries, computed once.  The
// owner's share is summed over the warp; the neighbour's goes into the
// neighbour's next free record as one 64-byte line (Atomic: is added to the
// outputs).
//
// Bounded by the load pipe (ncu: 70% of its wavefronts, FP64 33%): half of them
// are the 90 values that every entry reads by broadcast (512 bytes to a warp's
// registers each, four cycles), the rest the scattered records.  Tried: two
// entries a lane for each broadcast (2.30 ms: 12 warps per SM instead of 16); five
// lanes an entry, each with one of the five vector pairs in registers (2.96 ms:
// the entry's own values are then read five times over).  262,144 particles,
// 28 M entries: 2.17 ms, and 0.53 ms to collect the records.  Before, every
// entry was evaluated twice, by its owner's thread and by its neighbour's, each
// reading the owner's 736-byte stash from global memory word by word: 11.5 ms,
// 1.24 ms for the stash and 1.3 ms for a transpose of the table.
template <bool Walls, bool Atomic>
__global__ void __launch_bounds__(kAdjThreads, 4) operators_backward_kernel(const __grid_constant__ OperatorArgs a) {
  wait_for_previous();
  extern __shared__ __align__(16) unsigned char s_rows[];  // a StagedRow per warp
  __shared__ double s_r[kAdjWarps][82];      // 45 sums, the 36 cotangents of y
  __shared__ double2 s_st[kAdjWarps][5][9];  // {Rbar, y} of the four fields, {hhat, l}
  const unsigned all = 0xffffffffu;
  const int lane = threadIdx.x & (kWarp - 1), warp = threadIdx.x / kWarp;
  const index_t i = blockIdx.x * kAdjWarps + warp;
  if (i >= a.n) return;  // the whole warp
  const double* __restrict__ xv = a.inv_v + static_cast<size_t>(i) * 81;
  const double* __restrict__ xp = a.inv_p + static_cast<size_t>(i) * 81;
  const double4 pi = ld4(a.fp, i), ui = ld4(a.fv, i);
  const bool dir = Walls && dirichlet_row(a.label, i);
  const bool ppe = a.values != nullptr && !dir;
  const index_t nb = a.fo[i], ne = a.fo[i + 1];
  const double diag_bar = ppe ? a.values[i + nb] : 0.0;
  const double* ppe_bar = ppe ? a.values + (i + nb + 1) : nullptr;
  const double wrb = Walls && !dir ? opt(a.wall_rhs, i) - opt(a.rhs, i) : 0.0;
  StagedRow& row = reinterpret_cast<StagedRow*>(s_rows)[warp];
  double* R = s_r[warp];
  bool some = false;  // a positive trace
  {
    // R_f = sum w b dphi_f of the four fields and h = sum w b ab.  The two
    // halves of the warp take the same entries and three of the five
    // coefficients each, (dphi_0..2) and (dphi_3, ab, -): 27 sums a lane.
    stage_row(a, pi, ui, nb, min(kRowEntries, ne - nb), ppe_bar, diag_bar, !Atomic && ne - nb <= kRowEntries, row);
    __syncwarp();
    const int half = lane / 16, hl = lane % 16;
    const double(*phi)[kRowEntries] = row.phi + 3 * half;
    double r[27], b[9], s[3];
#pragma unroll
    for (int k = 0; k < 27; ++k) r[k] = 0.0;
    for (index_t first = nb; first < ne; first += kRowEntries) {
      const int many = min(kRowEntries, ne - first);
      if (first > nb) stage_row_again(a, pi, ui, first, many, ppe_bar + (ppe ? first - nb : 0), diag_bar, false, row);
#pragma unroll 1
      for (int e = hl; e < many; e += 16) {
        const double w = row.w[e];
        if (w <= 0.0) continue;
        basis_div(row.d[0][e], row.d[1][e], row.d[2][e], a.inv_re, b, s);
        if (!Walls) some |= w * (b[3] + b[4] + b[5]) > 0.0;
        const double c0 = w * phi[0][e], c1 = w * phi[1][e], c2 = half ? 0.0 : w * row.phi[2][e];
#pragma unroll
        for (int k = 0; k < 9; ++k) {
          r[k] = fma(c0, b[k], r[k]);
          r[9 + k] = fma(c1, b[k], r[9 + k]);
          r[18 + k] = fma(c2, b[k], r[18 + k]);
        }
      }
    }
    if (Walls) {
      const index_t we = a.wo[i + 1];
      for (index_t o = a.wo[i] + hl; o < we; o += 16) {
        const index_t j = a.wi[o];
        const double4 q = ld4(a.wp, j), v = ld4(a.wv, j), nrm = ld4(a.wn, j);
        const double dx = q.x - pi.x, dy = q.y - pi.y, dz = q.z - pi.z;
        const double w = lin_weight(sqrt(dx * dx + dy * dy + dz * dz), a.re);
        if (w <= 0.0) continue;
        const double om = a.lam_w * w;
        double c0 = om * (v.x - ui.x), c1 = om * (v.y - ui.y), c2 = om * (v.z - ui.z);
        if (half) {  // the wall Neumann vector, its gradient source and h's
          const double gn = a.gx * nrm.x + a.gy * nrm.y + a.gz * nrm.z;
          neumann_a(dx, dy, dz, nrm.x, nrm.y, nrm.z, a.inv_re, b);
          c0 = om * (a.re * a.rho * gn);
          c1 = 2.0 * om * gn * a.inv_re * wrb;
          c2 = 0.0;
        } else {
          basis_div(dx, dy, dz, a.inv_re, b, s);
        }
#pragma unroll
        for (int k = 0; k < 9; ++k) {
          r[k] = fma(c0, b[k], r[k]);
          r[9 + k] = fma(c1, b[k], r[9 + k]);
          r[18 + k] = fma(c2, b[k], r[18 + k]);
        }
      }
    }
    int base = 0, count = 27;
    lane_totals<27, 8>(r, base, count);  // over the 16 lanes of a half: at most 2 left a lane
#pragma unroll
    for (int k = 0; k < 2; ++k)
      if (k < count && 27 * half + base + k < 45) R[27 * half + base + k] = r[k];
  }
  // Cotangents of the y's: the divergence (and rhs = div / dt - wall_rhs) on
  // component c of field c, the Laplacian on components 3..5 (of the velocity
  // with walls, of the scalar without), the gradient on the scalar's 0..2.
  {
    const double dbar = dir ? 0.0 : (opt(a.div, i) + opt(a.rhs, i) * a.inv_dt) * a.inv_re;
    const double l2 = 2.0 * a.inv_re * a.inv_re;
    const bool spl = Walls && splash_row(a.label, i);
    for (int e = lane; e < 36; e += kWarp) {
      const int ft = e / 9, k = e % 9;
      double t = 0.0;
      if (ft < 3) {
        if (k == ft) t = dbar;
        if (Walls && k >= 3 && k <= 5) t = l2 * opt(a.lap_u[ft], i);
      } else {
        if (k < 3 && !spl) t = opt(a.grad[k], i) * a.inv_re;
        if (!Walls && k >= 3 && k <= 5) t = l2 * opt(a.lap_f, i);
      }
      R[45 + e] = t;
    }
    __syncwarp();
  }
  // y_f = X R_f and hhat = X h, Rbar_f = X t_f, l: 90 values over the lanes
  for (int e = lane; e < 90; e += kWarp) {
    const int v = e / 9, k = e % 9;  // 0..3 y, 4 hhat, 5..8 Rbar, 9 l
    const int g = v < 5 ? v : v - 5;
    double z = 0.0;
    if (v < 9) {
      const double* x = g < 3 ? xv : xp;
      const double* rr = v < 5 ? R + 9 * v : R + 45 + 9 * g;
#pragma unroll
      for (int c = 0; c < 9; ++c) z = fma(x[k + 9 * c], rr[c], z);
    } else {
      z = xp[3 + 9 * k] + xp[4 + 9 * k] + xp[5 + 9 * k];
    }
    double2& st = s_st[warp][g][k];
    if (v < 4 || v == 9)
      st.y = z;
    else
      st.x = z;
  }
  __syncwarp();
  const double2(*st)[9] = s_st[warp];
  // regularisation factors lambda / 9 sum Rbar . y (+ hhat . l) of the kinds
  double reg_v = 0.0, reg_p = 0.0;
  for (int e = lane; e < 45; e += kWarp) {
    const double2 p = st[e / 9][e % 9];
    (e < 27 ? reg_v : reg_p) += p.x * p.y;
  }
  reg_v = group_sum<kWarp>(reg_v, all);
  reg_p = group_sum<kWarp>(reg_p, all);
  const double lam9 = a.lambda / 9.0;
  some = Walls ? false : __any_sync(all, some) != 0;
  reg_v = (Walls ? a.tr_v[i] > 0.0 : some) ? reg_v * lam9 : 0.0;
  reg_p = (Walls ? a.tr_p[i] > 0.0 : some) ? reg_p * lam9 : 0.0;
  double acc[7];  // the owner's share: four fields, then the position
#pragma unroll
  for (int c = 0; c < 7; ++c) acc[c] = 0.0;
  for (index_t first = nb; first < ne; first += kRowEntries) {
    const int many = min(kRowEntries, ne - first);
    if (ne - nb > kRowEntries)
      stage_row_again(a, pi, ui, first, many, ppe_bar + (ppe ? first - nb : 0), diag_bar, !Atomic, row);
#pragma unroll 1
    for (int round = 0; round < many; round += kWarp) {
      // (also keeps the loads of the 90 values inside the loop: hoisted out of
      // it, they lived in spilled registers, 5.1 ms)
      __syncwarp();
      const int e = round + lane;
      if (e >= many) continue;
      const double w = row.w[e], rd = row.rdist[e];
      const bool live = !(w <= 0.0 || rd == 0.0);
      double t[4] = {0.0, 0.0, 0.0, 0.0}, g[3] = {0.0, 0.0, 0.0};
      if (live) {
        double b[9], s[3], beta[9];
        basis_div(row.d[0][e], row.d[1][e], row.d[2][e], a.inv_re, b, s);
        // alpha = dL/dw, beta = (dL/db) / w
        const double r2 = -2.0 * (reg_v + reg_p);
        double alpha = 0.5 * r2 * dot9(b, b);
#pragma unroll
        for (int k = 0; k < 9; ++k) beta[k] = r2 * b[k];
#pragma unroll
        for (int f = 0; f < 5; ++f) {
          double2 p[9];
          double px = 0.0, qy = 0.0;
#pragma unroll
          for (int k = 0; k < 9; ++k) {
            p[k] = st[f][k];
            px = fma(p[k].x, b[k], px);
            qy = fma(p[k].y, b[k], qy);
          }
          // field f: alpha += p (dphi - q), beta += Rbar (dphi - q) - p y;
          // PPE row: alpha += (ab - p) q, beta += (ab - p) l - q hhat
          const double phi = row.phi[f][e];
          const double ax = f < 4 ? phi - qy : -qy;
          const double ay = f < 4 ? -px : phi - px;
          alpha = f < 4 ? fma(px, ax, alpha) : fma(ay, qy, alpha);
          if (f < 4) t[f] = w * px;
#pragma unroll
          for (int k = 0; k < 9; ++k) beta[k] = fma(ax, p[k].x, fma(ay, p[k].y, beta[k]));
        }
        // dL/dd = (-alpha d/|d| + J_b(s)^T (w beta)) / r_e
        double jt[3];
        basis_jt(s, beta, jt);
        const double ad = -alpha * rd;
#pragma unroll
        for (int c = 0; c < 3; ++c) g[c] = fma(ad, row.d[c][e], w * jt[c]) * a.inv_re;
#pragma unroll
        for (int f = 0; f < 4; ++f) acc[f] -= t[f];
#pragma unroll
        for (int c = 0; c < 3; ++c) acc[4 + c] -= g[c];
      }
      if (Atomic) {
        if (!live) continue;
        const index_t j = row.j[e];
#pragma unroll
        for (int f = 0; f < 4; ++f)
          if (a.phibar[f]) atomicAdd(&a.phibar[f][j], t[f]);
#pragma unroll
        for (int c = 0; c < 3; ++c)
          if (a.xbar[c]) atomicAdd(&a.xbar[c][j], g[c]);
      } else if (row.record[e] >= 0) {
        double4* rec = a.records + 2 * static_cast<size_t>(row.record[e]);
        rec[0] = make_double4(t[0], t[1], t[2], t[3]);
        rec[1] = make_double4(g[0], g[1], g[2], __longlong_as_double(static_cast<long long>(first + e)));
      }
    }
  }
  if (Walls) {  // the wall row: only the owner's cotangents (walls are held fixed)
    const index_t we = a.wo[i + 1];
    for (index_t o = a.wo[i] + lane; o < we; o += kWarp) {
      const index_t j = a.wi[o];
      const double4 q = ld4(a.wp, j), v = ld4(a.wv, j), nrm = ld4(a.wn, j);
      const double dx = q.x - pi.x, dy = q.y - pi.y, dz = q.z - pi.z;
      const double dist = sqrt(dx * dx + dy * dy + dz * dz);
      const double w = lin_weight(dist, a.re);
      if (w <= 0.0 || dist <= 0.0) continue;
      const double om = a.lam_w * w;
      double b[9], s[3], beta[9], jt[3];
      // velocity kind, Dirichlet samples: alpha = dL/domega, beta = dL/db over omega
      basis_div(dx, dy, dz, a.inv_re, b, s);
      const double du[3] = {v.x - ui.x, v.y - ui.y, v.z - ui.z};
      double alpha = -reg_v * dot9(b, b);
#pragma unroll
      for (int k = 0; k < 9; ++k) beta[k] = -2.0 * reg_v * b[k];
#pragma unroll
      for (int f = 0; f < 3; ++f) {
        double2 p[9];
        double rb = 0.0, by = 0.0;
#pragma unroll
        for (int k = 0; k < 9; ++k) {
          p[k] = st[f][k];
          rb = fma(p[k].x, b[k], rb);
          by = fma(p[k].y, b[k], by);
        }
        const double e = du[f] - by;
        alpha = fma(rb, e, alpha);
#pragma unroll
        for (int k = 0; k < 9; ++k) beta[k] = fma(p[k].x, e, fma(-rb, p[k].y, beta[k]));
        acc[f] -= om * rb;
      }
      basis_jt(s, beta, jt);
      // pressure kind, Neumann terms and the PPE wall source, on q
      neumann_a(dx, dy, dz, nrm.x, nrm.y, nrm.z, a.inv_re, b);
      const double gn = a.gx * nrm.x + a.gy * nrm.y + a.gz * nrm.z;
      double rq = 0.0, qy = 0.0, hq = 0.0, lq = 0.0;
#pragma unroll
      for (int k = 0; k < 9; ++k) {
        const double2 p = st[3][k], h = st[4][k];
        rq = fma(p.x, b[k], rq);
        qy = fma(p.y, b[k], qy);
        hq = fma(h.x, b[k], hq);
        lq = fma(h.y, b[k], lq);
      }
      const double e = a.re * a.rho * gn - qy;
      const double m = 2.0 * gn * a.inv_re * wrb - hq;
      alpha += fma(rq, e, fma(m, lq, -reg_p * dot9(b, b)));
#pragma unroll
      for (int k = 3; k < 9; ++k) {  // J_q comes from q3..q8 (linear in s)
        const double2 p = st[3][k], h = st[4][k];
        beta[k] = fma(p.x, e, -rq * p.y) + fma(m, h.y, -lq * h.x) - 2.0 * reg_p * b[k];
      }
      jt[0] += 2.0 * nrm.x * beta[3] + nrm.y * beta[6] + nrm.z * beta[8];
      jt[1] += 2.0 * nrm.y * beta[4] + nrm.x * beta[6] + nrm.z * beta[7];
      jt[2] += 2.0 * nrm.z * beta[5] + nrm.y * beta[7] + nrm.x * beta[8];
      const double ad = -a.lam_w * alpha / dist;
      acc[4] -= fma(ad, dx, om * jt[0]) * a.inv_re;
      acc[5] -= fma(ad, dy, om * jt[1]) * a.inv_re;
      acc[6] -= fma(ad, dz, om * jt[2]) * a.inv_re;
    }
  }
  if (!Atomic && a.j0 != 0) return;  // a later pass over the same rows
  int base = 0, count = 7;
  lane_totals<7, 16>(acc, base, count);
  // lanes that differ in the last two exchanges hold the same total
  if (count == 0 || (lane & 3) != 0) return;
  if (Atomic) {
    double* out = base < 4 ? a.phibar[base] : a.xbar[base - 4];
    if (out) atomicAdd(&out[i], acc[0]);
  } else {
    a.own[8 * static_cast<size_t>(i) + base] = acc[0];
  }
}

// Entries ranked at a time in the last pass of the deterministic backward.
constexpr int kRankWindow = 128, kRankPer = kRankWindow / kWarp;

// The entry id of record e, and the place of the e-th in order where a row has more
// than kRankWindow records: the halves of a record's last double.
__device__ __forceinline__ int* record_half(double4* rec, int e, int upper) {
  return reinterpret_cast<int*>(rec + 2 * static_cast<size_t>(e) + 1) + 6 + upper;
}

// rank[k] += how many of ids[0 .. many - 1] come before mine[k] (past the end:
// INT32_MAX, before none).
__device__ __forceinline__ void add_ranks(const int* ids, int many, const int (&mine)[kRankPer], int (&rank)[kRankPer]) {
  for (int c = 0; c < many; c += 4) {
    const int4 v = *reinterpret_cast<const int4*>(ids + c);
#pragma unroll
    for (int k = 0; k < kRankPer; ++k)
      rank[k] += (v.x < mine[k]) + (v.y < mine[k]) + (v.z < mine[k]) + (v.w < mine[k]);
  }
}

// The order of more than kRankWindow records, into their upper halves.
__device__ __noinline__ void order_long_row(double4* rec, int count, int* ids) {
  const int lane = threadIdx.x & (kWarp - 1);
  for (int e0 = 0; e0 < count; e0 += kRankWindow) {
    int mine[kRankPer], rank[kRankPer];
#pragma unroll
    for (int k = 0; k < kRankPer; ++k) {
      const int e = e0 + k * kWarp + lane;
      mine[k] = e < count ? *record_half(rec, e, 0) : INT32_MAX;
      rank[k] = 0;
    }
    for (int c0 = 0; c0 < count; c0 += kRankWindow) {
      __syncwarp();
#pragma unroll
      for (int k = 0; k < kRankPer; ++k) {
        const int c = c0 + k * kWarp + lane;
        ids[k * kWarp + lane] = c < count ? *record_half(rec, c, 0) : INT32_MAX;
      }
      __syncwarp();
      add_ranks(ids, min(kRankWindow, count - c0), mine, rank);
    }
#pragma unroll
    for (int k = 0; k < kRankPer; ++k) {
      const int e = e0 + k * kWarp + lane;
      if (e < count) *record_half(rec, rank[k], 1) = e;
    }
  }
  __syncwarp();
}

// Deterministic form, last pass: particle j adds its incoming entries' terms
// in ascending entry order, whatever order their records arrived in (lane l
// takes the l-th, the (l + 32)-th, ..., then a fixed tree), to its own row's.
// One warp per particle; the arrival order is undone by ranking the entry ids.
// A row of 108 costs the ranking about 900 warp instructions, half of what the
// 64-byte records' own transfer takes; one of more than 128 is ranked 128 at a
// time against 128.  The whole backward of 64,000 particles with rows of 281
// entries 2.4 ms, of 956 10.4, of 4,000 with 3,999 10.1 (3.5, 42.7 and 260 with the
// ranks found anew for every 128 in order).
__global__ void __launch_bounds__(kAdjThreads) operators_collect_kernel(OperatorArgs a) {
  wait_for_previous();
  __shared__ __align__(16) int s_id[kAdjWarps][kRankWindow];
  __shared__ int s_at[kAdjWarps][kRankWindow];
  const int lane = threadIdx.x & (kWarp - 1), warp = threadIdx.x / kWarp;
  const index_t j = a.j0 + blockIdx.x * kAdjWarps + warp;
  if (j >= a.j1) return;  // the whole warp
  const size_t first = static_cast<size_t>(a.begin[j] - a.begin[a.j0]);
  const int count = a.begin[j + 1] - a.begin[j];
  const double4* rec = a.records + 2 * first;
  int* ids = s_id[warp];
  int* at = s_at[warp];
  const bool few = count <= kRankWindow;
  if (few) {
    int mine[kRankPer], rank[kRankPer];
#pragma unroll
    for (int k = 0; k < kRankPer; ++k) {
      const int e = k * kWarp + lane;
      mine[k] = e < count ? static_cast<int>(__double_as_longlong(rec[2 * static_cast<size_t>(e) + 1].w)) : INT32_MAX;
      rank[k] = 0;
      ids[e] = mine[k];
    }
    __syncwarp();
    add_ranks(ids, count, mine, rank);
#pragma unroll
    for (int k = 0; k < kRankPer; ++k) {
      const int e = k * kWarp + lane;
      if (e < count) at[rank[k]] = e;
    }
    __syncwarp();
  } else {
    order_long_row(a.records + 2 * first, count, ids);
  }
  double acc[7];
#pragma unroll
  for (int c = 0; c < 7; ++c) acc[c] = 0.0;
  for (int k = lane; k < count; k += kWarp) {
    const int e = few ? at[k] : __ldcg(record_half(a.records + 2 * first, k, 1));
    const double4 r0 = ld4(rec, 2 * e), r1 = ld4(rec, 2 * e + 1);
    acc[0] += r0.x;
    acc[1] += r0.y;
    acc[2] += r0.z;
    acc[3] += r0.w;
    acc[4] += r1.x;
    acc[5] += r1.y;
    acc[6] += r1.z;
  }
  int base = 0, left = 7;
  lane_totals<7, 16>(acc, base, left);
  if (left == 0 || (lane & 3) != 0) return;
  double* out = base < 4 ? a.phibar[base] : a.xbar[base - 4];
  if (out) out[j] = acc[0] + a.own[8 * static_cast<size_t>(j) + base];
}

// Incoming entries of every particle: count[j] += 1 for each entry that lists
// j (eight lanes per row).
__global__ void __launch_bounds__(kAdjThreads) incoming_count_kernel(const index_t* __restrict__ fo,
                                                                     const index_t* __restrict__ fi, index_t n,
                                                                     index_t* __restrict__ count) {
  wait_for_previous();
  const index_t i = static_cast<index_t>((static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) / 8);
  if (i >= n) return;
  const index_t ne = fo[i + 1];
  for (index_t o = fo[i] + (threadIdx.x & 7); o < ne; o += 8) {
    const index_t j = fi[o];
    if (j >= 0 && j < n) atomicAdd(&count[j], 1);
  }
}

// Most bytes of records that one pass over the rows may hold.  226 M entries
// (2 M particles) take 14.5 GB; a larger set is done in passes over the
// neighbours' index range, each evaluating every row's entries again.  (The
// bounds-checked build makes its passes small, so that its tests take several.)
#ifdef LSMPS_BOUNDS_CHECK
constexpr size_t kRecordBytes = size_t(1) << 20;
#else
constexpr size_t kRecordBytes = size_t(16) << 30;
#endif

constexpr size_t kStagedBytes = kAdjWarps * sizeof(StagedRow);  // 44 KB

template <bool Walls, bool Atomic>
void launch_rows(lsmps_ctx* ctx, const OperatorArgs& a) {
  cudaFuncSetAttribute(operators_backward_kernel<Walls, Atomic>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       static_cast<int>(kStagedBytes));
  launch_named(ctx, Walls ? "operators_backward_kernel<walls>" : "operators_backward_kernel<fluid>",
               operators_backward_kernel<Walls, Atomic>, dim3(div_up(a.n, kAdjWarps)), dim3(kAdjThreads), kStagedBytes, a);
}

}  // namespace

lsmps_status operators_forward(lsmps_ctx* ctx, const OperatorArgs& a, bool walls) {
  const dim3 grid(div_up(a.n, kAdjWarps)), block(kAdjThreads);
  if (walls)
    launch_named(ctx, "operators_forward_kernel<walls>", operators_forward_kernel<true>, grid, block, 0, a);
  else
    launch_named(ctx, "operators_forward_kernel<fluid>", operators_forward_kernel<false>, grid, block, 0, a);
  return check_launch(ctx, "operators forward");
}

lsmps_status operators_backward(lsmps_ctx* ctx, const lsmps_csr& fn, OperatorArgs a, bool walls) {
  const size_t n = static_cast<size_t>(a.n);
  a.j0 = 0;
  a.j1 = a.n;
  if (ctx->adjoint_atomic) {  // accumulates into the gradients: start from zero
    for (double* o : {a.phibar[0], a.phibar[1], a.phibar[2], a.phibar[3], a.xbar[0], a.xbar[1], a.xbar[2]})
      if (o) cudaMemsetAsync(o, 0, n * sizeof(double), ctx->stream);
    if (walls)
      launch_rows<true, true>(ctx, a);
    else
      launch_rows<false, true>(ctx, a);
    return check_launch(ctx, "operators backward");
  }
  index_t total = 0;
  if (cudaMemcpyAsync(&total, fn.offsets + n, sizeof(index_t), cudaMemcpyDeviceToHost, ctx->stream) != cudaSuccess ||
      cudaStreamSynchronize(ctx->stream) != cudaSuccess)
    return fail(ctx, LSMPS_CUDA_ERROR, "reading the neighbour count failed");
  if (total < 0 || static_cast<size_t>(total) > fn.neighbor_count)
    return fail(ctx, LSMPS_INVALID_ARGUMENT, "neighbour table offsets exceed its capacity");
  const size_t entry = 2 * sizeof(double4);
  const size_t fixed = 2 * (n + 1) * sizeof(index_t) + 8 * n * sizeof(double) + scan_scratch_bytes(n) + 4096;
  size_t most = std::min(kRecordBytes, static_cast<size_t>(total) * entry);
  if (ctx->record_limit && most > ctx->record_limit) {
    // memory was short before: no more is tried for (which would give up the scratch
    // at hand) until there is that much
    size_t room = 0, all = 0;
    if (cudaMemGetInfo(&room, &all) == cudaSuccess && room + ctx->scratch_bytes >= fixed + most + kScratchGrowth)
      ctx->record_limit = 0;
    else
      most = ctx->record_limit;
  }
  const size_t wanted = most;
  Scratch scratch(ctx);
  while (!scratch.reserve(fixed + most)) {  // less room: more passes
    most /= 2;
    if (most < (size_t(1) << 20)) return fail(ctx, LSMPS_CUDA_ERROR, "operator scratch allocation failed");
  }
  if (most < wanted) ctx->record_limit = most;
  index_t* begin = scratch.take<index_t>(n + 1);
  a.begin = begin;
  a.next = scratch.take<index_t>(n + 1);
  a.own = scratch.take<double>(8 * n);
  if (!begin || !a.next || !a.own) return fail(ctx, LSMPS_CUDA_ERROR, "operator scratch exhausted");
  cudaMemsetAsync(begin, 0, (n + 1) * sizeof(index_t), ctx->stream);
  launch(ctx, incoming_count_kernel, dim3(div_up(static_cast<long long>(n) * 8, kAdjThreads)), dim3(kAdjThreads), 0,
         a.fo, a.fi, a.n, begin);
  lsmps_status st = exclusive_scan_i32(ctx, scratch, begin, begin, n, nullptr, begin + n);
  if (st) return st;
  if (cudaMemcpyAsync(a.next, begin, n * sizeof(index_t), cudaMemcpyDeviceToDevice, ctx->stream) != cudaSuccess)
    return check_launch(ctx, "operators backward");
  a.records = scratch.take<double4>(most / sizeof(double4));
  if (!a.records) return fail(ctx, LSMPS_CUDA_ERROR, "operator scratch exhausted");
  std::vector<index_t> first;
  if (most < static_cast<size_t>(total) * entry) {
    try {
      first.resize(n + 1);
    } catch (const std::bad_alloc&) {
      return fail(ctx, LSMPS_CUDA_ERROR, "operator scratch allocation failed");
    }
    if (cudaMemcpyAsync(first.data(), begin, (n + 1) * sizeof(index_t), cudaMemcpyDeviceToHost, ctx->stream) !=
            cudaSuccess ||
        cudaStreamSynchronize(ctx->stream) != cudaSuccess)
      return fail(ctx, LSMPS_CUDA_ERROR, "reading the incoming counts failed");
  }
  const long long room = static_cast<long long>(most / entry);
  for (index_t j0 = 0; j0 < a.n; j0 = a.j1) {
    a.j0 = j0;
    if (!first.empty()) {
      const auto end = std::upper_bound(first.begin() + j0 + 1, first.end(), first[j0] + room,
                                        [](long long v, index_t f) { return v < static_cast<long long>(f); });
      a.j1 = static_cast<index_t>(end - first.begin()) - 1;
      if (a.j1 <= j0) return fail(ctx, LSMPS_CUDA_ERROR, "operator scratch allocation failed");
    }
    if (walls)
      launch_rows<true, false>(ctx, a);
    else
      launch_rows<false, false>(ctx, a);
    launch(ctx, operators_collect_kernel, dim3(div_up(a.j1 - j0, kAdjWarps)), dim3(kAdjThreads), 0, a);
  }
  return check_launch(ctx, "operators backward");
}

}  // namespace lsmps
