// step_adjoint.cu - the step's LSMPS operators with their wall terms as a
// forward/backward pair (no counterpart in the reference, which has no
// derivatives).
//
// Per fluid particle i, over its fluid row N(i) and wall row W(i), with
// s = d / r_e, w = 1 - |s| (moment_matrix.cu:145-150), b the Type-A basis,
// q the wall Neumann vector of the wall's normal n (moment_matrix.cu:177-201),
// lambda_w the wall weight scale and reg = lambda tr(S) / 9 (tr > 0) or lambda:
//   velocity kind   S_v = sum_N w b b^T + sum_W lambda_w w b b^T,
//                   R_c = sum_N w b (u_j,c - u_i,c) + sum_W lambda_w w b (u_w,c - u_i,c),
//                   y_c = (S_v + reg I)^-1 R_c
//                   lap_c = 2 / r_e^2 (y_c[3] + y_c[4] + y_c[5])   (explicit_update.cu:178-248)
//                   div   = sum_c y_c[c] / r_e                     (ppe_matrix.cu:355-361)
//   pressure kind   S_p = sum_N w b b^T + sum_W lambda_w w q q^T,
//                   R_p = sum_N w b (p_j - p_i) + sum_W lambda_w w q (r_e rho g.n),
//                   y_p = (S_p + reg I)^-1 R_p,  grad = y_p[0..2] / r_e  (pressure_correction.cu:200-276)
//                   L = rows 3 + 4 + 5 of (S_p + reg I)^-1; PPE row: a_ij = c w (L . b),
//                   c = 2 / (r_e^2 rho), diagonal -sum a_ij; wall_rhs = sum_W 2 lambda_w w (g.n) (L . q) / r_e;
//                   rhs = div / dt - wall_rhs                       (ppe_matrix.cu:243-370)
// Surface and Splash rows are Dirichlet rows (diagonal 1, neighbour slots 0,
// rhs = div = wall_rhs = 0); the gradient of a Splash particle is 0.
//
// Backward (labels, walls and both CSR tables fixed).  With the cotangents
// ybar of the y's, Rbar = M^-1 ybar for each field (M symmetric); the PPE
// rows' cotangent on L, h = sum_N c abar_ij w b + sum_W 2 lambda_w w (g.n)
// wrb q / r_e (abar_ij = the slot's cotangent minus the diagonal's,
// wrb = wall_rhs_bar - rhs_bar), gives hhat = M_p^-1 h.  The matrices'
// cotangents are -sum Rbar y^T (and -hhat L^T for M_p), plus, through the
// regularisation, lambda/9 times their trace on the diagonal (rho = sum
// Rbar . y (+ hhat . L) per kind).  A fluid entry (i, j) then contributes
// dL = alpha dw + beta . db with
//   alpha = sum_fields (Rbar . b)(dphi - b . y) - (hhat . b)(L . b) + c abar (L . b)
//           - (lambda/9)(rho_v + rho_p) |b|^2
//   beta  = w sum_fields [Rbar (dphi - b . y) - (Rbar . b) y] - w [(L . b) hhat + (hhat . b) L]
//           + c abar w L - 2 w (lambda/9)(rho_v + rho_p) b
// (fields: u_x, u_y, u_z on the velocity kind, p on the pressure kind), and
// its field cotangents w (Rbar . b) go to phibar_j and are taken from
// phibar_i.  A wall entry changes only its owner: with omega = lambda_w w,
// dL/domega = sum_c (Rbar_c . b)(du_c - b . y_c) - (lambda/9) rho_v |b|^2
//           + (Rbar_p . q)(r_e rho g.n - q . y_p) - (hhat . q)(L . q) - (lambda/9) rho_p |q|^2
//           + 2 (g.n)(L . q) wrb / r_e,
// and the cotangents of b and q follow the same pattern.  Positions: with
// d = x_j - x_i, dL/dd = (-(dL/dw) d / |d| + J_b^T dL/db + J_q^T dL/dq) / r_e,
// added to xbar_j (fluid neighbours) and taken from xbar_i.
//
// The inverses of both kinds are recomputed from the positions in the
// backward.  Deterministic form (default): every entry is evaluated once by
// its owner's warp, which keeps the owner's share (with its wall row's) and
// leaves the neighbour's as a record that the neighbour adds in entry order;
// atomic form (lsmps_ctx_set_adjoint_atomic): FP64 atomics into the
// neighbours.  The kernels are in operators.cu.
#include "adjoint.cuh"
#include "impl.cuh"
#include "packed.cuh"

namespace lsmps {
namespace {

lsmps_status check_step_inputs(lsmps_ctx* ctx, const lsmps_fluid& f, const lsmps_walls& w, const lsmps_csr& fn,
                               const lsmps_csr& wn, const lsmps_params& p) {
  if (!(p.support_radius > 0.0)) return fail(ctx, LSMPS_INVALID_ARGUMENT, "support radius must be positive");
  if (!(p.density > 0.0)) return fail(ctx, LSMPS_INVALID_ARGUMENT, "density must be positive");
  if (fn.particle_count < f.count || wn.particle_count < f.count)
    return fail(ctx, LSMPS_INVALID_ARGUMENT, "neighbour tables smaller than fluid");
  if (f.count && (!f.x || !f.y || !f.z || !f.vx || !f.vy || !f.vz || !f.pressure || !fn.offsets || !fn.indices ||
                  !wn.offsets || (wn.neighbor_count && !wn.indices)))
    return fail(ctx, LSMPS_INVALID_ARGUMENT, "step operator inputs missing");
  if (w.count && (!w.x || !w.y || !w.z || !w.vx || !w.vy || !w.vz || !w.normal_x || !w.normal_y || !w.normal_z))
    return fail(ctx, LSMPS_INVALID_ARGUMENT, "wall positions, velocities and normals are required");
  return check_neighbor_tables(ctx, f.count, w.count, fn, &wn);
}

// Both kinds' inverses (plain FP64) into the context's step-operator scratch,
// and the neighbour records.
lsmps_status prepare_step_ops(lsmps_ctx* ctx, const lsmps_fluid& f, const lsmps_walls& w, const lsmps_csr& fn,
                              const lsmps_csr& wn, const lsmps_params& p, const lsmps_step_operator_out& out,
                              OperatorArgs& a) {
  const size_t n = f.count;
  if (!ensure_step_ops(ctx, n) || !ensure_packs(ctx, n, w.count))
    return fail(ctx, LSMPS_CUDA_ERROR, "step operator scratch allocation failed");
  lsmps_moment m[2]{};
  const int kinds[2] = {LSMPS_MOMENT_VELOCITY_WALL_DIRICHLET_A, LSMPS_MOMENT_PRESSURE_WALL_NEUMANN_A};
  for (int k = 0; k < 2; ++k) {
    m[k].particle_count = n;
    m[k].matrix_size = 9;
    m[k].kind = kinds[k];
    m[k].support_radius = p.support_radius;
    m[k].wall_weight_scale = p.lsmps_wall_weight_scale;
    m[k].inverse_matrices = ctx->sop_inverse[k];
    m[k].moment_trace = ctx->sop_trace[k];
    m[k].regularization_added = ctx->sop_reg[k];
    m[k].info = ctx->sop_info[k];
    m[k].inversion_count = ctx->sop_count + k;
  }
  const int prec = ctx->precision;
  const int32_t* order = ctx->order;
  ctx->precision = LSMPS_PRECISION_PLAIN;
  ctx->order = nullptr;
  const lsmps_status st = prepare_moments_impl(ctx, f, w, fn, wn, p, m, 2);
  ctx->precision = prec;
  ctx->order = order;
  if (st) return st;
  pack4(ctx, f.x, f.y, f.z, f.pressure, n, ctx->pack_fluid[0]);
  pack4(ctx, f.vx, f.vy, f.vz, nullptr, n, ctx->pack_fluid[1]);
  pack4(ctx, w.x, w.y, w.z, nullptr, w.count, ctx->pack_wall[0]);
  pack4(ctx, w.vx, w.vy, w.vz, nullptr, w.count, ctx->pack_wall[1]);
  pack4(ctx, w.normal_x, w.normal_y, w.normal_z, nullptr, w.count, ctx->pack_wall[2]);
  a = OperatorArgs{};
  a.n = static_cast<index_t>(n);
  a.fp = ctx->pack_fluid[0];
  a.fv = ctx->pack_fluid[1];
  a.wp = ctx->pack_wall[0];
  a.wv = ctx->pack_wall[1];
  a.wn = ctx->pack_wall[2];
  a.fo = fn.offsets;
  a.fi = fn.indices;
  a.wo = wn.offsets;
  a.wi = wn.indices;
  a.label = f.surface_type;
  a.inv_v = ctx->sop_inverse[0];
  a.inv_p = ctx->sop_inverse[1];
  a.tr_v = ctx->sop_trace[0];
  a.tr_p = ctx->sop_trace[1];
  a.re = p.support_radius;
  a.inv_re = 1.0 / p.support_radius;
  a.lam_w = p.lsmps_wall_weight_scale;
  a.lambda = p.lsmps_regularization;
  a.rho = p.density;
  a.inv_dt = p.time_step > 0.0 ? 1.0 / p.time_step : 0.0;
  a.c_ppe = 2.0 / (p.support_radius * p.support_radius * p.density);
  a.gx = p.gravity[0];
  a.gy = p.gravity[1];
  a.gz = p.gravity[2];
  double* lap[3] = {out.lap_x, out.lap_y, out.lap_z};
  double* grad[3] = {out.grad_x, out.grad_y, out.grad_z};
  for (int c = 0; c < 3; ++c) {
    a.lap_u[c] = lap[c];
    a.grad[c] = grad[c];
  }
  a.div = out.divergence;
  a.rhs = out.ppe_rhs;
  a.wall_rhs = out.wall_rhs;
  a.values = out.ppe_values;
  a.row_offsets = out.ppe_row_offsets;
  a.columns = out.ppe_col_indices;
  return LSMPS_OK;
}

}  // namespace

// Context scratch of the step operator pair.
bool ensure_step_ops(lsmps_ctx* ctx, size_t n) {
  if (n <= ctx->sop_cap) return true;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  cudaStreamIsCapturing(ctx->stream, &cap);
  if (cap != cudaStreamCaptureStatusNone) return false;
  cudaStreamSynchronize(ctx->stream);
  free_step_ops(ctx);
  bool ok = cudaMalloc(&ctx->sop_count, 2 * sizeof(int32_t)) == cudaSuccess;
  for (int k = 0; k < 2 && ok; ++k)
    ok = cudaMalloc(&ctx->sop_inverse[k], n * 81 * sizeof(double)) == cudaSuccess &&
         cudaMalloc(&ctx->sop_trace[k], n * sizeof(double)) == cudaSuccess &&
         cudaMalloc(&ctx->sop_reg[k], n * sizeof(double)) == cudaSuccess &&
         cudaMalloc(&ctx->sop_info[k], n * sizeof(int32_t)) == cudaSuccess;
  if (!ok) {
    cudaGetLastError();
    free_step_ops(ctx);
    return false;
  }
  ctx->sop_cap = n;
  return true;
}

void free_step_ops(lsmps_ctx* ctx) {
  for (int k = 0; k < 2; ++k) {
    void* ps[] = {ctx->sop_inverse[k], ctx->sop_trace[k], ctx->sop_reg[k], ctx->sop_info[k]};
    for (void* p : ps)
      if (p) cudaFree(p);
    ctx->sop_inverse[k] = nullptr;
    ctx->sop_trace[k] = nullptr;
    ctx->sop_reg[k] = nullptr;
    ctx->sop_info[k] = nullptr;
  }
  if (ctx->sop_count) cudaFree(ctx->sop_count);
  ctx->sop_count = nullptr;
  ctx->sop_cap = 0;
}

}  // namespace lsmps

using namespace lsmps;

extern "C" lsmps_status lsmps_step_operators_forward(lsmps_ctx* ctx, const lsmps_fluid* fluid,
                                                     const lsmps_walls* walls, const lsmps_csr* fn,
                                                     const lsmps_csr* wn, const lsmps_params* params,
                                                     const lsmps_step_operator_out* out) {
  if (!ctx || !fluid || !walls || !fn || !wn || !params || !out) return LSMPS_INVALID_ARGUMENT;
  lsmps_status st = begin_call(ctx);
  if (st) return st;
  st = check_step_inputs(ctx, *fluid, *walls, *fn, *wn, *params);
  if (!st && out->count < fluid->count) st = fail(ctx, LSMPS_INVALID_ARGUMENT, "operator outputs too small");
  if (!st && fluid->count == 0) return end_call(ctx, LSMPS_OK);
  if (st) return end_call(ctx, st);
  OperatorArgs a;
  st = prepare_step_ops(ctx, *fluid, *walls, *fn, *wn, *params, *out, a);
  if (st) return end_call(ctx, st);
  return end_call(ctx, operators_forward(ctx, a, true));
}

extern "C" lsmps_status lsmps_step_operators_backward(lsmps_ctx* ctx, const lsmps_fluid* fluid,
                                                      const lsmps_walls* walls, const lsmps_csr* fn,
                                                      const lsmps_csr* wn, const lsmps_params* params,
                                                      const lsmps_step_operator_out* cotangent,
                                                      const lsmps_vector* u_bar, double* p_bar,
                                                      const lsmps_vector* x_bar) {
  if (!ctx || !fluid || !walls || !fn || !wn || !params || !cotangent) return LSMPS_INVALID_ARGUMENT;
  lsmps_status st = begin_call(ctx);
  if (st) return st;
  st = check_step_inputs(ctx, *fluid, *walls, *fn, *wn, *params);
  if (!st && cotangent->count < fluid->count) st = fail(ctx, LSMPS_INVALID_ARGUMENT, "cotangents too small");
  if (!st && ((u_bar && u_bar->count < fluid->count) || (x_bar && x_bar->count < fluid->count)))
    st = fail(ctx, LSMPS_INVALID_ARGUMENT, "gradient outputs too small");
  if (!st && fluid->count == 0) return end_call(ctx, LSMPS_OK);
  if (st) return end_call(ctx, st);
  OperatorArgs a;
  st = prepare_step_ops(ctx, *fluid, *walls, *fn, *wn, *params, *cotangent, a);
  if (st) return end_call(ctx, st);
  a.phibar[0] = u_bar ? u_bar->x : nullptr;
  a.phibar[1] = u_bar ? u_bar->y : nullptr;
  a.phibar[2] = u_bar ? u_bar->z : nullptr;
  a.phibar[3] = p_bar;
  a.xbar[0] = x_bar ? x_bar->x : nullptr;
  a.xbar[1] = x_bar ? x_bar->y : nullptr;
  a.xbar[2] = x_bar ? x_bar->z : nullptr;
  return end_call(ctx, operators_backward(ctx, *fn, a, true));
}
