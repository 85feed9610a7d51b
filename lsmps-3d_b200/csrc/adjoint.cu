// adjoint.cu - the LSMPS field operators and the fluid-only PPE rows as a
// forward/backward pair (no counterpart in the reference, which has no
// derivatives).
//
// Per fluid particle i over its fluid CSR row N(i), with s_ij = (x_j - x_i)/r_e,
// w_ij = 1 - |s_ij|, b_ij the Type-A basis (moment_matrix.cu:152-175) and the
// fluid-only Type-A moment matrix M_i = sum_j w_ij b_ij b_ij^T + reg_i I
// (moment_matrix.cu:254-309 with no wall term; reg_i = lambda tr/9):
//   R_i(phi) = sum_j w_ij b_ij (phi_j - phi_i),  y_i(phi) = M_i^-1 R_i(phi)
//   gradient    g_i   = y_i(f)[0..2] / r_e                (pressure_correction.cu:226-266)
//   Laplacian   lap_i = 2 / r_e^2 sum_{r=3..5} y_i(f)[r]    (explicit_update.cu:164-176)
//   divergence  div_i = sum_c y_i(v_c)[c] / r_e             (ppe_matrix.cu:355-361)
//   PPE row i   a_ij = 2 w_ij (l_i . b_ij) / (r_e^2 rho), l_i = sum_{r=3..5} M_i^-1[r, :],
//               diagonal -sum_j a_ij first, rhs_i = div_i / dt (ppe_matrix.cu:243-370
//               without the wall terms)
//
// Backward, for a loss L with cotangents of every output:
//   ybar_i(phi) is the cotangent of y_i(phi), Rbar_i(phi) = M_i^-1 ybar_i(phi)
//   (M symmetric), and for the PPE rows h_i = c sum_j abar_ij w_ij b_ij,
//   hhat_i = M_i^-1 h_i (abar_ij = the off-diagonal cotangent minus the
//   diagonal's).  Field cotangents: phibar_j += w_ij b_ij . Rbar_i(phi),
//   phibar_i -= the same.  Position cotangents: with d = x_j - x_i,
//   dL = alpha_ij dw_ij + beta_ij . db_ij, where
//     alpha = sum_phi (Rbar.b)(dphi - b.y) + c abar (l.b) - (hhat.b)(b.l)
//             - rho (lambda/9) |b|^2
//     beta  = w sum_phi [Rbar (dphi - b.y) - (Rbar.b) y] + c abar w l
//             - w [(b.l) hhat + (hhat.b) l] - rho (lambda/9) 2 w b
//   (rho = sum_phi Rbar.y + hhat.l; the lambda terms only when tr > 0), and
//   dL/dd = (-alpha d/|d| + J_b(s)^T beta) / r_e is added to xbar_j and
//   subtracted from xbar_i.
//
// The backward recomputes M_i^-1 from the positions (no stored inverse is
// needed) unless the caller passes the inverse the forward wrote.
//
// Each CSR entry (i, j) contributes to the cotangents of both its owner i and
// its neighbour j.  The default backward is deterministic: the owner's warp
// evaluates the entry once, keeps its own share and leaves the neighbour's as
// a record at the neighbour, which then adds its records in ascending entry
// order: repeated runs give the same bits.  lsmps_ctx_set_adjoint_atomic(ctx,
// 1) selects the scatter form instead (FP64 atomics into the neighbours; no
// records, but the result depends on the atomics' order at the rounding
// level).  The kernels are in operators.cu.
#include "adjoint.cuh"
#include "impl.cuh"
#include "packed.cuh"

namespace lsmps {

// Context scratch of the operator pair: the fluid-only inverse, its trace /
// regularisation / info.
bool ensure_adjoint(lsmps_ctx* ctx, size_t n) {
  if (n <= ctx->adj_cap) return true;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  cudaStreamIsCapturing(ctx->stream, &cap);
  if (cap != cudaStreamCaptureStatusNone) return false;
  cudaStreamSynchronize(ctx->stream);
  free_adjoint(ctx);
  bool ok = cudaMalloc(&ctx->adj_inverse, n * 81 * sizeof(double)) == cudaSuccess &&
            cudaMalloc(&ctx->adj_trace, n * sizeof(double)) == cudaSuccess &&
            cudaMalloc(&ctx->adj_reg, n * sizeof(double)) == cudaSuccess &&
            cudaMalloc(&ctx->adj_info, n * sizeof(int32_t)) == cudaSuccess &&
            cudaMalloc(&ctx->adj_count, sizeof(int32_t)) == cudaSuccess;
  if (!ok) {
    cudaGetLastError();
    free_adjoint(ctx);
    return false;
  }
  ctx->adj_cap = n;
  return true;
}

void free_adjoint(lsmps_ctx* ctx) {
  void* ps[] = {ctx->adj_inverse, ctx->adj_trace, ctx->adj_reg, ctx->adj_info, ctx->adj_count};
  for (void* p : ps)
    if (p) cudaFree(p);
  ctx->adj_inverse = nullptr;
  ctx->adj_trace = nullptr;
  ctx->adj_reg = nullptr;
  ctx->adj_info = nullptr;
  ctx->adj_count = nullptr;
  ctx->adj_cap = 0;
}

namespace {

lsmps_status check_inputs(lsmps_ctx* ctx, const lsmps_fluid& fl, const lsmps_csr& fn, const lsmps_params& p,
                          const double* f, const lsmps_vector& v) {
  if (!(p.support_radius > 0.0)) return fail(ctx, LSMPS_INVALID_ARGUMENT, "support radius must be positive");
  if (fn.particle_count < fl.count) return fail(ctx, LSMPS_INVALID_ARGUMENT, "neighbour table smaller than fluid");
  if (v.count < fl.count) return fail(ctx, LSMPS_INVALID_ARGUMENT, "vector field smaller than fluid");
  if (fl.count && (!fl.x || !fl.y || !fl.z || !f || !v.x || !v.y || !v.z || !fn.offsets || !fn.indices))
    return fail(ctx, LSMPS_INVALID_ARGUMENT, "operator inputs missing");
  return check_neighbor_tables(ctx, fl.count, 0, fn, nullptr);
}

// Fluid-only Type-A moments into the context's inverse (or `inverse`).
lsmps_status moments(lsmps_ctx* ctx, const lsmps_fluid& fl, const lsmps_csr& fn, const lsmps_params& p,
                     double* inverse) {
  lsmps_moment m{};
  m.particle_count = fl.count;
  m.matrix_size = 9;
  m.kind = LSMPS_MOMENT_FLUID_ONLY_A;
  m.support_radius = p.support_radius;
  m.wall_weight_scale = p.lsmps_wall_weight_scale;
  m.inverse_matrices = inverse;
  m.moment_trace = ctx->adj_trace;
  m.regularization_added = ctx->adj_reg;
  m.info = ctx->adj_info;
  m.inversion_count = ctx->adj_count;
  lsmps_walls none{};
  lsmps_csr wn{fl.count, 0, fn.offsets, fn.indices};  // unused by the fluid-only kind
  const int prec = ctx->precision;
  ctx->precision = LSMPS_PRECISION_PLAIN;
  const lsmps_status st = prepare_moments_impl(ctx, fl, none, fn, wn, p, &m, 1);
  ctx->precision = prec;
  return st;
}

OperatorArgs make_args(lsmps_ctx* ctx, const lsmps_fluid& fl, const lsmps_csr& fn, const lsmps_params& p, const double* f,
                       const lsmps_vector& v, const double* inverse, const lsmps_operator_out& out) {
  pack4(ctx, fl.x, fl.y, fl.z, f, fl.count, ctx->pack_fluid[0]);
  pack4(ctx, v.x, v.y, v.z, nullptr, fl.count, ctx->pack_fluid[1]);
  OperatorArgs a{};
  a.n = static_cast<index_t>(fl.count);
  a.fp = ctx->pack_fluid[0];
  a.fv = ctx->pack_fluid[1];
  a.fo = fn.offsets;
  a.fi = fn.indices;
  a.inv_v = inverse;
  a.inv_p = inverse;
  a.re = p.support_radius;
  a.inv_re = 1.0 / p.support_radius;
  a.c_ppe = 2.0 / (p.support_radius * p.support_radius * p.density);
  a.inv_dt = p.time_step > 0.0 ? 1.0 / p.time_step : 0.0;
  a.lambda = p.lsmps_regularization;
  a.grad[0] = out.grad_x;
  a.grad[1] = out.grad_y;
  a.grad[2] = out.grad_z;
  a.lap_f = out.laplacian;
  a.div = out.divergence;
  a.rhs = out.ppe_rhs;
  a.values = out.ppe_values;
  a.row_offsets = out.ppe_row_offsets;
  a.columns = out.ppe_col_indices;
  return a;
}

}  // namespace
}  // namespace lsmps

using namespace lsmps;

extern "C" lsmps_status lsmps_operators_forward(lsmps_ctx* ctx, const lsmps_fluid* fluid, const lsmps_csr* fn,
                                                const lsmps_params* params, const double* f, const lsmps_vector* v,
                                                const lsmps_operator_out* out, double* inverse_out) {
  if (!ctx || !fluid || !fn || !params || !v || !out) return LSMPS_INVALID_ARGUMENT;
  lsmps_status st = begin_call(ctx);
  if (st) return st;
  st = check_inputs(ctx, *fluid, *fn, *params, f, *v);
  if (!st && out->count < fluid->count) st = fail(ctx, LSMPS_INVALID_ARGUMENT, "operator outputs too small");
  if (!st && fluid->count == 0) return end_call(ctx, LSMPS_OK);
  if (!st && (!ensure_adjoint(ctx, fluid->count) || !ensure_packs(ctx, fluid->count, 0)))
    st = fail(ctx, LSMPS_CUDA_ERROR, "operator scratch allocation failed");
  if (st) return end_call(ctx, st);
  double* inverse = inverse_out ? inverse_out : ctx->adj_inverse;
  st = moments(ctx, *fluid, *fn, *params, inverse);
  if (st) return end_call(ctx, st);
  return end_call(ctx, operators_forward(ctx, make_args(ctx, *fluid, *fn, *params, f, *v, inverse, *out), false));
}

extern "C" lsmps_status lsmps_operators_backward(lsmps_ctx* ctx, const lsmps_fluid* fluid, const lsmps_csr* fn,
                                                 const lsmps_params* params, const double* f, const lsmps_vector* v,
                                                 const lsmps_operator_out* cotangent, const double* inverse,
                                                 double* f_bar, const lsmps_vector* v_bar,
                                                 const lsmps_vector* x_bar) {
  if (!ctx || !fluid || !fn || !params || !v || !cotangent) return LSMPS_INVALID_ARGUMENT;
  lsmps_status st = begin_call(ctx);
  if (st) return st;
  st = check_inputs(ctx, *fluid, *fn, *params, f, *v);
  if (!st && cotangent->count < fluid->count) st = fail(ctx, LSMPS_INVALID_ARGUMENT, "cotangents too small");
  if (!st && ((v_bar && v_bar->count < fluid->count) || (x_bar && x_bar->count < fluid->count)))
    st = fail(ctx, LSMPS_INVALID_ARGUMENT, "gradient outputs too small");
  if (!st && fluid->count == 0) return end_call(ctx, LSMPS_OK);
  if (!st && (!ensure_adjoint(ctx, fluid->count) || !ensure_packs(ctx, fluid->count, 0)))
    st = fail(ctx, LSMPS_CUDA_ERROR, "operator scratch allocation failed");
  if (st) return end_call(ctx, st);
  // The inverse is recomputed from the positions unless the caller kept the
  // forward's.
  if (!inverse) {
    st = moments(ctx, *fluid, *fn, *params, ctx->adj_inverse);
    if (st) return end_call(ctx, st);
  }
  OperatorArgs a = make_args(ctx, *fluid, *fn, *params, f, *v, inverse ? inverse : ctx->adj_inverse, *cotangent);
  a.phibar[0] = v_bar ? v_bar->x : nullptr;
  a.phibar[1] = v_bar ? v_bar->y : nullptr;
  a.phibar[2] = v_bar ? v_bar->z : nullptr;
  a.phibar[3] = f_bar;
  a.xbar[0] = x_bar ? x_bar->x : nullptr;
  a.xbar[1] = x_bar ? x_bar->y : nullptr;
  a.xbar[2] = x_bar ? x_bar->z : nullptr;
  return end_call(ctx, operators_backward(ctx, *fn, a, false));
}

extern "C" lsmps_status lsmps_ctx_set_adjoint_atomic(lsmps_ctx* ctx, int on) {
  if (!ctx || (on != 0 && on != 1)) return LSMPS_INVALID_ARGUMENT;
  ctx->adjoint_atomic = on != 0;
  return LSMPS_OK;
}
