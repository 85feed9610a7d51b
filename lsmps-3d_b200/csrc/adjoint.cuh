// adjoint.cuh - what the two differentiable operator pairs share (adjoint.cu:
// fluid-only operators; step_adjoint.cu: the step's operators with their wall
// terms): the arguments of their kernels and the queueing of them
// (operators.cu).
#pragma once

#include "common.cuh"

namespace lsmps {

struct OperatorArgs {
  index_t n;
  const double4* fp;  // fluid {x, y, z, scalar}
  const double4* fv;  // fluid {u_x, u_y, u_z, -}
  const double4* wp;  // walls {x, y, z, -}, velocities, normals (with walls)
  const double4* wv;
  const double4* wn;
  const index_t* fo;
  const index_t* fi;
  const index_t* wo;
  const index_t* wi;
  const int32_t* label;
  const double* inv_v;  // [n][81] column-major
  const double* inv_p;  // (= inv_v in the fluid-only pair)
  const double* tr_v;   // traces before regularisation
  const double* tr_p;
  double re;
  double inv_re;
  double lam_w;
  double lambda;
  double rho;
  double inv_dt;
  double c_ppe;  // 2 / (r_e^2 rho)
  double gx, gy, gz;
  // Forward: the outputs.  Backward: their cotangents.  NULL: not wanted / 0.
  double* lap_u[3];  // with walls
  double* lap_f;     // fluid-only
  double* grad[3];
  double* div;
  double* rhs;
  double* wall_rhs;  // with walls
  double* values;
  index_t* row_offsets;  // forward only
  index_t* columns;
  // Backward: gradients (x, y, z components of u, the scalar, positions).
  double* phibar[4];
  double* xbar[3];
  // Backward, deterministic form: per incoming entry of a particle a 64-byte
  // record {4 field terms, 3 position terms, entry id}, in the order the owners'
  // warps finish; next[j] the next free record of particle j, begin[j] its first
  // and begin[j + 1] its end; own[8 j ..] the terms of j's own row.  Only the
  // particles [j0, j1) have records in this pass, j0's first at records[0].
  index_t* next;
  const index_t* begin;
  double4* records;
  double* own;
  index_t j0, j1;
};

// Queue the forward (outputs in `a`), and the backward (cotangents in `a`,
// deterministic or atomic as the context is set; reads the entry count back in
// the deterministic form).  walls: the step's operators, else the fluid-only
// ones.  The moments and the packs of `a` are queued before.
lsmps_status operators_forward(lsmps_ctx* ctx, const OperatorArgs& a, bool walls);
lsmps_status operators_backward(lsmps_ctx* ctx, const lsmps_csr& fn, OperatorArgs a, bool walls);

}  // namespace lsmps
