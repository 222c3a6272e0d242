// The 3D pseudo-transient Newton step: right-preconditioned restarted GMRES with CGS2
// and Givens least squares (src/jaxrans/solvers/krylov.py:34-137), the relaxation, the
// acceptance test and the CFL ramp (src/jaxrans/solvers/implicit.py:54-168), driven on
// the host over vector operations `Ops` supplies.  On the device (newton3d.cu) the
// operations are kernels; a test-only host harness supplies loops, so this logic is
// checked against the reference without a GPU.
#pragma once
#include <cmath>
#include <vector>

namespace jr {

constexpr int MAX_RESTART3 = 64;   // krylov_subspace at most

struct Newton3Config {
  int restart, maxiter, preconditioner;   // preconditioner 0 none, 1 line_j, 2 line_j coupled
  double tol, success, max_relative_update;   // max_relative_update <= 0: none
  double cfl_min, cfl_max, cfl_growth, cfl_cutback;
};

// argmin |beta e1 - H y| by Givens rotations; pivots below rcond * the largest dropped
inline void givens_lstsq(const std::vector<double>& Hc, int m, double beta, double rcond, std::vector<double>& y) {
  // Hc: (m+1) x m, row-major
  std::vector<double> h(Hc), g(m + 1, 0.0), cs(m), sn(m);
  g[0] = beta;
  for (int j = 0; j < m; ++j) {
    for (int i = 0; i < j; ++i) {
      const double a = h[i * m + j], c = h[(i + 1) * m + j];
      h[i * m + j] = cs[i] * a + sn[i] * c;
      h[(i + 1) * m + j] = cs[i] * c - sn[i] * a;
    }
    const double a = h[j * m + j], c = h[(j + 1) * m + j];
    const double r = std::sqrt(a * a + c * c);
    const double safe = r > 0.0 ? r : 1.0;
    cs[j] = r > 0.0 ? a / safe : 1.0;
    sn[j] = r > 0.0 ? c / safe : 0.0;
    h[j * m + j] = r;
    h[(j + 1) * m + j] = 0.0;
    const double gj = g[j];
    g[j] = cs[j] * gj;
    g[j + 1] = -sn[j] * gj;
  }
  double largest = 0.0;
  for (int j = 0; j < m; ++j) largest = std::fmax(largest, std::fabs(h[j * m + j]));
  y.assign(m, 0.0);
  for (int j = m - 1; j >= 0; --j) {
    double rest = g[j];
    for (int k = j + 1; k < m; ++k) rest = rest - h[j * m + k] * y[k];
    y[j] = std::fabs(h[j * m + j]) > rcond * largest ? rest / h[j * m + j] : 0.0;
  }
}

// Ops: vectors by index -- RES_, B_, DU_, ACT_ (the step's) and T_ (work) -- each of the
// canvas length N = nvar * cells; the state U is the caller's.  Operations: prepare(U, cfl)
// (V/dt, the line factor, the linearisation), residual, nrm2, axpy, scale, density_norm,
// worst_ratio, physical_after, add_to_state; and gmres3(ops, U, cfl, c, B, X, ACTION), found by
// its argument: X of (V/dt + J) X = B by restarted GMRES, ACTION = A X by the Arnoldi relation
// (on the device newton3d.cu's, its scalars kept there).

// One Newton step on the state (U in place); returns |R| before the update.
template <class Ops>
double newton_step3(Ops& ops, double* U, double& cfl, double& res_prev, const Newton3Config& c) {
  ops.prepare(U, cfl);   // V/dt at (U, cfl), for the matrix-vector products of this step
  ops.residual(U, Ops::RES_);
  const double norm = ops.density_norm(Ops::RES_);
  ops.scale(-1.0, Ops::RES_, Ops::B_);
  gmres3(ops, U, cfl, c, Ops::B_, Ops::DU_, Ops::ACT_);
  double omega = 1.0;
  if (c.max_relative_update > 0.0) {
    const double worst = ops.worst_ratio(U, Ops::DU_);
    omega = std::fmin(1.0, c.max_relative_update / std::fmax(worst, 1e-300));
    ops.scale(omega, Ops::DU_, Ops::DU_);
  }
  ops.scale(omega, Ops::ACT_, Ops::T_);
  ops.axpy(1.0, Ops::RES_, Ops::T_);
  const double lin = ops.nrm2(Ops::T_) / std::fmax(ops.nrm2(Ops::RES_), 1e-300);
  const bool physical = ops.physical_after(U, Ops::DU_);
  const bool accept = physical && lin < 1.0;
  const double reduction = res_prev / std::fmax(norm, 1e-300);
  double next;
  if (accept && lin < c.success && omega >= 1.0) next = cfl * std::fmin(std::fmax(reduction, 1.0), c.cfl_growth);
  else if (accept) next = cfl;
  else next = cfl / c.cfl_cutback;
  if (accept) {
    ops.add_to_state(U, Ops::DU_);
    res_prev = norm;
  }
  cfl = std::fmin(std::fmax(next, c.cfl_min), c.cfl_max);
  return norm;
}

}  // namespace jr
