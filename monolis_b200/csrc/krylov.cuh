// krylov.cuh -- scalar steps of the CG and BiCGSTAB recurrences, shared by the
// kernel-per-phase solvers (solve.cu) and the one-kernel solvers (persist.cu).
#pragma once

#include "common.cuh"
#include "dev.h"

namespace mb {
namespace {

// ---------------------------------------------------------------------------
// Scalar updates run by the last block of a grid reduction.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void record(SolverState* st, double* hist, double resid) {
  st->resid = resid;
  if (hist) hist[st->iter] = resid;
}

// end of CG iteration `iter` (or the initial residual when iter == 0):
// rr = <r,r>, rz = <r,z> (= rho of the next iteration).
__device__ __forceinline__ void fin_cg(SolverState* st, double rr, double rz, double* hist) {
  if (st->iter == 0) {
    st->B2 = rr;
    if (rr == 0.0) { st->done = 1; st->status = kZeroRhs; return; }
    st->rho = rz;
    st->iter = 1;
    return;
  }
  const double resid = sqrt(rr / st->B2);  // src/linalg/mat_converge.f90:120
  record(st, hist, resid);
  if (resid < st->tol) { st->done = 1; st->status = kOk; return; }
  if (!isfinite(resid)) { st->done = 1; st->status = kNonFinite; return; }
  if (st->iter >= st->max_iter) { st->done = 1; st->status = kMaxIter; return; }
  st->rho1 = st->rho;
  st->rho = rz;
  st->beta = st->rho / st->rho1;  // src/iterative/CG.f90:79
  st->iter += 1;
}

// end of BiCGSTAB iteration: rr = <R,R>, rrt = <R,RT> (= rho of the next one)
__device__ __forceinline__ void fin_bicg(SolverState* st, double rr, double rrt, double* hist) {
  if (st->iter == 0) {
    st->B2 = rr;
    if (rr == 0.0) { st->done = 1; st->status = kZeroRhs; return; }
    st->rho = rrt;
    st->iter = 1;
    return;
  }
  const double resid = sqrt(rr / st->B2);
  record(st, hist, resid);
  if (resid < st->tol) { st->done = 1; st->status = kOk; return; }
  if (!isfinite(resid)) { st->done = 1; st->status = kNonFinite; return; }
  if (st->iter >= st->max_iter) { st->done = 1; st->status = kMaxIter; return; }
  st->rho1 = st->rho;
  st->rho = rrt;
  if (rrt == 0.0) { st->done = 1; st->status = kBreakdown; return; }
  st->beta = (st->rho / st->rho1) * (st->alpha / st->omega);  // src/iterative/BiCGSTAB.f90:96
  st->iter += 1;
}

// ---- mixed precision (FP32 loop, FP64 refresh) ----
__device__ __forceinline__ void fin_mixed_inner(SolverState* st, double rr, double rz, double* hist) {
  const double rn = sqrt(rr);
  const double resid = sqrt(rr / st->B2);
  record(st, hist, resid);
  st->rho1 = st->rho;
  if (!isfinite(resid)) { st->done = 1; st->status = kNonFinite; return; }
  if (rn > st->rmax) st->rmax = rn;
  if (rn < st->delta * st->rmax || resid < st->tol || st->iter >= st->max_iter ||
      (st->period > 0 && st->iter - st->last_refresh >= st->period)) {
    st->refresh = 1;  // the refresh kernel of this iteration finishes it
    return;
  }
  st->rho = rz;
  st->beta = st->rho / st->rho1;
  st->iter += 1;
}

// Mixed precision BiCGSTAB: the same scheme on src/iterative/BiCGSTAB.f90's
// recurrences. X + Y is the solution (Y accumulates alpha*PT + omega*ST in
// FP32); a refresh recomputes R = B - A (X + Y) in FP64 and continues with
// rho = <R,RT> of that residual, the shadow residual RT and P, V unchanged
// (the reference's own true-residual replacement, made adaptive).
__device__ __forceinline__ void fin_mixed_bicg(SolverState* st, double rr, double rrt, double* hist) {
  const double rn = sqrt(rr);
  const double resid = sqrt(rr / st->B2);
  record(st, hist, resid);
  st->rho1 = st->rho;
  if (!isfinite(resid)) { st->done = 1; st->status = kNonFinite; return; }
  if (rn > st->rmax) st->rmax = rn;
  if (rn < st->delta * st->rmax || resid < st->tol || st->iter >= st->max_iter ||
      (st->period > 0 && st->iter - st->last_refresh >= st->period)) {
    st->refresh = 1;
    return;
  }
  st->rho = rrt;
  if (rrt == 0.0) { st->done = 1; st->status = kBreakdown; return; }
  st->beta = (st->rho / st->rho1) * (st->alpha / st->omega);
  st->iter += 1;
}

// End of a refresh (or of the initial residual when iter == 0): rr = <r64,r64>,
// rz = <r,z> (CG) or <r,rt> (BiCGSTAB).
template <bool Bicg>
__device__ __forceinline__ void fin_mixed_refresh(SolverState* st, double rr, double rz, double* hist) {
  if (st->iter == 0) {
    st->B2 = rr;
    if (rr == 0.0) { st->done = 1; st->status = kZeroRhs; return; }
    st->rmax = sqrt(rr);
    st->rho = rz;
    st->iter = 1;
    return;
  }
  const double resid = sqrt(rr / st->B2);
  record(st, hist, resid);
  st->refresh = 0;
  st->fold = 1;
  st->n_refine += 1;
  st->last_refresh = st->iter;
  if (resid < st->tol) { st->done = 1; st->status = kOk; return; }
  if (!isfinite(resid)) { st->done = 1; st->status = kNonFinite; return; }
  if (st->iter >= st->max_iter) { st->done = 1; st->status = kMaxIter; return; }
  st->rmax = sqrt(rr);
  st->rho = rz;
  if (Bicg) {
    if (rz == 0.0) { st->done = 1; st->status = kBreakdown; return; }
    st->beta = (st->rho / st->rho1) * (st->alpha / st->omega);
  } else {
    st->beta = st->rho / st->rho1;
  }
  st->iter += 1;
}

}  // namespace
}  // namespace mb
