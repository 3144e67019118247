// The scalars of a Stokes solve on the device (mw_stokes::sc) and the decisions taken on them.  A
// loop's test runs in the block that finishes the sum it depends on, which also sets the loop's
// condition when the loop is a conditional node of a recorded graph.
#pragma once

#include "common.cuh"

namespace mw {

// Schur-residual reduction of a refinement sweep that starts at relative residual `rel`: the fixed
// sweep_reduction, or with target > 0 the smaller reduction target * tol / rel (at most 0.5).
MW_HD double sweep_target_reduction(double sweep_reduction, double target, double tol, double rel) {
  if (!(target > 0) || !(rel > 0)) return sweep_reduction;
  double r = target * tol / rel;
  if (r > 0.5) r = 0.5;
  return r > sweep_reduction ? r : sweep_reduction;
}

enum DevSlot {
  P_PAP = 64, P_RR, P_BB, P_IT, P_RZ2,                       // inner PCG; (r, z) by iteration parity at
                                                              // P_RZ2, P_RZ2 + 1
  U_RW2 = 70,                                                 // Schur CG; (r, w) by iteration parity
  U_DSD = 72, U_RR0, U_RR, U_IT, U_D2, U_Z2, U_M1, U_M2,     // ... the sums whose means are removed: U_M1, U_M2
  T_RV = 84, T_RP, T_REL,                                     // true residual
  S_BB = 88, S_BH, S_BNORM, S_REL0, S_NREF, S_RED,           // solve
  I_OUTER = 96, I_INNER, I_STATUS                             // info
};

// S_*, T_REL and I_* are the outcome of the last solve (mw_stokes_device_info): a call that is no solve
// leaves them alone.  A residual asked for by itself has scalars of its own, this far from the solve's.
constexpr int CALL_SCALARS = 128;

// Work caps of one solve on top of the per-loop caps: a stagnating solve ends with status 3 after
// this many inner (multigrid-PCG) or outer (Schur) iterations in total.
constexpr double DEV_INNER_BUDGET = 40000, DEV_OUTER_BUDGET = 4000;

// What ends a Schur iteration or a refinement sweep, and the condition it sets (device = 0: the host
// reads the scalars and decides)
struct LoopTest {
  int device;
  cudaGraphConditionalHandle handle;
  double tol;
  int max_count;
  int check_true;                          // Schur: stop on the true residual (computed before the test)
  double reduction;                        // Schur: residual reduction; < 0: this sweep's (S_RED)
  double sweep_reduction, sweep_target;    // refinement: the settings S_RED follows from
};

MW_D void schur_start(double* sc, const LoopTest& t) {
  sc[U_IT] = 0;
  if (t.device)
    cudaGraphSetConditional(t.handle, (t.max_count > 0 && isfinite(sc[U_RR0]) && sc[I_STATUS] == 0) ? 1u : 0u);
}

// one Schur iteration done: stop on a non-finite residual (status 2), on the FP64 true residual
// (check_true), on the Schur residual reduction, at max_count or at the work cap (status 3)
MW_D void schur_test(double* sc, const LoopTest& t) {
  if (!t.device) return;
  const double rr = sc[U_RR], red = t.reduction < 0 ? sc[S_RED] : t.reduction;
  bool go = sc[U_IT] < (double)t.max_count;
  if (!isfinite(rr)) { sc[I_STATUS] = 2; go = false; }
  if (sc[I_OUTER] >= DEV_OUTER_BUDGET && sc[I_STATUS] == 0) sc[I_STATUS] = 3;
  if (sc[I_STATUS] != 0) go = false;
  if (t.check_true && sc[T_REL] <= t.tol) go = false;
  if (rr <= red * red * sc[U_RR0]) go = false;
  cudaGraphSetConditional(t.handle, go ? 1u : 0u);
}

// what a true residual is computed for
enum ResidAction { RA_NONE = 0, RA_FIRST, RA_SWEEP, RA_SCHUR };

// sum of squares of the residual known: T_REL and, by action, the initial residual and the first
// sweep's condition, the next sweep's, or the Schur iteration's
MW_D void residual_done(double* sc, double sum, int action, const LoopTest& t) {
  sc[T_RV] = sum;
  sc[T_RP] = 0;
  const double r = sqrt(sum) / sc[S_BNORM];
  sc[T_REL] = r;
  if (action == RA_NONE) return;
  if (action == RA_SCHUR) {
    schur_test(sc, t);
    return;
  }
  if (action == RA_FIRST) sc[S_REL0] = r; else sc[S_NREF] += 1;
  sc[S_RED] = sweep_target_reduction(t.sweep_reduction, t.sweep_target, t.tol, r);
  const bool go = isfinite(r) && r > t.tol && sc[S_NREF] < (double)t.max_count &&
                  (action == RA_FIRST || sc[I_STATUS] == 0);
  if (t.device) cudaGraphSetConditional(t.handle, go ? 1u : 0u);
}

}  // namespace mw
