// wg_small.cuh -- a small simulation's output interval in one launch.
#pragma once
#include <cstdint>

#include "wg_bucket.cuh"

namespace wg {

// Most sheets one CTA takes: two per thread of the largest CTA.  At that size
// one CTA still beats the bucket kernel's launches (16.0 against 22.1 us per
// sub-step where every sub-step sorts, 8.1 against 16.5 where few sheets cross).
constexpr int kSmallSheets = 2048;
constexpr int kSmallExprSheets = 1536;  // the same with an expression force

struct SmallArgs {
  const StateTable* table;  // current set: the sheets in any order, in place
  int n;
  int nleap;
  int ends;                 // (filled in) the last sub-step ends the call
  double dt;
  double pre;               // opening half drift
  uint64_t T_lo, T_hi;      // totmass in fixed point
  int E;
  int has_omega;
  double omega2;
  ExtForce ext;
  const double* t_seq;      // [nleap] times (forces that depend on the time only)
  double* x_out;            // outputs in original order
  double* v_out;
  double* a_out;            // optional: accelerations of the last force evaluation
  SheetRec* xi_out;         // optional: (idx, x) in the last sub-step's sorted order
  StepFlags* flag;          // receives full sorts, n and the last sub-step's largest |v|
};

// nleap sub-steps (with the opening and closing half drifts) of a simulation
// of at most kSmallSheets sheets; the sheets end in the current set, sorted
// by their positions at the last force evaluation.
// Returns the launches made.
int launch_small_run(const SmallArgs& a, cudaStream_t s);

}  // namespace wg
