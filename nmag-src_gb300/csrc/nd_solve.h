// nd_solve.h -- data of the direct Poisson solver (nd_solve.cu).
#pragma once
#include <cstdint>

namespace nmg {

// CG iteration caps below this keep the CG, whose cap they are.
constexpr int kNdMinMaxits = 1000;
// A handle gets its factors once the CG's solves, those it has done and those
// that are certain to come, are worth 3/4 of what the factors cost, so that a
// program pays at most about twice what the better of the two would have taken,
// whenever it stops.  Both are estimates, the same in every run: from the CG's
// iteration counts, and from the mesh (nd_cost).  No handle is looked at before
// its fourth demag evaluation.
constexpr int kNdEvals = 4;
constexpr double kNdShare = 0.75;
// What is certain: an integration's first steps (64 evaluations; 100
// iterations of the CG each, it takes 23 to 650), RK4's four evaluations a step.
constexpr int kNdIntegration = 64, kNdIters = 100;
constexpr int kNdResponseIters = 40;   // a Jacobian's demag response, solved to 1e-3

struct NdFront {    // a part of the separator tree eliminated together
  int pos, k, nb, s;      // pivots [pos, pos + k) of the elimination order, boundary size, k + nb
  int uoff, boff, moff;   // its slices of u, the boundary list, the child maps (nch lists of s entries)
  int nch;                // children
  long long off;          // its factor entries: k rows of s, then nb rows of k
};
struct NdTask { int front, start, count; };      // rows of a front (upwards: of its nb, downwards: of its k)
struct NdLevel { int t0, t1, cs, pad; };         // one phase of a sweep: its tasks, warps sharing a row

// What the next kernels of the demag pipeline read, written with the answer
// (all may be null): its values at the boundary nodes, and sum = add + x.
struct NdOut {
  double *bnd = nullptr;
  const double *add = nullptr;
  double *sum = nullptr;
};

}  // namespace nmg
