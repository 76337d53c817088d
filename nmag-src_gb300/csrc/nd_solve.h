// nd_solve.h -- data of the direct Poisson solver (nd_solve.cu).
#pragma once
#include <cstdint>

namespace nmg {

// CG iteration caps below this keep the CG, whose cap they are.
constexpr int kNdMinMaxits = 1000;
// Demag evaluations after which a handle that has only evaluated fields gets
// its factors: they cost as much as 6 to 15 evaluations save (film: 24 ms
// against 3.2 ms each at 1e-12; cube: 6.5 ms against 1.1), so a program that
// looks at one field does not pay for them.  Integrations, whose many
// evaluations are certain, factor at their start.
constexpr int kNdEvals = 4;

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
