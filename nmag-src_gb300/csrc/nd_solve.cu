// nd_solve.cu -- direct Poisson solves: nested dissection of the P1 stiffness
// matrix, factored once per mesh, applied by one persistent kernel.
//
// The reference solves K phi1 = rho (constant null space removed) and
// K_II phi2_I = -K_IB phi2_B with PETSc Krylov solvers (nmag_lam.py:614-634,
// nsim.ml:2210-2262).  An iterative solve of these systems on the GPU is a
// chain of grid barriers, two or three per iteration: the 30,753-node film
// took 1.1 ms (warm start, 1e-10) to 3.3 ms (1e-12) per Neumann solve and a
// 1,331-node cube 0.34 to 0.88 ms, whatever the bandwidth.  The matrix never
// changes, so it is factored once and a solve becomes two sweeps over a
// separator tree, with one barrier per level.
//
// Tree.  Nodes are split recursively at the median plane of the longest
// extent; the nodes of one side that touch the other are the separator.
// Consecutive tree levels are merged into groups; a "front" is the part of a
// subtree inside one group, with k pivots (its separators, or whole leaves)
// and nb boundary nodes (the ancestors' pivots the subtree touches).  With the
// front's matrix [A11 A12; A21 A22] after its children's Schur complements
// are added, the factor keeps two dense blocks, rows contiguous:
//   down  [P | W^T]  (k x (k + nb)),  P = A11^-1,  W = A21 P,   up  W  (nb x k).
// Solve: upwards  u = v2 - W v1  (v: right-hand side plus the children's u,
// gathered in a fixed order, so results repeat bit for bit), downwards
// x1 = [P | W^T] . [v1; -x2].  Both are dense row products, no recurrences.
// A level costs a barrier and the latency of one task in either direction
// (kLevelSec), fewer levels cost more entries; nd_plan groups the levels by
// that cost, so that up to ~1,000 nodes the whole matrix is one front, and
// the film has five levels.
//
// The Neumann matrix is singular: the root's block, whose null space is the
// constant vector, gets alpha 1 1^T added, which leaves the solution of a
// centred right-hand side unchanged up to the constant that is removed.
//
// Every solve ends with the FP64 residual b - A x; while it exceeds the
// tolerance the residual is solved for and added (FP64 factors: none needed
// down to ~1e-13; FP32 factors: each pass gains 4 to 6 digits, less on long
// wires, whose condition number is the square of their length in elements).
// A residual that no longer falls is the answer's rounding once it is as small
// as that of |A||x| + |b|, and ends the solve as well (kNdRound): on a wire of
// L x 1 x 1 cells, magnetised along it, that is 1.5e-12 of |b| for L = 500,
// 1e-11 for 2,000, 1e-10 for 8,000, and no FP64 answer has a smaller one.  (The
// FP64 CG's recurrence runs on below it and meets any tolerance; the
// mixed-precision CG measures its residual and refuses one below rounding, and
// so do FP32 factors, but for the few units by which two answers' rounding differs.)
#include <algorithm>
#include <array>
#include <cmath>
#include <cstring>
#include <vector>

#include "nd_solve.h"
#include "nmg_internal.h"

namespace nmg {
namespace {

constexpr int kNdThreads = 512;              // two workers of 256 threads per block
constexpr int kNdWorker = 256;
constexpr int nd_chunk(int mb) { return mb == 8 ? 1024 : 2048; }   // vector entries a worker keeps in shared memory
constexpr int kNdPanel = 32;                 // pivots eliminated per factorisation step
constexpr int kNdMaxPass = 11;
constexpr int kNdProbePass = 8;              // passes the setup's probes may take; more: the CG
// Residuals that have stopped falling lie at 0.5 to 3 units of rounding
// (2^-53) of |A||x| + |b|, at 20 on a wire of 16,000 cells.
constexpr double kNdRound = 64.0 / 9007199254740992.0;
constexpr int kNdChildren = 8;               // children of a front at most (three merged tree levels)
constexpr double kLevelSec = 3.5e-6, kEntriesPerSec = 0.3e12;   // the plan's cost model
constexpr unsigned kNdSpinLimit = 1u << 25;  // seconds; then the error flag ends every block

inline int nblk(long long n, int t) { return (int)((n + t - 1) / t); }

// ---------------------------------------------------------------- ordering

struct TreeNode {
  int lo, hi, sep, depth;   // positions [lo, hi) of the subtree, pivots of this node [sep, hi)
  int child[2];
  std::vector<int> bnd;     // positions >= hi adjacent to the subtree, ascending
};

struct Orderer {
  const std::vector<int32_t> &rp, &ci;
  const std::vector<double> &X;
  const std::vector<int32_t> &local;   // node -> 0 (active) or -1
  std::vector<int> node;               // active nodes, permuted in place into elimination order
  std::vector<int> side, stamp;        // per mesh node
  std::vector<TreeNode> tree;
  int leaf, tick = 0;

  Orderer(const std::vector<int32_t> &rp_, const std::vector<int32_t> &ci_, const std::vector<double> &X_,
          const std::vector<int32_t> &act, int leaf_)
      : rp(rp_), ci(ci_), X(X_), local(act), side(act.size(), 0), stamp(act.size(), 0), leaf(leaf_) {
    for (size_t i = 0; i < act.size(); ++i)
      if (act[i] >= 0) node.push_back((int)i);
  }

  // Split [lo, hi) at the median plane of the longest extent: left, right,
  // separator (the side with fewer nodes touching the other).
  bool split(int lo, int hi, int &nl, int &nr) {
    double mn[3] = {1e300, 1e300, 1e300}, mx[3] = {-1e300, -1e300, -1e300};
    for (int i = lo; i < hi; ++i)
      for (int d = 0; d < 3; ++d) {
        const double v = X[3 * (size_t)node[i] + d];
        mn[d] = std::min(mn[d], v);
        mx[d] = std::max(mx[d], v);
      }
    int order[3] = {0, 1, 2};
    std::sort(order, order + 3, [&](int a, int b) { return mx[a] - mn[a] > mx[b] - mn[b]; });
    std::vector<double> c(hi - lo);
    for (int t = 0; t < 3; ++t) {
      const int ax = order[t];
      if (!(mx[ax] > mn[ax])) return false;
      for (int i = lo; i < hi; ++i) c[i - lo] = X[3 * (size_t)node[i] + ax];
      const size_t mid = c.size() / 2;
      std::nth_element(c.begin(), c.begin() + mid, c.end());
      const double v = c[mid];
      size_t less = 0, leq = 0;
      for (double w : c) { less += w < v; leq += w <= v; }
      // the cut nearer to the middle of the two the median value allows
      const size_t half = c.size() / 2;
      const bool incl = (leq > half ? leq - half : half - leq) < (half > less ? half - less : less - half);
      const size_t nleft = incl ? leq : less;
      if (nleft == 0 || nleft == c.size()) continue;
      const int now = ++tick;
      for (int i = lo; i < hi; ++i) {
        const double w = X[3 * (size_t)node[i] + ax];
        stamp[node[i]] = now;
        side[node[i]] = (incl ? w <= v : w < v) ? 0 : 1;
      }
      size_t touch[2] = {0, 0};
      for (int i = lo; i < hi; ++i) {
        const int a = node[i], s = side[a];
        for (int q = rp[a]; q < rp[a + 1]; ++q) {
          const int b = ci[q];
          if (stamp[b] == now && (side[b] & 1) != s) { ++touch[s]; break; }
        }
      }
      const int from = touch[1] <= touch[0] ? 1 : 0;   // the separator leaves this side
      for (int i = lo; i < hi; ++i) {
        const int a = node[i];
        if ((side[a] & 1) != from) continue;
        for (int q = rp[a]; q < rp[a + 1]; ++q) {
          const int b = ci[q];
          if (stamp[b] == now && (side[b] & 1) != from) { side[a] |= 2; break; }
        }
      }
      std::vector<int> part[3];
      for (int i = lo; i < hi; ++i) {
        const int s = side[node[i]];
        part[s & 2 ? 2 : s].push_back(node[i]);
      }
      nl = (int)part[0].size();
      nr = (int)part[1].size();
      if (nl == 0 || nr == 0) continue;   // the separator swallowed a side: try the next axis
      int o = lo;
      for (auto &p : part)
        for (int a : p) node[o++] = a;
      return true;
    }
    return false;
  }

  int rec(int lo, int hi, int depth) {
    const int id = (int)tree.size();
    tree.push_back({lo, hi, lo, depth, {-1, -1}, {}});
    int nl = 0, nr = 0;
    if (hi - lo > leaf && depth < 24 && split(lo, hi, nl, nr)) {
      const int a = rec(lo, lo + nl, depth + 1);
      const int b = rec(lo + nl, lo + nl + nr, depth + 1);
      tree[id].child[0] = a;
      tree[id].child[1] = b;
      tree[id].sep = lo + nl + nr;
    }
    return id;
  }

  // bnd of every tree node, children first (they follow their parent in `tree`)
  void boundaries(const std::vector<int32_t> &pos) {
    std::vector<int> seen(node.size(), -1);
    for (int t = (int)tree.size() - 1; t >= 0; --t) {
      TreeNode &f = tree[t];
      auto take = [&](int p) {
        if (p >= f.hi && seen[p] != t) { seen[p] = t; f.bnd.push_back(p); }
      };
      for (int c : f.child)
        if (c >= 0)
          for (int p : tree[c].bnd) take(p);
      for (int p = f.sep; p < f.hi; ++p) {
        const int a = node[p];
        for (int q = rp[a]; q < rp[a + 1]; ++q)
          if (local[ci[q]] >= 0) take(pos[ci[q]]);
      }
      std::sort(f.bnd.begin(), f.bnd.end());
    }
  }
};

// ---------------------------------------------------------------- factorisation

// F (s x s per front) = the children's Schur complements, gathered through the
// front's maps (entry of a child's boundary for each local index, or -1).
__global__ void k_nd_assemble(const NdFront *__restrict__ fr, int f0, const int32_t *__restrict__ map,
                              const long long *__restrict__ foff, const double *__restrict__ Fc,
                              const int *__restrict__ child, double *__restrict__ F) {
  const NdFront f = fr[f0 + blockIdx.y];
  double *out = F + foff[f0 + blockIdx.y];
  const int *ch = child + (size_t)kNdChildren * (f0 + blockIdx.y);
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < (long long)f.s * f.s;
       e += (long long)gridDim.x * blockDim.x) {
    const int r = (int)(e / f.s), c = (int)(e - (long long)r * f.s);
    double v = 0.0;
    for (int q = 0; q < f.nch; ++q) {
      const NdFront g = fr[ch[q]];
      const int a = map[f.moff + (size_t)q * f.s + r], b = map[f.moff + (size_t)q * f.s + c];
      if (a >= 0 && b >= 0)
        v += Fc[foff[ch[q]] + (size_t)(g.k + a - g.uoff) * g.s + (g.k + b - g.uoff)];
    }
    out[e] = v;
  }
}

// The matrix entries of the front's pivot rows (entries towards descendants
// were added in their fronts).
__global__ void k_nd_entries(const NdFront *__restrict__ fr, int f0, const long long *__restrict__ foff,
                             const int32_t *__restrict__ prow, const int32_t *__restrict__ pcol,
                             const double *__restrict__ pK, const int32_t *__restrict__ bnd, double *__restrict__ F) {
  const NdFront f = fr[f0 + blockIdx.y];
  double *out = F + foff[f0 + blockIdx.y];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= f.k) return;
  const int32_t *B = bnd + f.boff;
  for (int q = prow[f.pos + i]; q < prow[f.pos + i + 1]; ++q) {
    const int o = pcol[q];
    if (o < f.pos) continue;
    if (o < f.pos + f.k) {
      out[(size_t)i * f.s + (o - f.pos)] += pK[q];
    } else {
      int lo = 0, hi = f.nb;
      while (lo < hi) { const int mid = (lo + hi) >> 1; if (B[mid] < o) lo = mid + 1; else hi = mid; }
      if (lo >= f.nb || B[lo] != o) continue;   // never: the boundary holds every later neighbour
      out[(size_t)i * f.s + f.k + lo] += pK[q];
      out[((size_t)f.k + lo) * f.s + i] += pK[q];
    }
  }
}

// Root of the singular (Neumann) system: + (mean diagonal / k) 1 1^T.
__global__ void k_nd_regularise(int k, double *__restrict__ F) {
  __shared__ double sm[32];
  double t = 0.0;
  for (int i = threadIdx.x; i < k; i += blockDim.x) t += F[(size_t)i * k + i];
  for (int o = 16; o; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = t;
  __syncthreads();
  t = 0.0;
  for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += sm[w];
  const double a = t / k / k;
  for (long long e = threadIdx.x; e < (long long)k * k; e += blockDim.x) F[e] += a;
}

// One elimination step of every front of a level, in the symmetric sweep form
// (all rows, eliminated ones included): with D = F[p,p], C = F[:,p],
// E = C D^-1: F[p,p] -> -D^-1, F[:,p] -> E, the rest -= E C^T.  After the k
// pivots the front holds [-P, W^T; W, Schur complement].  k_nd_panel forms D^-1,
// C and E (a block inverts D by itself, 32 dependent FP64 steps, ~7 us);
// k_nd_update applies them: 64 x 64 tiles, FP64-pipe-bound, the lower
// triangle of tiles computed and mirrored.
__global__ void __launch_bounds__(256) k_nd_panel(const NdFront *__restrict__ fr, int f0, int p0,
                                                  const long long *__restrict__ foff,
                                                  const long long *__restrict__ eoff, const double *__restrict__ F,
                                                  double *__restrict__ C, double *__restrict__ E,
                                                  double *__restrict__ Dn) {
  __shared__ double D[kNdPanel][kNdPanel + 1], Cs[64][kNdPanel + 1];
  const NdFront f = fr[f0 + blockIdx.y];
  const int r0 = blockIdx.x * 64;
  if (p0 >= f.k || r0 >= f.s) return;
  const double *A = F + foff[f0 + blockIdx.y];
  const int w = min(kNdPanel, f.k - p0), tid = threadIdx.x;
  for (int e = tid; e < kNdPanel * kNdPanel; e += 256) {
    const int i = e / kNdPanel, j = e % kNdPanel;
    D[i][j] = (i < w && j < w) ? A[(size_t)(p0 + i) * f.s + p0 + j] : (i == j ? 1.0 : 0.0);
  }
  for (int e = tid; e < 64 * kNdPanel; e += 256) {
    const int i = e / kNdPanel, j = e % kNdPanel;
    Cs[i][j] = (r0 + i < f.s && j < w) ? A[(size_t)(r0 + i) * f.s + p0 + j] : 0.0;
  }
  __syncthreads();
  for (int q = 0; q < w; ++q) {
    const double inv = 1.0 / D[q][q];
    double v[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const int e = tid + 256 * t, i = e / kNdPanel, j = e % kNdPanel;
      if (i == q && j == q) v[t] = -inv;
      else if (i == q) v[t] = D[q][j] * inv;
      else if (j == q) v[t] = D[i][q] * inv;
      else v[t] = D[i][j] - D[i][q] * inv * D[q][j];
    }
    __syncthreads();
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const int e = tid + 256 * t;
      D[e / kNdPanel][e % kNdPanel] = v[t];
    }
    __syncthreads();
  }
  const size_t eo = (size_t)eoff[f0 + blockIdx.y] * kNdPanel;
  for (int e = tid; e < 64 * kNdPanel; e += 256) {
    const int i = e / kNdPanel, j = e % kNdPanel;
    if (r0 + i >= f.s) break;
    double t = 0.0;
    for (int q = 0; q < w; ++q) t -= Cs[i][q] * D[q][j];   // D is -inverse here
    const size_t o = eo + (size_t)(r0 + i) * kNdPanel + j;
    C[o] = Cs[i][j];
    E[o] = j < w ? t : 0.0;
  }
  if (blockIdx.x == 0)
    for (int e = tid; e < kNdPanel * kNdPanel; e += 256)
      Dn[(size_t)blockIdx.y * kNdPanel * kNdPanel + e] = D[e / kNdPanel][e % kNdPanel];
}

__global__ void __launch_bounds__(256) k_nd_update(const NdFront *__restrict__ fr, int f0, int p0,
                                                   const long long *__restrict__ foff,
                                                   const long long *__restrict__ eoff, double *__restrict__ F,
                                                   const double *__restrict__ C, const double *__restrict__ E,
                                                   const double *__restrict__ Dn) {
  __shared__ double Es[64][kNdPanel + 1], Cs[kNdPanel][64 + 1];
  const NdFront f = fr[f0 + blockIdx.z];
  const int ti = blockIdx.y, tj = blockIdx.x;
  if (p0 >= f.k || tj > ti || ti * 64 >= f.s) return;
  double *A = F + foff[f0 + blockIdx.z];
  const size_t eo = (size_t)eoff[f0 + blockIdx.z] * kNdPanel;
  const double *dn = Dn + (size_t)blockIdx.z * kNdPanel * kNdPanel;
  const int tid = threadIdx.x, w = min(kNdPanel, f.k - p0);
  for (int e = tid; e < 64 * kNdPanel; e += 256) {
    const int i = e / kNdPanel, j = e % kNdPanel;
    Es[i][j] = ti * 64 + i < f.s ? E[eo + (size_t)(ti * 64 + i) * kNdPanel + j] : 0.0;
    Cs[j][i] = tj * 64 + i < f.s ? C[eo + (size_t)(tj * 64 + i) * kNdPanel + j] : 0.0;
  }
  __syncthreads();
  const int tx = tid & 15, ty = tid >> 4;
  double acc[4][4] = {};
  for (int q = 0; q < w; ++q) {
    double a[4], b[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) { a[i] = Es[ty + 16 * i][q]; b[i] = Cs[q][tx + 16 * i]; }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = fma(a[i], b[j], acc[i][j]);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int r = ti * 64 + ty + 16 * i, c = tj * 64 + tx + 16 * j;
      if (r >= f.s || c >= f.s) continue;
      const bool rp = r >= p0 && r < p0 + w, cp = c >= p0 && c < p0 + w;
      double v;
      if (rp && cp) v = dn[(r - p0) * kNdPanel + (c - p0)];
      else if (rp) v = E[eo + (size_t)c * kNdPanel + (r - p0)];
      else if (cp) v = E[eo + (size_t)r * kNdPanel + (c - p0)];
      else v = A[(size_t)r * f.s + c] - acc[i][j];
      A[(size_t)r * f.s + c] = v;
      if (ti != tj) A[(size_t)c * f.s + r] = v;
    }
}

// [P | W^T] (the first k rows) and W (the other rows' first k columns) to the factor.
__global__ void k_nd_store(const NdFront *__restrict__ fr, int f0, const long long *__restrict__ foff,
                           const double *__restrict__ F, double *__restrict__ out) {
  const NdFront f = fr[f0 + blockIdx.y];
  const double *A = F + foff[f0 + blockIdx.y];
  const long long nd = (long long)f.k * f.s, n = nd + (long long)f.nb * f.k;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n;
       e += (long long)gridDim.x * blockDim.x) {
    if (e < nd) {
      const int c = (int)(e % f.s);
      out[f.off + e] = c < f.k ? -A[e] : A[e];
    } else {
      const long long q = e - nd;
      const int j = (int)(q / f.k), i = (int)(q - (long long)j * f.k);
      out[f.off + e] = A[((size_t)f.k + j) * f.s + i];
    }
  }
}

__global__ void k_nd_f32(long long n, const double *__restrict__ a, float *__restrict__ b) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    b[i] = (float)a[i];
}

// The active part of K in elimination order.
__global__ void k_nd_rows(int n, const int32_t *__restrict__ perm, const int32_t *__restrict__ posof,
                          const int32_t *__restrict__ row_ptr, const int32_t *__restrict__ col_idx,
                          const double *__restrict__ K, const int32_t *__restrict__ prow, int32_t *__restrict__ pcol,
                          double *__restrict__ pK) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  int o = prow[p];
  const int a = perm[p];
  for (int q = row_ptr[a]; q < row_ptr[a + 1]; ++q) {
    const int c = posof[col_idx[q]];
    if (c < 0) continue;
    pcol[o] = c;
    pK[o] = K[q];
    ++o;
  }
}

// The setup's right-hand sides: 1 everywhere, one without structure, one that
// rises along an axis (the smoothest, whose answer is the largest).
enum { kProbeOne, kProbeHash, kProbeRise, kProbes };
__global__ void k_nd_probe(int n, double *__restrict__ b, int kind, const double *__restrict__ X, int axis,
                           double middle) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (kind == kProbeOne) b[i] = 1.0;
  else if (kind == kProbeHash) b[i] = (double)((unsigned)i * 2654435761u >> 8) / 16777216.0 - 0.5;
  else b[i] = X[3 * (size_t)i + axis] - middle;
}

// one = x (elimination order), kone = K x.
__global__ void k_nd_one(int n, const int32_t *__restrict__ prow,
                         const int32_t *__restrict__ pcol, const double *__restrict__ pK,
                         const double *__restrict__ x, double *__restrict__ one, double *__restrict__ kone) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  double s = 0.0;
  for (int q = prow[p]; q < prow[p + 1]; ++q) s = fma(pK[q], x[pcol[q]], s);
  one[p] = x[p];
  kone[p] = s;
}

// ---------------------------------------------------------------- solve

struct NdArgs {
  int N, n, nlev, mode, nm;   // mesh nodes, active nodes, tree levels, system, members
  const NdFront *front;
  const NdLevel *phase;       // 2 nlev - 1: upwards levels nlev - 1 .. 1, downwards 0 .. nlev - 1
  const NdTask *task;
  const int32_t *bnd, *map, *perm, *prow, *pcol, *b_of_node;
  const double *pK;
  const void *fac;
  const double *b;
  const double *one, *kone;   // mode 0: the sweeps' answer to b = 1 and K times it (null: sweeps alone, x as they give it)
  double *x, *xw, *r, *part;
  NdOut out;
  int nbnd;
  void *u, *d;
  unsigned *bar;
  int *err, *iters;
  double rtol, atol;
  bool probe;                 // whatever the tolerance, down to rounding will do
};

__device__ __forceinline__ unsigned nd_ld_acquire(const unsigned *p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Grid barrier in two halves, so that a block can fetch what does not depend
// on the others in between: one release add per block, then thread 0 polls
// with acquire loads.  The error word is looked at every 1024 polls only, and
// the outcome reaches the block through the closing __syncthreads, not through
// another load.
__device__ __forceinline__ void nd_arrive(const NdArgs &a) {
  __syncthreads();
  if (gridDim.x > 1 && threadIdx.x == 0)
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(a.bar) : "memory");
}
__device__ __forceinline__ bool nd_wait(const NdArgs &a, unsigned &epoch) {
  if (gridDim.x == 1) return true;   // nd_arrive's __syncthreads was the barrier
  int ok = 1;
  ++epoch;
  if (threadIdx.x == 0) {
    const unsigned target = epoch * gridDim.x;
    unsigned spins = 0;
    while (nd_ld_acquire(a.bar) < target) {
      if ((++spins & 1023u) == 0u && (spins > kNdSpinLimit || (*(volatile int *)a.err & ERR_BARRIER))) {
        atomicOr(a.err, ERR_BARRIER);
        ok = 0;
        break;
      }
    }
  }
  return __syncthreads_and(ok) != 0;
}

// The last block to leave clears the counters for the next launch.
__device__ __forceinline__ void nd_leave(const NdArgs &a) {
  if (gridDim.x > 1 && threadIdx.x == 0 && atomicAdd(a.bar + 1, 1u) == gridDim.x - 1) {
    a.bar[0] = 0u;
    a.bar[1] = 0u;
  }
}

__device__ __forceinline__ void worker_sync(int half) {
  asm volatile("bar.sync %0, %1;" ::"r"(half + 1), "n"(kNdWorker) : "memory");
}

// MB consecutive values written by another block of this launch.
template <typename T, int MB>
__device__ __forceinline__ void ld_members(const T *p, T (&v)[MB]) {
  if constexpr (sizeof(T) * MB % 16 == 0) {
    constexpr int PER = 16 / sizeof(T);
#pragma unroll
    for (int q = 0; q < MB / PER; ++q) {
      const float4 t = __ldcg(reinterpret_cast<const float4 *>(p) + q);
      memcpy(&v[q * PER], &t, 16);
    }
  } else {
#pragma unroll
    for (int m = 0; m < MB; ++m) v[m] = __ldcg(p + m);
  }
}

// Sum each of NV values over the warp by recursive halving; lane L ends with
// the total of value L >> (5 - log2 NV).
template <typename T, int NV>
__device__ __forceinline__ T nd_transpose_sum(T (&v)[NV]) {
  const int lane = threadIdx.x & 31;
  int n = NV;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    if (n > 1) {
      const bool up = (lane & o) != 0;
#pragma unroll
      for (int i = 0; i < NV / 2; ++i) {
        if (i >= n / 2) break;
        const T send = up ? v[i] : v[i + n / 2];
        const T keep = up ? v[i + n / 2] : v[i];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
      }
      n >>= 1;
    } else {
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    }
  }
  return v[0];
}

// Sums over the grid, in a fixed order and identical in every block, of two
// values for each of MB members; a thread brings MW members' (member
// MW (thread mod MB / MW) first): v[0..MW) and v[MW..2 MW).  nd_partial leaves
// the block's share in `slot`, nd_total adds the shares after a barrier; res
// (shared): [value][member].  sm: 16 x 2 MB scratch.
template <int MB, int MW>
__device__ __forceinline__ void nd_partial(const double (&v)[2 * MW], double *sm, double *slot) {
  constexpr int Q = MB / MW, NV = 2 * MB, NW = kNdThreads / 32;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int j = 0; j < 2 * MW; ++j) {
    double s = v[j];
#pragma unroll
    for (int o = 16; o >= Q; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane < Q) sm[wid * NV + (j / MW) * MB + lane * MW + j % MW] = s;
  }
  __syncthreads();
  if (wid < NV) {
    double s = lane < NW ? sm[lane * NV + wid] : 0.0;
#pragma unroll
    for (int o = NW / 2; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) slot[(size_t)wid * gridDim.x + blockIdx.x] = s;
  }
  __syncthreads();   // sm may be used again
}
template <int MB>
__device__ __forceinline__ void nd_total(const double *slot, double *res) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (wid < 2 * MB) {
    double s = 0.0;
#pragma unroll 5
    for (unsigned b = lane; b < gridDim.x; b += 32) s += __ldcg(slot + (size_t)wid * gridDim.x + b);
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) res[wid] = s;
  }
  __syncthreads();
}

// One solve of nm <= MB right-hand sides (member m at b + m N), factors and
// sweeps in T (see the head of the file).  Bound by the latency of a task and
// a barrier per level and direction; a worker fetches its next task's
// descriptors and gather lists before it waits.
template <typename T, int MB>
__global__ void __launch_bounds__(kNdThreads, 1) k_nd_solve(NdArgs a) {
  constexpr int RW = MB == 8 ? 4 : 8;              // rows a warp takes at once
  constexpr int NV = RW * MB;                      // 8, 16 or 32 sums per warp
  constexpr int SH = NV == 32 ? 0 : (NV == 16 ? 1 : 2);
  constexpr int MW = MB >= 2 ? 2 : 1, Q = MB / MW; // row work outside the sweeps: Q threads per row, MW members each
  extern __shared__ char nd_dyn[];
  __shared__ double s_res[2 * MB], s_mean[MB], s_tol[MB], s_last[MB];
  __shared__ double s_size[2 * MB];
  __shared__ int s_state;
  __shared__ double s_sm[kNdThreads / 32 * 2 * MB];
  const int tid = threadIdx.x, half = tid / kNdWorker, wt = tid % kNdWorker;
  const int lane = tid & 31, ww = wt >> 5;
  constexpr int kNdChunk = nd_chunk(MB);
  T *vs = reinterpret_cast<T *>(nd_dyn) + (size_t)half * (kNdChunk + kNdWorker) * MB;   // vector chunk
  T *rs = vs + (size_t)kNdChunk * MB;                                                   // partial sums
  const T *fac = static_cast<const T *>(a.fac);
  T *U = static_cast<T *>(a.u), *Dv = static_cast<T *>(a.d);
  const int nworker = 2 * gridDim.x, worker = half * gridDim.x + blockIdx.x;
  const int gt = blockIdx.x * kNdThreads + tid, gn = gridDim.x * kNdThreads;
  unsigned epoch = 0;

  // the blocks' shares of the right-hand sides' sums and squares (added up
  // when the first residual needs them); Dirichlet rows pass through
  double *slot0 = a.part, *slot1 = a.part + 2 * MB * (size_t)gridDim.x;
  if (a.one || a.mode == 1) {
    double v[2 * MW];
#pragma unroll
    for (int q = 0; q < 2 * MW; ++q) v[q] = 0.0;
    const int m0 = gt % Q * MW;
    for (int i = gt / Q; i < a.N; i += gn / Q) {
      const bool fixed = a.mode == 1 && a.perm[i] < 0;
#pragma unroll
      for (int w = 0; w < MW; ++w) {
        const int m = m0 + w;
        const double t = m < a.nm ? a.b[(size_t)m * a.N + i] : 0.0;
        v[w] += t;
        v[MW + w] += t * t;
        if (fixed && m < a.nm) {
          const size_t o = (size_t)m * a.N + i;
          a.x[o] = t;
          if (a.out.sum) a.out.sum[o] = a.out.add[o] + t;
        }
      }
    }
    nd_partial<MB, MW>(v, s_sm, slot0);
  }
  if (a.nlev == 0) nd_arrive(a);

  int pass = 0;
  int failed = 0;
  // the vector entry a task's row products need at local index c of front f:
  // right-hand side plus the children's u (c < k), the solution's negative
  // (downwards, c >= k)
  auto gather = [&](const NdFront &f, int c, T (&v)[MB]) {
    if (c < f.k) {
      if (pass == 0) {
        const int i = __ldg(a.perm + a.N + f.pos + c);
#pragma unroll
        for (int m = 0; m < MB; ++m) v[m] = m < a.nm ? (T)a.b[(size_t)m * a.N + i] : T(0);
      } else {
        double t[MB];
        ld_members<double, MB>(a.r + ((size_t)f.pos + c) * MB, t);
#pragma unroll
        for (int m = 0; m < MB; ++m) v[m] = (T)t[m];
      }
      constexpr int GB = 8 / MB;   // children's values in flight
      for (int q0 = 0; q0 < f.nch; q0 += GB) {
        int i[GB];
        T w[GB][MB];
#pragma unroll
        for (int q = 0; q < GB; ++q)
          i[q] = q0 + q < f.nch ? __ldg(a.map + f.moff + (size_t)(q0 + q) * f.s + c) : -1;
#pragma unroll
        for (int q = 0; q < GB; ++q)
          if (i[q] >= 0) ld_members<T, MB>(U + (size_t)i[q] * MB, w[q]);
#pragma unroll
        for (int q = 0; q < GB; ++q)   // (an FP64 add costs its warp 16 cycles of the pipe: none for nothing)
          if (i[q] >= 0)
#pragma unroll
            for (int m = 0; m < MB; ++m) v[m] += w[q][m];
      }
    } else {
      ld_members<T, MB>(Dv + (size_t)__ldg(a.bnd + f.boff + c - f.k) * MB, v);
#pragma unroll
      for (int m = 0; m < MB; ++m) v[m] = -v[m];
    }
  };
  for (;; ++pass) {
    for (int ph = 0; ph < 2 * a.nlev - 1; ++ph) {
      const NdLevel lv = a.phase[ph];
      const bool up = ph < a.nlev - 1;
      const int cs = lv.cs, group = ww / cs, part = ww % cs, rows = RW * (8 / cs);
      NdTask tk = {0, 0, 0};
      NdFront f = {};
      int t = lv.t0 + worker;
      if (t < lv.t1) {
        tk = a.task[t];
        f = a.front[tk.front];
        // the gather lists and the rows to L1 before the wait
        const int len = up ? f.k : f.s;
        const char *M0 = reinterpret_cast<const char *>(fac + f.off + (up ? (size_t)f.k * f.s : 0) +
                                                        (size_t)tk.start * len);
        const int bytes = min(tk.count * len * (int)sizeof(T), 48 * 1024);
        for (int o = wt * 128; o < bytes; o += kNdWorker * 128)
          asm volatile("prefetch.global.L1 [%0];" ::"l"(M0 + o));
        for (int c = wt; c < len; c += kNdWorker) {
          const int32_t *l = c < f.k ? a.map + f.moff + c : a.bnd + f.boff + c - f.k;
          for (int q = 0; q < (c < f.k ? f.nch : 1); ++q)
            asm volatile("prefetch.global.L1 [%0];" ::"l"(l + (size_t)q * f.s));
        }
      }
      if ((ph > 0 || pass > 0) && !nd_wait(a, epoch)) return;
      for (; t < lv.t1; t += nworker) {
        if (t >= lv.t0 + nworker) {
          tk = a.task[t];
          f = a.front[tk.front];
        }
        const int len = up ? f.k : f.s;   // row length
        const T *M = fac + f.off + (up ? (size_t)f.k * f.s : 0);
        const int nrow = up ? f.nb : f.k;
        for (int sub = 0; sub < tk.count; sub += rows) {
          const int row0 = tk.start + sub + group * RW;
          // upwards: the value this thread's output starts from, in flight early
          T base = T(0);
          const int oi = wt / MB, om = wt % MB;
          const bool out = wt < rows * MB && sub + oi < tk.count;
          if (up && out) {
            const int c = f.k + tk.start + sub + oi;
            int i[kNdChildren];
#pragma unroll
            for (int q = 0; q < kNdChildren; ++q)
              i[q] = q < f.nch ? __ldg(a.map + f.moff + (size_t)q * f.s + c) : -1;
            T w[kNdChildren];
#pragma unroll
            for (int q = 0; q < kNdChildren; ++q)
              if (i[q] >= 0) w[q] = __ldcg(U + (size_t)i[q] * MB + om);
#pragma unroll
            for (int q = 0; q < kNdChildren; ++q)
              if (i[q] >= 0) base += w[q];
          }
          const T *rp[RW];
#pragma unroll
          for (int r = 0; r < RW; ++r) rp[r] = M + (size_t)min(row0 + r, nrow - 1) * len;
          T acc[NV];
#pragma unroll
          for (int q = 0; q < NV; ++q) acc[q] = T(0);
          for (int c0 = 0; c0 < len; c0 += kNdChunk) {
            const int n = min(kNdChunk, len - c0);
            if (sub == 0 || len > kNdChunk) {
              for (int e = wt; e < n; e += kNdWorker) {
                T v[MB];
                gather(f, c0 + e, v);
#pragma unroll
                for (int m = 0; m < MB; ++m) vs[e * MB + m] = v[m];
              }
              worker_sync(half);
            }
#pragma unroll 2
            for (int e = part * 32 + lane; e < n; e += 32 * cs) {
              T z[MB];
#pragma unroll
              for (int m = 0; m < MB; ++m) z[m] = vs[e * MB + m];
#pragma unroll
              for (int r = 0; r < RW; ++r) {
                const T w = __ldg(rp[r] + c0 + e);
#pragma unroll
                for (int m = 0; m < MB; ++m) acc[r * MB + m] = fma(w, z[m], acc[r * MB + m]);
              }
            }
            if (len > kNdChunk) worker_sync(half);
          }
          const T tot = nd_transpose_sum<T, NV>(acc);
          if ((lane & ((1 << SH) - 1)) == 0) rs[ww * NV + (lane >> SH)] = tot;
          worker_sync(half);
          if (out) {
            const int g = oi / RW, q = (oi % RW) * MB + om, row = tk.start + sub + oi;
            T s = T(0);
            for (int p = 0; p < cs; ++p) s += rs[(g * cs + p) * NV + q];
            if (up) {
              U[((size_t)f.uoff + row) * MB + om] = base - s;
            } else {
              const size_t o = ((size_t)f.pos + row) * MB + om;
              Dv[o] = s;
              a.xw[o] = pass == 0 ? (double)s : __ldcg(a.xw + o) + (double)s;
            }
          }
          worker_sync(half);
        }
      }
      nd_arrive(a);
    }
    if (!nd_wait(a, epoch)) return;
    if (pass == 0 && (a.one || a.mode == 1)) {
      nd_total<MB>(slot0, s_res);
      if (tid < MB) {
        const double mean = a.mode == 0 ? s_res[tid] / a.N : 0.0;
        const double bn = sqrt(fmax(s_res[MB + tid] - a.N * mean * mean, 0.0));
        s_mean[tid] = mean;
        s_tol[tid] = fmax(a.rtol * bn, a.atol);
        s_last[tid] = 0.0;
      }
      __syncthreads();
    }
    if (a.mode == 0 && !a.one) break;   // the sweeps alone
    // ---- residual: Q threads per row, MW members each.  The sweeps took b as
    // it is; its mean's share, mean * one, leaves the answer here ----
    double v[2 * MW];
#pragma unroll
    for (int q = 0; q < 2 * MW; ++q) v[q] = 0.0;
    const int m0 = gt % Q * MW;
    for (int p = gt / Q; p < a.n; p += gn / Q) {
      double s[MW], t[MW], x0[MW], rb[MW];
      const int q1 = a.prow[p + 1], i = a.perm[a.N + p];
      const double k1 = a.mode == 0 ? a.kone[p] : 0.0, w1 = a.mode == 0 ? a.one[p] : 0.0;
      ld_members<double, MW>(a.xw + (size_t)p * MB + m0, x0);
#pragma unroll
      for (int w = 0; w < MW; ++w) {
        s[w] = 0.0;
        rb[w] = m0 + w < a.nm ? a.b[(size_t)(m0 + w) * a.N + i] : 0.0;
      }
#pragma unroll 4
      for (int q = a.prow[p]; q < q1; ++q) {
        ld_members<double, MW>(a.xw + (size_t)a.pcol[q] * MB + m0, t);
        const double kv = a.pK[q];
#pragma unroll
        for (int w = 0; w < MW; ++w) s[w] = fma(kv, t[w], s[w]);
      }
#pragma unroll
      for (int w = 0; w < MW; ++w) {
        const int m = m0 + w;
        const double mean = m < a.nm ? s_mean[m] : 0.0;
        const double r = (rb[w] - mean) - (s[w] - mean * k1);
        a.r[(size_t)p * MB + m] = r;
        v[w] += r * r;
        v[MW + w] += x0[w] - mean * w1;
      }
    }
    nd_partial<MB, MW>(v, s_sm, slot1);
    nd_arrive(a);
    if (!nd_wait(a, epoch)) return;
    nd_total<MB>(slot1, s_res);
    if (tid == 0) {
      int st = 1;   // 1 done, 0 another pass, 2 not finite, 3 done if what is left is rounding
      for (int m = 0; m < a.nm; ++m) {
        const double rn = sqrt(s_res[m]);
        if (!(rn == rn) || isinf(rn)) st = 2;
        else if (!(rn <= s_tol[m]) && st != 2)
          st = st != 0 && pass > 0 && (rn > 0.25 * s_last[m] || pass + 1 >= kNdMaxPass) ? 3 : 0;
        s_last[m] = rn;
      }
      s_state = st;
    }
    __syncthreads();
    int st = s_state;
    if (st == 3) {   // the same in every block
#pragma unroll
      for (int q = 0; q < 2 * MW; ++q) v[q] = 0.0;
      for (int p = gt / Q; p < a.n; p += gn / Q) {
        double t[MW], s[MW];
        const int i = a.perm[a.N + p];
#pragma unroll
        for (int w = 0; w < MW; ++w) s[w] = m0 + w < a.nm ? fabs(a.b[(size_t)(m0 + w) * a.N + i]) : 0.0;
        for (int q = a.prow[p]; q < a.prow[p + 1]; ++q) {
          ld_members<double, MW>(a.xw + (size_t)a.pcol[q] * MB + m0, t);
          const double kv = fabs(a.pK[q]);
#pragma unroll
          for (int w = 0; w < MW; ++w) s[w] = fma(kv, fabs(t[w]), s[w]);
        }
#pragma unroll
        for (int w = 0; w < MW; ++w) v[w] += s[w] * s[w];
      }
      nd_partial<MB, MW>(v, s_sm, slot0);   // (read in the first pass only)
      nd_arrive(a);
      if (!nd_wait(a, epoch)) return;
      nd_total<MB>(slot0, s_size);
      if (tid == 0) {
        st = 1;
        for (int m = 0; m < a.nm; ++m) {
          double floor = kNdRound * sqrt(s_size[m]);
          if (sizeof(T) == 4 && !a.probe) floor = fmin(floor, 4.0 * s_tol[m]);
          if (!(s_last[m] <= fmax(s_tol[m], floor))) st = 0;
        }
        s_state = st;
      }
      __syncthreads();
      st = s_state;
    }
    if (st == 2) failed = ERR_NONFINITE;
    else if (st == 0 && pass + 1 >= kNdMaxPass) failed = ERR_CG_MAXITS;
    if (st != 0 || failed) break;
    nd_arrive(a);   // slot1 is free, r is complete
  }
  {
    const int m0 = gt % Q * MW;
    for (int p = gt / Q; p < a.n; p += gn / Q) {
      const int i = a.perm[a.N + p];
      const double w1 = a.one ? a.one[p] : 0.0;
#pragma unroll
      for (int w = 0; w < MW; ++w) {
        const int m = m0 + w;
        if (m >= a.nm) continue;
        double t = __ldcg(a.xw + (size_t)p * MB + m);
        if (a.one) t = (t - s_mean[m] * w1) - s_res[MB + m] / a.N;   // mode 0
        const size_t o = (size_t)m * a.N + i;
        a.x[o] = t;
        if (a.out.sum) a.out.sum[o] = a.out.add[o] + t;
        if (a.out.bnd) {
          const int bi = a.b_of_node[i];
          if (bi >= 0) a.out.bnd[(size_t)m * a.nbnd + bi] = t;
        }
      }
    }
  }
  if (gt == 0) {
    a.iters[a.mode] = pass + 1;
    a.iters[2 + a.mode] += pass + 1;
    if (failed) atomicOr(a.err, failed);
  }
  nd_leave(a);
}

template <typename T>
const void *nd_kernel(int nm) {
  return nm <= 1   ? (const void *)k_nd_solve<T, 1>
         : nm <= 2 ? (const void *)k_nd_solve<T, 2>
         : nm <= 4 ? (const void *)k_nd_solve<T, 4>
                   : (const void *)k_nd_solve<T, 8>;
}
int nd_members(int nm) { return nm <= 1 ? 1 : (nm <= 2 ? 2 : (nm <= 4 ? 4 : 8)); }
size_t nd_smem(int mb, size_t elem) { return 2 * (size_t)(nd_chunk(mb) + kNdWorker) * mb * elem; }

// The host side of one system's solver: the tree cut at the chosen depth, the
// sweeps' index lists and tasks.
struct NdPlan {
  int n = 0, nfront = 0, nlev = 0, grid = 1;
  int first[33] = {0};               // fronts of level d: [first[d], first[d + 1])
  long long entries = 0, nu = 0;
  std::vector<NdFront> fr;
  std::vector<int> child;            // kNdChildren per front
  std::vector<int32_t> bnd, map, pos, perm, prow;   // pos: of a node, perm: node of a position
  std::vector<NdTask> task;
  std::vector<NdLevel> phase;
};

// Shares of the rows of the fronts [f0, f1) (nb rows of k upwards, k rows of s
// downwards) for `workers` workers: the split of a row among a worker's warps
// that leaves the least over.
void nd_tasks(const NdPlan &P, int f0, int f1, bool up, int workers, NdLevel &L, std::vector<NdTask> &out) {
  double bv = 1e300;
  L.cs = 1;
  L.pad = 0;
  for (int cs : {1, 2, 4, 8}) {
    const int rows = 64 / cs;
    long long nt = 0;
    int lmax = 0;
    for (int f = f0; f < f1; ++f) {
      const int n = up ? P.fr[f].nb : P.fr[f].k, len = up ? P.fr[f].k : P.fr[f].s;
      nt += (n + rows - 1) / rows;
      if (n) lmax = std::max(lmax, len);
    }
    const double v = std::ceil((double)nt / workers) * (1.5e-6 + lmax * (1.0e-9 + rows / 1.9e9));
    if (nt && v < bv) { bv = v; L.cs = cs; }
  }
  const int rows = 64 / L.cs;
  L.t0 = (int)out.size();
  for (int f = f0; f < f1; ++f) {
    const int n = up ? P.fr[f].nb : P.fr[f].k;
    for (int i = 0; i < n; i += rows) out.push_back({f, i, std::min(rows, n - i)});
  }
  L.t1 = (int)out.size();
}

// 0: planned; -1: the direct solver does not apply (a Neumann mesh of several
// parts has one null vector each; a factor too large to pay for itself).
int nd_plan(int mode, int sm_count, const std::vector<int32_t> &rp, const std::vector<int32_t> &ci,
            const std::vector<double> &X, const std::vector<int32_t> &bon, NdPlan &P) {
  const int N = (int)rp.size() - 1;
  std::vector<int32_t> act(N, 0);
  if (mode == 1)
    for (int i = 0; i < N; ++i) act[i] = bon[i] >= 0 ? -1 : 0;
  Orderer od(rp, ci, X, act, 40);
  const int n = P.n = (int)od.node.size();
  P.pos.assign(N, -1);
  if (n == 0) {   // every node on the boundary: the solve copies the boundary values
    P.grid = std::min(sm_count, nblk(N, kNdThreads));
    return 0;
  }
  if (mode == 0) {
    std::vector<int> stack{0};
    std::vector<char> seen(N, 0);
    seen[0] = 1;
    int cnt = 1;
    while (!stack.empty()) {
      const int v = stack.back();
      stack.pop_back();
      for (int q = rp[v]; q < rp[v + 1]; ++q)
        if (!seen[ci[q]]) { seen[ci[q]] = 1; ++cnt; stack.push_back(ci[q]); }
    }
    if (cnt != N) return -1;
  }
  od.rec(0, n, 0);
  for (int p = 0; p < n; ++p) P.pos[od.node[p]] = p;
  od.boundaries(P.pos);
  const std::vector<TreeNode> &tree = od.tree;
  const int nt = (int)tree.size();
  int maxd = 0;
  for (const TreeNode &t : tree) maxd = std::max(maxd, t.depth);
  // own[t][g]: pivots of t's subtree within g tree levels (g = 0: the whole subtree)
  std::vector<std::array<int, 4>> own(nt);
  for (int t = nt - 1; t >= 0; --t) {
    own[t][0] = tree[t].hi - tree[t].lo;
    own[t][1] = tree[t].child[0] < 0 ? own[t][0] : tree[t].hi - tree[t].sep;
    for (int g = 2; g <= 3; ++g) {
      own[t][g] = own[t][1];
      if (tree[t].child[0] >= 0) own[t][g] += own[tree[t].child[0]][g - 1] + own[tree[t].child[1]][g - 1];
    }
  }
  // grouping of the tree levels: cost[d] = the cheapest continuation from
  // depth d on, len[d] = the levels merged there (0: the subtrees are leaves).
  // The factorisation counts over a few thousand solves (a nanosecond of
  // simulated time takes ten times that).
  std::vector<double> cost(maxd + 2, 1e300);
  std::vector<int> len(maxd + 2, 0);
  for (int d = maxd; d >= 0; --d)
    for (int g = 0; g <= 3; ++g) {
      if (g > 0 && d + g > maxd) continue;
      double e = 0.0, fl = 0.0;
      for (int t = 0; t < nt; ++t) {
        if (tree[t].depth != d) continue;
        const double k = own[t][g], nb = (double)tree[t].bnd.size(), s = k + nb;
        e += k * (s + nb);
        fl += k * s * s;
      }
      if (e > (double)(1ll << 28) || fl > 4e11) continue;
      const double v = (d > 0 ? 2 : 1) * kLevelSec + e / kEntriesPerSec + fl / 0.2e12 / 2000.0 +
                       (g > 0 ? cost[d + g] : 0.0);
      if (v < cost[d]) { cost[d] = v; len[d] = g; }
    }
  if (cost[0] > 1e299) return -1;
  // fronts, level by level, and the elimination order they ask for
  std::vector<int> tid, front_of(nt, -1);
  for (int d = 0;; d += len[d]) {
    P.first[P.nlev++] = (int)tid.size();
    for (int t = 0; t < nt; ++t)
      if (tree[t].depth == d) { front_of[t] = (int)tid.size(); tid.push_back(t); }
    if (len[d] == 0) break;
  }
  const int nf = P.nfront = P.first[P.nlev] = (int)tid.size();
  P.fr.resize(nf);
  P.child.assign((size_t)kNdChildren * nf, -1);
  P.perm.reserve(n);
  std::vector<int> order;   // node of each position, children first
  auto place = [&](auto &&self, int f) -> void {
    const int g = len[tree[tid[f]].depth];
    std::vector<int> piv;
    int nch = 0;
    auto walk = [&](auto &&down, int t, int left) -> void {
      const bool leaf = tree[t].child[0] < 0;
      if (g > 0 && !leaf) {
        for (int c : tree[t].child) {
          if (left > 1) {
            down(down, c, left - 1);
          } else {
            P.child[(size_t)kNdChildren * f + nch++] = front_of[c];
            self(self, front_of[c]);
          }
        }
      }
      for (int p = (g == 0 || leaf) ? tree[t].lo : tree[t].sep; p < tree[t].hi; ++p) piv.push_back(od.node[p]);
    };
    walk(walk, tid[f], g);
    P.fr[f].pos = (int)order.size();
    P.fr[f].k = (int)piv.size();
    P.fr[f].nch = nch;
    order.insert(order.end(), piv.begin(), piv.end());
  };
  place(place, 0);
  if ((int)order.size() != n) return -1;   // never: every node is a pivot once
  const std::vector<int> old = od.node;
  P.perm.assign(order.begin(), order.end());
  for (int p = 0; p < n; ++p) P.pos[P.perm[p]] = p;
  std::vector<std::vector<int>> bnd(nf);
  for (int f = 0; f < nf; ++f) {
    NdFront &q = P.fr[f];
    for (int p : tree[tid[f]].bnd) bnd[f].push_back(P.pos[old[p]]);
    std::sort(bnd[f].begin(), bnd[f].end());
    q.nb = (int)bnd[f].size();
    q.s = q.k + q.nb;
    q.off = P.entries;
    q.uoff = (int)P.nu;
    q.boff = (int)P.bnd.size();
    P.entries += (long long)q.k * (q.s + q.nb);
    P.nu += q.nb;
    P.bnd.insert(P.bnd.end(), bnd[f].begin(), bnd[f].end());
  }
  for (int f = 0; f < nf; ++f) {
    NdFront &q = P.fr[f];
    q.moff = (int)P.map.size();
    P.map.resize(P.map.size() + (size_t)q.nch * q.s, -1);
    for (int c = 0; c < q.nch; ++c) {
      const int g = P.child[(size_t)kNdChildren * f + c];
      size_t w = 0;
      for (size_t j = 0; j < bnd[g].size(); ++j) {
        int loc;
        if (bnd[g][j] < q.pos + q.k) {
          loc = bnd[g][j] - q.pos;
        } else {
          while (w < bnd[f].size() && bnd[f][w] < bnd[g][j]) ++w;
          if (w == bnd[f].size() || bnd[f][w] != bnd[g][j]) return -1;
          loc = q.k + (int)w;
        }
        if (loc < 0) return -1;   // never: a child's boundary lies in its parent's front
        P.map[q.moff + (size_t)c * q.s + loc] = P.fr[g].uoff + (int)j;
      }
    }
  }
  // blocks: one where it holds the whole solve (its barriers are free), else
  // as many as the widest phase has use for
  const bool one = n <= 96 && N <= 512;
  const int workers = one ? 2 : 2 * sm_count;
  int most = 1;
  for (int ph = 0; ph < 2 * P.nlev - 1; ++ph) {
    const bool up = ph < P.nlev - 1;
    const int d = up ? P.nlev - 1 - ph : ph - (P.nlev - 1);
    NdLevel L;
    nd_tasks(P, P.first[d], P.first[d + 1], up, workers, L, P.task);
    P.phase.push_back(L);
    most = std::max(most, L.t1 - L.t0);
  }
  P.grid = one ? 1 : std::max(1, std::min(sm_count, std::max((most + 1) / 2, N / 2048)));
  P.prow.assign(n + 1, 0);
  for (int p = 0; p < n; ++p) {
    int c = 0;
    for (int q = rp[P.perm[p]]; q < rp[P.perm[p] + 1]; ++q) c += P.pos[ci[q]] >= 0;
    P.prow[p + 1] = P.prow[p] + c;
  }
  return 0;
}

}  // namespace

// The direct solver of one system (mode 0: K with the constant null space, 1:
// the interior block).  Returns 0 with S.ready unset where it does not apply.
static int nd_build(nmg_handle *h, int mode, const std::vector<int32_t> &rp, const std::vector<int32_t> &ci,
                    const std::vector<double> &X, const std::vector<int32_t> &bon, bool f32, std::string &err) {
  Mesh &M = h->mesh;
  NdSystem &S = h->nd.sys[mode];
  cudaStream_t st = h->stream;
  NdPlan P;
  if (nd_plan(mode, h->sm_count, rp, ci, X, bon, P)) return 0;
  const int n = P.n, nf = P.nfront;
  S.n = n; S.nlev = P.nlev; S.grid = P.grid; S.entries = P.entries; S.nu = P.nu;
  P.prow.resize(n + 1, 0);
  auto up = [&](auto &dst, const auto &v) {
    if (dst.alloc(std::max<size_t>(v.size(), 1)) != cudaSuccess) return false;
    return v.empty() || cudaMemcpyAsync(dst.p, v.data(), v.size() * sizeof(v[0]), cudaMemcpyHostToDevice, st) == cudaSuccess;
  };
  // numeric factorisation, deepest level first: where each front's matrix and
  // panel rows lie within its level's buffers
  std::vector<long long> foff(nf), eoff(nf);
  long long emax = 0, lmax = 0;
  int nfmax = 0;
  for (int d = 0; d < P.nlev; ++d) {
    long long o = 0, e = 0;
    for (int f = P.first[d]; f < P.first[d + 1]; ++f) {
      foff[f] = o;
      eoff[f] = e;
      o += (long long)P.fr[f].s * P.fr[f].s;
      e += P.fr[f].s;
    }
    emax = std::max(emax, e);
    lmax = std::max(lmax, o);
    nfmax = std::max(nfmax, P.first[d + 1] - P.first[d]);
  }
  DevBuf<int> dchild;
  DevBuf<long long> dfoff, deoff;
  DevBuf<double> F[2], C, E, Dn;
  std::vector<int32_t> perm(P.pos);   // of every node its position (or -1), then of every position its node
  perm.insert(perm.end(), P.perm.begin(), P.perm.end());
  if (!up(S.front, P.fr) || !up(S.bnd, P.bnd) || !up(S.map, P.map) || !up(S.perm, perm) || !up(S.prow, P.prow) ||
      !up(S.task, P.task) || !up(S.phase, P.phase) || !up(dchild, P.child) ||
      !up(dfoff, foff) || !up(deoff, eoff) || S.pcol.alloc(P.prow[n]) || S.pK.alloc(P.prow[n]) ||
      S.f64.alloc((size_t)P.entries) || (f32 && S.f32.alloc((size_t)P.entries)) || F[0].alloc(lmax) ||
      F[1].alloc(P.nlev > 1 ? lmax : 0) || C.alloc(emax * kNdPanel) || E.alloc(emax * kNdPanel) ||
      Dn.alloc((size_t)nfmax * kNdPanel * kNdPanel)) {
    cudaGetLastError();
    cudaStreamSynchronize(st);
    S.release();
    return 0;   // no room: the CG needs less
  }
  if (n > 0)
    k_nd_rows<<<nblk(n, 256), 256, 0, st>>>(n, S.perm.p + M.N, S.perm, M.row_ptr, M.col_idx, M.K, S.prow, S.pcol, S.pK);
  constexpr int kGridYZ = 32768;   // fronts per launch (grid.y and grid.z end at 65,535)
  for (int d = P.nlev - 1; d >= 0; --d) {
    const int f0 = P.first[d], nl = P.first[d + 1] - f0;
    int smax = 0, kmax = 0;
    for (int f = f0; f < f0 + nl; ++f) { smax = std::max(smax, P.fr[f].s); kmax = std::max(kmax, P.fr[f].k); }
    if (smax == 0) continue;
    double *cur = F[d & 1], *prev = F[(d + 1) & 1];
    const int tiles = (smax + 63) / 64;
    for (int y0 = 0; y0 < nl; y0 += kGridYZ) {
      const int ny = std::min(kGridYZ, nl - y0);
      k_nd_assemble<<<dim3(std::min(256, nblk((long long)smax * smax, 256)), ny), 256, 0, st>>>(
          S.front, f0 + y0, S.map, dfoff, prev, dchild, cur);
      if (kmax > 0)
        k_nd_entries<<<dim3(nblk(kmax, 128), ny), 128, 0, st>>>(S.front, f0 + y0, dfoff, S.prow, S.pcol, S.pK, S.bnd,
                                                               cur);
      if (d == 0 && mode == 0) k_nd_regularise<<<1, 1024, 0, st>>>(P.fr[0].k, cur);
      for (int p0 = 0; p0 < kmax; p0 += kNdPanel) {
        k_nd_panel<<<dim3(tiles, ny), 256, 0, st>>>(S.front, f0 + y0, p0, dfoff, deoff, cur, C, E, Dn);
        k_nd_update<<<dim3(tiles, tiles, ny), 256, 0, st>>>(S.front, f0 + y0, p0, dfoff, deoff, cur, C, E, Dn);
      }
      if (kmax > 0)
        k_nd_store<<<dim3(std::min(256, nblk(2LL * kmax * smax, 256)), ny), 256, 0, st>>>(S.front, f0 + y0, dfoff,
                                                                                          cur, S.f64);
    }
  }
  if (f32 && n > 0) k_nd_f32<<<h->sm_count * 4, 256, 0, st>>>(P.entries, S.f64, S.f32);
  NMG_CUDA_TRY(cudaGetLastError(), "nested dissection");
  NMG_CUDA_TRY(cudaStreamSynchronize(st), "nested dissection");   // the host arrays and temporaries are in use until here
  S.ready = true;
  return 0;
}

bool nd_available(const nmg_handle *h, int mode, bool fp32) {
  const NdSystem &S = h->nd.sys[mode];
  return S.ready && (S.n == 0 || (fp32 ? S.f32.p != nullptr : S.f64.p != nullptr));   // (n = 0: nothing but the boundary)
}

// with64: FP64 factors stay beside (or in place of) the FP32 ones.
static int nd_setup(nmg_handle *h, bool with64, std::string &err) {
  Mesh &M = h->mesh;
  Workspace &W = h->ws;
  NdSolver &D = h->nd;
  const int N = M.N;
  std::vector<int32_t> rp(N + 1), ci(M.nnz), bon(N);
  std::vector<double> X(3 * (size_t)N);
  cudaStream_t st = h->stream;
  NMG_CUDA_TRY(cudaMemcpyAsync(rp.data(), M.row_ptr.p, sizeof(int32_t) * (N + 1), cudaMemcpyDeviceToHost, st), "d2h");
  NMG_CUDA_TRY(cudaMemcpyAsync(ci.data(), M.col_idx.p, sizeof(int32_t) * M.nnz, cudaMemcpyDeviceToHost, st), "d2h");
  NMG_CUDA_TRY(cudaMemcpyAsync(X.data(), M.coords.p, sizeof(double) * 3 * N, cudaMemcpyDeviceToHost, st), "d2h");
  NMG_CUDA_TRY(cudaMemcpyAsync(bon.data(), M.b_of_node.p, sizeof(int32_t) * N, cudaMemcpyDeviceToHost, st), "d2h");
  NMG_CUDA_TRY(cudaStreamSynchronize(st), "direct solver setup");
  for (int mode = 0; mode < 2; ++mode)
    if (int rc = nd_build(h, mode, rp, ci, X, bon, h->mixed_cg(), err)) return rc;
  if (!D.sys[0].ready && !D.sys[1].ready) return 0;
  const int MB = nd_members(std::min(h->nrep, kChunk));
  const long long nu = std::max(D.sys[0].nu, D.sys[1].nu);
  DevBuf<double> pb, px;   // the probes, and counters and error word of their own
  DevBuf<int> iters, errw;
  if (D.u.alloc(std::max<size_t>((size_t)nu * MB, 1)) || D.d.alloc((size_t)N * MB) || D.xw.alloc((size_t)N * MB) ||
      D.r.alloc((size_t)N * MB) || D.part.alloc(2 * 2 * (size_t)kChunk * h->sm_count) || D.bar.alloc(2) ||
      pb.alloc(N) || px.alloc(N) || iters.alloc(4) || errw.alloc(1)) {
    cudaGetLastError();   // no room: the CG needs less
    D.release();
    return 0;
  }
  NMG_CUDA_TRY(cudaMemsetAsync(D.bar.p, 0, 2 * sizeof(unsigned), st), "memset");
  NMG_CUDA_TRY(cudaMemsetAsync(iters.p, 0, 4 * sizeof(int), st), "memset");
  NMG_CUDA_TRY(cudaMemsetAsync(errw.p, 0, sizeof(int), st), "memset");
  for (int nm : {1, 2, 4, 8}) {
    cudaFuncSetAttribute(nd_kernel<double>(nm), cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)nd_smem(nm, sizeof(double)));
    cudaFuncSetAttribute(nd_kernel<float>(nm), cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)nd_smem(nm, sizeof(float)));
  }
  cudaGetLastError();
  W.iters.swap(iters);
  W.err.swap(errw);
  double mn[3] = {1e300, 1e300, 1e300}, mx[3] = {-1e300, -1e300, -1e300};
  for (int i = 0; i < N; ++i)
    for (int d = 0; d < 3; ++d) {
      mn[d] = std::min(mn[d], X[3 * (size_t)i + d]);
      mx[d] = std::max(mx[d], X[3 * (size_t)i + d]);
    }
  int axis = 0;
  for (int d = 1; d < 3; ++d)
    if (mx[d] - mn[d] > mx[axis] - mn[axis]) axis = d;
  auto probe = [&](int kind) {
    k_nd_probe<<<nblk(N, 256), 256, 0, st>>>(N, pb, kind, M.coords, axis, 0.5 * (mn[axis] + mx[axis]));
  };
  int rc = 0;
  if (D.sys[0].ready) {   // the Neumann sweeps' answer to b = 1, and K times it
    NdSystem &S = D.sys[0];
    DevBuf<double> w;
    rc = w.alloc(N) || S.kone.alloc(N) ? 100 : 0;
    if (!rc) {
      probe(kProbeOne);
      rc = nd_solve(h, 0, 1, pb, px, 1e-9, 1e-50, false);
    }
    if (!rc) {
      k_nd_one<<<nblk(N, 256), 256, 0, st>>>(N, S.prow, S.pcol, S.pK, D.xw, w, S.kone);
      rc = cudaStreamSynchronize(st) == cudaSuccess ? 0 : 100;
      S.one.swap(w);
    }
  }
  // a system whose factor does not solve the probes to the handle's tolerance,
  // in fewer passes than a solve may take, stays with the CG
  for (int kind = kProbeHash; kind < kProbes && !rc; ++kind) {
    probe(kind);
    for (int mode = 0; mode < 2 && !rc; ++mode)
      for (int f32 = 0; f32 < (h->mixed_cg() ? 2 : 1) && D.sys[mode].ready; ++f32) {
        int flag = 0, passes[2] = {0, 0};
        rc = nd_solve(h, mode, 1, pb, px, std::min(1e-9, mode ? h->opt.dbc_rtol : h->opt.nbc_rtol), 1e-50, f32 == 1,
                      NdOut(), true);
        if (!rc && (cudaMemcpyAsync(&flag, W.err.p, sizeof(int), cudaMemcpyDeviceToHost, st) ||
                    cudaMemcpyAsync(passes, W.iters.p, sizeof(passes), cudaMemcpyDeviceToHost, st) ||
                    cudaStreamSynchronize(st)))
          rc = 100;
        if (rc || flag || passes[mode] > kNdProbePass) {
          D.sys[mode].release();
          cudaMemsetAsync(W.err.p, 0, sizeof(int), st);
          nd_reset_barrier(h);
        }
      }
  }
  W.iters.swap(iters);
  W.err.swap(errw);
  if (rc || cudaGetLastError() != cudaSuccess || cudaStreamSynchronize(st) != cudaSuccess) {
    err = "direct Poisson solver: setup failed";
    return 100;
  }
  if (!with64)
    for (NdSystem &s : D.sys) s.f64.release();
  if (!D.sys[0].ready && !D.sys[1].ready) D.release();
  return 0;
}

// Iteration caps are the CG's: a caller that sets a small one, or chooses a
// form of the CG's preconditioner, gets the CG.
static bool nd_applies(const nmg_handle *h) {
  const nmg_options &o = h->opt;
  return o.do_demag && h->mesh.nb > 0 && !o.cg_no_coarse && o.cg_local_sweeps <= 1 && o.nbc_maxits >= kNdMinMaxits &&
         o.dbc_maxits >= kNdMinMaxits;
}

int nd_prepare(nmg_handle *h, bool adjoint) {
  if (h->pot) return nd_prepare(h->pot, adjoint);   // several materials: the potential mesh's solves
  NdSolver &D = h->nd;
  const nmg_options &o = h->opt;
  // who solves in FP64; the other handles keep the FP32 factors alone
  const bool with64 = D.with64 || o.cg_precision != 1 || (adjoint && o.adjoint_cg_precision != 1);
  if (D.tried && with64 == D.with64) return 0;
  const bool again = D.tried && (D.sys[0].ready || D.sys[1].ready);
  if (!nd_applies(h) || (D.tried && !again)) {
    D.tried = true;
    D.with64 = with64;
    return 0;
  }
  D.release();
  D.tried = true;
  D.with64 = with64;
  std::string err;
  if (nd_setup(h, with64, err)) {
    // refused by the device: nothing is kept, and the CG answers, if the device still does
    D.release();
    cudaGetLastError();
    if (cudaStreamSynchronize(h->stream) != cudaSuccess) {
      h->last_error = err;
      return 100;
    }
  }
  return 0;
}

// Seconds of an iteration of the CG: grid barriers, which take longer with more
// blocks, and a little for the nodes.  A fit (us measured, formula): 60 nodes 8.0
// (8.2), 1,331 8.6 (8.9), slab of 11,163 10.9 (10.7), film of 30,753 12.7 (12.6),
// cubes of 17,576 9.7 (11.4), 68,921 12.8 (14.8) and 132,651 19.4 (17.5).
static double nd_iteration(const nmg_handle *h) { return 8e-6 + 2.6e-8 * std::sqrt((double)h->mesh.N); }

// Seconds of nd_prepare, a fit to measured ones (ms, this formula in brackets):
// 60 nodes 0.7 (1.2), 343 2.4 (2.1), 1,331 5.9 (5.9), slab of 11,163 14.5 (13.8),
// box of 11,193 23 (23), film of 30,753 24 (29), cubes of 17,576 39 (36), 68,921
// 158 (161) and 132,651 427 (382).  Thin meshes have small separators.
static double nd_cost(const nmg_handle *h) {
  const double N = h->mesh.N, in = N - h->mesh.nb;
  return 1e-3 + 2.5e-6 * std::min(N, 2000.0) + 2e-6 * (N - 0.95 * h->mesh.nb) + 1e-11 * in * in;
}

int nd_note(nmg_handle *h) {
  NdSolver &D = h->nd;
  if (++D.evals < kNdEvals || D.tried) return 0;
  if (!nd_applies(h)) return nd_prepare(h);
  int total[2] = {0, 0};
  if (cudaMemcpyAsync(total, h->ws.iters.p + 2, sizeof(total), cudaMemcpyDeviceToHost, h->stream) ||
      cudaStreamSynchronize(h->stream)) {
    h->last_error = "direct Poisson solver: reading the iteration counts failed";
    return 100;
  }
  const double spent = ((double)total[0] + total[1]) * nd_iteration(h);
  return spent + D.responses + D.certain >= kNdShare * nd_cost(h) ? nd_prepare(h) : 0;
}

int nd_response(nmg_handle *h) {
  if (h->pot) return nd_response(h->pot);
  NdSolver &D = h->nd;
  D.responses += 2 * kNdResponseIters * nd_iteration(h);
  return nd_note(h);
}

int nd_expect(nmg_handle *h, long long evals) {
  if (h->pot) return nd_expect(h->pot, evals);
  NdSolver &D = h->nd;
  D.certain = std::max(D.certain, (double)evals * kNdIters * nd_iteration(h));
  return !D.tried && nd_applies(h) && D.certain >= kNdShare * nd_cost(h) ? nd_prepare(h) : 0;
}

void nd_reset_barrier(nmg_handle *h) {
  if (h->nd.bar.p) cudaMemsetAsync(h->nd.bar.p, 0, 2 * sizeof(unsigned), h->stream);
}

int nd_solve(nmg_handle *h, int mode, int nm, const double *b, double *x, double rtol, double atol, bool fp32,
             const NdOut &out, bool probe) {
  NdSolver &D = h->nd;
  NdSystem &S = D.sys[mode];
  Workspace &W = h->ws;
  NdArgs a;
  a.N = h->mesh.N; a.n = S.n; a.nlev = S.nlev; a.mode = mode; a.nm = nm;
  a.front = S.front; a.phase = S.phase; a.task = S.task;
  a.bnd = S.bnd; a.map = S.map; a.perm = S.perm; a.prow = S.prow; a.pcol = S.pcol; a.b_of_node = h->mesh.b_of_node;
  a.pK = S.pK;
  a.fac = fp32 ? (const void *)S.f32.p : (const void *)S.f64.p;
  a.out = out; a.nbnd = h->mesh.nb;
  a.b = b; a.x = x; a.xw = D.xw; a.r = D.r; a.part = D.part; a.u = D.u.p; a.d = D.d.p;
  a.bar = D.bar; a.err = W.err; a.iters = W.iters;
  a.one = mode == 0 ? S.one.p : nullptr;
  a.kone = S.kone;
  a.rtol = rtol; a.atol = atol; a.probe = probe;
  void *args[] = {&a};
  const int mb = nd_members(nm);
  const void *fn = fp32 ? nd_kernel<float>(nm) : nd_kernel<double>(nm);
  NMG_PROF_BEGIN(h, 1 + mode);
  const cudaError_t e = cudaLaunchCooperativeKernel(fn, dim3(S.grid), dim3(kNdThreads), args,
                                                    nd_smem(mb, fp32 ? sizeof(float) : sizeof(double)), h->stream);
  NMG_PROF_END(h);
  ++h->launches;
  if (e != cudaSuccess) {
    h->last_error = std::string("direct Poisson solve: launch failed: ") + cudaGetErrorString(e);
    return 100;
  }
  return 0;
}

}  // namespace nmg
