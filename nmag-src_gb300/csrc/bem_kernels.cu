// bem_kernels.cu -- dense Lindholm double-layer BEM on the device.
//
// Replaces the reference's BEM fill: nas_partially_fill_bem_matrix_row_constrained
// (src/bem3d.ml:938-1047) driving caml_bem3d_raw_lindholm_block_pbc
// (src/bem3d_stubs.c:413-610) for every (surface triangle, observer row), then
// adding Omega_i/(4 pi) - 1 on the diagonal (bem3d.ml:1040-1043).
//
// The formula's parts that neighbouring triangles share are formed once: for a
// chunk of observers the distances to the boundary nodes, the logarithms of
// the surface edges, and every triangle's solid angle and distance from its
// plane; then one thread per (column, observer) adds the column's triangles in
// the reference's order, so every entry is accumulated in exactly that order
// with no atomics and written once.  A warp holds 32 observers of one node,
// edge, triangle or column, so geometry loads are uniform and every other
// access is coalesced.  The chunk is as large as keeps its arrays (8 bytes per
// observer and node, edge, and twice per triangle) in L2.
//
// Bound by the FP64 pipe: ~165 operations a pair, against ~350 with three
// logarithms, an arc cosine and three distances per triangle and one thread
// per observer row (which left the chip half idle below ~20,000 rows).  8,562
// x 17,120 pairs: 245 ms before, 30 now (angles 51 %, edges 27 %, columns 16 %,
// distances 6 %); the film's 8.8e8: a handle in 1,086 ms before, 280 now; the
// 30 nm cube's in 23, 2.4 now.  The expressions the angle's rounding depends on
// (it is the arc cosine of a number near 1) follow the reference's operation
// order; this file is compiled with --fmad=false, and fma() is written where it
// is wanted.
//
// The columns leave as a[c*nb + k] = B[k][c] (k = observer row); a tiled
// transpose then stores the matrix row-major with the row stride padded to a
// multiple of 8 (bem[k*ld + c]), the layout the matrix-vector product streams.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <numeric>
#include <type_traits>
#include <vector>

#include "nmg_internal.h"

namespace nmg {
namespace {

constexpr double kPi = 3.141592653589793;

// Per-triangle constants of the Lindholm formula (bem3d_stubs.c:466-525).
__global__ void k_tri_setup(int ntri, const int32_t *__restrict__ tri, const double *__restrict__ tri_normal,
                            const int32_t *__restrict__ node_of_b, const double *__restrict__ X,
                            TriGeo *__restrict__ geo) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= ntri) return;
  TriGeo g;
  double s[3][3], xi[3][3];
  g.ok = 0;
  g.maxgeo = 0.0;
  for (int k = 0; k < 3; ++k)
    for (int d = 0; d < 3; ++d) {
      g.p[k][d] = X[3 * (size_t)node_of_b[tri[3 * (size_t)t + k]] + d];
      double ax = fabs(g.p[k][d]);
      if (ax > g.maxgeo) g.maxgeo = ax;
    }
  for (int d = 0; d < 3; ++d) {
    s[0][d] = g.p[2][d] - g.p[1][d]; s[1][d] = g.p[0][d] - g.p[2][d]; s[2][d] = g.p[1][d] - g.p[0][d];
  }
  bool ok = true;
  for (int k = 0; k < 3; ++k) {
    g.s_l[k] = sqrt(s[k][0] * s[k][0] + s[k][1] * s[k][1] + s[k][2] * s[k][2]);
    if (g.s_l[k] == 0.0) { ok = false; g.s_l[k] = 1.0; }
    double inv = 1.0 / g.s_l[k];
    for (int d = 0; d < 3; ++d) xi[k][d] = s[k][d] * inv;
  }
  double z[3];
  z[0] = s[1][1] * s[2][2] - s[1][2] * s[2][1];
  z[1] = s[1][2] * s[2][0] - s[1][0] * s[2][2];
  z[2] = s[1][0] * s[2][1] - s[1][1] * s[2][0];
  double len = sqrt(z[0] * z[0] + z[1] * z[1] + z[2] * z[2]);
  if (len == 0.0) { ok = false; len = 1.0; }
  double area = 0.5 * len, inv = 1.0 / len;
  for (int d = 0; d < 3; ++d) g.zeta_v[d] = z[d] * inv;
  g.gam01 = xi[0][0] * xi[1][0] + xi[0][1] * xi[1][1] + xi[0][2] * xi[1][2];
  g.gam12 = xi[1][0] * xi[2][0] + xi[1][1] * xi[2][1] + xi[1][2] * xi[2][2];
  g.gam20 = xi[2][0] * xi[0][0] + xi[2][1] * xi[0][1] + xi[2][2] * xi[0][2];
  for (int k = 0; k < 3; ++k) {
    const double *zv = g.zeta_v;
    g.eta[k][0] = zv[1] * xi[k][2] - zv[2] * xi[k][1];
    g.eta[k][1] = zv[2] * xi[k][0] - zv[0] * xi[k][2];
    g.eta[k][2] = zv[0] * xi[k][1] - zv[1] * xi[k][0];
  }
  double f = 1.0 * (1.0 / (8.0 * kPi * area));
  const double *n = tri_normal + 3 * (size_t)t;
  if (g.zeta_v[0] * n[0] + g.zeta_v[1] * n[1] + g.zeta_v[2] * n[2] < 0.0) f = -f;
  g.factor = f;
  g.ok = ok ? 1 : 0;
  geo[t] = g;
}

// Running maximum of |observer coordinate| in row order: the reference's
// geo_eps = 1e-13 * max over the triangle and the observers visited so far
// within one block call (bem3d_stubs.c:531-533).
// One block: tiles of its threads, a shuffle scan in each.
__global__ void __launch_bounds__(1024) k_observer_prefix_max(int nb, const int32_t *__restrict__ node_of_b,
                                                              const double *__restrict__ X,
                                                              double *__restrict__ out) {
  __shared__ double wmax[32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  double run = 0.0;
  for (int base = 0; base < nb; base += blockDim.x) {
    const int k = base + threadIdx.x;
    double a = 0.0;
    if (k < nb) {
      const double *o = X + 3 * (size_t)node_of_b[k];
      for (int d = 0; d < 3; ++d) { const double v = fabs(o[d]); if (v > a) a = v; }
    }
    for (int s = 1; s < 32; s <<= 1) {
      const double v = __shfl_up_sync(0xffffffffu, a, s);
      if (lane >= s && v > a) a = v;
    }
    if (lane == 31) wmax[w] = a;
    __syncthreads();
    for (int q = 0; q < w; ++q) if (wmax[q] > a) a = wmax[q];
    if (run > a) a = run;
    if (k < nb) out[k] = a;
    for (int q = 0; q < (int)(blockDim.x >> 5); ++q) if (wmax[q] > run) run = wmax[q];
    __syncthreads();
  }
}

// What the sums need of a triangle's vertex v: eta_v and the triangle's height
// eta_v . (p_(v+1) - p_v), f s_v, and the direction cosines between edge v and
// the two after it.
struct VertexGeo {
  double eta[3], height, fs, ga, gb;
};
__global__ void k_vertex_geo(int ntri, const TriGeo *__restrict__ geo, VertexGeo *__restrict__ out) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= 3 * ntri) return;
  const TriGeo &g = geo[e / 3];
  const int v = e % 3, n = v == 2 ? 0 : v + 1;
  VertexGeo o;
  for (int d = 0; d < 3; ++d) o.eta[d] = g.eta[v][d];
  o.height = g.eta[v][0] * (g.p[n][0] - g.p[v][0]) + g.eta[v][1] * (g.p[n][1] - g.p[v][1]) +
             g.eta[v][2] * (g.p[n][2] - g.p[v][2]);
  o.fs = g.factor * g.s_l[v];
  o.ga = v == 0 ? g.gam01 : (v == 1 ? g.gam12 : g.gam20);   // edges v, v + 1
  o.gb = v == 0 ? g.gam20 : (v == 1 ? g.gam01 : g.gam12);   // edges v, v + 2
  out[e] = o;
}

// The observers [k0, k0 + kc) of a chunk; arrays are [item][kc].
struct FillArgs {
  int nb, ne, ntri, k0, kc;
  const int32_t *node_of_b, *tri, *edge, *tri_edge, *col_ptr, *col_tri;   // col_tri: 3 triangle + vertex, ascending
  const double *X, *edge_len, *obs_max, *solid_angle;
  const TriGeo *geo;
  const VertexGeo *vgeo;
  double *dist, *lg, *ang, *zeta, *bem;
  int *touch;   // set where an observer lies on an edge, or next to it
};
// The upper words of 28 and of infinity.  A logarithm of 28 or more: (a + b - s) / s
// below 1.4e-12, infinite or not a number.
constexpr unsigned k28 = 0x403c0000u, kInf = 0x7ff00000u;

// Distance of every boundary node from every observer of the chunk.
__global__ void __launch_bounds__(256) k_fill_dist(FillArgs a) {
  const int k = blockIdx.x * 32 + (threadIdx.x & 31), v = blockIdx.y * 8 + (threadIdx.x >> 5);
  if (k >= a.kc || v >= a.nb || a.k0 + k >= a.nb) return;
  const double *o = a.X + 3 * (size_t)a.node_of_b[a.k0 + k], *p = a.X + 3 * (size_t)a.node_of_b[v];
  const double r0 = p[0] - o[0], r1 = p[1] - o[1], r2 = p[2] - o[2];
  a.dist[(size_t)v * a.kc + k] = sqrt(r0 * r0 + r1 * r1 + r2 * r2);
}

// kExact in the next three: every entry as the reference's operation order
// rounds it, for matrices that are then rounded to 24 bits (the particle batch,
// whose adaptive steps one entry rounded the other way moves by 1e-6; the FP32
// and the split-BF16 forms, whose products it moves by 1e-7 in its row).

// log((a + b + s) / (a + b - s)) of every surface edge (length s, its ends at
// distances a and b): 2 artanh(s / (a + b)), by its series where the edge is
// far (the truncation is below 2^-58), by the logarithm where it is near.
template <bool kExact>
__global__ void __launch_bounds__(256) k_fill_edges(FillArgs a) {
  const int k = blockIdx.x * 32 + (threadIdx.x & 31), e = blockIdx.y * 8 + (threadIdx.x >> 5);
  if (k >= a.kc || e >= a.ne || a.k0 + k >= a.nb) return;
  const double da = a.dist[(size_t)a.edge[2 * e] * a.kc + k], db = a.dist[(size_t)a.edge[2 * e + 1] * a.kc + k];
  const double L = da + db;
  const double s = a.edge_len[e];
  double v;
  if (!kExact && 8.0 * s <= L) {
    const double x = s / L, y = x * x;
    double t = 1.0 / 17.0;
    t = fma(t, y, 1.0 / 15.0); t = fma(t, y, 1.0 / 13.0); t = fma(t, y, 1.0 / 11.0); t = fma(t, y, 1.0 / 9.0);
    t = fma(t, y, 1.0 / 7.0);  t = fma(t, y, 1.0 / 5.0);  t = fma(t, y, 1.0 / 3.0);
    v = 2.0 * fma(x * y, t, x);
  } else {
    v = log((L + s) / (L - s));
    if ((unsigned)__double2hiint(v) >= k28 && da != 0.0 && db != 0.0) *a.touch = 1;   // (not an end of the edge)
  }
  a.lg[(size_t)e * a.kc + k] = v;
}

// Signed solid angle and distance from the plane of every triangle; angle
// infinite: the triangle adds nothing (degenerate, the observer one of its
// vertices or in its plane, bem3d_stubs.c:531-600).  In the plane the reference
// adds 0 times the formula, which is not a number where the observer lies on an
// edge (a node on another part's edge): with kTouch such an entry stays NaN, to
// be noticed.  (Looking for it in every triangle of an observer's plane took 1 to
// 2 of the 57 ms of an 8,562-node handle; k_fill_edges tells which mesh needs it.)
template <bool kExact, bool kTouch>
__global__ void __launch_bounds__(256) k_fill_angles(FillArgs a) {
  const int k = blockIdx.x * 32 + (threadIdx.x & 31), t = blockIdx.y * 8 + (threadIdx.x >> 5);
  if (k >= a.kc || t >= a.ntri || a.k0 + k >= a.nb) return;
  const TriGeo &g = a.geo[t];
  const int32_t *tv = a.tri + 3 * (size_t)t;
  const double *o = a.X + 3 * (size_t)a.node_of_b[a.k0 + k];
  const double ox = o[0], oy = o[1], oz = o[2], omax = a.obs_max[a.k0 + k];
  double r[3][3], rl[3];
  for (int v = 0; v < 3; ++v) {
    r[v][0] = g.p[v][0] - ox; r[v][1] = g.p[v][1] - oy; r[v][2] = g.p[v][2] - oz;
    rl[v] = a.dist[(size_t)tv[v] * a.kc + k];
  }
  const double kNothing = HUGE_VAL;
  double angle = kNothing;
  const double zeta = g.zeta_v[0] * r[0][0] + g.zeta_v[1] * r[0][1] + g.zeta_v[2] * r[0][2];
  const double geo_eps = (g.maxgeo > omax ? g.maxgeo : omax) * 1e-13;
  const bool plane = fabs(zeta) < geo_eps;
  auto edge = [&](unsigned least) {   // on an edge or next to it: elsewhere in the plane the formula is finite
    const int32_t *te = a.tri_edge + 3 * (size_t)t;
    bool any = false;
#pragma unroll
    for (int v = 0; v < 3; ++v) any |= (unsigned)__double2hiint(a.lg[(size_t)te[v] * a.kc + k]) >= least;
    return any;
  };
  if (g.ok && !(rl[0] <= 0.0 || rl[1] <= 0.0 || rl[2] <= 0.0) && (!plane || (kTouch && edge(k28)))) {
    const double sp01 = r[0][0] * r[1][0] + r[0][1] * r[1][1] + r[0][2] * r[1][2];
    const double sp12 = r[1][0] * r[2][0] + r[1][1] * r[2][1] + r[1][2] * r[2][2];
    const double sp20 = r[2][0] * r[0][0] + r[2][1] * r[0][1] + r[2][2] * r[0][2];
    const double num = rl[0] * rl[1] * rl[2] + rl[0] * sp12 + rl[1] * sp20 + rl[2] * sp01;
    const double den = sqrt(2.0 * (rl[1] * rl[2] + sp12) * (rl[2] * rl[0] + sp20) * (rl[0] * rl[1] + sp01));
    if (den != 0.0) {
      double q = num / den;
      q = q < -1.0 ? -1.0 : (q > 1.0 ? 1.0 : q);
      const double y = 0.5 * (1.0 - q);   // exact for q >= 1/2
      if (!kExact && y < 0.0078125) {   // acos q = 2 asin sqrt y, the arc sine's series (truncation below 2^-58)
        double p = 143.0 / 10240.0;
        p = fma(p, y, 231.0 / 13312.0); p = fma(p, y, 63.0 / 2816.0); p = fma(p, y, 35.0 / 1152.0);
        p = fma(p, y, 5.0 / 112.0);     p = fma(p, y, 3.0 / 40.0);    p = fma(p, y, 1.0 / 6.0);
        const double s = sqrt(y);
        angle = 4.0 * fma(s * y, p, s);
      } else {
        angle = 2.0 * acos(q);
      }
      if (zeta < 0.0) angle = -angle;
      if (kTouch && plane) angle = angle != angle || edge(kInf) ? nan("") : kNothing;
    }
  }
  a.ang[(size_t)t * a.kc + k] = angle;
  a.zeta[(size_t)t * a.kc + k] = zeta;
}

// Entry (observer, column): the column's triangles in order.
template <bool kExact>
__global__ void __launch_bounds__(256) k_fill_columns(FillArgs a) {
  const int k = blockIdx.x * 32 + (threadIdx.x & 31), c = blockIdx.y * 8 + (threadIdx.x >> 5);
  if (k >= a.kc || c >= a.nb || a.k0 + k >= a.nb) return;
  const double *o = a.X + 3 * (size_t)a.node_of_b[a.k0 + k];
  const double ox = o[0], oy = o[1], oz = o[2];
  const double *pc = a.X + 3 * (size_t)a.node_of_b[c];
  const double c0 = pc[0] - ox, c1 = pc[1] - oy, c2 = pc[2] - oz;
  double acc = 0.0;
  for (int q = a.col_ptr[c]; q < a.col_ptr[c + 1]; ++q) {
    const int e = a.col_tri[q], t = e / 3, v = e - 3 * t, n = v == 2 ? 0 : v + 1, m = n == 2 ? 0 : n + 1;
    const double angle = a.ang[(size_t)t * a.kc + k], zeta = a.zeta[(size_t)t * a.kc + k];
    if (isinf(angle)) continue;
    const VertexGeo &g = a.vgeo[e];
    const int32_t *te = a.tri_edge + 3 * (size_t)t;
    const double lv = a.lg[(size_t)te[v] * a.kc + k], ln = a.lg[(size_t)te[n] * a.kc + k],
                 lm = a.lg[(size_t)te[m] * a.kc + k];
    if (kExact) {   // the three products of a row of the direction cosines in the reference's order
      const double *p = a.X + 3 * (size_t)a.node_of_b[a.tri[3 * (size_t)t + n]];
      const double r0 = p[0] - ox, r1 = p[1] - oy, r2 = p[2] - oz;
      const double e0 = g.eta[0] * r0 + g.eta[1] * r1 + g.eta[2] * r2;
      const double gl = v == 0 ? lv + g.ga * ln + g.gb * lm : (v == 1 ? g.gb * lm + lv + g.ga * ln : g.ga * ln + g.gb * lm + lv);
      acc += g.fs * (angle * e0 - zeta * gl);
      continue;
    }
    const double gl = fma(g.gb, lm, fma(g.ga, ln, lv));
    // eta . (p_(v+1) - o), from differences of coordinates alone: with eta . p - eta . o
    // entries of an 18-unit box were off by 9e-14 of the largest at 1e4 from the origin, by 2e-12 at 4e5 (1e-15 so)
    const double en = fma(g.eta[0], c0, fma(g.eta[1], c1, fma(g.eta[2], c2, g.height)));
    acc = fma(g.fs, fma(angle, en, -(zeta * gl)), acc);
  }
  if (c == a.k0 + k) acc += a.solid_angle[c] / (4.0 * kPi) - 1.0;
  a.bem[(size_t)c * a.nb + a.k0 + k] = acc;
}

// Column-major fill buffer (a[c*nb + k]) -> row-major matrix with padded row
// stride ld (b[k*ld + c], pad columns zero), 32x32 tiles through shared memory.
__global__ void k_transpose_pad(int nb, int ld, const double *__restrict__ a, double *__restrict__ b) {
  __shared__ double tile[32][33];
  const int c0 = blockIdx.x * 32, k0 = blockIdx.y * 32;
  for (int j = threadIdx.y; j < 32; j += blockDim.y) {
    const int c = c0 + j, k = k0 + threadIdx.x;
    tile[j][threadIdx.x] = (c < nb && k < nb) ? a[(size_t)c * nb + k] : 0.0;
  }
  __syncthreads();
  for (int j = threadIdx.y; j < 32; j += blockDim.y) {
    const int k = k0 + j, c = c0 + threadIdx.x;
    if (k < nb && c < ld) b[(size_t)k * ld + c] = tile[threadIdx.x][j];
  }
}

// BF16 bits of the FP32 rounding residual B - fp32(B) (round to nearest even).
__global__ void k_split_lo(size_t n, const double *__restrict__ a, const float *__restrict__ hi,
                           uint16_t *__restrict__ lo) {
  size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (; i < n; i += stride) {
    const __nv_bfloat16 v = __float2bfloat16_rn((float)(a[i] - (double)hi[i]));
    lo[i] = *reinterpret_cast<const uint16_t *>(&v);
  }
}

// FP32 copy of the row-major matrix (same padded stride).
__global__ void k_to_f32(size_t n, const double *__restrict__ a, float *__restrict__ b) {
  size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (; i < n; i += stride) b[i] = (float)a[i];
}

// max |B| as float bits (non-negative floats order like their bit patterns).
__global__ void k_absmax_f32(long long n, const float *__restrict__ v, unsigned *__restrict__ out) {
  unsigned m = 0u;
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x)
    m = max(m, __float_as_uint(fabsf(v[k])));
  for (int o = 16; o; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0 && m) atomicMax(out, m);
}

// FP16 copy of B (times scale) in the A-operand fragment order of
// mma.m16n8k16 (row-major): tile (rb, kb) holds rows 16 rb .. +15 and
// columns 16 kb .. +15 as 32 lanes x 8 halves; lane 4 g + t carries
// (g, 2t), (g, 2t+1), (g+8, 2t), (g+8, 2t+1), (g, 2t+8), (g, 2t+9),
// (g+8, 2t+8), (g+8, 2t+9) -- the PTX fragment elements a0..a7 -- so one
// 16-byte load per lane fills the operand.  Entries beyond nb are 0.
__global__ void k_pack_bem16f(int nb, int ld, int KT, long long ntiles, const float *__restrict__ B32, float scale,
                              uint4 *__restrict__ out) {
  const long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (g >= ntiles * 32) return;
  const long long tile = g >> 5;
  const int lane = (int)(g & 31);
  const int rb = (int)(tile / KT), kb = (int)(tile - (long long)rb * KT);
  const int gq = lane >> 2, t = lane & 3;
  unsigned w[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    float v[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int i = 2 * j + h;
      const int r = 16 * rb + gq + ((i & 2) ? 8 : 0);
      const int c = 16 * kb + 2 * t + (i & 1) + (i >= 4 ? 8 : 0);
      v[h] = (r < nb && c < nb) ? B32[(size_t)r * ld + c] * scale : 0.f;
    }
    const __half2 p = __floats2half2_rn(v[0], v[1]);   // v[0] in the low half
    memcpy(&w[j], &p, sizeof(unsigned));
  }
  out[g] = make_uint4(w[0], w[1], w[2], w[3]);
}

}  // namespace

int fill_bem(nmg_handle *h, std::string &err, bool exact) {
  Mesh &M = h->mesh;
  cudaStream_t s = h->stream;
  if (M.nb == 0) return 0;
  exact = exact || h->opt.bem_precision == 1 || h->opt.bem_precision == 3;
  const size_t nb = M.nb;
  if (M.ld != (M.nb + 7) / 8 * 8) {
    err = "BEM row stride not set up by the workspace";
    return 3;
  }
  NMG_CUDA_TRY(M.trigeo.alloc(M.ntri), "alloc trigeo");
  NMG_CUDA_TRY(M.obs_max.alloc(M.nb), "alloc obs_max");
  {
    // The fill accumulates column-major (coalesced, reference order) into a
    // temporary; one tiled transpose then gives the row-major product layout.
    DevBuf<double> colmajor;
    NMG_CUDA_TRY(colmajor.alloc(nb * nb), "alloc BEM fill buffer (nb^2 doubles)");
    k_tri_setup<<<(M.ntri + 127) / 128, 128, 0, s>>>(M.ntri, M.tri, M.tri_normal, M.node_of_b, M.coords, M.trigeo);
    k_observer_prefix_max<<<1, 1024, 0, s>>>(M.nb, M.node_of_b, M.coords, M.obs_max);
    // the surface's edges and every column's triangles
    const int nt = M.ntri;
    std::vector<int32_t> tri(3 * (size_t)nt);
    std::vector<TriGeo> geo(nt);
    NMG_CUDA_TRY(cudaMemcpyAsync(tri.data(), M.tri.p, sizeof(int32_t) * tri.size(), cudaMemcpyDeviceToHost, s), "d2h");
    NMG_CUDA_TRY(cudaMemcpyAsync(geo.data(), M.trigeo.p, sizeof(TriGeo) * nt, cudaMemcpyDeviceToHost, s), "d2h");
    NMG_CUDA_TRY(cudaStreamSynchronize(s), "surface triangles");
    std::vector<std::pair<uint64_t, int32_t>> key(3 * (size_t)nt);
    for (int t = 0; t < nt; ++t)
      for (int v = 0; v < 3; ++v) {   // edge v faces vertex v
        const uint64_t x = tri[3 * (size_t)t + (v + 1) % 3], y = tri[3 * (size_t)t + (v + 2) % 3];
        key[3 * (size_t)t + v] = {std::min(x, y) << 32 | std::max(x, y), 3 * t + v};
      }
    std::sort(key.begin(), key.end());
    std::vector<int32_t> edge, tri_edge(3 * (size_t)nt), col_ptr(nb + 1, 0), col_tri(3 * (size_t)nt);
    std::vector<double> edge_len;
    for (size_t q = 0; q < key.size(); ++q) {
      if (q == 0 || key[q].first != key[q - 1].first) {
        edge.push_back((int32_t)(key[q].first >> 32));
        edge.push_back((int32_t)(key[q].first & 0xffffffffu));
        edge_len.push_back(geo[key[q].second / 3].s_l[key[q].second % 3]);   // the same from either side, bit for bit
      }
      tri_edge[key[q].second] = (int32_t)edge_len.size() - 1;
    }
    for (int32_t c : tri) ++col_ptr[c + 1];
    std::partial_sum(col_ptr.begin(), col_ptr.end(), col_ptr.begin());
    {
      std::vector<int32_t> at(col_ptr.begin(), col_ptr.end() - 1);
      for (int32_t e = 0; e < 3 * nt; ++e) col_tri[at[tri[e]]++] = e;
    }
    const int ne = (int)edge_len.size();
    const size_t per = nb + ne + 2 * (size_t)nt;   // doubles per observer of a chunk
    int kc = (int)std::min<size_t>((nb + 31) / 32 * 32, std::max<size_t>(32, (72u << 20) / (8 * per) / 32 * 32));
    DevBuf<int32_t> dedge, dte, dcp, dct;
    DevBuf<double> dlen, work;
    DevBuf<VertexGeo> vg;
    NMG_CUDA_TRY(dedge.alloc(std::max<size_t>(edge.size(), 1)), "alloc");
    NMG_CUDA_TRY(dte.alloc(std::max<size_t>(tri_edge.size(), 1)), "alloc");
    NMG_CUDA_TRY(dcp.alloc(nb + 1), "alloc");
    NMG_CUDA_TRY(dct.alloc(std::max<size_t>(col_tri.size(), 1)), "alloc");
    NMG_CUDA_TRY(dlen.alloc(std::max(ne, 1)), "alloc");
    NMG_CUDA_TRY(vg.alloc(std::max(3 * (size_t)nt, (size_t)1)), "alloc");
    NMG_CUDA_TRY(work.alloc(per * kc), "alloc BEM fill chunk");
    NMG_CUDA_TRY(cudaMemcpyAsync(dedge.p, edge.data(), sizeof(int32_t) * edge.size(), cudaMemcpyHostToDevice, s), "h2d");
    NMG_CUDA_TRY(cudaMemcpyAsync(dte.p, tri_edge.data(), sizeof(int32_t) * tri_edge.size(), cudaMemcpyHostToDevice, s), "h2d");
    NMG_CUDA_TRY(cudaMemcpyAsync(dcp.p, col_ptr.data(), sizeof(int32_t) * (nb + 1), cudaMemcpyHostToDevice, s), "h2d");
    NMG_CUDA_TRY(cudaMemcpyAsync(dct.p, col_tri.data(), sizeof(int32_t) * col_tri.size(), cudaMemcpyHostToDevice, s), "h2d");
    NMG_CUDA_TRY(cudaMemcpyAsync(dlen.p, edge_len.data(), sizeof(double) * ne, cudaMemcpyHostToDevice, s), "h2d");
    if (nt > 0) k_vertex_geo<<<(3 * nt + 127) / 128, 128, 0, s>>>(nt, M.trigeo, vg);
    FillArgs a;
    a.nb = M.nb; a.ne = ne; a.ntri = nt; a.kc = kc;
    a.node_of_b = M.node_of_b; a.tri = M.tri; a.edge = dedge; a.tri_edge = dte; a.col_ptr = dcp; a.col_tri = dct;
    a.X = M.coords; a.edge_len = dlen; a.obs_max = M.obs_max; a.solid_angle = M.solid_angle;
    a.geo = M.trigeo; a.vgeo = vg;
    a.dist = work; a.lg = a.dist + nb * kc; a.ang = a.lg + (size_t)ne * kc; a.zeta = a.ang + (size_t)nt * kc;
    a.bem = colmajor;
    // grid.y ends at 65,535: eight items a block
    if ((std::max<size_t>(std::max<size_t>(nb, ne), nt) + 7) / 8 > 65535) {
      err = "BEM fill: surface too large (more than 524,280 nodes, edges or triangles)";
      return 3;
    }
    DevBuf<int> touch;
    NMG_CUDA_TRY(touch.alloc(1), "alloc");
    NMG_CUDA_TRY(cudaMemsetAsync(touch.p, 0, sizeof(int), s), "memset");
    a.touch = touch;
    auto fill = [&](auto ex, auto touching) {
      constexpr bool kExact = decltype(ex)::value, kTouch = decltype(touching)::value;
      for (a.k0 = 0; a.k0 < M.nb; a.k0 += kc) {
        const unsigned gx = (unsigned)((std::min(kc, M.nb - a.k0) + 31) / 32);
        const dim3 ge(gx, (ne + 7) / 8), gt(gx, (nt + 7) / 8), gc(gx, (M.nb + 7) / 8);
        k_fill_dist<<<gc, 256, 0, s>>>(a);
        if (ne > 0) k_fill_edges<kExact><<<ge, 256, 0, s>>>(a);
        if (nt > 0) k_fill_angles<kExact, kTouch><<<gt, 256, 0, s>>>(a);
        k_fill_columns<kExact><<<gc, 256, 0, s>>>(a);
      }
    };
    if (exact) fill(std::true_type(), std::false_type());
    else fill(std::false_type(), std::false_type());
    int touching = 0;   // parts that touch with unlike cells, which is rare: once more, looking at edges
    NMG_CUDA_TRY(cudaMemcpyAsync(&touching, touch.p, sizeof(int), cudaMemcpyDeviceToHost, s), "d2h");
    NMG_CUDA_TRY(cudaStreamSynchronize(s), "bem fill");
    if (touching) {
      if (exact) fill(std::true_type(), std::true_type());
      else fill(std::false_type(), std::true_type());
    }
    NMG_CUDA_TRY(cudaGetLastError(), "bem fill launch");
    NMG_CUDA_TRY(M.bem.alloc(nb * M.ld), "alloc BEM (nb x ld doubles)");
    dim3 tb(32, 8), tg((M.ld + 31) / 32, (M.nb + 31) / 32);
    k_transpose_pad<<<tg, tb, 0, s>>>(M.nb, M.ld, colmajor, M.bem);
    NMG_CUDA_TRY(cudaGetLastError(), "bem transpose launch");
    NMG_CUDA_TRY(cudaStreamSynchronize(s), "bem fill");
  }
  if (h->opt.bem_precision == 3) {   // tensor-core product: BF16 planes of the FP64 matrix
    if (int rc = bem_tc_setup(h, err)) return rc;
  }
  if (h->opt.bem_precision == 1 || h->opt.bem_precision == 2) {
    NMG_CUDA_TRY(M.bem32.alloc(nb * M.ld), "alloc FP32 BEM");
    k_to_f32<<<h->sm_count * 8, 256, 0, s>>>(nb * M.ld, M.bem, M.bem32);
  }
  if (h->opt.bem_precision == 2) {
    NMG_CUDA_TRY(M.bem16lo.alloc(nb * M.ld), "alloc BEM residual (BF16)");
    k_split_lo<<<h->sm_count * 8, 256, 0, s>>>(nb * M.ld, M.bem, M.bem32, M.bem16lo);
  }
  if (h->opt.bem_precision == 2 && h->opt.bem_anchor_tol > 0.0 && h->nrep > 1 && h->opt.anchor_product == 1) {
    // FP16 fragment copy for the anchored ensemble product, scaled by a power
    // of two that puts max|B| in [2^13, 2^14) (FP16 normal range for the rest)
    DevBuf<unsigned> amax;
    NMG_CUDA_TRY(amax.alloc(1), "alloc");
    NMG_CUDA_TRY(cudaMemsetAsync(amax.p, 0, sizeof(unsigned), s), "zero");
    k_absmax_f32<<<h->sm_count * 4, 256, 0, s>>>((long long)nb * M.ld, M.bem32, amax);
    unsigned bits = 0;
    NMG_CUDA_TRY(cudaMemcpyAsync(&bits, amax.p, sizeof(unsigned), cudaMemcpyDeviceToHost, s), "copy");
    NMG_CUDA_TRY(cudaStreamSynchronize(s), "absmax");
    float mx;
    std::memcpy(&mx, &bits, sizeof(float));
    int e = 0;
    if (mx > 0.f && std::isfinite(mx)) std::frexp(mx, &e);
    M.h16_scale = std::ldexp(1.f, 14 - e);
    M.h16_kt = (nb + 15) / 16;
    const long long ntiles = (long long)M.h16_kt * M.h16_kt;   // row blocks = column tiles
    NMG_CUDA_TRY(M.bem16f.alloc((size_t)ntiles * 256), "alloc FP16 fragment BEM");
    k_pack_bem16f<<<(unsigned)((ntiles * 32 + 255) / 256), 256, 0, s>>>(
        nb, M.ld, M.h16_kt, ntiles, M.bem32, M.h16_scale, reinterpret_cast<uint4 *>(M.bem16f.p));
    NMG_CUDA_TRY(cudaGetLastError(), "pack FP16 fragment BEM");
  }
  NMG_CUDA_TRY(cudaStreamSynchronize(s), "bem fill");
  return 0;
}

}  // namespace nmg
