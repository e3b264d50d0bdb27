// Static integrals of tetrahedron pairs sharing 2, 3 or 4 vertices (the
// singular near-field pairs), computed once per geometry as 24 moments per
// ordered pair:
//   per kernel K in {1/(4 pi r), 1/(4 pi), r/(8 pi)}:
//     int K,  int K (x - o),  int K (y - o),  int K (x - o).(y - o)
// in the unit-simplex measure, o = the first common vertex.
//
// The reference integrates these pairs with its generalised Taylor-Duffy code
// and an adaptive cubature at relative tolerance 1e-6 (TTaylorDuffy.cc:284-343,
// tolerance set at SWGGeometry.cc:46-47; called from GMatrixElements.cc:174-263,
// 343-353).  Here the rule is a relative-coordinate polar rule: barycentrics
// lambda (row tetrahedron A) and mu (column tetrahedron B), common vertices
// first; d = (lambda_k - mu_k | lambda_A-own | -mu_B-own) makes x - y linear
// and homogeneous in d; the admissible d form the polytope {sum d = 0,
// |d|_1 <= 2} whose faces away from the origin are Delta_{p-1} x Delta_{q-1},
// one per sign pattern S of the common components.  With d = rho zeta the
// remaining common barycentrics span a (c-1)-simplex of size 1 - rho and
//   dlambda dmu = rho^{m-1} (1 - rho)^{c-1} drho dzeta dt,  m = 7 - c,
// so the t- and rho-integrals are closed-form Beta integrals and only the
// 6 - c angular dimensions of each face cube [0,1]^{6-c} need a rule.
//
// Two stages:
//  * k_sing_fixed, one CTA per pair: collapsed Gauss-Legendre product rules
//    of orders n and n + 2 over every face cube.  Where all 24 moments of the
//    two orders agree to flag_tol of their scale (|M0|, |M0| h, |M0| h^2 for
//    the zeroth, first and second moments of each kernel, h = diameter of A)
//    the order n + 2 values are final; otherwise the pair is queued.
//  * refinement (k_sgr_*): each face cube of a queued pair is refined level by
//    level, all pairs of a batch together.  Every open box is halved along
//    each of its dimensions in turn (a 6^{6-c}-point rule per half); the split
//    that changes the box value most is taken; the box closes when that change
//    is within tol of the scale (its two halves are kept) or stays open as two
//    boxes for the next level.  At most SG_MAXBOX boxes of a pair are open per
//    level and SG_MAXLEVEL levels are run; a box that cannot be opened for lack
//    of room, or is still open after the last level, keeps its halves and sets
//    bit 0 / bit 1 of the pair's status (never silently: the bits are OR-ed
//    into the geometry's status word, bg_geometry_singular_stats).
// Points are not evaluated one by one: along the last dimension of the rule
// only one of the two points moves, on a straight line, so a thread takes one
// line of n points, R = Q + u D, and keeps four sums on it (1/R, u/R, R, u R);
// the eight raw sums per kernel power follow from them once per line.  About
// 45 instructions a point in place of 350 (barycentrics, table look-ups and 24
// accumulations per point).  FP64-pipe bound.
// With the fixed rule only (bg_geometry_set_singular_refine off) the order n
// values are kept for every pair, as before refinement existed.
//
// Every sum has a fixed order (thread-strided points, fixed shuffle trees,
// boxes closed in level and box order), so results are deterministic.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "devmath.cuh"
#include "internal.h"

namespace bg {

#define SG_THREADS 256
#define SG_NG 6            // Gauss points per dimension of a refinement box
#define SG_MAXBOX 2048     // boxes open per level, at most (per pair)
#define SG_MAXLEVEL 40
#define SG_REC 34          // doubles per box record: lo[4], hi[4], val[24], S, pair slot
#define SG_RES 48          // doubles per evaluated box: the two halves of the split taken

// Gauss-Legendre rules on [0,1]: row n holds the n-point rule (n <= 16)
__constant__ double c_sgx[17][16], c_sgw[17][16];
static bool s_sg_tables = false;

static int sg_tables() {
  if (s_sg_tables) return BG_OK;
  static double x[17][16], w[17][16];
  for (int n = 1; n <= 16; n++) gauss_legendre01(n, x[n], w[n]);
  BG_CUDA_TRY(cudaMemcpyToSymbol(c_sgx, x, sizeof x));
  BG_CUDA_TRY(cudaMemcpyToSymbol(c_sgw, w, sizeof w));
  BG_CUDA_TRY(uploads_done());
  s_sg_tables = true;
  return BG_OK;
}

// per-pair data: vertices relative to the first common vertex, the closed-form
// moments of the common simplex (ub, W) and the Beta factors G
struct SgPair {
  double VA[4][3], VB[4][3];
  double ub[3], W;
  double G[3][3];
  int c;
};

__device__ __forceinline__ double sg_fact(int n) {
  double r = 1.0;
  for (int i = 2; i <= n; i++) r *= i;
  return r;
}

__device__ void sg_setup(const DevGeom &g, int4 oa, int4 ob, int c, SgPair &X) {
  const int via[4] = {oa.x, oa.y, oa.z, oa.w}, vib[4] = {ob.x, ob.y, ob.z, ob.w};
  double o[3] = {g.V4[4 * (size_t)via[0]], g.V4[4 * (size_t)via[0] + 1], g.V4[4 * (size_t)via[0] + 2]};
  for (int i = 0; i < 4; i++)
    for (int k = 0; k < 3; k++) {
      X.VA[i][k] = g.V4[4 * (size_t)via[i] + k] - o[k];
      X.VB[i][k] = g.V4[4 * (size_t)vib[i] + k] - o[k];
    }
  c = c < 2 ? 2 : c > 4 ? 4 : c;   // two tetrahedra share at most 4 vertices
  X.c = c;
  int nn = c - 1, m = 7 - c;
  double s2 = 0, sv[3] = {0, 0, 0};
  for (int i = 0; i < c; i++)
    for (int k = 0; k < 3; k++) { sv[k] += X.VA[i][k]; s2 += X.VA[i][k] * X.VA[i][k]; }
  for (int k = 0; k < 3; k++) X.ub[k] = sv[k] / (nn + 1);
  X.W = (s2 + sv[0] * sv[0] + sv[1] * sv[1] + sv[2] * sv[2]) / ((nn + 1.0) * (nn + 2.0));
  for (int p = 0; p < 3; p++)
    for (int j = 0; j < 3; j++) {
      int a = m - 2 + p;   // m - 1 + (p - 1)
      X.G[p][j] = sg_fact(a + j) / sg_fact(a + j + nn + 1);
    }
}

__device__ __forceinline__ double sel4(const double *a, int i) {
  return i == 0 ? a[0] : i == 1 ? a[1] : i == 2 ? a[2] : a[3];
}

// Barycentrics of the collapsed map of u[0..k-1] (k <= 3) onto Delta_k with the
// Jacobian (1-u0)^{k-1} (1-u1)^{k-2} ...  With line set, the last coordinate is
// left open: the point is b + u (e_{k-1} - e_k) rest, u in [0, 1].
__device__ __forceinline__ double sg_collapse(int k, const double *u, double *b, bool line, double &rest) {
  double J = 1.0;
  rest = 1.0;
#pragma unroll
  for (int i = 0; i < 4; i++) b[i] = 0.0;
  const int kk = line ? k - 1 : k;
#pragma unroll
  for (int i = 0; i < 3; i++)
    if (i < kk) {
      b[i] = rest * u[i];
      rest *= 1.0 - u[i];
      if (i < k - 1) J *= rest;
    }
#pragma unroll
  for (int i = 0; i < 4; i++)
    if (i == k) b[i] = rest;
  return J;
}

// One line of the product rule on face S: the coordinates u[0..K-2] fixed
// (ka of the K collapsed coordinates map onto A's simplex, the others onto
// B's; A1, B1: the points of A and B relative to the first common vertex,
// which is the origin, so VA[0] = 0), the last one over the n Gauss points
// x of [lo, lo + h] with weights wx.  The 24 moments are linear in eight raw
// sums per kernel power R^p (p = -1, 0, 1): sum w R^p, sum w R^p A1,
// sum w R^p B1, sum w R^p A1.B1; sg_raw_to_moment applies the Beta factors and
// the common-simplex moments once per box.  w: weight of the fixed coordinates.
template <int C>
__device__ __forceinline__ void sg_line(const SgPair &X, int S, int ka, const double *u, double w, int n,
                                        const double *x, const double *wx, double lo, double h, double raw[24]) {
  constexpr int K = 6 - C;
  const int kb = K - ka;
  const bool varB = kb >= 1;
  double uA[3], uB[3];
#pragma unroll
  for (int e = 0; e < 3; e++) {
    uA[e] = e < K - 1 ? u[e < K - 1 ? e : 0] : 0.0;
    double v = 0.0;
#pragma unroll
    for (int d = 0; d < K - 1; d++)
      if (d - ka == e) v = u[d];
    uB[e] = v;
  }
  double al[4], be[4], ra, rb;
  w *= sg_collapse(ka, uA, al, !varB, ra);
  w *= sg_collapse(kb, uB, be, varB, rb);
  // vertices in order: common ones by the sign pattern, then the own ones
  const int kv = varB ? kb : ka;
  const double rest = varB ? rb : ra;
  double A1[3] = {0, 0, 0}, B1[3] = {0, 0, 0}, D[3] = {0, 0, 0};
  int ja = 0, jb = 0;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const bool onA = k < C ? (S >> k) & 1 : true, onB = k < C ? !onA : true;
    if (onA) {
      const double z = sel4(al, ja), zd = varB ? 0.0 : (ja == kv - 1 ? rest : (ja == kv ? -rest : 0.0));
      ja++;
      if (k > 0)
#pragma unroll
        for (int q = 0; q < 3; q++) {
          const double P = X.VA[k][q];
          A1[q] = fma(z, P, A1[q]);
          D[q] = fma(zd, P, D[q]);
        }
    }
    if (onB) {
      const double z = sel4(be, jb), zd = varB ? (jb == kv - 1 ? rest : (jb == kv ? -rest : 0.0)) : 0.0;
      jb++;
      if (k > 0)
#pragma unroll
        for (int q = 0; q < 3; q++) {
          const double P = k < C ? X.VA[k][q] : X.VB[k][q];
          B1[q] = fma(z, P, B1[q]);
          D[q] = fma(zd, P, D[q]);
        }
    }
  }
  // F fixed, V + u D moving
  double Q[3];
#pragma unroll
  for (int q = 0; q < 3; q++) Q[q] = varB ? B1[q] - A1[q] : A1[q] - B1[q];
  double T0 = 0, U0 = 0, T2 = 0, U2 = 0;
#pragma unroll 2
  for (int i = 0; i < n; i++) {
    const double uu = fma(h, x[i], lo), wi = wx[i];
    const double R0 = fma(uu, D[0], Q[0]), R1 = fma(uu, D[1], Q[1]), R2 = fma(uu, D[2], Q[2]);
    const double r2 = fma(R0, R0, fma(R1, R1, R2 * R2)), ir = rsqrt_fast(r2);
    const double a = wi * ir, b = a * r2;
    T0 += a;
    U0 = fma(a, uu, U0);
    T2 += b;
    U2 = fma(b, uu, U2);
  }
  w *= h;
  // R^0: the rule integrates 1 and u exactly
  const double T[3] = {w * T0, w, w * T2}, U[3] = {w * U0, w * fma(0.5, h, lo), w * U2};
#pragma unroll
  for (int pk = 0; pk < 3; pk++) {
    double ab = 0.0;
    raw[8 * pk] += T[pk];
#pragma unroll
    for (int q = 0; q < 3; q++) {
      const double F = varB ? A1[q] : B1[q], V = varB ? B1[q] : A1[q];
      const double Y = fma(T[pk], V, U[pk] * D[q]), TF = T[pk] * F;
      raw[8 * pk + 1 + q] += varB ? TF : Y;
      raw[8 * pk + 4 + q] += varB ? Y : TF;
      ab = fma(F, Y, ab);
    }
    raw[8 * pk + 7] += ab;
  }
}

// moment i of the pair from the raw sums (Beta factors G, common-simplex
// moments ub and W)
__device__ __forceinline__ double sg_raw_to_moment(const SgPair &X, const double *raw, int i) {
  int pk = i / 8, j = i % 8;
  double G0 = X.G[pk][0], G1 = X.G[pk][1], G2 = X.G[pk][2];
  const double *r = raw + 8 * pk;
  if (j == 0) return G0 * r[0];
  if (j < 4) return G1 * r[j] + X.ub[j - 1] * (G0 - G1) * r[0];
  if (j < 7) return G1 * r[j] + X.ub[j - 4] * (G0 - G1) * r[0];
  double uAB = X.ub[0] * (r[1] + r[4]) + X.ub[1] * (r[2] + r[5]) + X.ub[2] * (r[3] + r[6]);
  return G2 * r[7] + (G1 - G2) * uAB + X.W * (G0 - 2.0 * G1 + G2) * r[0];
}

// all 24 moments from raw sums held in registers (constant indices only)
__device__ __forceinline__ void sg_moments_from_raw(const SgPair &X, const double raw[24], double out[24]) {
#pragma unroll
  for (int pk = 0; pk < 3; pk++) {
    double G0 = X.G[pk][0], G1 = X.G[pk][1], G2 = X.G[pk][2];
    const double *r = raw + 8 * pk;
    double *m = out + 8 * pk;
    m[0] = G0 * r[0];
#pragma unroll
    for (int x = 0; x < 3; x++) {
      m[1 + x] = G1 * r[1 + x] + X.ub[x] * (G0 - G1) * r[0];
      m[4 + x] = G1 * r[4 + x] + X.ub[x] * (G0 - G1) * r[0];
    }
    double uAB = X.ub[0] * (r[1] + r[4]) + X.ub[1] * (r[2] + r[5]) + X.ub[2] * (r[3] + r[6]);
    m[7] = G2 * r[7] + (G1 - G2) * uAB + X.W * (G0 - 2.0 * G1 + G2) * r[0];
  }
}


__device__ __forceinline__ int sg_face_S(int c, int f) { return c == 4 ? f + 1 : f; }
__device__ __forceinline__ int sg_nfaces(int c) { return c == 4 ? 14 : (1 << c); }

__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// sums part[24] over the block into out[24] (shared) in a fixed order
__device__ void sg_block_sum(double part[24], double (*red)[24], double *out) {
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int i = 0; i < 24; i++) {
    double v = warp_sum_d(part[i]);
    if (lane == 0) red[wid][i] = v;
  }
  __syncthreads();
  if (threadIdx.x < 24) {
    double s = 0.0;
    for (int w = 0; w < SG_THREADS / 32; w++) s += red[w][threadIdx.x];
    out[threadIdx.x] = s;
  }
  __syncthreads();
}

__constant__ double c_sg_gpre[3] = {0.25 / M_PI, 0.25 / M_PI, 0.125 / M_PI};

// whole-face product rule of order n (points x, weights wx of [0, 1] in shared
// memory), lines strided over the block (raw sums)
template <int C>
__device__ void sg_fixed_pass(const SgPair &X, int n, const double *x, const double *wx, double raw[24]) {
  constexpr int nown = 4 - C, K = 6 - C, nf = C == 4 ? 14 : (1 << C);
  int per = 1;
#pragma unroll
  for (int i = 0; i < K - 1; i++) per *= n;
#pragma unroll
  for (int i = 0; i < 24; i++) raw[i] = 0.0;
#pragma unroll 1
  for (int f = threadIdx.x; f < nf * per; f += SG_THREADS) {
    int face = f / per, t = f - face * per;
    int S = sg_face_S(C, face), ns = __popc(S);
    double u[K], w = 1.0;
#pragma unroll
    for (int d = 0; d < K - 1; d++) {
      const int q = t / n, i = t - q * n;
      t = q;
      u[d] = x[i];
      w *= wx[i];
    }
    sg_line<C>(X, S, ns + nown - 1, u, w, n, x, wx, 0.0, 1.0, raw);
  }
}

// h^2 = squared diameter of tetrahedron A; scales of the 24 moments from the
// order n + 2 values f1 (which include the kernel prefactors)
__device__ void sg_scales(const SgPair &X, const double *f1, double *scale) {
  double h2 = 0.0;
  for (int i = 0; i < 4; i++)
    for (int j = 0; j < 4; j++) {
      double s2 = 0.0;
      for (int x = 0; x < 3; x++) s2 += (X.VA[i][x] - X.VA[j][x]) * (X.VA[i][x] - X.VA[j][x]);
      h2 = fmax(h2, s2);
    }
  double h = sqrt(h2);
  for (int pk = 0; pk < 3; pk++) {
    double m0 = fabs(f1[8 * pk]) / c_sg_gpre[pk];
    scale[8 * pk] = m0;
    for (int x = 1; x < 7; x++) scale[8 * pk + x] = m0 * h;
    scale[8 * pk + 7] = m0 * h2;
  }
}

struct SgLists {
  int *list;        // flagged pair indices, by class (c = 2, 3, 4) at start[c-2]
  int *cnt;         // 3 counters
  int start[3];
  unsigned char *flag;   // per singular pair: bit 0 flagged, bits 1-2 refinement status
  unsigned int *status;
};

template <int C>
__device__ void sg_fixed_pair(const SgPair &X, int pidx, int first, double *mom, int n, int refine,
                              double flag_tol, const SgLists &L, const double (*tab)[16], double (*red)[24],
                              double *f0, double *f1) {
  double part[24];
  sg_fixed_pass<C>(X, n, tab[0], tab[1], part);
  sg_block_sum(part, red, f1);
  if (threadIdx.x < 24) f0[threadIdx.x] = sg_raw_to_moment(X, f1, threadIdx.x) * c_sg_gpre[threadIdx.x / 8];
  __syncthreads();
  if (!refine) {
    if (threadIdx.x < 24) mom[24 * (size_t)pidx + threadIdx.x] = f0[threadIdx.x];
    return;
  }
  sg_fixed_pass<C>(X, n + 2, tab[2], tab[3], part);
  sg_block_sum(part, red, f1);
  double m1 = threadIdx.x < 24 ? sg_raw_to_moment(X, f1, threadIdx.x) * c_sg_gpre[threadIdx.x / 8] : 0.0;
  __syncthreads();
  if (threadIdx.x < 24) f1[threadIdx.x] = m1;
  __syncthreads();
  if (threadIdx.x == 0) {
    double scale[24];
    sg_scales(X, f1, scale);
    double flag = 0.0;
    for (int i = 0; i < 24; i++) flag = fmax(flag, fabs(f1[i] - f0[i]) / c_sg_gpre[i / 8] / scale[i]);
    for (int i = 0; i < 24; i++) mom[24 * (size_t)pidx + i] = f1[i];
    bool flagged = !(flag <= flag_tol);
    L.flag[pidx - first] = flagged ? 1 : 0;
    if (flagged) {
      int pos = atomicAdd(&L.cnt[C - 2], 1);
      L.list[L.start[C - 2] + pos] = pidx;
    }
  }
}

__global__ void __launch_bounds__(SG_THREADS, 2) k_sing_fixed(DevGeom g, const int4 *tp, const int4 *ordA,
                                                              const int4 *ordB, int first, double *mom, int n,
                                                              int refine, double flag_tol, SgLists L) {
  __shared__ SgPair X;
  __shared__ double red[SG_THREADS / 32][24];
  __shared__ double f0[24], f1[24], tab[4][16];   // points and weights of orders n and n + 2
  const int pidx = first + blockIdx.x;
  if (threadIdx.x < 64) {
    const int r = threadIdx.x >> 4, i = threadIdx.x & 15, o = r < 2 ? n : min(n + 2, 16);
    tab[r][i] = r & 1 ? c_sgw[o][i] : c_sgx[o][i];
  }
  if (threadIdx.x == 0) sg_setup(g, ordA[pidx], ordB[pidx], tp[pidx].z, X);
  __syncthreads();
  switch (X.c) {
    case 2: sg_fixed_pair<2>(X, pidx, first, mom, n, refine, flag_tol, L, tab, red, f0, f1); break;
    case 3: sg_fixed_pair<3>(X, pidx, first, mom, n, refine, flag_tol, L, tab, red, f0, f1); break;
    default: sg_fixed_pair<4>(X, pidx, first, mom, n, refine, flag_tol, L, tab, red, f0, f1); break;
  }
}

// ------------------------------------------------------------- refinement
// A batch of flagged pairs of one class, all levels together: box lists in
// HBM, the boxes of a pair contiguous and in order.  Per level: k_sgr_eval
// evaluates the 2K halves of every box and decides, k_sgr_count and
// k_sgr_scan place every pair's children, k_sgr_next writes them in order and
// adds the closed boxes to the pair's moments, in level and box order.  One
// CTA per pair left the pairs with many levels running alone, at 9.6 % FP64-pipe
// activity.  Jittered sphere, N = 5,760: refinement 201 -> 54 ms, the fixed
// passes 55 -> 13.7 ms.
struct SgrPair {
  SgPair X;
  double scale[24], acc[24];
  int pidx, status;
  int beg, n;              // its boxes of this level
  int nopen, nbeg;         // open ones (children / 2), first child
};

struct SgrBatch {
  SgrPair *pair;
  double *cur, *nxt, *res;       // SG_REC, SG_REC, SG_RES doubles per box
  int *open;                     // per box: split dimension of an open box, -1 closed; closed ones in cd
  int *cd;                       // split dimension taken
  int *total;                    // boxes of the next level
  int np, cap;
};

__global__ void k_sgr_setup(DevGeom g, const int4 *tp, const int4 *ordA, const int4 *ordB, const double *mom,
                            const int *list, SgrBatch B, int nf) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= B.np) return;
  SgrPair &Q = B.pair[p];
  const int pidx = list[p];
  SgPair X;
  sg_setup(g, ordA[pidx], ordB[pidx], tp[pidx].z, X);
  Q.X = X;
  double f1[24], scale[24];
  for (int i = 0; i < 24; i++) f1[i] = mom[24 * (size_t)pidx + i];
  sg_scales(X, f1, scale);
  for (int i = 0; i < 24; i++) { Q.scale[i] = scale[i]; Q.acc[i] = 0.0; }
  Q.pidx = pidx;
  Q.status = 0;
  Q.beg = p * nf;
  Q.n = nf;
}

// Moments of one task (a box): its lines over the G lanes of a group, a fixed
// shuffle tree, the result in every lane of the group
template <int C, int G>
__device__ __forceinline__ void sgr_task(const SgPair &X, int S, const double *lo, const double *hi, int gl,
                                         const double *x, const double *wx, double out[24]) {
  constexpr int K = 6 - C, nown = 4 - C;
  constexpr int LN = SG_NG * (K > 2 ? SG_NG : 1) * (K > 3 ? SG_NG : 1);   // lines: 6^{K-1}
  const int ka = __popc(S) + nown - 1;
  double raw[24];
#pragma unroll
  for (int i = 0; i < 24; i++) raw[i] = 0.0;
#pragma unroll 1
  for (int t0 = gl; t0 < LN; t0 += G) {
    int t = t0;
    double u[K], w = 1.0;
#pragma unroll
    for (int d = 0; d < K - 1; d++) {
      const int i = t % SG_NG;
      t /= SG_NG;
      const double h = hi[d] - lo[d];
      u[d] = fma(h, x[i], lo[d]);
      w *= h * wx[i];
    }
    sg_line<C>(X, S, ka, u, w, SG_NG, x, wx, lo[K - 1], hi[K - 1] - lo[K - 1], raw);
  }
#pragma unroll
  for (int i = 0; i < 24; i++)
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) raw[i] += __shfl_xor_sync(0xffffffffu, raw[i], o);
  sg_moments_from_raw(X, raw, out);
}

template <int C> struct SgrCfg;
template <> struct SgrCfg<2> { static constexpr int G = 32, NB = 1; };    // 8 halves a box: 256 lanes
template <> struct SgrCfg<3> { static constexpr int G = 4, NB = 10; };    // 6 halves: 24 lanes
template <> struct SgrCfg<4> { static constexpr int G = 2, NB = 32; };    // 4 halves: 8 lanes

// level 0: the whole face cubes of every pair
template <int C>
__global__ void __launch_bounds__(SG_THREADS) k_sgr_init(SgrBatch B) {
  constexpr int K = 6 - C, nf = C == 4 ? 14 : (1 << C), G = SgrCfg<C>::G, NT = SG_THREADS / G;
  __shared__ double tx[SG_NG], tw[SG_NG];
  if (threadIdx.x < SG_NG) { tx[threadIdx.x] = c_sgx[SG_NG][threadIdx.x]; tw[threadIdx.x] = c_sgw[SG_NG][threadIdx.x]; }
  __syncthreads();
  const int gl = threadIdx.x % G, grp = threadIdx.x / G, total = B.np * nf;
  for (int base = blockIdx.x * NT; base < total; base += gridDim.x * NT) {
    const int b = min(base + grp, total - 1);      // idle groups repeat the last box
    const int p = b / nf, S = sg_face_S(C, b - p * nf);
    double lo[4] = {0, 0, 0, 0}, hi[4] = {1, 1, 1, 1}, m[24];
    sgr_task<C, G>(B.pair[p].X, S, lo, hi, gl, tx, tw, m);
    if (gl == 0 && base + grp < total) {
      double *r = B.cur + (size_t)b * SG_REC;
      for (int d = 0; d < 4; d++) { r[d] = 0.0; r[4 + d] = 1.0; }
#pragma unroll
      for (int i = 0; i < 24; i++) r[8 + i] = m[i];
      r[32] = (double)S;
      r[33] = (double)p;
    }
  }
  (void)K;
}

// halves of every box, the split that changes it most, open or closed
template <int C>
__global__ void __launch_bounds__(SG_THREADS, 2) k_sgr_eval(SgrBatch B, int nbox, double tol) {
  constexpr int K = 6 - C, G = SgrCfg<C>::G, NB = SgrCfg<C>::NB, LB = 2 * K * G;   // lanes per box
  extern __shared__ __align__(16) double sm[];
  double *sres = sm;                             // NB x 2K x 24 moments
  double *sbox = sres + NB * 2 * K * 24;         // NB x SG_REC
  double *serr = sbox + NB * SG_REC;             // NB x K
  SgPair *sX = (SgPair *)(serr + NB * K);        // NB pairs
  __shared__ double tx[SG_NG], tw[SG_NG];
  __shared__ int sd[NB];
  const int tid = threadIdx.x;
  if (tid < SG_NG) { tx[tid] = c_sgx[SG_NG][tid]; tw[tid] = c_sgw[SG_NG][tid]; }
  for (int base = blockIdx.x * NB; base < nbox; base += gridDim.x * NB) {
    const int nb = min(NB, nbox - base);
    __syncthreads();
    for (int e = tid; e < nb * SG_REC; e += SG_THREADS) sbox[e] = B.cur[(size_t)base * SG_REC + e];
    constexpr int XD = sizeof(SgPair) / 8;
    __syncthreads();
    for (int e = tid; e < nb * XD; e += SG_THREADS) {
      const int j = e / XD;
      ((double *)&sX[j])[e - j * XD] = ((const double *)&B.pair[(int)sbox[j * SG_REC + 33]].X)[e - j * XD];
    }
    __syncthreads();
    {
      // lanes past the last box repeat it (the shuffles need whole warps)
      const int jb = tid / LB, j = min(jb, nb - 1), task = (tid % LB) / G, gl = tid % G;
      const double *r = sbox + j * SG_REC;
      const int sdim = task >> 1;
      double lo[K], hi[K];
#pragma unroll
      for (int d = 0; d < K; d++) {
        lo[d] = r[d];
        hi[d] = r[4 + d];
        if (d == sdim) {
          const double mid = 0.5 * (lo[d] + hi[d]);
          if (task & 1) lo[d] = mid; else hi[d] = mid;
        }
      }
      double m[24];
      sgr_task<C, G>(sX[j], (int)r[32], lo, hi, gl, tx, tw, m);
      if (gl == 0 && jb < nb)
#pragma unroll
        for (int i = 0; i < 24; i++) sres[(j * 2 * K + task) * 24 + i] = m[i];
    }
    __syncthreads();
    if (tid < nb * K) {
      const int j = tid / K, d = tid - j * K;
      const double *v0 = sres + (j * 2 * K + 2 * d) * 24, *v1 = v0 + 24, *val = sbox + j * SG_REC + 8;
      const double *scale = B.pair[(int)sbox[j * SG_REC + 33]].scale;
      double e = 0.0;
      for (int i = 0; i < 24; i++) e = fmax(e, fabs(v0[i] + v1[i] - val[i]) / scale[i]);
      serr[tid] = e;
    }
    __syncthreads();
    if (tid < nb) {
      double best = -1.0;
      int bd = 0;
      for (int d = 0; d < K; d++)
        if (serr[tid * K + d] > best) { best = serr[tid * K + d]; bd = d; }
      sd[tid] = bd;
      B.cd[base + tid] = bd;
      B.open[base + tid] = best > tol;
    }
    __syncthreads();
    for (int e = tid; e < nb * SG_RES; e += SG_THREADS) {
      const int j = e / SG_RES, f = e - j * SG_RES;
      B.res[(size_t)(base + j) * SG_RES + f] = sres[(j * 2 * K + 2 * sd[j]) * 24 + f];
    }
  }
}

// open boxes of every pair, in order up to the limits
__global__ void k_sgr_count(SgrBatch B, int last) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= B.np) return;
  SgrPair &Q = B.pair[p];
  int n = 0, status = 0;
  for (int b = Q.beg; b < Q.beg + Q.n; b++)
    if (B.open[b]) {
      if (2 * n + 2 > SG_MAXBOX) { status |= 1; B.open[b] = 0; }
      else if (last) { status |= 2; B.open[b] = 0; }
      else n++;
    }
  Q.nopen = n;
  Q.status |= status;
}

__global__ void __launch_bounds__(1024) k_sgr_scan(SgrBatch B) {
  __shared__ int wsum[32], carry;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  if (tid == 0) carry = 0;
  __syncthreads();
  for (int base = 0; base < B.np; base += 1024) {
    const int p = base + tid, v = p < B.np ? 2 * B.pair[p].nopen : 0;
    int x = v;
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) wsum[wid] = x;
    __syncthreads();
    if (wid == 0) {
      int s = wsum[lane];
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, s, o);
        if (lane >= o) s += y;
      }
      wsum[lane] = s;
    }
    __syncthreads();
    if (p < B.np) B.pair[p].nbeg = carry + (wid ? wsum[wid - 1] : 0) + x - v;
    __syncthreads();
    if (tid == 0) carry += wsum[31];
    __syncthreads();
  }
  if (tid == 0) *B.total = carry;
}

// children and closed sums of every pair, one warp per pair, in box order
__global__ void __launch_bounds__(256) k_sgr_next(SgrBatch B) {
  const int p = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (p >= B.np) return;
  SgrPair &Q = B.pair[p];
  if (*B.total > B.cap) return;          // the host splits the batch
  double a = lane < 24 ? Q.acc[lane] : 0.0;
  int pos = Q.nbeg;
  const int beg = Q.beg, n = Q.n;
  // the flags of 32 boxes at a time; the loads of the boxes do not depend on
  // one another
  for (int b0 = beg; b0 < beg + n; b0 += 32) {
    const int nb = min(32, beg + n - b0);
    const unsigned op = __ballot_sync(0xffffffffu, lane < nb && __ldg(B.open + b0 + lane));
    const int cd = lane < nb ? __ldg(B.cd + b0 + lane) : 0;
#pragma unroll 4
    for (int j = 0; j < nb; j++) {
      const double *v = B.res + (size_t)(b0 + j) * SG_RES, *r = B.cur + (size_t)(b0 + j) * SG_REC;
      const int d = __shfl_sync(0xffffffffu, cd, j);
      if (!(op >> j & 1)) {
        if (lane < 24) a += __ldg(v + lane) + __ldg(v + 24 + lane);
        continue;
      }
      const int at = pos + 2 * __popc(op & ((1u << j) - 1));
      const double mid = 0.5 * (__ldg(r + d) + __ldg(r + 4 + d));
#pragma unroll
      for (int e0 = 0; e0 < 96; e0 += 32) {
        const int e = e0 + lane, h = e / SG_REC, f = e - h * SG_REC;
        if (e >= 2 * SG_REC) break;
        double x = f < 8 || f >= 32 ? __ldg(r + f) : __ldg(v + 24 * h + f - 8);
        if (h == 0 && f == 4 + d) x = mid;
        if (h == 1 && f == d) x = mid;
        B.nxt[(size_t)(at + h) * SG_REC + f] = x;
      }
    }
    pos += 2 * __popc(op);
  }
  if (lane < 24) Q.acc[lane] = a;
  if (lane == 0) { Q.beg = Q.nbeg; Q.n = 2 * Q.nopen; }
}

__global__ void k_sgr_store(SgrBatch B, int first, double *mom, SgLists L) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= B.np) return;
  const SgrPair &Q = B.pair[p];
  for (int i = 0; i < 24; i++) mom[24 * (size_t)Q.pidx + i] = Q.acc[i] * c_sg_gpre[i / 8];
  L.flag[Q.pidx - first] |= (unsigned char)(Q.status << 1);
  if (Q.status) atomicOr(L.status, (unsigned int)Q.status);
}

template <int C>
static int sgr_smem() {
  constexpr int K = 6 - C, NB = SgrCfg<C>::NB;
  return (int)(sizeof(double) * (NB * 2 * K * 24 + NB * SG_REC + NB * K) + NB * sizeof(SgPair));
}

// refines list[0 .. np); halves the batch while its boxes outgrow the lists
template <int C>
static int sgr_run(bg_geometry *g, const int *list, int np, SgrBatch B, const SgLists &L, long long *evals) {
  NearData &nd = g->near;
  constexpr int K = 6 - C, nf = C == 4 ? 14 : (1 << C), NB = SgrCfg<C>::NB;
  constexpr long long P = (long long)SG_NG * SG_NG * (K > 2 ? SG_NG : 1) * (K > 3 ? SG_NG : 1);
  static bool attr = false;
  if (!attr) {
    BG_CUDA_TRY(cudaFuncSetAttribute(k_sgr_eval<C>, cudaFuncAttributeMaxDynamicSharedMemorySize, sgr_smem<C>()));
    attr = true;
  }
  B.np = np;
  const int pb = (np + 127) / 128;
  k_sgr_setup<<<pb, 128, 0, stream()>>>(g->dev, nd.tp, nd.tpOrdA, nd.tpOrdB, nd.tpMom, list, B, nf);
  BG_LAUNCHED();
  const int grid = 148 * 4;
  constexpr int NT = SG_THREADS / SgrCfg<C>::G;
  k_sgr_init<C><<<std::min(grid, (np * nf + NT - 1) / NT), SG_THREADS, 0, stream()>>>(B);
  BG_LAUNCHED();
  long long ev = (long long)np * nf * P;
  int nbox = np * nf;
  for (int level = 0; level < SG_MAXLEVEL && nbox > 0; level++) {
    k_sgr_eval<C><<<std::min(grid, (nbox + NB - 1) / NB), SG_THREADS, sgr_smem<C>(), stream()>>>(B, nbox, g->sing_tol);
    BG_LAUNCHED();
    ev += (long long)nbox * 2 * K * P;
    k_sgr_count<<<pb, 128, 0, stream()>>>(B, level == SG_MAXLEVEL - 1);
    BG_LAUNCHED();
    k_sgr_scan<<<1, 1024, 0, stream()>>>(B);
    BG_LAUNCHED();
    k_sgr_next<<<(np + 7) / 8, 256, 0, stream()>>>(B);
    BG_LAUNCHED();
    BG_CUDA_TRY(cudaMemcpyAsync(&nbox, B.total, sizeof(int), cudaMemcpyDeviceToHost, stream()));
    BG_CUDA_TRY(cudaStreamSynchronize(stream()));
    if (nbox > B.cap) {
      const int h = np / 2;              // one pair holds at most SG_MAXBOX <= cap boxes
      int st = sgr_run<C>(g, list, h, B, L, evals);
      return st ? st : sgr_run<C>(g, list + h, np - h, B, L, evals);
    }
    std::swap(B.cur, B.nxt);
  }
  k_sgr_store<<<pb, 128, 0, stream()>>>(B, nd.ntp_reg, nd.tpMom, L);
  BG_LAUNCHED();
  *evals += ev;
  return BG_OK;
}

// all flagged pairs of the three classes, in batches
static int sgr_refine(bg_geometry *g, const SgLists &L, const int cnt[3], long long *evals) {
  const int most = std::max(cnt[0], std::max(cnt[1], cnt[2]));
  if (most <= 0) return BG_OK;
  // 32 boxes a pair on average (8-14 start, about 30 at the widest level)
  const int batch = std::min(most, 8192);
  SgrBatch B{};
  B.cap = std::max(2 * SG_MAXBOX, 32 * batch);
  const size_t nb = (size_t)B.cap;
  const size_t bytes = sizeof(double) * nb * (2 * SG_REC + SG_RES) + sizeof(SgrPair) * (size_t)batch + 2 * sizeof(int) * nb + 64;
  char *blk = nullptr;
  if (cudaMallocAsync((void **)&blk, bytes, stream()) != cudaSuccess) {
    cudaGetLastError();
    set_error("singular near-field precompute: cannot allocate the refinement box lists");
    return BG_ERR_NOMEM;
  }
  char *q = blk;
  B.cur = (double *)q; q += sizeof(double) * nb * SG_REC;
  B.nxt = (double *)q; q += sizeof(double) * nb * SG_REC;
  B.res = (double *)q; q += sizeof(double) * nb * SG_RES;
  B.pair = (SgrPair *)q; q += sizeof(SgrPair) * (size_t)batch;
  B.open = (int *)q; q += sizeof(int) * nb;
  B.cd = (int *)q; q += sizeof(int) * nb;
  B.total = (int *)q;
  int st = BG_OK;
  for (int cls = 0; cls < 3 && !st; cls++)
    for (int b = 0; b < cnt[cls] && !st; b += batch) {
      const int n = std::min(batch, cnt[cls] - b);
      const int *list = L.list + L.start[cls] + b;
      st = cls == 0 ? sgr_run<2>(g, list, n, B, L, evals)
         : cls == 1 ? sgr_run<3>(g, list, n, B, L, evals) : sgr_run<4>(g, list, n, B, L, evals);
    }
  cudaFreeAsync(blk, stream());
  return st;
}

// Singular pairs of the near table: [ntp_reg, ntp), sorted by class (2, 3, 4
// common vertices).  Fills tpMom and the geometry's singular statistics.
int singular_precompute(bg_geometry *g) {
  NearData &nd = g->near;
  const int nsing = nd.ntp - nd.ntp_reg;
  for (int i = 0; i < 6; i++) g->sing_stats[i] = 0;
  if (nsing <= 0) return BG_OK;
  int st = sg_tables();
  if (st) return st;
  const int n = g->singular_order;
  const bool refine = g->sing_refine;
  // points of the fixed passes (host arithmetic, per class)
  long long fixed_pts = 0;
  for (int cls = 0; cls < 3; cls++) {
    int c = cls + 2, nf = c == 4 ? 14 : (1 << c);
    long long p0 = 1, p1 = 1;
    for (int i = 0; i < 6 - c; i++) { p0 *= n; p1 *= n + 2; }
    fixed_pts += (long long)nd.nsing_c[cls] * nf * (p0 + (refine ? p1 : 0));
  }
  g->sing_stats[0] = nsing;
  g->sing_stats[2] = fixed_pts;
  // small device block: counters (3), status, then the list and the per-pair
  // flags
  size_t hdr = 64, bytes = hdr + sizeof(int) * (size_t)nsing + (size_t)nsing;
  char *blk = nullptr;
  BG_CUDA_TRY(cudaMallocAsync((void **)&blk, bytes, stream()));
  SgLists L;
  L.cnt = (int *)blk;
  L.status = (unsigned int *)(blk + 16);
  L.list = (int *)(blk + hdr);
  L.flag = (unsigned char *)(blk + hdr + sizeof(int) * (size_t)nsing);
  L.start[0] = 0;
  L.start[1] = nd.nsing_c[0];
  L.start[2] = nd.nsing_c[0] + nd.nsing_c[1];
  int rc = BG_OK;
  long long evals = 0;
  do {
    if (cudaMemsetAsync(blk, 0, bytes, stream()) != cudaSuccess) { rc = BG_ERR_CUDA; break; }
    k_sing_fixed<<<nsing, SG_THREADS, 0, stream()>>>(g->dev, nd.tp, nd.tpOrdA, nd.tpOrdB, nd.ntp_reg, nd.tpMom, n,
                                                     refine ? 1 : 0, g->sing_flag_tol, L);
    if (cudaGetLastError() != cudaSuccess) { rc = BG_ERR_CUDA; break; }
    g_launches.fetch_add(1, std::memory_order_relaxed);
    struct { int cnt[4]; unsigned int status; } h;
    if (cudaMemcpyAsync(&h, blk, sizeof h, cudaMemcpyDeviceToHost, stream()) != cudaSuccess ||
        cudaStreamSynchronize(stream()) != cudaSuccess) { rc = BG_ERR_CUDA; break; }
    if (refine) {
      // the order of a list comes from an atomic counter and its pairs are
      // independent of one another: no result depends on it
      if ((rc = sgr_refine(g, L, h.cnt, &evals))) break;
      if (cudaMemcpyAsync(&h, blk, sizeof h, cudaMemcpyDeviceToHost, stream()) != cudaSuccess) { rc = BG_ERR_CUDA; break; }
    }
    if (!nd.tpFlag && cudaMallocAsync((void **)&nd.tpFlag, (size_t)nsing, stream()) != cudaSuccess) {
      set_error("singular near-field precompute: cannot allocate the pair flags");
      rc = BG_ERR_NOMEM;
      break;
    }
    if (cudaMemcpyAsync(nd.tpFlag, L.flag, (size_t)nsing, cudaMemcpyDeviceToDevice, stream()) != cudaSuccess) {
      rc = BG_ERR_CUDA;
      break;
    }
    if (cudaStreamSynchronize(stream()) != cudaSuccess) { rc = BG_ERR_CUDA; break; }
    g->sing_stats[1] = (long long)h.cnt[0] + h.cnt[1] + h.cnt[2];
    g->sing_stats[3] = evals;
    g->sing_stats[4] = h.status;
    g->sing_stats[5] = refine ? 1 : 0;
  } while (0);
  if (rc == BG_ERR_CUDA) set_error("singular near-field precompute: %s", cudaGetErrorString(cudaGetLastError()));
  cudaFreeAsync(blk, stream());
  if (rc == BG_OK) BG_CUDA_TRY(cudaStreamSynchronize(stream()));
  return rc;
}

}  // namespace bg
