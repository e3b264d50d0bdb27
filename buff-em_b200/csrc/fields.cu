// Fields of the solved currents at evaluation points: SWGGeometry::GetFields
// (GetFields.cc:287-382) with Get1BFFields (GetFields.cc:265-281) and the
// volume integrand GetFields_VIntegrand (GetFields.cc:176-201).
//
// The reference sums, per point X and basis function a, J_a times the fields
// of b_a integrated over both tetrahedra with the 4-point rule when
// |X - centroid_a| / radius_a > 10, else the 16-point rule.  Both rules are
// fully symmetric, so their points depend only on the tetrahedron, and the
// sum over the (up to four) basis functions living on one tetrahedron T is a
// single linear current per rule:
//
//   sum_a J_a b_a(y) * 6 vol_T = sum_k g_k (y - V_k),   g_k = 2 s_k A_k J_k
//
// (k runs over T's faces that carry a basis function, V_k is the vertex
// opposite face k, s_k = +1 on the basis function's P side, -1 on its M side,
// A_k the face area).  The kernel therefore walks tetrahedra, not basis
// functions: each (point, tetrahedron) pair costs 4 quadrature points when all
// of T's faces are far from X, and 4 + 16 (split by face) otherwise --
// a quarter of the per-basis-function work, with the same quadrature points
// and the same rule choice per basis function as the reference.
//
// Field kernels (e^{-i w t}, vacuum, g = e^{ikr}/(4 pi r), R = X - y, Rh = R/r):
//   E = i w Z0 g [(1 + i/kr - 1/kr^2) J + (-1 - 3i/kr + 3/kr^2) (Rh.J) Rh]
//   H = g (ik - 1/r) Rh x J
// which are the G and C dyadics of the reference's CalcGC with its prefactors.
// The incident plane wave adds E0 e^{ik nhat.X} and nhat x E / Z0.
//
// HBM layout (per tetrahedron, built once per geometry):
//   (all in the order of field_tables, which follows the doubles of fieldTet)
//   fieldTet  16 doubles: V0..V3 (12), centroid (3), R_all (1), where
//             |X - centroid| > R_all implies every face of T is far from X
//   fieldFace 16 doubles: per local face k, (centroid, radius), radius 0 if the
//             face carries no basis function
//   coef       8 doubles per call: g_k (4 complex) from J
// Work split: a block owns 128 x tpt tetrahedra (tpt = 1 with the
// tetrahedron's data held in registers across the points while the partials
// stay small; else tpt grows to ~8 blocks per SM) and 32 points; each
// warp reduces its lanes per point into shared memory and the block writes one
// partial per (tetrahedron block, point), summed in a fixed order by the
// finishing kernel (deterministic).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "devmath.cuh"
#include "internal.h"

namespace bg {
namespace {

constexpr int FTHREADS = 128;
constexpr int FPCH = 32;           // points per block
constexpr double ZVAC_F = 376.73031346177;

// 16-point rule (TetCR.cc): orbit patterns as in the assembly kernels
__constant__ double c_fr16[64];
static bool s_fr16_ok = false;

int init_rule16() {
  if (s_fr16_ok) return BG_OK;
  const double v[5] = {0.771642902067237, 0.076119032644254315, 0.07183164526766925, 0.11970052779780202,
                       0.40423391346726440};
  const char *pat[2] = {"ABB BAB BBA BBB", "CDE CED CEE DCE DEC DEE ECD ECE EDC EDE EEC EED"};
  const double w[2] = {8.3956323500204695e-3, 0.011090344772215399};
  double h[64];
  int np = 0;
  for (int o = 0; o < 2; o++)
    for (const char *p = pat[o]; *p;) {
      if (*p == ' ') { p++; continue; }
      h[4 * np] = v[p[0] - 'A']; h[4 * np + 1] = v[p[1] - 'A']; h[4 * np + 2] = v[p[2] - 'A'];
      h[4 * np + 3] = w[o];
      np++;
      p += 3;
    }
  BG_CUDA_TRY(cudaMemcpyToSymbol(c_fr16, h, sizeof h));
  BG_CUDA_TRY(uploads_done());
  s_fr16_ok = true;
  return BG_OK;
}

struct z { double r, i; };
__device__ __forceinline__ z zmul(z a, z b) { return z{a.r * b.r - a.i * b.i, a.r * b.i + a.i * b.r}; }

struct FieldK {
  z k;       // wavenumber (= omega in the reference's units)
  z invik;   // 1 / (i k)
  z ik;      // i k
};

// phase of a tetrahedron's points: e^{ikr} = e^{ik rc} e^{i(k r - k rc)}, rc the
// distance of its centroid
struct FieldPhase { double k, krc; z ec; };

// One quadrature point: current alpha y - beta at y with weight w.  MODE 3:
// complex k.  For real k, with a = 1/kr,
//   E += g [((1 - a^2) + ia) J + ((3 a^2 - 1) - 3ia) (R.J) R / r^2],
//   H += g (ik - 1/r) R x J / r,
// and e^{ikr} is the tetrahedron's common phase times a short series (MODE 2:
// |k| |y - centroid| <= 1/4, MODE 1: <= 1) or a sincos (MODE 0).  A point at x
// itself (r < 1e-12) gets weight 0: no branch, so points are in flight together.
// FP64-pipe bound; 4,225 points of a plane through the body, N = 57,222:
// 15.9 -> 11.3 ms.
template <int MODE>
__device__ __forceinline__ void field_point(const FieldK &K, const FieldPhase &F, const double *x, const double *y,
                                            double w, z al, const z *be, double *acc) {
  z J[3];
#pragma unroll
  for (int c = 0; c < 3; c++) J[c] = z{al.r * y[c] - be[c].r, al.i * y[c] - be[c].i};
  const double R[3] = {x[0] - y[0], x[1] - y[1], x[2] - y[2]};
  const double rr = R[0] * R[0] + R[1] * R[1] + R[2] * R[2];
  const bool on = !(rr < 1e-24);            // a NaN stays one
  const double r2 = on ? rr : 1.0, ir = rsqrt_fast(r2), r = r2 * ir, m = on ? w * ir : 0.0;
  z A, Bc, C;      // factors of J, (R.J) R and R x J
  if (MODE == 3) {
    double s, c;
    sincos(K.k.r * r, &s, &c);
    const double me = m * exp(-K.k.i * r);
    const z g{me * c, me * s};               // w e^{ikr} / r
    const z u{K.invik.r * ir, K.invik.i * ir}, u2 = zmul(u, u);   // 1/(ikr)
    A = zmul(g, z{1.0 - u.r + u2.r, -u.i + u2.i});
    Bc = zmul(g, z{(-1.0 + 3.0 * (u.r - u2.r)) * (ir * ir), 3.0 * (u.i - u2.i) * (ir * ir)});
    C = zmul(g, z{(K.ik.r - ir) * ir, K.ik.i * ir});
  } else {
    z g;
    if (MODE == 0) {
      double s, c;
      sincos(K.k.r * r, &s, &c);
      g = z{m * c, m * s};
    } else {
      z e;
      const double th = fma(F.k, r, -F.krc);
      if (MODE == 2) cossin_small_short(th, e.r, e.i);
      else cossin_small(th, e.r, e.i);
      e = zmul(F.ec, e);
      g = z{m * e.r, m * e.i};
    }
    const double a = -K.invik.i * ir, a2 = a * a, ir2 = ir * ir, t1 = 1.0 - a2;
    A = z{g.r * t1 - g.i * a, g.r * a + g.i * t1};
    const double br = fma(3.0, a2, -1.0) * ir2, bi = -3.0 * a * ir2, ci = K.ik.i * ir;
    Bc = z{g.r * br - g.i * bi, g.r * bi + g.i * br};
    C = z{-g.r * ir2 - g.i * ci, g.r * ci - g.i * ir2};
  }
  const z RJ{R[0] * J[0].r + R[1] * J[1].r + R[2] * J[2].r, R[0] * J[0].i + R[1] * J[1].i + R[2] * J[2].i};
  const z c2 = zmul(Bc, RJ);
#pragma unroll
  for (int q = 0; q < 3; q++) {
    acc[2 * q] = fma(A.r, J[q].r, fma(-A.i, J[q].i, fma(c2.r, R[q], acc[2 * q])));
    acc[2 * q + 1] = fma(A.r, J[q].i, fma(A.i, J[q].r, fma(c2.i, R[q], acc[2 * q + 1])));
  }
#pragma unroll
  for (int q = 0; q < 3; q++) {
    const int q1 = (q + 1) % 3, q2 = (q + 2) % 3;
    const z X{R[q1] * J[q2].r - R[q2] * J[q1].r, R[q1] * J[q2].i - R[q2] * J[q1].i};
    acc[6 + 2 * q] = fma(C.r, X.r, fma(-C.i, X.i, acc[6 + 2 * q]));
    acc[7 + 2 * q] = fma(C.r, X.i, fma(C.i, X.r, acc[7 + 2 * q]));
  }
}

template <int MODE>
__device__ __forceinline__ void rule4(const FieldK &K, const FieldPhase &F, const double *x, const double (*V)[3],
                                      z al, const z *be, double *acc) {
  // barycentric (B, A, A, A) and permutations, weight 1/24 (TetCR.cc 4-point rule)
  const double A = 0.13819660112501051, B = 0.58541019662496850;
  double S[3];
#pragma unroll
  for (int c = 0; c < 3; c++) S[c] = A * (V[0][c] + V[1][c] + V[2][c] + V[3][c]);
#pragma unroll
  for (int i = 0; i < 4; i++) {
    double y[3];
#pragma unroll
    for (int c = 0; c < 3; c++) y[c] = S[c] + (B - A) * V[i][c];
    field_point<MODE>(K, F, x, y, 1.0 / 24.0, al, be, acc);
  }
}

template <int MODE>
__device__ __forceinline__ void rule16(const FieldK &K, const FieldPhase &F, const double *x, const double (*V)[3],
                                       z al, const z *be, double *acc) {
#pragma unroll 2
  for (int i = 0; i < 16; i++) {
    const double *u = c_fr16 + 4 * i;
    double y[3];
#pragma unroll
    for (int c = 0; c < 3; c++)
      y[c] = V[0][c] + u[0] * (V[1][c] - V[0][c]) + u[1] * (V[2][c] - V[0][c]) + u[2] * (V[3][c] - V[0][c]);
    field_point<MODE>(K, F, x, y, u[3], al, be, acc);
  }
}

// g_k per tetrahedron from the basis-function coefficients
__global__ void k_fields_coef(DevGeom g, const int *order, const z *J, z *coef) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= g.NT) return;
  const int t = order[i];
  int4 fi = g.tetFI[t];
  int f[4] = {fi.x, fi.y, fi.z, fi.w};
#pragma unroll
  for (int k = 0; k < 4; k++) {
    z v{0.0, 0.0};
    int a = f[k];
    if (a >= 0) {
      double s = (g.bfTet[a].x == t ? 2.0 : -2.0) * g.bfArea[a];
      z Ja = J[a];
      v = z{s * Ja.r, s * Ja.i};
    }
    coef[4 * (size_t)i + k] = v;
  }
}

// one tetrahedron's data for the field sums: vertices, the all-faces-far
// sphere, and the linear current alpha y - beta of all its basis functions
struct TetData {
  double V[4][3], ctr[3], Rall;
  z al, be[3];
};

__device__ __forceinline__ void load_tet(const double *__restrict__ tetT, const z *__restrict__ coef, int t,
                                         TetData &T) {
  const double2 *T2 = reinterpret_cast<const double2 *>(tetT + 16 * (size_t)t);
  double2 a0 = T2[0], a1 = T2[1], a2 = T2[2], a3 = T2[3], a4 = T2[4], a5 = T2[5], a6 = T2[6], a7 = T2[7];
  T.V[0][0] = a0.x; T.V[0][1] = a0.y; T.V[0][2] = a1.x; T.V[1][0] = a1.y; T.V[1][1] = a2.x; T.V[1][2] = a2.y;
  T.V[2][0] = a3.x; T.V[2][1] = a3.y; T.V[2][2] = a4.x; T.V[3][0] = a4.y; T.V[3][1] = a5.x; T.V[3][2] = a5.y;
  T.ctr[0] = a6.x; T.ctr[1] = a6.y; T.ctr[2] = a7.x; T.Rall = a7.y;
  T.al = z{0.0, 0.0};
#pragma unroll
  for (int c = 0; c < 3; c++) T.be[c] = z{0.0, 0.0};
#pragma unroll
  for (int k = 0; k < 4; k++) {
    z gk = coef[4 * (size_t)t + k];
    T.al.r += gk.r; T.al.i += gk.i;
#pragma unroll
    for (int c = 0; c < 3; c++) { T.be[c].r += gk.r * T.V[k][c]; T.be[c].i += gk.i * T.V[k][c]; }
  }
}

// fields at x of tetrahedron t (data T): the 4-point rule for all of it when
// every face is far, else split by face with the reference's rule choice
template <int MODE>
__device__ __forceinline__ void tet_point(const FieldK &K, const double *x, const TetData &T,
                                          const double *__restrict__ tetF, const z *__restrict__ coef, int t,
                                          double *acc) {
  double d2 = (x[0] - T.ctr[0]) * (x[0] - T.ctr[0]) + (x[1] - T.ctr[1]) * (x[1] - T.ctr[1]) +
              (x[2] - T.ctr[2]) * (x[2] - T.ctr[2]);
  FieldPhase F{K.k.r, 0.0, {1.0, 0.0}};
  if (MODE == 1 || MODE == 2) {
    F.krc = K.k.r * sqrt(d2);
    sincos(F.krc, &F.ec.i, &F.ec.r);
    // beyond, k r - k rc is rounding only and would leave the range of the series: one phase
    if (!(fabs(F.krc) < 0x1p48)) F.k = F.krc = 0.0;
  }
  if (d2 > T.Rall * T.Rall) {
    rule4<MODE>(K, F, x, T.V, T.al, T.be, acc);
    return;
  }
  // per face: the reference's rule choice |X - centroid| / radius > 10
  z a4{0.0, 0.0}, b4[3] = {{0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}};
  z a16{0.0, 0.0}, b16[3] = {{0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}};
  bool any4 = false, any16 = false;
  const double4 *F4 = reinterpret_cast<const double4 *>(tetF + 16 * (size_t)t);
#pragma unroll
  for (int k = 0; k < 4; k++) {
    double4 f = F4[k];
    z gk = coef[4 * (size_t)t + k];
    double dx = x[0] - f.x, dy = x[1] - f.y, dz = x[2] - f.z;
    bool live = f.w != 0.0;
    bool far = live && sqrt(dx * dx + dy * dy + dz * dz) / f.w > 10.0;
    bool near = live && !far;
    double m4 = far ? 1.0 : 0.0, m16 = near ? 1.0 : 0.0;
    a4.r += m4 * gk.r; a4.i += m4 * gk.i;
    a16.r += m16 * gk.r; a16.i += m16 * gk.i;
#pragma unroll
    for (int c = 0; c < 3; c++) {
      b4[c].r += m4 * gk.r * T.V[k][c]; b4[c].i += m4 * gk.i * T.V[k][c];
      b16[c].r += m16 * gk.r * T.V[k][c]; b16[c].i += m16 * gk.i * T.V[k][c];
    }
    any4 |= far;
    any16 |= near;
  }
  if (any4) rule4<MODE>(K, F, x, T.V, a4, b4, acc);
  if (any16) rule16<MODE>(K, F, x, T.V, a16, b16, acc);
}

// warp sum of the 12 accumulators of point p into the warp's shared slot: the
// lanes' tree of pairs l, l ^ 16, l ^ 8, ... with each exchange halving the
// values a lane still carries (12, 6, 3, 2, 1: 26 shuffles in place of 120,
// beside about 300 other instructions of a far point: 11.3 -> 10.9 ms for 4,225
// points of a plane, N = 57,222)
__device__ __forceinline__ void warp_flush(double *acc, double (*slot)[12], int p, int lane) {
  double v[6], u[4], w[2];
#pragma unroll
  for (int q = 0; q < 6; q++) {
    const bool up = lane & 16;
    v[q] = (up ? acc[q + 6] : acc[q]) + __shfl_xor_sync(0xffffffffu, up ? acc[q] : acc[q + 6], 16);
  }
#pragma unroll
  for (int q = 0; q < 3; q++) {
    const bool up = lane & 8;
    u[q] = (up ? v[q + 3] : v[q]) + __shfl_xor_sync(0xffffffffu, up ? v[q] : v[q + 3], 8);
  }
  u[3] = 0.0;
#pragma unroll
  for (int q = 0; q < 2; q++) {
    const bool up = lane & 4;
    w[q] = (up ? u[q + 2] : u[q]) + __shfl_xor_sync(0xffffffffu, up ? u[q] : u[q + 2], 4);
  }
  const bool up = lane & 2;
  double r = (up ? w[1] : w[0]) + __shfl_xor_sync(0xffffffffu, up ? w[0] : w[1], 2);
  r += __shfl_xor_sync(0xffffffffu, r, 1);
  const int k = (lane >> 1) & 3;
  if (!(lane & 1) && k < 3) slot[p][6 * (lane >> 4) + 3 * ((lane >> 3) & 1) + k] = r;
}

template <int MODE, bool ONE>
__global__ void __launch_bounds__(FTHREADS, 3)
k_fields(const double *__restrict__ tetT, const double *__restrict__ tetF, const z *__restrict__ coef, int NT,
         int tpt, const double *__restrict__ X, int P, FieldK K, double *__restrict__ part) {
  __shared__ double sx[FPCH][3];
  __shared__ double sacc[FTHREADS / 32][FPCH][12];
  int p0 = blockIdx.x * FPCH, np = min(FPCH, P - p0);
  for (int i = threadIdx.x; i < 3 * np; i += FTHREADS) sx[i / 3][i % 3] = X[3 * p0 + i];
  __syncthreads();
  int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int tbase = blockIdx.y * FTHREADS * tpt + threadIdx.x;
  if (ONE) {
    // one tetrahedron per thread: its data stays in registers for all points
    bool live = tbase < NT;
    TetData T;
    if (live) load_tet(tetT, coef, tbase, T);
    for (int p = 0; p < np; p++) {
      double x[3] = {sx[p][0], sx[p][1], sx[p][2]};
      double acc[12];
#pragma unroll
      for (int q = 0; q < 12; q++) acc[q] = 0.0;
      if (live) tet_point<MODE>(K, x, T, tetF, coef, tbase, acc);
      warp_flush(acc, sacc[warp], p, lane);
    }
  } else {
    for (int p = 0; p < np; p++) {
      double x[3] = {sx[p][0], sx[p][1], sx[p][2]};
      double acc[12];
#pragma unroll
      for (int q = 0; q < 12; q++) acc[q] = 0.0;
      for (int j = 0; j < tpt; j++) {
        int t = tbase + j * FTHREADS;
        if (t >= NT) break;
        TetData T;
        load_tet(tetT, coef, t, T);
        tet_point<MODE>(K, x, T, tetF, coef, t, acc);
      }
      warp_flush(acc, sacc[warp], p, lane);
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 12 * np; i += FTHREADS) {
    int p = i / 12, q = i % 12;
    double s = 0.0;
#pragma unroll
    for (int w = 0; w < FTHREADS / 32; w++) s += sacc[w][p][q];
    part[((size_t)blockIdx.y * P + p0 + p) * 12 + q] = s;
  }
}

struct FieldInc { z E0[3]; double nh[3]; int on; };

__global__ void k_fields_finish(const double *__restrict__ part, int nblk, int P, const double *__restrict__ X,
                                FieldK K, z epre, FieldInc inc, z *out) {
  int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= P) return;
  double s[12];
  for (int q = 0; q < 12; q++) s[q] = 0.0;
  for (int b = 0; b < nblk; b++)
    for (int q = 0; q < 12; q++) s[q] += part[((size_t)b * P + p) * 12 + q];
  z F[6];
  const double inv4pi = 0.25 / M_PI;
  for (int c = 0; c < 3; c++) {
    F[c] = zmul(epre, z{s[2 * c], s[2 * c + 1]});
    F[3 + c] = z{inv4pi * s[6 + 2 * c], inv4pi * s[7 + 2 * c]};
  }
  if (inc.on) {
    double ph = inc.nh[0] * X[3 * p] + inc.nh[1] * X[3 * p + 1] + inc.nh[2] * X[3 * p + 2];
    double sn, cs;
    sincos(K.k.r * ph, &sn, &cs);
    double m = K.k.i == 0.0 ? 1.0 : exp(-K.k.i * ph);
    z e{m * cs, m * sn}, E[3];
    for (int c = 0; c < 3; c++) E[c] = zmul(inc.E0[c], e);
    const double *n = inc.nh;
    z H[3] = {{(n[1] * E[2].r - n[2] * E[1].r) / ZVAC_F, (n[1] * E[2].i - n[2] * E[1].i) / ZVAC_F},
              {(n[2] * E[0].r - n[0] * E[2].r) / ZVAC_F, (n[2] * E[0].i - n[0] * E[2].i) / ZVAC_F},
              {(n[0] * E[1].r - n[1] * E[0].r) / ZVAC_F, (n[0] * E[1].i - n[1] * E[0].i) / ZVAC_F}};
    for (int c = 0; c < 3; c++) {
      F[c].r += E[c].r; F[c].i += E[c].i;
      F[3 + c].r += H[c].r; F[3 + c].i += H[c].i;
    }
  }
  for (int c = 0; c < 6; c++) out[6 * (size_t)p + c] = F[c];
}

}  // namespace

// per-tetrahedron field tables, built on first use
static int field_tables(bg_geometry *g) {
  if (g->d_fieldTet && g->d_fieldFace) return BG_OK;
  double rmax = 0.0;      // largest distance of a vertex from its tetrahedron's centroid
  // Order of the tetrahedra: by place (bits of the centroid's grid coordinates
  // interleaved), so that the 32 of a warp are neighbours in space and take the
  // same rule for most points.  In mesh order (rows of cells) 24.6 of 32 lanes
  // were active on average, now 26.4: 10.9 -> 9.8 ms for 4,225 points of a plane,
  // N = 57,222.
  double lo[3] = {HUGE_VAL, HUGE_VAL, HUGE_VAL}, hi[3] = {-HUGE_VAL, -HUGE_VAL, -HUGE_VAL};
  for (const Object &o : g->objs)
    for (size_t i = 0; i < o.V.size(); i++) {
      lo[i % 3] = std::fmin(lo[i % 3], o.V[i]);
      hi[i % 3] = std::fmax(hi[i % 3], o.V[i]);
    }
  const double ext = std::fmax(std::fmax(hi[0] - lo[0], hi[1] - lo[1]), hi[2] - lo[2]);
  const double cells = ext > 0 ? 1023.0 / ext : 0.0;
  auto spread = [](uint64_t x) {      // 10 bits to every third place
    x = (x | x << 16) & 0x030000ff;
    x = (x | x << 8) & 0x0300f00f;
    x = (x | x << 4) & 0x030c30c3;
    return (x | x << 2) & 0x09249249;
  };
  std::vector<uint64_t> order;
  order.reserve(g->NT);
  std::vector<std::pair<const Object *, int>> where;
  where.reserve(g->NT);
  for (const Object &o : g->objs)
    for (int t = 0; t < o.nt; t++) {
      uint64_t key = 0;
      for (int c = 0; c < 3; c++) {
        double v = 0;
        for (int k = 0; k < 4; k++) v += 0.25 * o.V[3 * o.VI[4 * t + k] + c];
        key |= spread((uint64_t)std::fmin(1023.0, std::fmax(0.0, (v - lo[c]) * cells))) << c;
      }
      order.push_back(key << 32 | (uint64_t)where.size());
      where.push_back({&o, t});
    }
  std::sort(order.begin(), order.end());
  std::vector<double> T(16 * (size_t)g->NT + ((size_t)g->NT + 1) / 2), F(16 * (size_t)g->NT);
  int *idx = (int *)(T.data() + 16 * (size_t)g->NT);      // the order, behind the tables
  for (int i = 0; i < g->NT; i++) {
    idx[i] = (int)(uint32_t)order[i];
    const Object &o = *where[idx[i]].first;
    const int t = where[idx[i]].second;
    double *Ti = &T[16 * (size_t)i], *Fi = &F[16 * (size_t)i];
    double ctr[3] = {0, 0, 0};
    for (int k = 0; k < 4; k++)
      for (int c = 0; c < 3; c++) {
        double v = o.V[3 * o.VI[4 * t + k] + c];
        Ti[3 * k + c] = v;
        ctr[c] += 0.25 * v;
      }
    double Rall = 0.0;
    for (int k = 0; k < 4; k++) {
      const double *v = Ti + 3 * k;
      rmax = std::fmax(rmax, std::sqrt((v[0] - ctr[0]) * (v[0] - ctr[0]) + (v[1] - ctr[1]) * (v[1] - ctr[1]) +
                                       (v[2] - ctr[2]) * (v[2] - ctr[2])));
    }
    for (int k = 0; k < 4; k++) {
      int f = o.FI[4 * t + k];
      if (f >= 0 && f < o.nif) {
        const Face &Fc = o.F[f];
        double d = std::sqrt((Fc.cen[0] - ctr[0]) * (Fc.cen[0] - ctr[0]) + (Fc.cen[1] - ctr[1]) * (Fc.cen[1] - ctr[1]) +
                             (Fc.cen[2] - ctr[2]) * (Fc.cen[2] - ctr[2]));
        Rall = std::fmax(Rall, 10.0 * Fc.radius + d);
        Fi[4 * k] = Fc.cen[0];
        Fi[4 * k + 1] = Fc.cen[1];
        Fi[4 * k + 2] = Fc.cen[2];
        Fi[4 * k + 3] = Fc.radius;
      }
    }
    // margin so that rounding never calls a face far that the per-face test would not
    Rall = Rall * (1.0 + 1e-12) + 1e-300;
    for (int c = 0; c < 3; c++) Ti[12 + c] = ctr[c];
    Ti[15] = Rall;
  }
  double *dT = nullptr, *dF = nullptr;
  cudaError_t e = cudaMalloc(&dT, sizeof(double) * T.size());
  if (e == cudaSuccess) e = cudaMalloc(&dF, sizeof(double) * F.size());
  if (e == cudaSuccess) e = cudaMemcpy(dT, T.data(), sizeof(double) * T.size(), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(dF, F.data(), sizeof(double) * F.size(), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = uploads_done();
  if (e != cudaSuccess) {
    // both tables or neither: a failed build leaves the geometry as it was
    cudaFree(dT);
    cudaFree(dF);
    set_error("GetFields tables: %s", cudaGetErrorString(e));
    return BG_ERR_CUDA;
  }
  g->field_rmax = rmax;
  g->d_fieldTet = dT;
  g->d_fieldFace = dF;
  return BG_OK;
}

int get_fields(bg_geometry *g, double wr, double wi, const void *dJ, const double *E0, const double *nhat,
               int npts, const double *dX, void *dOut) {
  int st = upload_geometry(g);
  if (st || (st = init_rule16()) || (st = field_tables(g))) return st;
  if (npts == 0) return BG_OK;
  FieldK K;
  K.k = z{wr, wi};
  K.ik = z{-wi, wr};
  double d = wr * wr + wi * wi;
  K.invik = z{-wi / d, -wr / d};      // 1/(ik) = -i/k
  // i w Z0 / (4 pi)
  const double f = ZVAC_F * 0.25 / M_PI;
  z epre{-wi * f, wr * f};
  FieldInc inc{};
  if (E0 && nhat) {
    inc.on = 1;
    for (int c = 0; c < 3; c++) { inc.E0[c] = z{E0[2 * c], E0[2 * c + 1]}; inc.nh[c] = nhat[c]; }
  }
  int NT = g->NT;
  int ny = (npts + FPCH - 1) / FPCH, tpt = 1;
  int nbx = dJ ? (NT + FTHREADS - 1) / FTHREADS : 0;
  // one tetrahedron per thread (data in registers) while the partial sums
  // (96 bytes per tetrahedron block and point) stay under 256 MiB; beyond
  // that, longer tetrahedron blocks until the grid is about 8 blocks per SM,
  // which amortises the per-point warp reductions over many tetrahedra
  bool one = 96.0 * nbx * npts <= 268435456.0 && nbx <= 65535;
  while (!one && (nbx > 65535 || (nbx > 1 && (long)nbx * ny > 8L * 148))) {
    tpt *= 2;
    nbx = (NT + FTHREADS * tpt - 1) / (FTHREADS * tpt);
  }
  double *part = nullptr;
  z *coef = nullptr;
  if (nbx) {
    BG_CUDA_TRY(cudaMallocAsync(&part, sizeof(double) * 12 * (size_t)nbx * npts, stream()));
    cudaError_t e = cudaMallocAsync(&coef, sizeof(z) * 4 * (size_t)NT, stream());
    if (e != cudaSuccess) {
      cudaFreeAsync(part, stream());
      set_error("GetFields scratch: %s", cudaGetErrorString(e));
      return BG_ERR_CUDA;
    }
    k_fields_coef<<<(NT + 255) / 256, 256, 0, stream()>>>(
        g->dev, (const int *)(g->d_fieldTet + 16 * (size_t)NT), (const z *)dJ, coef);
    BG_LAUNCHED();
    dim3 grid(ny, nbx);
    // the largest |k| |y - centroid| of any quadrature point (see field_point)
    const double span = std::fabs(wr) * g->field_rmax;
    const int mode = wi != 0.0 ? 3 : (span <= 0.25 ? 2 : (span <= 1.0 ? 1 : 0));
    auto kern = mode == 3 ? (one ? k_fields<3, true> : k_fields<3, false>)
              : mode == 2 ? (one ? k_fields<2, true> : k_fields<2, false>)
              : mode == 1 ? (one ? k_fields<1, true> : k_fields<1, false>)
                          : (one ? k_fields<0, true> : k_fields<0, false>);
    kern<<<grid, FTHREADS, 0, stream()>>>(g->d_fieldTet, g->d_fieldFace, coef, NT, tpt, dX, npts, K, part);
    BG_LAUNCHED();
  }
  k_fields_finish<<<(npts + 127) / 128, 128, 0, stream()>>>(part, nbx, npts, dX, K, epre, inc, (z *)dOut);
  BG_LAUNCHED();
  if (part) cudaFreeAsync(part, stream());
  if (coef) cudaFreeAsync(coef, stream());
  return BG_OK;
}

}  // namespace bg
