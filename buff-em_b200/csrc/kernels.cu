// sm_100a kernels of the VIE assembly path: far-field G entries, the
// frequency-independent near-field integrals (regular 16x16 rule and the
// singular relative-coordinate rule, both as tetrahedron-pair moments), the
// per-frequency near entries, V^-1 Gram blocks, plane-wave RHS and the
// absorbed/scattered power (EMT and overlap).
//
// Reference semantics (HomerReid/buff-em, src/libs/libbuff):
//   GMatrixElements.cc:59-167,270-424   kernels and dispatcher
//   Cubature.cc:161-527, TetCR.cc:35-95 fixed tetrahedron rules
//   VIEMatrix.cc:51-72,122-316,321-460  Gram blocks and assembly
//   RHSVector.cc:62-124                 plane-wave RHS
//   EMTPFT.cc:151-493, OPFT.cc:62-119   power
#include <cuda_runtime.h>

#include <cmath>
#include <cstdio>
#include <vector>

#include "devmath.cuh"
#include "internal.h"

namespace bg {

// ----------------------------------------------------------------- tables
// Fixed tetrahedron rules (TetCR.cc:35-95): points (u1,u2,u3) in the unit
// simplex, weights summing to 1/6.  All orbits are complete, so the point set
// does not depend on which vertex is taken as origin.
__constant__ double c_tcr16[64];
__constant__ double c_tcr33[132];
static double h_tcr16[64], h_tcr33[132];
static int s_tables_ok = 0;

static void fill_rule(double *dst, const char *pat, const double *vals, double w, int *np) {
  for (const char *p = pat; *p;) {
    if (*p == ' ') { p++; continue; }
    double *q = dst + 4 * (*np);
    q[0] = vals[p[0] - 'A']; q[1] = vals[p[1] - 'A']; q[2] = vals[p[2] - 'A']; q[3] = w;
    (*np)++;
    p += 3;
  }
}

static int init_tables() {
  if (s_tables_ok) return BG_OK;
  int np;
  const double v16[5] = {0.771642902067237, 0.076119032644254315, 0.07183164526766925, 0.11970052779780202,
                         0.40423391346726440};
  np = 0;
  fill_rule(h_tcr16, "ABB BAB BBA BBB", v16, 8.3956323500204695e-3, &np);
  fill_rule(h_tcr16, "CDE CED CEE DCE DEC DEE ECD ECE EDC EDE EEC EED", v16, 0.011090344772215399, &np);
  const double v33[11] = {0.25, 0.31407428362944793, 0.05777714911165610, 0.06254680497480394,
                          0.81235958507558810, 0.04120213879937276, 0.30021473119185615, 0.61738099120939840,
                          0.05292032110257111, 0.25198057383388334, 0.44311853122966216};
  np = 0;
  fill_rule(h_tcr33, "AAA", v33, 0.017783308938202055, &np);
  fill_rule(h_tcr33, "BBB CBB BCB BBC", v33, -0.019099406118263309, &np);
  fill_rule(h_tcr33, "DDD EDD DED DDE", v33, 3.8252276536630236e-3, &np);
  fill_rule(h_tcr33, "FFG FFH FGF FGH FHF FHG GFF GFH GHF HFF HFG HGF", v33, 0.0035475499144103266, &np);
  fill_rule(h_tcr33, "IJJ IJK IKJ JIJ JIK JJI JJK JKI JKJ KIJ KJI KJJ", v33, 0.013950789384495153, &np);
  BG_CUDA_TRY(cudaMemcpyToSymbol(c_tcr16, h_tcr16, sizeof h_tcr16));
  BG_CUDA_TRY(cudaMemcpyToSymbol(c_tcr33, h_tcr33, sizeof h_tcr33));
  BG_CUDA_TRY(uploads_done());
  s_tables_ok = 1;
  return BG_OK;
}

void gauss_legendre01(int n, double *x, double *w) {
  for (int i = 0; i < n; i++) {
    double z = std::cos(M_PI * (i + 0.75) / (n + 0.5)), pp = 0.0;
    for (int it = 0; it < 100; it++) {
      double p1 = 1.0, p2 = 0.0;
      for (int j = 1; j <= n; j++) {
        double p3 = p2;
        p2 = p1;
        p1 = ((2.0 * j - 1.0) * z * p2 - (j - 1.0) * p3) / j;
      }
      pp = n * (z * p1 - p2) / (z * z - 1.0);
      double z1 = z;
      z = z1 - p1 / pp;
      if (std::fabs(z - z1) < 1e-16) break;
    }
    x[i] = 0.5 * (1.0 - z);
    w[i] = 1.0 / ((1.0 - z * z) * pp * pp);
  }
}

// ----------------------------------------------------------------- complex
struct cd { double r, i; };
__device__ __forceinline__ cd cmk(double r, double i) { return cd{r, i}; }
__device__ __forceinline__ cd cadd(cd a, cd b) { return cd{a.r + b.r, a.i + b.i}; }
__device__ __forceinline__ cd csub(cd a, cd b) { return cd{a.r - b.r, a.i - b.i}; }
__device__ __forceinline__ cd cmul(cd a, cd b) { return cd{a.r * b.r - a.i * b.i, a.r * b.i + a.i * b.r}; }
__device__ __forceinline__ cd cscale(cd a, double s) { return cd{a.r * s, a.i * s}; }
__device__ __forceinline__ cd cdiv(cd a, cd b) {
  double d = b.r * b.r + b.i * b.i;
  return cd{(a.r * b.r + a.i * b.i) / d, (a.i * b.r - a.r * b.i) / d};
}
__device__ __forceinline__ double cnorm2(cd a) { return a.r * a.r + a.i * a.i; }
// exp(i k r) for complex k
__device__ __forceinline__ cd expikr(cd k, double r) {
  double s, c;
  sincos(k.r * r, &s, &c);
  double m = (k.i == 0.0) ? 1.0 : exp(-k.i * r);
  return cd{m * c, m * s};
}

__device__ __forceinline__ cd expi_small(double x) {
  cd e;
  cossin_small(x, e.r, e.i);
  return e;
}
__device__ __forceinline__ cd expi_small_short(double x) {
  cd e;
  cossin_small_short(x, e.r, e.i);
  return e;
}

// e^x - 1 - x - x^2/2: GetExpRelTable(x,3,3), GMatrixElements.cc:59-93 -- the
// series from n=4 is stopped once |term|^2 < 1e-16 |sum|^2 (or n = 100).
__device__ __forceinline__ cd exprel3(cd x) {
  cd term = cmul(cscale(x, 0.5), x);   // x^2/2
  term = cmul(term, cscale(x, 1.0 / 3.0));
  cd first = term, sum = cmk(0, 0);
  for (int n = 4; n < 100; n++) {
    term = cmul(term, cscale(x, 1.0 / n));
    sum = cadd(sum, term);
    if (cnorm2(term) < 1.0e-16 * cnorm2(sum)) break;
  }
  return cadd(first, sum);
}

// complex functions of the SVTENSOR programs, from their definitions in
// terms of the real exp, log, sincos, sinh, cosh, sqrt, hypot and atan2
__device__ cd cx_exp(cd z) {
  double s, c, e = exp(z.r);
  sincos(z.i, &s, &c);
  return cd{e * c, e * s};
}
__device__ cd cx_log(cd z) { return cd{log(hypot(z.r, z.i)), atan2(z.i, z.r)}; }
__device__ cd cx_sqrt(cd z) {   // principal branch
  double r = hypot(z.r, z.i);
  if (r == 0.0) return cd{0.0, 0.0};
  if (z.r >= 0.0) {
    double t = sqrt(0.5 * (r + z.r));
    return cd{t, z.i / (2.0 * t)};
  }
  double t = sqrt(0.5 * (r - z.r));
  return cd{fabs(z.i) / (2.0 * t), copysign(t, z.i)};
}
__device__ cd cx_sin(cd z) {
  double s, c;
  sincos(z.r, &s, &c);
  return cd{s * cosh(z.i), c * sinh(z.i)};
}
__device__ cd cx_cos(cd z) {
  double s, c;
  sincos(z.r, &s, &c);
  return cd{c * cosh(z.i), -s * sinh(z.i)};
}
__device__ cd cx_sinh(cd z) {
  double s, c;
  sincos(z.i, &s, &c);
  return cd{sinh(z.r) * c, cosh(z.r) * s};
}
__device__ cd cx_cosh(cd z) {
  double s, c;
  sincos(z.i, &s, &c);
  return cd{cosh(z.r) * c, sinh(z.r) * s};
}
// asin z = -i log(iz + sqrt(1 - z^2)), acos z = pi/2 - asin z,
// atan z = (i/2) [log(1 - iz) - log(1 + iz)]
__device__ cd cx_asin(cd z) {
  cd w = cx_log(cadd(cd{-z.i, z.r}, cx_sqrt(csub(cd{1.0, 0.0}, cmul(z, z)))));
  return cd{w.i, -w.r};
}
__device__ cd cx_atan(cd z) {
  cd a = cx_log(cd{1.0 + z.i, -z.r}), b = cx_log(cd{1.0 - z.i, z.r});
  cd d = csub(a, b);
  return cd{-0.5 * d.i, 0.5 * d.r};
}
__device__ cd cx_pow(cd x, cd y) {
  // integer powers by repeated squaring, as the host evaluator (matprop.cpp)
  if (y.i == 0.0 && y.r == floor(y.r) && fabs(y.r) <= 64.0) {
    long n = (long)y.r;
    bool inv = n < 0;
    unsigned long m = inv ? (unsigned long)(-n) : (unsigned long)n;
    cd r{1.0, 0.0};
    while (m) {
      if (m & 1) r = cmul(r, x);
      x = cmul(x, x);
      m >>= 1;
    }
    return inv ? cdiv(cd{1.0, 0.0}, r) : r;
  }
  return cx_exp(cmul(y, cx_log(x)));
}

// one component program of a compiled SVTENSOR (DevExpr) at point x
__device__ cd expr_eval(const DevExpr &e, int comp, const double *x) {
  cd st[BG_EXPR_STACK];
  int sp = 0;
  const int b = e.start[comp], n = e.len[comp];
  for (int k = 0; k < n; k++) {
    const int w = e.op[b + k], code = w >> 16, arg = w & 0xffff;
    switch (code) {
      case 0: st[sp++] = cd{e.con[2 * arg], e.con[2 * arg + 1]}; break;
      case 1: {
        double v;
        if (arg < 3) v = x[arg];
        else if (arg == 3) v = sqrt(x[0] * x[0] + x[1] * x[1] + x[2] * x[2]);
        else if (arg == 4) v = atan2(sqrt(x[0] * x[0] + x[1] * x[1]), x[2]);
        else v = atan2(x[1], x[0]);
        st[sp++] = cd{v, 0.0};
        break;
      }
      case 2: st[sp - 1] = csub(cd{0.0, 0.0}, st[sp - 1]); break;
      case 8: {
        cd a = st[sp - 1], r;
        switch (arg) {
          case 0: r = cx_exp(a); break;
          case 1: r = cx_log(a); break;
          case 2: r = cx_sqrt(a); break;
          case 3: r = cx_sin(a); break;
          case 4: r = cx_cos(a); break;
          case 5: r = cdiv(cx_sin(a), cx_cos(a)); break;
          case 6: r = cx_sinh(a); break;
          case 7: r = cx_cosh(a); break;
          case 8: r = cdiv(cx_sinh(a), cx_cosh(a)); break;
          case 9: r = cx_asin(a); break;
          case 10: r = csub(cd{0.5 * M_PI, 0.0}, cx_asin(a)); break;
          case 11: r = cx_atan(a); break;
          case 12: r = cd{hypot(a.r, a.i), 0.0}; break;
          default: r = cd{a.r < 0.0 ? 0.0 : 1.0, 0.0}; break;
        }
        st[sp - 1] = r;
        break;
      }
      default: {
        cd bb = st[--sp], aa = st[sp - 1];
        st[sp - 1] = code == 3 ? cadd(aa, bb) : code == 4 ? csub(aa, bb) : code == 5 ? cmul(aa, bb)
                   : code == 6 ? cdiv(aa, bb) : cx_pow(aa, bb);
        break;
      }
    }
  }
  return st[0];
}

// permittivity functor (SVTensor::Evaluate semantics, SVTensor.cc:306-373);
// ex: the object's compiled program when m.kind == BG_MAT_EXPR
__device__ __noinline__ void mat_eval_expr(const DevExpr *ex, const double *x, cd E[3][3]) {
  // components not given keep the identity, off-diagonal pairs are
  // averaged, yy and zz follow xx when only xx is given (SVTensor.cc:344-372)
  for (int i = 0; i < 3; i++)
    for (int j = 0; j < 3; j++)
      E[i][j] = ex->len[3 * i + j] ? expr_eval(*ex, 3 * i + j, x) : cmk(i == j ? 1.0 : 0.0, 0.0);
  for (int mu = 0; mu < 3; mu++) {
    int nu = (mu + 1) % 3;
    cd a = cscale(cadd(E[mu][nu], E[nu][mu]), 0.5);
    E[mu][nu] = E[nu][mu] = a;
  }
  if (ex->len[0]) {
    if (!ex->len[4]) E[1][1] = E[0][0];
    if (!ex->len[8]) E[2][2] = E[0][0];
  }
}
// the fixed functors inline: a kernel calls out for compiled programs only
__device__ __forceinline__ void mat_eval(const bg_material &m, const DevExpr *ex, const double *x, cd E[3][3]) {
  if (m.kind == BG_MAT_EXPR) {
    cd T[3][3];
    mat_eval_expr(ex, x, T);
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int j = 0; j < 3; j++) E[i][j] = T[i][j];
    return;
  }
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) E[i][j] = cmk(0, 0);
  if (m.kind == BG_MAT_CONST_TENSOR) {
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int j = 0; j < 3; j++) E[i][j] = cmk(m.eps[2 * (3 * i + j)], m.eps[2 * (3 * i + j) + 1]);
#pragma unroll
    for (int mu = 0; mu < 3; mu++) {
      int nu = (mu + 1) % 3;
      cd a = cscale(cadd(E[mu][nu], E[nu][mu]), 0.5);
      E[mu][nu] = E[nu][mu] = a;
    }
    return;
  }
  cd e;
  if (m.kind == BG_MAT_CONST_ISO) e = cmk(m.eps[0], m.eps[1]);
  else if (m.kind == BG_MAT_JANUS_Z) e = (x[2] > m.center[2]) ? cmk(m.eps[0], m.eps[1]) : cmk(m.eps2[0], m.eps2[1]);
  else {
    double d0 = x[0] - m.center[0], d1 = x[1] - m.center[1], d2 = x[2] - m.center[2];
    double r2 = (d0 * d0 + d1 * d1 + d2 * d2) / (m.width * m.width);
    double g = exp(-r2);
    e = cmk(m.eps[0] + m.amp[0] * g, m.eps[1] + m.amp[1] * g);
  }
  E[0][0] = E[1][1] = E[2][2] = e;
}

// Invert3x3Matrix, VIEMatrix.cc:51-72
__device__ __forceinline__ void inv3(cd M[3][3], cd W[3][3]) {
  cd M11 = M[0][0], M12 = M[0][1], M13 = M[0][2];
  cd M21 = M[1][0], M22 = M[1][1], M23 = M[1][2];
  cd M31 = M[2][0], M32 = M[2][1], M33 = M[2][2];
  cd Det = csub(csub(csub(cadd(cadd(cmul(cmul(M12, M23), M31), cmul(cmul(M13, M21), M32)), cmul(cmul(M11, M22), M33)),
                          cmul(cmul(M13, M22), M31)),
                     cmul(cmul(M11, M23), M32)),
                cmul(cmul(M12, M21), M33));
  W[0][0] = cdiv(csub(cmul(M22, M33), cmul(M23, M32)), Det);
  W[0][1] = cdiv(csub(cmul(M13, M32), cmul(M12, M33)), Det);
  W[0][2] = cdiv(csub(cmul(M12, M23), cmul(M13, M22)), Det);
  W[1][0] = cdiv(csub(cmul(M23, M31), cmul(M21, M33)), Det);
  W[1][1] = cdiv(csub(cmul(M11, M33), cmul(M13, M31)), Det);
  W[1][2] = cdiv(csub(cmul(M13, M21), cmul(M11, M23)), Det);
  W[2][0] = cdiv(csub(cmul(M21, M32), cmul(M22, M31)), Det);
  W[2][1] = cdiv(csub(cmul(M12, M31), cmul(M11, M32)), Det);
  W[2][2] = cdiv(csub(cmul(M11, M22), cmul(M12, M21)), Det);
}

__device__ __forceinline__ void load3(const double *V4, int v, double *x) {
  x[0] = V4[4 * v]; x[1] = V4[4 * v + 1]; x[2] = V4[4 * v + 2];
}

__device__ __forceinline__ double warp_sum(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// =========================================================================
// far field (GetGME_BFBFInt, GMatrixElements.cc:270-288; BFBFInt,
// Cubature.cc:476-527): for a basis-function pair (a, b) with no common
// vertex, 4 tetrahedron pairs x 4x4 points of the Helmholtz kernel.  With
// w = 6V w_i (w_i = 1/24) and b = +-A/(3V)(x - Q) the volume cancels:
//   w_a b_a . w_b b_b = s_a s_b A_a A_b (x-Q_a).(y-Q_b)/144,
//   w_a Div b_a w_b Div b_b = s_a s_b A_a A_b / 16,
// so with x~ = x - o_A, y~ = y - o_B (o = tetrahedron centroid) and
// q = Q - o each tetrahedron pair contributes through 8 complex moments of
// phi = exp(ikr)/(4 pi r):
//   M0 = sum phi, M1 = sum x~ phi, M1' = sum y~ phi, M2 = sum x~.y~ phi,
//   entry += s s' A A' [M2/144 - M0/(16k^2) - q'.M1/144 - q.M1'/144 + q.q' M0/144].
// The moments depend on the two tetrahedra only, and a tile of 32
// consecutive basis functions touches about 29 distinct tetrahedra (face
// numbering follows the mesh), so a CTA computes each distinct tetrahedron
// pair of its 32 x 32 tile once (about 850 instead of 4096 pairs of 16
// kernel evaluations).  The thread that computes a pair's 8 moments forms,
// while they are in registers, the terms of every basis-function pair of
// the tile that uses it (side sa of row ra on tetrahedron iA, side sb of
// column rb on tetrahedron jB: term slot (ra, rb, 2 sa + sb), written by
// exactly one thread); after one barrier each basis-function pair adds its
// four slots in a fixed order.
// Phase: for real k, exp(ikr) = exp(ik rc) exp(ik (r - rc)) with rc the
// centroid distance and |r - rc| <= rA + rB (triangle inequality, rA the
// largest distance of a rule point from its centroid); when |k| (rA + rB)
// <= 1 the second factor is a short Taylor series (expi_small), so one
// sincos serves the 16 point pairs.
// =========================================================================
#define FT 16        // PFT tiles (k_pft_far): 16 x 16 basis functions
#define FTF BG_FAR_TILE
#define FTT BG_FAR_TILE_TETS
#define FTHR 256     // threads of the far kernel
#define FPS 13       // doubles per staged tetrahedron (odd: conflict-free 8-byte reads)

struct FarSmem {
  // term (sa, sb) of the basis-function pair (row ra, column rb) of the tile:
  // a plane per (sa, sb), rows padded, so that the lanes of a warp (columns
  // rb running) store to different banks
  double2 slot[4][FTF][FTF + 1];
  double pA[FTT][FPS], pB[FTT][FPS];   // 4 points x 3, padded: lanes read different tetrahedra
  double oA[FTT][3], oB[FTT][3];
  double rA[FTT], rB[FTT];      // largest distance of a rule point from its centroid
  double uA[FTF][2][4], uB[FTF][2][4];   // s A (1, Q - o) per side
  int lA[FTF][2], lB[FTF][2];            // tile-local tetrahedron of each side, -1 past N
  int vA[FTF][5], vB[FTF][5];
  unsigned char sA[FTT][4], sB[FTT][4];  // sides on each tetrahedron: row << 1 | side
  int nsA[FTT], nsB[FTT];
};

// Frequency-parameterised launches: when fq (device, {Re w, Im w}) is
// given, the kernels below read omega from it instead of their by-value
// arguments, so that one captured CUDA graph serves every frequency.
__device__ __forceinline__ cd dev_invk2(double wr, double wi) {
  double d = (wr * wr - wi * wi) * (wr * wr - wi * wi) + 4 * wr * wr * wi * wi;
  return cd{(wr * wr - wi * wi) / d, -2 * wr * wi / d};
}

__device__ void far_stage_tets(const DevGeom &g, int tile, double (*P)[FPS], int tid) {
  int nt = g.tileNT[tile];
  for (int e = tid; e < nt * 12; e += FTHR) {
    int t = e / 12, r = e % 12;
    int tet = g.tileTet[(size_t)tile * FTT + t];
    P[t][r] = g.tetP4[16 * (size_t)tet + 4 * (r / 3) + (r % 3)];
  }
}

__device__ void far_stage_bfs(const DevGeom &g, int tile, double (*P)[FPS], double (*u)[2][4], int (*l)[2],
                              int (*v)[5], int tid) {
  if (tid < 2 * FTF) {
    int r = tid >> 1, s = tid & 1;
    int bf = tile * FTF + r;
    l[r][s] = -1;
    if (bf < g.N) {
      int2 loc = g.bfTileLoc[bf];
      int lt = s == 0 ? loc.x : loc.y;
      int2 qq = g.bfQ[bf];
      double Q[3];
      load3(g.V4, s == 0 ? qq.x : qq.y, Q);
      double coef = (s == 0 ? 1.0 : -1.0) * g.bfArea[bf];
      u[r][s][0] = coef;
      for (int c = 0; c < 3; c++) {
        double o = 0.25 * (P[lt][c] + P[lt][3 + c] + P[lt][6 + c] + P[lt][9 + c]);
        u[r][s][1 + c] = coef * (Q[c] - o);
      }
      l[r][s] = lt;
      if (s == 0) {
        int4 vv = g.bfV[bf];
        v[r][0] = qq.x; v[r][1] = vv.x; v[r][2] = vv.y; v[r][3] = vv.z; v[r][4] = qq.y;
      }
    }
  }
}

// centroid, point radius and the sides resting on tetrahedron t of a tile
__device__ void far_stage_tet_info(int t, const double (*P)[FPS], double (*o)[3], double *rad, const int (*l)[2],
                                   unsigned char (*sides)[4], int *ns) {
  for (int c = 0; c < 3; c++) o[t][c] = 0.25 * (P[t][c] + P[t][3 + c] + P[t][6 + c] + P[t][9 + c]);
  double r2 = 0.0;
  for (int i = 0; i < 4; i++) {
    double a2 = 0.0;
    for (int c = 0; c < 3; c++) {
      double d = P[t][3 * i + c] - o[t][c];
      a2 += d * d;
    }
    r2 = fmax(r2, a2);
  }
  rad[t] = sqrt(r2);
  int n = 0;
  for (int r = 0; r < FTF; r++)
    for (int s = 0; s < 2; s++)
      if (l[r][s] == t && n < 4) sides[t][n++] = (unsigned char)(r << 1 | s);
  ns[t] = n;
}

// The 8 moments of one tetrahedron pair (1/(4 pi) included): row points pA
// about oA, column points pB about oB.  MODE as in k_far, without 3.  No
// branch per point (coincident points, r < 1e-12, get factor 0), so the four
// columns of a row are in flight together.  FP64-pipe bound (54 % active, the
// rest barriers of the tile's four rounds and shared-memory latency): 24.6 ->
// 17.7 ms at N = 19,872, 100 -> 73 ms at N = 39,150 (with the term
// factorisation and the padded shared layouts of k_far).
template <int MODE>
__device__ __forceinline__ void far_moments(cd k, const double *pA, const double *oA, const double *pB,
                                            const double *oB, cd m[8]) {
  const double inv4pi = 0.25 / M_PI;
#pragma unroll
  for (int q = 0; q < 8; q++) m[q] = cmk(0, 0);
  const double e0 = oA[0] - oB[0], e1 = oA[1] - oB[1], e2 = oA[2] - oB[2];
  const double rc = sqrt(e0 * e0 + e1 * e1 + e2 * e2);
  // exp(ikr) = exp(ik rc) e: the first factor is common to all points and
  // multiplies the moments at the end
  const cd ec = MODE ? cscale(expikr(k, rc), inv4pi) : cmk(inv4pi, 0.0);
  const double krc = k.r * rc;
  double yt[4][3];
#pragma unroll
  for (int j = 0; j < 4; j++)
#pragma unroll
    for (int c = 0; c < 3; c++) yt[j][c] = pB[3 * j + c] - oB[c];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const double x0 = pA[3 * i] - oA[0], x1 = pA[3 * i + 1] - oA[1], x2 = pA[3 * i + 2] - oA[2];
    // x - y from the points themselves: differences of the centroid-relative
    // coordinates would add two roundings to every distance
    const double z0 = pA[3 * i], z1 = pA[3 * i + 1], z2 = pA[3 * i + 2];
    cd ph = cmk(0, 0), W[3] = {cmk(0, 0), cmk(0, 0), cmk(0, 0)};   // sums over the columns: phi, phi y~
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const double R0 = z0 - pB[3 * j], R1 = z1 - pB[3 * j + 1], R2 = z2 - pB[3 * j + 2];
      const double r2 = fma(R0, R0, fma(R1, R1, R2 * R2));
      const double ir = r2 < 1.0e-24 ? 0.0 : rsqrt_fast(r2), r = r2 * ir;
      const cd e = MODE == 2 ? expi_small_short(fma(k.r, r, -krc))
                             : (MODE == 1 ? expi_small(fma(k.r, r, -krc)) : expikr(k, r));
      const cd phi = cscale(e, ir);
      ph = cadd(ph, phi);
#pragma unroll
      for (int c = 0; c < 3; c++) W[c] = cmk(fma(phi.r, yt[j][c], W[c].r), fma(phi.i, yt[j][c], W[c].i));
    }
    m[0] = cadd(m[0], ph);
    m[1] = cadd(m[1], cscale(ph, x0));
    m[2] = cadd(m[2], cscale(ph, x1));
    m[3] = cadd(m[3], cscale(ph, x2));
#pragma unroll
    for (int c = 0; c < 3; c++) m[4 + c] = cadd(m[4 + c], W[c]);
    m[7] = cmk(fma(W[0].r, x0, fma(W[1].r, x1, fma(W[2].r, x2, m[7].r))),
               fma(W[0].i, x0, fma(W[1].i, x1, fma(W[2].i, x2, m[7].i))));
  }
#pragma unroll
  for (int q = 0; q < 8; q++) m[q] = MODE ? cmul(ec, m[q]) : cscale(m[q], inv4pi);
}

// one CTA per 32 x 32 tile of basis-function pairs (upper triangle of tiles).
// MODE, the phase of exp(ikr) per point pair, fixed per launch so that one
// code path is compiled into each instantiation: 2 = ec * (short series)
// (|k| (rA + rB) <= 1/4 for every pair of the mesh), 1 = ec * (series)
// (<= 1), 0 = sincos per point pair (complex k or coarse pairs), 3 = chosen
// per tetrahedron pair (launches that read omega from device memory, whose
// frequency the host does not know when it launches them).
template <int MODE>
__global__ void __launch_bounds__(FTHR, 2) k_far(DevGeom g, cd k, cd invk2, cd *M, size_t ld, const double *fq,
                                                  float2 *F, size_t ldf) {
  if (fq) {
    k = cd{fq[0], fq[1]};
    invk2 = dev_invk2(fq[0], fq[1]);
  }
  int bx = blockIdx.x, by = blockIdx.y;
  if (bx > by) return;
  extern __shared__ __align__(16) unsigned char far_smem_raw[];
  FarSmem &S = *reinterpret_cast<FarSmem *>(far_smem_raw);
  const int tid = threadIdx.x;
  const int nA = g.tileNT[bx], nB = g.tileNT[by];
  far_stage_tets(g, bx, S.pA, tid);
  far_stage_tets(g, by, S.pB, tid);
  __syncthreads();
  far_stage_bfs(g, bx, S.pA, S.uA, S.lA, S.vA, tid);
  far_stage_bfs(g, by, S.pB, S.uB, S.lB, S.vB, tid);
  __syncthreads();
  if (tid < FTT) {
    if (tid < nA) far_stage_tet_info(tid, S.pA, S.oA, S.rA, S.lA, S.sA, S.nsA);
  } else if (tid < 2 * FTT) {
    if (tid - FTT < nB) far_stage_tet_info(tid - FTT, S.pB, S.oB, S.rB, S.lB, S.sB, S.nsB);
  }
  __syncthreads();
  for (int p = tid; p < nA * nB; p += FTHR) {
    const int iA = p / nB, tB = p - iA * nB;
    cd m[8];
    if (MODE != 3) {
      far_moments<MODE == 3 ? 0 : MODE>(k, S.pA[iA], S.oA[iA], S.pB[tB], S.oB[tB], m);
    } else {
      // phase about the centroid distance (see above): short series, series or
      // sincos per point pair, by the span of this pair
      const double span = fabs(k.r) * (S.rA[iA] + S.rB[tB]);
      if (k.i != 0.0 || span > 1.0) far_moments<0>(k, S.pA[iA], S.oA[iA], S.pB[tB], S.oB[tB], m);
      else if (span > 0.25) far_moments<1>(k, S.pA[iA], S.oA[iA], S.pB[tB], S.oB[tB], m);
      else far_moments<2>(k, S.pA[iA], S.oA[iA], S.pB[tB], S.oB[tB], m);
    }
    // terms of the basis-function pairs on (iA, tB):
    //   s s' A A' [M2/144 - M0/(16 k^2) - q'.M1/144 - q.M1'/144 + q.q' M0/144]
    // = u0 c + u.g - u0 v0 M0/(16 k^2) with, per column side,
    // c = (v0 M2 - v.M1)/144 and g = (v M0 - v0 M1')/144.  The last term is
    // the largest and cancels between the four tetrahedron pairs of a
    // basis-function pair, so it is added once, at the end.
    const cd kM0 = cscale(cmul(invk2, m[0]), 1.0 / 16.0);
#pragma unroll
    for (int q = 0; q < 8; q++) m[q] = cscale(m[q], 1.0 / 144.0);
    const int na = S.nsA[iA], nb = S.nsB[tB];
    for (int ib = 0; ib < nb; ib++) {
      const int cb = S.sB[tB][ib], rb = cb >> 1, sb = cb & 1;
      const double *v = S.uB[rb][sb];
      const double v0 = v[0], v1 = v[1], v2 = v[2], v3 = v[3];
      cd c = cscale(m[7], v0), gv[3];
      c = cmk(fma(-v1, m[1].r, fma(-v2, m[2].r, fma(-v3, m[3].r, c.r))),
              fma(-v1, m[1].i, fma(-v2, m[2].i, fma(-v3, m[3].i, c.i))));
      gv[0] = cmk(fma(v1, m[0].r, -v0 * m[4].r), fma(v1, m[0].i, -v0 * m[4].i));
      gv[1] = cmk(fma(v2, m[0].r, -v0 * m[5].r), fma(v2, m[0].i, -v0 * m[5].i));
      gv[2] = cmk(fma(v3, m[0].r, -v0 * m[6].r), fma(v3, m[0].i, -v0 * m[6].i));
      for (int ia = 0; ia < na; ia++) {
        const int ca = S.sA[iA][ia], ra = ca >> 1, sa = ca & 1;
        const double *u = S.uA[ra][sa];
        const double u0 = u[0], u1 = u[1], u2 = u[2], u3 = u[3];
        const double uv = u0 * v0;
        const double tr = fma(u0, c.r, fma(u1, gv[0].r, fma(u2, gv[1].r, u3 * gv[2].r)));
        const double ti = fma(u0, c.i, fma(u1, gv[0].i, fma(u2, gv[1].i, u3 * gv[2].i)));
        S.slot[2 * sa + sb][ra][rb] = make_double2(fma(-uv, kM0.r, tr), fma(-uv, kM0.i, ti));
      }
    }
  }
  __syncthreads();
  // this thread's 2 x 2 basis-function pairs: rows tx, tx + 16; columns ty, ty + 16
  const int tx = tid & 15, ty = tid >> 4;
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int j = 0; j < 2; j++) {
      int ra = tx + 16 * i, rb = ty + 16 * j;
      int a = bx * FTF + ra, b = by * FTF + rb;
      if (!(a < g.N && b < g.N && a <= b)) continue;
      // CompareBFs (SWGVolume.cc:295-344): pairs with a common vertex are near
      int ncv = 0;
      for (int p = 0; p < 5; p++)
        for (int q = 0; q < 5; q++) ncv += (S.vA[ra][p] == S.vB[rb][q]);
      if (ncv) continue;
      const double2 s0 = S.slot[0][ra][rb], s1 = S.slot[1][ra][rb], s2 = S.slot[2][ra][rb], s3 = S.slot[3][ra][rb];
      const cd v = cmk(s0.x + s1.x + s2.x + s3.x, s0.y + s1.y + s2.y + s3.y);
      M[(size_t)a + (size_t)b * ld] = v;
      if (a != b) M[(size_t)b + (size_t)a * ld] = v;
      if (F) {   // the complex64 copy, as k_c128_to_c64 would convert it
        const float2 f = make_float2((float)v.r, (float)v.i);
        F[(size_t)a + (size_t)b * ldf] = f;
        if (a != b) F[(size_t)b + (size_t)a * ldf] = f;
      }
    }
}

int assemble_far(bg_geometry *g, double wr, double wi, void *M, size_t ld, const double *fq, void *F, size_t ldf) {
  int st = init_tables();
  if (st) return st;
  cd k{wr, wi};
  // 1/k^2
  double d = (wr * wr - wi * wi) * (wr * wr - wi * wi) + 4 * wr * wr * wi * wi;
  cd invk2{(wr * wr - wi * wi) / d, -2 * wr * wi / d};
  int nb = (g->N + FTF - 1) / FTF;
  dim3 grid(nb, nb);
  static bool attr = false;
  if (!attr) {
    const int sm = (int)sizeof(FarSmem);
    BG_CUDA_TRY(cudaFuncSetAttribute(k_far<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm));
    BG_CUDA_TRY(cudaFuncSetAttribute(k_far<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm));
    BG_CUDA_TRY(cudaFuncSetAttribute(k_far<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm));
    BG_CUDA_TRY(cudaFuncSetAttribute(k_far<3>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm));
    attr = true;
  }
  // the largest phase span |k| (rA + rB) of any tetrahedron pair of the mesh
  const double span = std::fabs(wr) * 2.0 * g->rule_rmax;
  const int mode = fq ? 3 : (wi != 0.0 ? 0 : (span <= 0.25 ? 2 : (span <= 1.0 ? 1 : 0)));
  const size_t sm = sizeof(FarSmem);
  switch (mode) {
    case 0: k_far<0><<<grid, FTHR, sm, stream()>>>(g->dev, k, invk2, (cd *)M, ld, fq, (float2 *)F, ldf); break;
    case 1: k_far<1><<<grid, FTHR, sm, stream()>>>(g->dev, k, invk2, (cd *)M, ld, fq, (float2 *)F, ldf); break;
    case 2: k_far<2><<<grid, FTHR, sm, stream()>>>(g->dev, k, invk2, (cd *)M, ld, fq, (float2 *)F, ldf); break;
    default: k_far<3><<<grid, FTHR, sm, stream()>>>(g->dev, k, invk2, (cd *)M, ld, fq, (float2 *)F, ldf); break;
  }
  BG_LAUNCHED();
  return BG_OK;
}

// =========================================================================
// near field, frequency independent: tetrahedron-pair moments
//   M0 = sum K,  M1 = sum K (x-o_A),  M1' = sum K (y-o_B),  M2 = sum K (x-o_A).(y-o_B)
// for K in {1/(4 pi r), 1/(4 pi), r/(8 pi)} (GMEIntegrand KERNEL_STATIC,
// GMatrixElements.cc:153-165), in the unit-simplex measure (rule weights sum
// to 1/6 per tetrahedron).  Layout: 24 doubles per pair, [kernel][M0, M1(3),
// M1'(3), M2].  The per-basis-function-pair numbers of
// GetGME_TetTetInt(KERNEL_STATIC) follow from
//   int (x-Q).(y-Q') K = M2 - q.M1' - q'.M1 + q.q' M0,  q = Q-o_A, q' = Q'-o_B.
// =========================================================================

// regular pairs (<= 1 common vertex): 16x16 rule (GMatrixElements.cc:329-341),
// one warp per tetrahedron pair, origins o_A, o_B = first vertex of each tet.
__global__ void k_tp_regular(DevGeom g, const int4 *tp, int ntp, double *mom) {
  int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= ntp) return;
  int4 p = tp[warp];
  int4 A = g.tetVI[p.x], B = g.tetVI[p.y];
  double oA[3], oB[3], LA[3][3], LB[3][3];
  load3(g.V4, A.x, oA); load3(g.V4, B.x, oB);
  int va[3] = {A.y, A.z, A.w}, vb[3] = {B.y, B.z, B.w};
  for (int i = 0; i < 3; i++) {
    double t[3];
    load3(g.V4, va[i], t);
    for (int c = 0; c < 3; c++) LA[i][c] = t[c] - oA[c];
    load3(g.V4, vb[i], t);
    for (int c = 0; c < 3; c++) LB[i][c] = t[c] - oB[c];
  }
  double d0 = oA[0] - oB[0], d1 = oA[1] - oB[1], d2 = oA[2] - oB[2];
  double acc[24];
#pragma unroll
  for (int i = 0; i < 24; i++) acc[i] = 0.0;
  const double inv4pi = 0.25 / M_PI, inv8pi = 0.125 / M_PI;
  for (int idx = lane; idx < 256; idx += 32) {
    int i = idx >> 4, j = idx & 15;
    double xa[3], yb[3];
    for (int c = 0; c < 3; c++) {
      xa[c] = c_tcr16[4 * i] * LA[0][c] + c_tcr16[4 * i + 1] * LA[1][c] + c_tcr16[4 * i + 2] * LA[2][c];
      yb[c] = c_tcr16[4 * j] * LB[0][c] + c_tcr16[4 * j + 1] * LB[1][c] + c_tcr16[4 * j + 2] * LB[2][c];
    }
    double w = c_tcr16[4 * i + 3] * c_tcr16[4 * j + 3];
    double R0 = d0 + xa[0] - yb[0], R1 = d1 + xa[1] - yb[1], R2 = d2 + xa[2] - yb[2];
    double r = sqrt(R0 * R0 + R1 * R1 + R2 * R2);
    if (r < 1.0e-12) continue;
    double K[3] = {inv4pi / r, inv4pi, r * inv8pi};
    double xy = xa[0] * yb[0] + xa[1] * yb[1] + xa[2] * yb[2];
#pragma unroll
    for (int pk = 0; pk < 3; pk++) {
      double wk = w * K[pk];
      acc[8 * pk] += wk;
      acc[8 * pk + 1] += wk * xa[0]; acc[8 * pk + 2] += wk * xa[1]; acc[8 * pk + 3] += wk * xa[2];
      acc[8 * pk + 4] += wk * yb[0]; acc[8 * pk + 5] += wk * yb[1]; acc[8 * pk + 6] += wk * yb[2];
      acc[8 * pk + 7] += wk * xy;
    }
  }
#pragma unroll
  for (int i = 0; i < 24; i++) acc[i] = warp_sum(acc[i]);
  if (lane == 0)
    for (int i = 0; i < 24; i++) mom[24 * (size_t)warp + i] = acc[i];
}

// singular pairs (2..4 common vertices): singular.cu (singular_precompute)

// combine the 4 tetrahedron pairs of each near basis-function pair into the
// 6 numbers of GetGME_TetTetInt(KERNEL_STATIC) (GMatrixElements.cc:295-365):
// per kernel {4 A A' int (x-Q).(y-Q') K, 36 A A' int K} with sign +1 for PP/MM,
// -1 for PM/MP.
__device__ __forceinline__ void tp_origin(const DevGeom &g, const int4 *tp, const int4 *ordA, int id, bool first,
                                          double *o) {
  int4 p = tp[id];
  if (p.z >= 2) load3(g.V4, ordA[id].x, o);
  else load3(g.V4, first ? g.tetVI[p.x].x : g.tetVI[p.y].x, o);
}

__global__ void k_fibbi_combine(DevGeom g, NearData nd) {
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nd.npairs) return;
  int2 ab = nd.pairs[k];
  int a = ab.x, b = ab.y;
  int4 t4 = nd.pairTP[k];
  int tid[4] = {t4.x, t4.y, t4.z, t4.w};
  int2 qa = g.bfQ[a], qb = g.bfQ[b];
  double AA = g.bfArea[a] * g.bfArea[b];
  double out[6] = {0, 0, 0, 0, 0, 0};
  for (int sa = 0; sa < 2; sa++)
    for (int sb = 0; sb < 2; sb++) {
      int code = tid[2 * sa + sb];
      bool sw = (code >> 30) & 1;
      int id = code & ~(1 << 30);
      const double *M = nd.tpMom + 24 * (size_t)id;
      double ox[3], oy[3], Q[3], QP[3];
      tp_origin(g, nd.tp, nd.tpOrdA, id, !sw, ox);
      tp_origin(g, nd.tp, nd.tpOrdA, id, sw, oy);
      load3(g.V4, sa == 0 ? qa.x : qa.y, Q);
      load3(g.V4, sb == 0 ? qb.x : qb.y, QP);
      double q[3] = {Q[0] - ox[0], Q[1] - ox[1], Q[2] - ox[2]};
      double qp[3] = {QP[0] - oy[0], QP[1] - oy[1], QP[2] - oy[2]};
      double s = (sa == sb) ? 1.0 : -1.0;
      for (int pk = 0; pk < 3; pk++) {
        const double *m = M + 8 * pk;
        const double *m1 = sw ? m + 4 : m + 1;   // moment of the x (row) tetrahedron
        const double *m1p = sw ? m + 1 : m + 4;  // moment of the y (column) tetrahedron
        double J = m[7] - (q[0] * m1p[0] + q[1] * m1p[1] + q[2] * m1p[2]) -
                   (qp[0] * m1[0] + qp[1] * m1[1] + qp[2] * m1[2]) +
                   (q[0] * qp[0] + q[1] * qp[1] + q[2] * qp[2]) * m[0];
        out[2 * pk] += s * 4.0 * AA * J;
        out[2 * pk + 1] += s * 36.0 * AA * m[0];
      }
    }
  for (int i = 0; i < 6; i++) nd.fibbi[6 * (size_t)k + i] = out[i];
}

int precompute_near(bg_geometry *g) {
  int st = init_tables();
  if (st) return st;
  NearData &nd = g->near;
  if (nd.ntp_reg > 0) {
    int threads = 256, blocks = (nd.ntp_reg * 32 + threads - 1) / threads;
    k_tp_regular<<<blocks, threads, 0, stream()>>>(g->dev, nd.tp, nd.ntp_reg, nd.tpMom);
    BG_LAUNCHED();
  }
  if ((st = singular_precompute(g))) return st;
  if (nd.npairs > 0) {
    k_fibbi_combine<<<(nd.npairs + 127) / 128, 128, 0, stream()>>>(g->dev, nd);
    BG_LAUNCHED();
  }
  BG_CUDA_TRY(cudaStreamSynchronize(stream()));
  return BG_OK;
}

// =========================================================================
// near field per frequency: desingularised 64-point BF-pair integral plus the
// cached static numbers (GetGMatrixElement, GMatrixElements.cc:400-420):
//   G = BFBFInt[(e^{ikr}-1-ikr-(ikr)^2/2)/4 pi r] + (F0-F1/k^2) + ik(F2-F3/k^2)
//       + (ik)^2 (F4-F5/k^2)
// =========================================================================
__global__ void k_near(DevGeom g, NearData nd, cd k, cd invk2, cd *M, size_t ld, const double *fq, float2 *Fc,
                       size_t ldf) {
  if (fq) {
    k = cd{fq[0], fq[1]};
    invk2 = dev_invk2(fq[0], fq[1]);
  }
  // four lanes per pair, one per tetrahedron pair (PP, PM, MP, MM); the sum
  // keeps that order (88 -> 26 us at N = 72, where 2,600 threads did not fill
  // the SMs; 398 -> 375 us at N = 4,494)
  const int id = blockIdx.x * blockDim.x + threadIdx.x, kk = id >> 2;
  const bool live = kk < nd.npairs;
  const int2 ab = nd.pairs[live ? kk : 0];
  const int a = ab.x, b = ab.y, sa = (id >> 1) & 1, sb = id & 1;
  const int2 ta = g.bfTet[a], tb = g.bfTet[b], qa = g.bfQ[a], qb = g.bfQ[b];
  const double Aa = g.bfArea[a], Ab = g.bfArea[b];
  const double inv4pi = 0.25 / M_PI;
  const cd ik = cmk(-k.i, k.r);
  cd part = cmk(0, 0);
  if (live) {
    const int t1 = sa == 0 ? ta.x : ta.y, t2 = sb == 0 ? tb.x : tb.y;
    double Q[3], QP[3];
    load3(g.V4, sa == 0 ? qa.x : qa.y, Q);
    load3(g.V4, sb == 0 ? qb.x : qb.y, QP);
    const double cc = (sa == sb ? 1.0 : -1.0) * Aa * Ab;
    for (int i = 0; i < 4; i++) {
      const double *x = g.tetP4 + 16 * (size_t)t1 + 4 * i;
      for (int j = 0; j < 4; j++) {
        const double *y = g.tetP4 + 16 * (size_t)t2 + 4 * j;
        double R0 = x[0] - y[0], R1 = x[1] - y[1], R2 = x[2] - y[2];
        double r = sqrt(R0 * R0 + R1 * R1 + R2 * R2);
        if (r < 1.0e-12) continue;
        double dot = (x[0] - Q[0]) * (y[0] - QP[0]) + (x[1] - Q[1]) * (y[1] - QP[1]) + (x[2] - Q[2]) * (y[2] - QP[2]);
        cd phi = cscale(exprel3(cscale(ik, r)), inv4pi / r);
        cd pe = cmk(dot * (1.0 / 144.0) - invk2.r * (1.0 / 16.0), -invk2.i * (1.0 / 16.0));
        part = cadd(part, cmul(pe, phi));
      }
    }
    part = cscale(part, cc);
  }
  const int l0 = threadIdx.x & 28;
  cd acc = cmk(0, 0);
#pragma unroll
  for (int q = 0; q < 4; q++)
    acc = cadd(acc, cmk(__shfl_sync(0xffffffffu, part.r, l0 + q), __shfl_sync(0xffffffffu, part.i, l0 + q)));
  if (!live) return;
  const double *F = nd.fibbi + 6 * (size_t)kk;
  cd t0 = cadd(cmk(F[0], 0), cscale(invk2, -F[1]));
  cd t1 = cmul(ik, cadd(cmk(F[2], 0), cscale(invk2, -F[3])));
  cd t2 = cmul(cmul(ik, ik), cadd(cmk(F[4], 0), cscale(invk2, -F[5])));
  acc = cadd(acc, cadd(t0, cadd(t1, t2)));
  // the four lanes write the entry, its mirror and their complex64 copies
  const int w = id & 3;
  if (w == 0) M[(size_t)a + (size_t)b * ld] = acc;
  if (w == 1 && a != b) M[(size_t)b + (size_t)a * ld] = acc;
  if (Fc) {
    const float2 f = make_float2((float)acc.r, (float)acc.i);
    if (w == 2) Fc[(size_t)a + (size_t)b * ldf] = f;
    if (w == 3 && a != b) Fc[(size_t)b + (size_t)a * ldf] = f;
  }
}

int assemble_near(bg_geometry *g, double wr, double wi, void *M, size_t ld, const double *fq, void *F, size_t ldf) {
  NearData &nd = g->near;
  if (nd.npairs == 0) return BG_OK;
  double d = (wr * wr - wi * wi) * (wr * wr - wi * wi) + 4 * wr * wr * wi * wi;
  cd invk2{(wr * wr - wi * wi) / d, -2 * wr * wi / d};
  k_near<<<(int)((4LL * nd.npairs + 127) / 128), 128, 0, stream()>>>(g->dev, nd, cd{wr, wi}, invk2, (cd *)M, ld, fq,
                                                       (float2 *)F, ldf);
  BG_LAUNCHED();
  return BG_OK;
}

// =========================================================================
// V^-1 Gram block of one row (GetOverlaps, VIEMatrix.cc:200-316):
//   -(1/w^2) int_T F_a . (eps(x)-1)^-1 . F_b, 33-point rule with w = 6V w_i,
// w = real(omega), over the faces of both tetrahedra of basis function a.
// Added to M(a,b) and M(b,a) for b >= a (the reference adds the full row and
// its symmetric fill then overwrites the lower triangle with the upper).
// =========================================================================
//
// A half warp per tetrahedron of the row (lanes 0-15 the plus side, 16-31 the
// minus side), its lanes over the 33 points: eps(x) and its 3 x 3 inverse are
// formed once per point and serve the four faces, and the four sums come out
// of a 16-lane shuffle tree.  One thread per row walked 2 x 4 x 33 points in
// series, inverse included: 0.58-0.66 ms whatever N; now 20 us at N = 72 and
// 50 us at N = 4,494.
__global__ void __launch_bounds__(128) k_gram(DevGeom g, double w, cd *M, size_t ld, const double *fq, float2 *F,
                                              size_t ldf) {
  if (fq) w = fq[0];
  const int a = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (a >= g.N) return;
  const int side = lane >> 4, l = lane & 15;
  const int2 tt = g.bfTet[a], qq = g.bfQ[a];
  const double pre = -1.0 / (w * w);
  const int t = side == 0 ? tt.x : tt.y;
  const int obj = g.tetObj[t];
  const bg_material &mat = g.mats[obj];
  const DevExpr *mex = g.expr ? g.expr + obj : nullptr;
  const double vol = g.tetVol[t];
  const double pa = (side == 0 ? 1.0 : -1.0) * g.bfArea[a] / (3.0 * vol);
  double QA[3], V[4][3];
  load3(g.V4, side == 0 ? qq.x : qq.y, QA);
  const int4 vi = g.tetVI[t], fi = g.tetFI[t];
  const int vv[4] = {vi.x, vi.y, vi.z, vi.w}, fl[4] = {fi.x, fi.y, fi.z, fi.w};
  double pb[4];
#pragma unroll
  for (int f = 0; f < 4; f++) {
    load3(g.V4, vv[f], V[f]);     // the vertex opposite face f is its Q
    pb[f] = fl[f] < 0 ? 0.0 : (g.bfTet[fl[f]].x == t ? 1.0 : -1.0) * g.bfArea[fl[f]] / (3.0 * vol);
  }
  cd acc[4] = {cmk(0, 0), cmk(0, 0), cmk(0, 0), cmk(0, 0)};
  for (int i = l; i < 33; i += 16) {
    const double *u = c_tcr33 + 4 * i;
    const double wt = pre * (6.0 * vol * u[3]);
    double x[3], FA[3];
#pragma unroll
    for (int c = 0; c < 3; c++) {
      x[c] = V[0][c] + u[0] * (V[1][c] - V[0][c]) + u[1] * (V[2][c] - V[0][c]) + u[2] * (V[3][c] - V[0][c]);
      FA[c] = pa * (x[c] - QA[c]);
    }
    cd E[3][3], Ei[3][3], r[3];
    mat_eval(mat, mex, x, E);
    E[0][0].r -= 1.0; E[1][1].r -= 1.0; E[2][2].r -= 1.0;
    inv3(E, Ei);
#pragma unroll
    for (int nu = 0; nu < 3; nu++)
      r[nu] = cscale(cadd(cadd(cscale(Ei[0][nu], FA[0]), cscale(Ei[1][nu], FA[1])), cscale(Ei[2][nu], FA[2])), wt);
#pragma unroll
    for (int f = 0; f < 4; f++)
#pragma unroll
      for (int nu = 0; nu < 3; nu++) acc[f] = cadd(acc[f], cscale(r[nu], pb[f] * (x[nu] - V[f][nu])));
  }
#pragma unroll
  for (int f = 0; f < 4; f++)
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {
      acc[f].r += __shfl_xor_sync(0xffffffffu, acc[f].r, o);
      acc[f].i += __shfl_xor_sync(0xffffffffu, acc[f].i, o);
    }
  // the diagonal sums both sides; every other face belongs to one side
  cd diag = cmk(0, 0);
#pragma unroll
  for (int f = 0; f < 4; f++)
    if (fl[f] == a) diag = acc[f];
  const cd other = cmk(__shfl_xor_sync(0xffffffffu, diag.r, 16), __shfl_xor_sync(0xffffffffu, diag.i, 16));
  if (l >= 4) return;
  const int b = l == 0 ? fl[0] : l == 1 ? fl[1] : l == 2 ? fl[2] : fl[3];
  cd val = l == 0 ? acc[0] : l == 1 ? acc[1] : l == 2 ? acc[2] : acc[3];
  if (b < a || (b == a && side == 1)) return;   // also faces of the surface, b = -1
  if (b == a) val = cadd(diag, other);
  cd *p = M + (size_t)a + (size_t)b * ld;
  const cd v = cadd(*p, val);
  *p = v;
  cd vt = v;
  if (b != a) {
    cd *q = M + (size_t)b + (size_t)a * ld;
    vt = cadd(*q, val);
    *q = vt;
  }
  if (F) {   // the final value of these entries: the complex64 copy
    F[(size_t)a + (size_t)b * ldf] = make_float2((float)v.r, (float)v.i);
    if (b != a) F[(size_t)b + (size_t)a * ldf] = make_float2((float)vt.r, (float)vt.i);
  }
}

int assemble_gram(bg_geometry *g, double wr, double wi, void *M, size_t ld, const double *fq, void *F, size_t ldf) {
  if (g->dispersive && fq) { set_error("frequency-dependent materials need a host frequency"); return BG_ERR_ARG; }
  int st = refresh_materials(g, wr, wi);
  if (st) return st;
  k_gram<<<(g->N + 3) / 4, 128, 0, stream()>>>(g->dev, wr, (cd *)M, ld, fq, (float2 *)F, ldf);
  BG_LAUNCHED();
  return BG_OK;
}

// =========================================================================
// plane-wave RHS (RHSVector.cc:85-124): v_a = -1/(i w Z0) BFInt[b . E],
// E = E0 exp(i k nhat.x), 33-point rule on both tetrahedra of a.
// =========================================================================
struct PWave { cd E0[3]; double nh[3]; cd k; };

// 16 lanes per basis function, over the 2 x 33 points (one thread per basis
// function evaluated them in series: 19-24 us; now 8-11 us)
__global__ void k_rhs(DevGeom g, PWave pw, cd pre, cd *out, const double *fq) {
  if (fq) {
    // -1/(i w Z0) = i/(w Z0)
    double wr = fq[0], wi = fq[1], d = (wr * wr + wi * wi) * 376.73031346177;
    pw.k = cd{wr, wi};
    pre = cd{wi / d, wr / d};
  }
  const int a = (blockIdx.x * blockDim.x + threadIdx.x) >> 4, l = threadIdx.x & 15;
  const bool live = a < g.N;
  cd tot = cmk(0, 0);
  if (live) {
    const int2 tt = g.bfTet[a], qq = g.bfQ[a];
    const double Aa = g.bfArea[a];
#pragma unroll 1
    for (int side = 0; side < 2; side++) {
      const int t = side == 0 ? tt.x : tt.y;
      const int4 vi = g.tetVI[t];
      double Q[3], V[4][3];
      load3(g.V4, side == 0 ? qq.x : qq.y, Q);
      load3(g.V4, vi.x, V[0]); load3(g.V4, vi.y, V[1]); load3(g.V4, vi.z, V[2]); load3(g.V4, vi.w, V[3]);
      const double vol = g.tetVol[t], pf = (side == 0 ? 1.0 : -1.0) * Aa / (3.0 * vol);
      for (int i = l; i < 33; i += 16) {
        const double *u = c_tcr33 + 4 * i;
        const double wt = 6.0 * vol * u[3] * pf;
        double x[3];
#pragma unroll
        for (int c = 0; c < 3; c++)
          x[c] = V[0][c] + u[0] * (V[1][c] - V[0][c]) + u[1] * (V[2][c] - V[0][c]) + u[2] * (V[3][c] - V[0][c]);
        const cd e = expikr(pw.k, pw.nh[0] * x[0] + pw.nh[1] * x[1] + pw.nh[2] * x[2]);
        const cd be = cadd(cadd(cscale(pw.E0[0], x[0] - Q[0]), cscale(pw.E0[1], x[1] - Q[1])), cscale(pw.E0[2], x[2] - Q[2]));
        tot = cadd(tot, cscale(cmul(be, e), wt));
      }
    }
  }
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) {
    tot.r += __shfl_xor_sync(0xffffffffu, tot.r, o);
    tot.i += __shfl_xor_sync(0xffffffffu, tot.i, o);
  }
  if (live && l == 0) out[a] = cmul(pre, tot);
}

static PWave make_pw(double wr, double wi, const double *E0, const double *nhat) {
  PWave pw;
  for (int i = 0; i < 3; i++) { pw.E0[i] = cd{E0[2 * i], E0[2 * i + 1]}; pw.nh[i] = nhat[i]; }
  pw.k = cd{wr, wi};
  return pw;
}

int rhs_planewave(bg_geometry *g, double wr, double wi, const double *E0, const double *nhat, void *out,
                  const double *fq) {
  int st = init_tables();
  if (st) return st;
  PWave pw = make_pw(wr, wi, E0, nhat);
  // -1/(i w Z0) = i/(w Z0)
  const double Z0 = 376.73031346177;
  double d = (wr * wr + wi * wi) * Z0;
  cd pre{wi / d, wr / d};
  k_rhs<<<(g->N + 7) / 8, 128, 0, stream()>>>(g->dev, pw, pre, (cd *)out, fq);
  BG_LAUNCHED();
  return BG_OK;
}

// =========================================================================
// EMT power (EMTPFT.cc:324-493): PScat = sum_{a<=b} Re(Z0 J_a^* J_b) Im Q_ab
// (same object; Im Q = w BFBFInt[PEFIE sin(kr)/(4 pi r)], series for kr<2e-2)
// and -1/2 Re(Z0 J_a^* J_b i Q_ab) across objects (full e^{ikr}/(4 pi r));
// rule 4/16/33 points by common vertices and kR>5 (EMTPFT.cc:305-313).
// Extinction 1/2 Re(J_a^* BFInt[b.E_inc]) (EMTPFT.cc:151-211).
// Partial sums per block and object pair are reduced on the host in a fixed
// order.
// =========================================================================
struct PftArgs {
  DevGeom g;
  const cd *J;
  double w;      // real(omega)
  double absw;   // |omega|
  int nobj;
  const cd *DR = nullptr;   // dressed Rytov matrix (column-major, ldr) in place of J
  size_t ldr = 0;
};

__device__ __forceinline__ void rule_point(int npts, int i, double *u) {
  if (npts == 16) { u[0] = c_tcr16[4 * i]; u[1] = c_tcr16[4 * i + 1]; u[2] = c_tcr16[4 * i + 2]; u[3] = c_tcr16[4 * i + 3]; }
  else { u[0] = c_tcr33[4 * i]; u[1] = c_tcr33[4 * i + 1]; u[2] = c_tcr33[4 * i + 2]; u[3] = c_tcr33[4 * i + 3]; }
}

// Full EMT PFT (EMTPFT.cc:85-127 extinction, 216-291 scattered, 396-491 sum).
// Ten quantities per pair, NPQ order: PScat, force (3), torque from b_A x b_B
// (3), torque from (x_A - c_A) x R (3); c_A = torque centre (object origin).
#define NPQ 10
#define TEN_THIRDS (10.0 / 3.0)

// BFBFInt of the scattered integrand (EMTPFT.cc:216-291); lanes [lane, nl)
// split the point pairs; q: this lane's partial integrals
__device__ void scat_q(const PftArgs &P, int a, int b, int npts, bool same, int lane, int nl, cd q[NPQ]) {
  const DevGeom &g = P.g;
  int2 ta = g.bfTet[a], tb = g.bfTet[b], la = g.bfLoc[a], lb = g.bfLoc[b];
  double k = P.w, k2 = k * k;
  for (int n = 0; n < NPQ; n++) q[n] = cmk(0, 0);
  const double inv4pi = 0.25 / M_PI;
  int oa = g.bfV[a].w;
  const double *tc = g.objOrigin + 3 * oa;
  for (int sa = 0; sa < 2; sa++)
    for (int sb = 0; sb < 2; sb++) {
      int t1 = sa == 0 ? ta.x : ta.y, t2 = sb == 0 ? tb.x : tb.y;
      int i1 = sa == 0 ? la.x : la.y, i2 = sb == 0 ? lb.x : lb.y;
      int4 v1 = g.tetVI[t1], v2 = g.tetVI[t2];
      int va[4] = {v1.x, v1.y, v1.z, v1.w}, vb[4] = {v2.x, v2.y, v2.z, v2.w};
      double Q1[3], Q2[3], L1[3][3], L2[3][3];
      load3(g.V4, va[i1], Q1);
      load3(g.V4, vb[i2], Q2);
      for (int i = 0; i < 3; i++) {
        double tmp[3];
        load3(g.V4, va[(i1 + 1 + i) % 4], tmp);
        for (int c = 0; c < 3; c++) L1[i][c] = tmp[c] - Q1[c];
        load3(g.V4, vb[(i2 + 1 + i) % 4], tmp);
        for (int c = 0; c < 3; c++) L2[i][c] = tmp[c] - Q2[c];
      }
      double V1 = g.tetVol[t1], V2 = g.tetVol[t2];
      double p1 = (sa == 0 ? 1.0 : -1.0) * g.bfArea[a] / (3.0 * V1);
      double p2 = (sb == 0 ? 1.0 : -1.0) * g.bfArea[b] / (3.0 * V2);
      int np2 = npts * npts;
      for (int idx = lane; idx < np2; idx += nl) {
        int i = idx / npts, j = idx % npts;
        double u[4], v[4];
        if (npts == 4) {
          const double qa = 0.13819660112501051, qb = 0.58541019662496850;
          u[0] = (i == 1) ? qb : qa; u[1] = (i == 2) ? qb : qa; u[2] = (i == 3) ? qb : qa; u[3] = 1.0 / 24.0;
          v[0] = (j == 1) ? qb : qa; v[1] = (j == 2) ? qb : qa; v[2] = (j == 3) ? qb : qa; v[3] = 1.0 / 24.0;
        } else {
          rule_point(npts, i, u);
          rule_point(npts, j, v);
        }
        double xa[3], xb[3], ba[3], bb[3];
        for (int c = 0; c < 3; c++) {
          ba[c] = u[0] * L1[0][c] + u[1] * L1[1][c] + u[2] * L1[2][c];
          xa[c] = Q1[c] + ba[c];
          ba[c] *= p1;
          bb[c] = v[0] * L2[0][c] + v[1] * L2[1][c] + v[2] * L2[2][c];
          xb[c] = Q2[c] + bb[c];
          bb[c] *= p2;
        }
        double wt = 6.0 * V1 * u[3] * 6.0 * V2 * v[3];
        double R[3] = {xa[0] - xb[0], xa[1] - xb[1], xa[2] - xb[2]};
        double r2 = R[0] * R[0] + R[1] * R[1] + R[2] * R[2], r = sqrt(r2), kr = k * r;
        double pefie = ba[0] * bb[0] + ba[1] * bb[1] + ba[2] * bb[2] - (3.0 * p1) * (3.0 * p2) / k2;
        cd phi, psi;
        if (same) {
          double imphi, impsi;
          if (fabs(kr) < 2.0e-2) {
            imphi = (1.0 - kr * kr / 6.0) * k * inv4pi;
            impsi = -(1.0 - kr * kr / 10.0) * k2 * k / (12.0 * M_PI);
          } else {
            double s, c;
            sincos(kr, &s, &c);
            imphi = s * inv4pi / r;
            impsi = (kr * c - s) * inv4pi / (r * r2);
          }
          phi = cmk(0, imphi);
          psi = cmk(0, impsi);
        } else {
          double s, c;
          sincos(kr, &s, &c);
          phi = cmk(c * inv4pi / r, s * inv4pi / r);
          psi = cscale(cmul(phi, cmk(-1.0, kr)), 1.0 / r2);     // phi (ikr - 1) / r^2
        }
        double XT[3] = {xa[0] - tc[0], xa[1] - tc[1], xa[2] - tc[2]};
        q[0] = cadd(q[0], cscale(phi, P.w * pefie * wt));
        cd pp = cscale(psi, TEN_THIRDS * pefie * wt), pf = cscale(phi, TEN_THIRDS * wt);
        for (int m = 0; m < 3; m++) {
          int m1 = (m + 1) % 3, m2 = (m + 2) % 3;
          q[1 + m] = cadd(q[1 + m], cscale(pp, R[m]));
          q[4 + m] = cadd(q[4 + m], cscale(pf, ba[m1] * bb[m2] - ba[m2] * bb[m1]));
          q[7 + m] = cadd(q[7 + m], cscale(pp, XT[m1] * R[m2] - XT[m2] * R[m1]));
        }
      }
    }
}

// contributions of pair (a, b) to the per-object-pair sums (EMTPFT.cc:416-436)
__device__ __forceinline__ void scat_terms(const PftArgs &P, int a, int b, const cd q[NPQ], bool same, double d[NPQ]) {
  const double Z0 = 376.73031346177;
  // u0JJ = Z0 GetJJ(a, b) (GetPFT.cc:108-115): Z0 DR(b, a) for a dressed
  // Rytov matrix, else Z0 conj(Ja) Jb
  cd u;
  if (P.DR) {
    cd v = P.DR[(size_t)b + (size_t)a * P.ldr];
    u = cmk(Z0 * v.r, Z0 * v.i);
  } else {
    cd Ja = P.J[a], Jb = P.J[b];
    u = cmk(Z0 * (Ja.r * Jb.r + Ja.i * Jb.i), Z0 * (Ja.r * Jb.i - Ja.i * Jb.r));
  }
  if (same) {
    d[0] = u.r * q[0].i;
    for (int n = 1; n < NPQ; n++) d[n] = a != b ? u.i * q[n].i : 0.0;
  } else {
    // -0.5 Re(u i q) = 0.5 Im(u q);  -0.5 Im(u i q) = -0.5 Re(u q)
    cd uq = cmul(u, q[0]);
    d[0] = 0.5 * uq.i;
    for (int n = 1; n < NPQ; n++) d[n] = -0.5 * cmul(u, q[n]).r;
  }
}

#define PMAXOBJ 4
// far pairs (no common vertex): one thread per pair; partial sums per block
// and object pair: part[block][noa*NO + nob][NPQ]
__global__ void __launch_bounds__(FT * FT) k_pft_far(PftArgs P, double *part) {
  int bx = blockIdx.x, by = blockIdx.y;
  int a = bx * FT + threadIdx.x, b = by * FT + threadIdx.y;
  const DevGeom &g = P.g;
  double d[NPQ];
  for (int n = 0; n < NPQ; n++) d[n] = 0.0;
  int pairid = 0;
  if (bx <= by && a < g.N && b < g.N && a <= b) {
    int4 va = g.bfV[a], vb = g.bfV[b];
    int2 qa = g.bfQ[a], qb = g.bfQ[b];
    int A5[5] = {qa.x, va.x, va.y, va.z, qa.y}, B5[5] = {qb.x, vb.x, vb.y, vb.z, qb.y};
    int ncv = 0;
    for (int i = 0; i < 5; i++)
      for (int j = 0; j < 5; j++) ncv += A5[i] == B5[j];
    if (ncv == 0) {
      double kR = P.absw * fmax(g.bfRadius[a], g.bfRadius[b]);
      int npts = kR > 5.0 ? 16 : 4;
      bool same = va.w == vb.w;
      cd q[NPQ];
      scat_q(P, a, b, npts, same, 0, 1, q);
      scat_terms(P, a, b, q, same, d);
      pairid = va.w * P.nobj + vb.w;
    }
  }
  __shared__ double red[FT * FT / 32][PMAXOBJ * PMAXOBJ][NPQ];
  int tid = threadIdx.y * FT + threadIdx.x, lane = tid & 31, wid = tid >> 5;
  for (int pid = 0; pid < P.nobj * P.nobj; pid++)
    for (int n = 0; n < NPQ; n++) {
      double v = warp_sum(pid == pairid ? d[n] : 0.0);
      if (lane == 0) red[wid][pid][n] = v;
    }
  __syncthreads();
  int nv = P.nobj * P.nobj * NPQ;
  for (int e = tid; e < nv; e += FT * FT) {
    int pid = e / NPQ, n = e % NPQ;
    double s = 0;
    for (int w = 0; w < FT * FT / 32; w++) s += red[w][pid][n];
    part[((size_t)by * gridDim.x + bx) * nv + e] = s;
  }
}

// near pairs (same object, common vertex): one warp per pair, lanes split the
// point pairs; partial sums per block and object: part[block][no][NPQ]
__global__ void k_pft_near(PftArgs P, NearData nd, double *part) {
  int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  double d[NPQ];
  for (int n = 0; n < NPQ; n++) d[n] = 0.0;
  if (warp < nd.npairs) {
    int2 ab = nd.pairs[warp];
    const DevGeom &g = P.g;
    double kR = P.absw * fmax(g.bfRadius[ab.x], g.bfRadius[ab.y]);
    int npts = kR > 5.0 ? 33 : 16;
    cd q[NPQ];
    scat_q(P, ab.x, ab.y, npts, true, lane, 32, q);
    for (int n = 0; n < NPQ; n++) {
      q[n].r = warp_sum(q[n].r);
      q[n].i = warp_sum(q[n].i);
    }
    if (lane == 0) scat_terms(P, ab.x, ab.y, q, true, d);
  }
  __shared__ double red[8][NPQ];
  __shared__ int objs[8];
  int wid = threadIdx.x >> 5;
  if (lane == 0) {
    for (int n = 0; n < NPQ; n++) red[wid][n] = d[n];
    objs[wid] = (warp < nd.npairs) ? P.g.bfV[nd.pairs[warp].x].w : 0;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < P.nobj * NPQ; e += blockDim.x) {
    int o = e / NPQ, n = e % NPQ;
    double s = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++)
      if (objs[w] == o) s += red[w][n];
    part[(size_t)blockIdx.x * P.nobj * NPQ + e] = s;
  }
}

// total current sum J_a b_a(x) of tetrahedron t (its up to four basis functions)
__device__ __forceinline__ void tet_current(const DevGeom &g, const cd *J, int t, const double (*V)[3],
                                            const double *x, cd j[3]) {
  const int4 fi = g.tetFI[t];
  const int f[4] = {fi.x, fi.y, fi.z, fi.w};
  const double iv = 1.0 / (3.0 * g.tetVol[t]);
  j[0] = j[1] = j[2] = cmk(0, 0);
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const int a = f[q];
    if (a < 0) continue;
    const cd Ja = cscale(J[a], (g.bfTet[a].x == t ? 1.0 : -1.0) * g.bfArea[a] * iv);
#pragma unroll
    for (int c = 0; c < 3; c++) j[c] = cadd(j[c], cscale(Ja, x[c] - V[q][c]));
  }
}
__device__ __forceinline__ void tet_point33(const DevGeom &g, int t, int i, double (*V)[3], double *x, double &wt) {
  const int4 vi = g.tetVI[t];
  load3(g.V4, vi.x, V[0]); load3(g.V4, vi.y, V[1]); load3(g.V4, vi.z, V[2]); load3(g.V4, vi.w, V[3]);
  const double *u = c_tcr33 + 4 * i;
#pragma unroll
  for (int c = 0; c < 3; c++)
    x[c] = V[0][c] + u[0] * (V[1][c] - V[0][c]) + u[1] * (V[2][c] - V[0][c]) + u[2] * (V[3][c] - V[0][c]);
  wt = 6.0 * g.tetVol[t] * u[3];
}

// extinction (EMTPFT.cc:85-127, 151-211) for a plane wave (grad E = ik nhat E).
// Linear in conj(J_a), so one thread per point of the 33-point rule takes the
// tetrahedron's total current j: with be = conj(j).E and xt = x - c
// (torque centre), e[0] = Re be, e[1+i] = Im(ik nhat_i be),
// e[4+i] = Im(conj(j) x E)_i, e[7+i] = Im(ik be (xt x nhat)_i); partial sums
// per block and object.  33 NT independent threads in place of N threads of
// 66 points each (24-28 us at N = 72 and 4,494; now 6-10 us).
__global__ void __launch_bounds__(128) k_pft_ext(PftArgs P, PWave pw, double *part) {
  const DevGeom &g = P.g;
  const int id = blockIdx.x * blockDim.x + threadIdx.x, t = id / 33;
  double e[NPQ];
  for (int n = 0; n < NPQ; n++) e[n] = 0.0;
  int obj = 0;
  if (t < g.NT) {
    obj = g.tetObj[t];
    const double *tc = g.objOrigin + 3 * obj;
    double V[4][3], x[3], wt;
    tet_point33(g, t, id - 33 * t, V, x, wt);
    cd j[3], E[3];
    tet_current(g, P.J, t, V, x, j);
    const cd ph = cscale(expikr(pw.k, pw.nh[0] * x[0] + pw.nh[1] * x[1] + pw.nh[2] * x[2]), wt);
#pragma unroll
    for (int c = 0; c < 3; c++) { E[c] = cmul(pw.E0[c], ph); j[c].i = -j[c].i; }
    const cd be = cadd(cadd(cmul(j[0], E[0]), cmul(j[1], E[1])), cmul(j[2], E[2]));
    const cd ikbe = cmul(cmk(-pw.k.i, pw.k.r), be);
    e[0] = be.r;
#pragma unroll
    for (int i = 0; i < 3; i++) {
      const int i1 = (i + 1) % 3, i2 = (i + 2) % 3;
      e[1 + i] = ikbe.i * pw.nh[i];
      e[4 + i] = csub(cmul(j[i1], E[i2]), cmul(j[i2], E[i1])).i;
      e[7 + i] = ikbe.i * ((x[i1] - tc[i1]) * pw.nh[i2] - (x[i2] - tc[i2]) * pw.nh[i1]);
    }
  }
  __shared__ double red[4][PMAXOBJ][NPQ];
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int o = 0; o < P.nobj; o++)
    for (int n = 0; n < NPQ; n++) {
      double v = warp_sum(o == obj ? e[n] : 0.0);
      if (lane == 0) red[wid][o][n] = v;
    }
  __syncthreads();
  for (int x = threadIdx.x; x < P.nobj * NPQ; x += blockDim.x) {
    int o = x / NPQ, n = x % NPQ;
    double s = 0;
    for (int w = 0; w < 4; w++) s += red[w][o][n];
    part[(size_t)blockIdx.x * P.nobj * NPQ + x] = s;
  }
}

// The overlap power of point i of tetrahedron t where eps may jump between two
// points (Janus, expressions): a basis function's rule starts at its own vertex
// Q, and the points are rounded as QA + (u . L); a point that lies on the jump
// takes the side this rounding gives it, for each of the four faces by itself.
__device__ __noinline__ double opft_point_by_face(const DevGeom &g, const cd *J, int t, int i, int obj, cd pre) {
  const int4 vi = g.tetVI[t], fi = g.tetFI[t];
  const int v[4] = {vi.x, vi.y, vi.z, vi.w}, fl[4] = {fi.x, fi.y, fi.z, fi.w};
  const double *u = c_tcr33 + 4 * i;
  const double vol = g.tetVol[t], wt = 6.0 * vol * u[3];
  double V[4][3], contrib = 0.0;
  for (int q = 0; q < 4; q++) load3(g.V4, v[q], V[q]);
  for (int q = 0; q < 4; q++) {
    const int a = fl[q];
    if (a < 0) continue;
    double QA[3], L[3][3], bA[3], x[3];
    load3(g.V4, v[q], QA);
    for (int m = 0; m < 3; m++) {
      double tmp[3];
      load3(g.V4, v[(q + 1 + m) % 4], tmp);
      for (int c = 0; c < 3; c++) L[m][c] = tmp[c] - QA[c];
    }
    for (int c = 0; c < 3; c++) {
      bA[c] = u[0] * L[0][c] + u[1] * L[1][c] + u[2] * L[2][c];
      x[c] = bA[c] + QA[c];
    }
    cd j[3], E[3][3], Ei[3][3], s = cmk(0, 0);
    tet_current(g, J, t, V, x, j);
    mat_eval(g.mats[obj], g.expr ? g.expr + obj : nullptr, x, E);
    E[0][0].r -= 1.0; E[1][1].r -= 1.0; E[2][2].r -= 1.0;
    inv3(E, Ei);
    const double pa = (g.bfTet[a].x == t ? 1.0 : -1.0) * g.bfArea[a] / (3.0 * vol);
    for (int mu = 0; mu < 3; mu++) {
      const cd r = cadd(cadd(cmul(Ei[mu][0], j[0]), cmul(Ei[mu][1], j[1])), cmul(Ei[mu][2], j[2]));
      s = cadd(s, cscale(r, pa * bA[mu]));
    }
    const cd Ja = J[a];
    contrib += cmul(cmul(cscale(pre, 0.5 * wt), cmk(Ja.r, -Ja.i)), s).r;
  }
  return contrib;
}

// OPFT absorbed power (OPFT.cc:62-119, OverlapIntegrand_PFT PAbs term,
// OverlapIntegrals.cc:79-170,242-298): sum Re(conj(Ja) Jb ME_ab),
// ME_ab = 1/2 int b_a . (i Z0/w)(eps-1)^-1 . b_b on the shared tetrahedron.
// The sum over the faces of a tetrahedron is 1/2 int conj(j).(i Z0/w)
// (eps-1)^-1.j of its total current, so one thread takes one of its 33 points
// (one eps(x) and one inverse).  One thread per row walked 2 x 4 x 33 points
// with an inverse each: 0.55-0.62 ms at any N; now 11 us at N = 72 and 20 us at 4,494.
__global__ void __launch_bounds__(128) k_opft(PftArgs P, cd omega, double *part, const double *fq) {
  if (fq) omega = cd{fq[0], fq[1]};
  const DevGeom &g = P.g;
  const int id = blockIdx.x * blockDim.x + threadIdx.x, t = id / 33;
  double contrib = 0.0;
  int obj = 0;
  // a tetrahedron without a basis function adds nothing, whatever eps is there
  // (eps = 1 has no inverse)
  const int4 fi = t < g.NT ? g.tetFI[t] : make_int4(-1, -1, -1, -1);
  if (max(max(fi.x, fi.y), max(fi.z, fi.w)) >= 0) {
    obj = g.tetObj[t];
    const cd pre0 = cdiv(cmk(0, 376.73031346177), omega);
    const int kind = g.mats[obj].kind;
    if (kind != BG_MAT_CONST_ISO && kind != BG_MAT_CONST_TENSOR && kind != BG_MAT_GAUSSIAN) {
      contrib = opft_point_by_face(g, P.J, t, id - 33 * t, obj, pre0);
    } else {
      double V[4][3], x[3], wt;
      tet_point33(g, t, id - 33 * t, V, x, wt);
      cd j[3];
      tet_current(g, P.J, t, V, x, j);
      const cd pre = cscale(pre0, 0.5 * wt);
      cd E[3][3], Ei[3][3], s = cmk(0, 0);
      mat_eval(g.mats[obj], g.expr ? g.expr + obj : nullptr, x, E);
      E[0][0].r -= 1.0; E[1][1].r -= 1.0; E[2][2].r -= 1.0;
      inv3(E, Ei);
#pragma unroll
      for (int mu = 0; mu < 3; mu++) {
        const cd r = cadd(cadd(cmul(Ei[mu][0], j[0]), cmul(Ei[mu][1], j[1])), cmul(Ei[mu][2], j[2]));
        s = cadd(s, cmul(cmk(j[mu].r, -j[mu].i), r));
      }
      contrib = cmul(pre, s).r;
    }
  }
  __shared__ double red[4][PMAXOBJ];
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int o = 0; o < P.nobj; o++) {
    double v = warp_sum(o == obj ? contrib : 0.0);
    if (lane == 0) red[wid][o] = v;
  }
  __syncthreads();
  if (threadIdx.x < P.nobj) {
    double s = 0;
    for (int w = 0; w < 4; w++) s += red[w][threadIdx.x];
    part[(size_t)blockIdx.x * P.nobj + threadIdx.x] = s;
  }
}

// blocks (and rows of partial sums) of k_opft and k_pft_ext
int pft_point_blocks(const bg_geometry *g) { return (int)((33LL * g->NT + 127) / 128); }

#include "emt_pairs.cuh"

static int ensure_scratch(bg_geometry *g, size_t bytes) {
  if (g->scratch_bytes >= bytes) return BG_OK;
  if (g->d_scratch) cudaFree(g->d_scratch);
  g->d_scratch = nullptr;
  g->scratch_bytes = 0;
  BG_CUDA_TRY(cudaMalloc(&g->d_scratch, bytes));
  g->scratch_bytes = bytes;
  return BG_OK;
}

__global__ void k_opft_reduce(int nrow, int nobj, const double *part, double *out) {
  int o = blockIdx.x;
  double s = 0;
  for (int b = threadIdx.x; b < nrow; b += blockDim.x) s += part[(size_t)b * nobj + o];
  s = warp_sum(s);
  __shared__ double red[8];
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += red[w];
    out[o] = t;
  }
}

int pft(bg_geometry *g, double wr, double wi, const void *dJ, const double *E0, const double *nhat, int method,
        double *out) {
  int st = init_tables();
  if (st) return st;
  int NO = (int)g->objs.size();
  if (NO > PMAXOBJ) { set_error("PFT supports at most %d objects", PMAXOBJ); return BG_ERR_ARG; }
  if (method == BG_PFT_OVERLAP) {
    if ((st = refresh_materials(g, wr, wi))) return st;
    const int nblk = pft_point_blocks(g);
    if ((st = ensure_scratch(g, sizeof(double) * ((size_t)nblk + 1) * NO))) return st;
    double *sum = g->d_scratch, h[PMAXOBJ];
    if ((st = opft_enqueue(g, wr, wi, dJ, nullptr, sum + NO, sum))) return st;
    BG_CUDA_TRY(cudaMemcpyAsync(h, sum, sizeof(double) * NO, cudaMemcpyDeviceToHost, stream()));
    BG_CUDA_TRY(cudaStreamSynchronize(stream()));
    for (int o = 0; o < NO; o++) {
      out[2 * o] = h[o];
      out[2 * o + 1] = 0.0;
    }
    return BG_OK;
  }
  double full[8 * PMAXOBJ];
  if ((st = pft_emt_full(g, wr, wi, dJ, E0, nhat, full))) return st;
  for (int o = 0; o < NO; o++) {
    out[2 * o] = full[8 * o];
    out[2 * o + 1] = full[8 * o + 1];
  }
  return BG_OK;
}

// Taylor coefficients of Im(phi), Im(psi) in r^2 (emt_pairs.cuh)
static EmtKernel emt_kernel(double k) {
  EmtKernel K{};
  K.k = k;
  K.k2 = k * k;
  K.tiny2 = (2.0e-2 / k) * (2.0e-2 / k);
  double f = 1.0, p = 1.0;   // (2n + 1)!, (-k^2)^n
  for (int n = 0; n < EMT_MAXT; n++) {
    if (n) { f *= (2.0 * n) * (2.0 * n + 1.0); p *= -K.k2; }
    K.c[n] = p / f;
    K.d[n] = -p * (2.0 * n + 2.0) / (f * (2.0 * n + 2.0) * (2.0 * n + 3.0));
  }
  return K;
}
// terms that reach 2e-17 of the value at r = 0 up to |k| r = x; 0: no polynomial
static int emt_terms(double x) { return x <= 1.0 ? 9 : (x <= 2.0 ? 12 : (x <= 4.0 ? 16 : 0)); }

static int emt_add_job(EmtReduce &R, const double *src, long long rows, int width, double *dst) {
  if (rows > 0) {
    R.src[R.n] = src; R.rows[R.n] = rows; R.width[R.n] = width; R.dst[R.n] = dst;
    R.wmax = std::max(R.wmax, width);
    R.n++;
  }
  return 0;
}

// pair sums through tetrahedra: far (job per object pair), near and self
// partials into the scratch from `s` on; the sums' places are sums[0..]:
// NO*NO*NPQ far, NO*NPQ near, NO self
static int emt_tet_sums(bg_geometry *g, const PftArgs &P, double *s, double *sums, EmtReduce &R,
                        const EmtBlockMap &bm, int nfar, int near_blocks, int near_per, int self_blocks) {
  const int NO = P.nobj;
  const EmtKernel K = emt_kernel(P.w);
  const bool dr = P.DR != nullptr;
  const int nt_far = emt_terms(std::fabs(P.w) * g->obj_diam);
  const int nt_near = emt_terms(std::fabs(P.w) * std::min(g->obj_diam, 4.01 * g->bf_rmax));
  // the points first: they are read as 16-byte pairs (s is 16-byte aligned)
  double *pts = s, *pfar = pts + (dr ? 0 : (size_t)4 * g->NT * EMT_PT), *pnear = pfar + (size_t)nfar * NPQ,
         *pself = pnear + (size_t)near_blocks * NO * NPQ;
  if (!dr) {
    k_emt_points<<<(4 * g->NT + 127) / 128, 128, 0, stream()>>>(g->dev, P.J, 1.0 / P.w, pts);
    BG_LAUNCHED();
    switch (nt_far) {
      case 9: k_emt_far<9><<<nfar, EMT_JT, 0, stream()>>>(g->dev, K, bm, pts, pfar); break;
      case 12: k_emt_far<12><<<nfar, EMT_JT, 0, stream()>>>(g->dev, K, bm, pts, pfar); break;
      case 16: k_emt_far<16><<<nfar, EMT_JT, 0, stream()>>>(g->dev, K, bm, pts, pfar); break;
      default: k_emt_far<0><<<nfar, EMT_JT, 0, stream()>>>(g->dev, K, bm, pts, pfar); break;
    }
  } else {
    switch (nt_far) {
      case 9: k_emt_far_dr<9><<<nfar, EMT_DJ, 0, stream()>>>(P, K, bm, pfar); break;
      case 12: k_emt_far_dr<12><<<nfar, EMT_DJ, 0, stream()>>>(P, K, bm, pfar); break;
      case 16: k_emt_far_dr<16><<<nfar, EMT_DJ, 0, stream()>>>(P, K, bm, pfar); break;
      default: k_emt_far_dr<0><<<nfar, EMT_DJ, 0, stream()>>>(P, K, bm, pfar); break;
    }
  }
  BG_LAUNCHED();
  for (int m = 0; m < bm.nmap; m++)
    emt_add_job(R, pfar + (size_t)bm.first[m] * NPQ, (m + 1 < bm.nmap ? bm.first[m + 1] : nfar) - bm.first[m], NPQ,
                sums + (size_t)(bm.oa[m] * NO + bm.ob[m]) * NPQ);
  if (near_blocks > 0) {
    const int T = EMT_NG * 16;
#define EMT_NEAR(n)                                                                                              \
  case n:                                                                                                        \
    if (dr) k_emt_near<n, true><<<near_blocks, T, 0, stream()>>>(P, g->near, K, near_per, pnear);                \
    else k_emt_near<n, false><<<near_blocks, T, 0, stream()>>>(P, g->near, K, near_per, pnear);                  \
    break;
    switch (nt_near) { EMT_NEAR(9) EMT_NEAR(12) EMT_NEAR(16) EMT_NEAR(0) }
#undef EMT_NEAR
    BG_LAUNCHED();
    emt_add_job(R, pnear, near_blocks, NO * NPQ, sums + (size_t)NO * NO * NPQ);
  }
  if (self_blocks > 0) {
    k_emt_self<<<self_blocks, 256, 0, stream()>>>(P, pself);
    BG_LAUNCHED();
    emt_add_job(R, pself, self_blocks, NO, sums + (size_t)(NO * NO + NO) * NPQ);
  }
  return BG_OK;
}

// GetPFTMatrix with EMT (GetPFT.cc:133-189, EMTPFT.cc:324-493): out[8*no + c],
// c = PAbs, PScat, Fx, Fy, Fz, Tx, Ty, Tz (force and torque in the
// reference's units, TENTHIRDS = 10/3), plane-wave incident field.
// The pair sums go through tetrahedra (emt_pairs.cuh) while every basis
// function stays below the rule switch |omega| R = 5; above it pairs of one
// tetrahedron pair ask for different rules and are taken one by one.  All
// partial sums are added on the device in a fixed order; one small copy
// returns them.
static int pft_emt_impl(bg_geometry *g, double wr, double wi, const void *dJ, const void *dDR, size_t ldr,
                        const double *E0, const double *nhat, double *out) {
  int st = init_tables();
  if (st) return st;
  int NO = (int)g->objs.size();
  if (NO > PMAXOBJ) { set_error("PFT supports at most %d objects", PMAXOBJ); return BG_ERR_ARG; }
  PftArgs P{g->dev, (const cd *)dJ, wr, std::sqrt(wr * wr + wi * wi), NO, (const cd *)dDR, ldr};
  const int nrow = pft_point_blocks(g);
  if ((st = build_near_lists(g))) return st;
  const bool tets = P.absw * g->bf_rmax <= 5.0;
  const int NP2 = NO * NO * NPQ;
  // block partials of the far, near and self sums
  size_t nfar = 0, nnear = 0, nself = 0, npts = 0;
  EmtBlockMap bm{};
  int far_blocks = 0, near_blocks = 0, near_per = 1, self_blocks = 0;
  const int nb = (g->N + FT - 1) / FT;
  if (tets) {
    const int q = dDR ? 1 : 4, jt = dDR ? EMT_DJ : EMT_JT;
    // short chunks while there are few points, so that every SM has blocks
    bm.ic = dDR ? EMT_DI : (4 * g->NT <= 8192 ? EMT_JT : 4 * EMT_JT);
    for (int oa = 0; oa < NO; oa++)
      for (int ob = oa; ob < NO; ob++) {
        const int m = bm.nmap;
        bm.first[m] = far_blocks;
        bm.oa[m] = oa; bm.ob[m] = ob;
        bm.i0[m] = q * g->tOffset[oa]; bm.i1[m] = q * (g->tOffset[oa] + g->objs[oa].nt);
        bm.j0[m] = q * g->tOffset[ob]; bm.j1[m] = q * (g->tOffset[ob] + g->objs[ob].nt);
        bm.nj[m] = (bm.j1[m] - bm.j0[m] + jt - 1) / jt;
        const long long nblk = (long long)bm.nj[m] * ((bm.i1[m] - bm.i0[m] + bm.ic - 1) / bm.ic);
        if (nblk == 0) continue;
        if (far_blocks + nblk > 0x7fffffffLL) { set_error("PFT: geometry too large"); return BG_ERR_ARG; }
        far_blocks += (int)nblk;
        bm.nmap++;
      }
    if (g->near.ntp > 0) {
      near_blocks = std::min(148 * 8, (g->near.ntp + 4 * EMT_NG - 1) / (4 * EMT_NG));
      near_per = (g->near.ntp + near_blocks * EMT_NG - 1) / (near_blocks * EMT_NG);
    }
    self_blocks = (g->N + 15) / 16;
    nfar = (size_t)far_blocks * NPQ;
    nnear = (size_t)near_blocks * NO * NPQ;
    nself = (size_t)self_blocks * NO;
    npts = dDR ? 0 : (size_t)4 * g->NT * EMT_PT;
  } else {
    near_blocks = (g->near.npairs * 32 + 255) / 256;
    nfar = (size_t)nb * nb * NP2;
    nnear = (size_t)near_blocks * NO * NPQ;
  }
  const size_t next = (size_t)nrow * NO * NPQ;
  // sums first: far [NO][NO][NPQ], near [NO][NPQ], self [NO], extinction [NO][NPQ]
  const size_t nsum = (size_t)NP2 + (size_t)NO * NPQ + NO + (size_t)NO * NPQ;
  const size_t nsum_pad = (nsum + 1) / 2 * 2;     // the points are read as pairs
  const size_t nparts = nfar + nnear + nself;
  if ((st = ensure_scratch(g, sizeof(double) * (nsum_pad + nparts + npts + next)))) return st;
  double *sums = g->d_scratch, *part = sums + nsum_pad, *pext = part + nparts + npts;
  double *sext = sums + (size_t)NP2 + (size_t)NO * NPQ + NO;
  BG_CUDA_TRY(cudaMemsetAsync(sums, 0, sizeof(double) * nsum, stream()));
  EmtReduce R{};
  if (tets) {
    if ((st = emt_tet_sums(g, P, part, sums, R, bm, far_blocks, near_blocks, near_per, self_blocks))) return st;
  } else {
    k_pft_far<<<dim3(nb, nb), dim3(FT, FT), 0, stream()>>>(P, part);
    BG_LAUNCHED();
    emt_add_job(R, part, (long long)nb * nb, NP2, sums);
    if (g->near.npairs > 0) {
      k_pft_near<<<near_blocks, 256, 0, stream()>>>(P, g->near, part + nfar);
      BG_LAUNCHED();
      emt_add_job(R, part + nfar, near_blocks, NO * NPQ, sums + NP2);
    }
  }
  if (E0) {
    PWave pw = make_pw(wr, wi, E0, nhat);
    k_pft_ext<<<nrow, 128, 0, stream()>>>(P, pw, pext);
    BG_LAUNCHED();
    emt_add_job(R, pext, nrow, NO * NPQ, sext);
  }
  if (R.n) {
    k_emt_reduce<<<dim3(R.n, R.wmax), 256, 0, stream()>>>(R);
    BG_LAUNCHED();
  }
  std::vector<double> h(nsum);
  BG_CUDA_TRY(cudaMemcpyAsync(h.data(), sums, sizeof(double) * nsum, cudaMemcpyDeviceToHost, stream()));
  BG_CUDA_TRY(cudaStreamSynchronize(stream()));
  const double *scat = h.data(), *near = scat + NP2, *self = near + NO * NPQ, *ext = self + NO;
  double ftf = 0.5 * TEN_THIRDS / wr;
  for (int o = 0; o < NO; o++) {
    double s[NPQ] = {0};
    for (int ob = 0; ob < NO; ob++)
      for (int n = 0; n < NPQ; n++) s[n] += scat[((size_t)o * NO + ob) * NPQ + n];
    for (int n = 0; n < NPQ; n++) s[n] += near[o * NPQ + n];
    s[0] += self[o];
    const double *e = ext + (size_t)o * NPQ;
    double *r = out + 8 * o;
    r[0] = 0.5 * e[0] - s[0];
    r[1] = s[0];
    for (int i = 0; i < 3; i++) {
      r[2 + i] = ftf * e[1 + i] - s[1 + i];
      r[5 + i] = ftf * (e[4 + i] + e[7 + i]) - s[4 + i] - s[7 + i];
    }
  }
  return BG_OK;
}

int pft_emt_full(bg_geometry *g, double wr, double wi, const void *dJ, const double *E0, const double *nhat,
                 double *out) {
  return pft_emt_impl(g, wr, wi, dJ, nullptr, 0, E0, nhat, out);
}

// GetPFTMatrix(0, Omega, {EMT, DRMatrix}) as buff-neq calls it (GetFlux.cc:391-399):
// the pair sums with JJ = DR(b, a) and no incident field
int pft_emt_dr(bg_geometry *g, double wr, double wi, const void *dDR, size_t ldr, double *out) {
  return pft_emt_impl(g, wr, wi, nullptr, dDR, ldr, nullptr, nullptr, out);
}

// =========================================================================
// Overlap blocks for buff-neq (GetOverlaps, VIEMatrix.cc:122-316, and
// GetOverlapElements, SWGVolume.cc:405-481), row a: up to 7 columns b with
//   S_ab  = int b_a . b_b (closed form),
//   V_ab  = -w^2 int b_a . (eps - 1) b_b,
//   R_ab  = 4 w / (pi Z0) int b_a . Im(eps - 1) b_b   (uniform temperature),
// w = real(omega), the V and R integrals by the 33-point rule on each
// tetrahedron of a.  Slot 0 is the diagonal; cnt[a] is the number of slots.
// =========================================================================
__global__ void k_neq_overlaps(DevGeom g, double w, int *idx, double *S, cd *V, double *R, int *cnt) {
  int a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= g.N) return;
  int2 tt = g.bfTet[a], qq = g.bfQ[a];
  int4 fv = g.bfV[a];
  double Aa = g.bfArea[a];
  double cen[3], P1[3], P2[3], P3[3];
  load3(g.V4, fv.x, P1); load3(g.V4, fv.y, P2); load3(g.V4, fv.z, P3);
  for (int c = 0; c < 3; c++) cen[c] = (P1[c] + P2[c] + P3[c]) / 3.0;
  int nnz = 1;
  int ix[8];
  double sv[8], rv[8];
  cd vv[8];
  ix[0] = a; sv[0] = 0.0; rv[0] = 0.0; vv[0] = cmk(0, 0);
  const double rpre = 4.0 * w / (M_PI * 376.73031346177), vpre = -w * w;
  for (int side = 0; side < 2; side++) {
    int t = side == 0 ? tt.x : tt.y;
    double sa = side == 0 ? 1.0 : -1.0;
    const bg_material &mat = g.mats[g.tetObj[t]];
    const DevExpr *mex = g.expr ? g.expr + g.tetObj[t] : nullptr;
    double vol = g.tetVol[t];
    double QA[3];
    load3(g.V4, side == 0 ? qq.x : qq.y, QA);
    // closed-form Gram terms of this tetrahedron
    double L2s = 0.0, XmQ[3], XmQ2 = 0.0;
    for (int c = 0; c < 3; c++) {
      double d1 = P1[c] - QA[c], d2 = P2[c] - QA[c], d3 = P3[c] - QA[c];
      L2s += d1 * d1 + d2 * d2 + d3 * d3;
      XmQ[c] = cen[c] - QA[c];
      XmQ2 += XmQ[c] * XmQ[c];
    }
    sv[0] += Aa * Aa * (XmQ2 / 20.0 + L2s / 180.0) / vol;
    double pa = sa * Aa / (3.0 * vol);
    int4 vi = g.tetVI[t];
    double V0[3], L[3][3];
    load3(g.V4, vi.x, V0);
    int vq[3] = {vi.y, vi.z, vi.w};
    for (int i = 0; i < 3; i++) {
      double tmp[3];
      load3(g.V4, vq[i], tmp);
      for (int c = 0; c < 3; c++) L[i][c] = tmp[c] - V0[c];
    }
    int4 fi = g.tetFI[t];
    int fl[4] = {fi.x, fi.y, fi.z, fi.w};
    for (int ifb = 0; ifb < 4; ifb++) {
      int b = fl[ifb];
      if (b < 0) continue;
      int2 tb = g.bfTet[b], qb = g.bfQ[b];
      double QB[3], pb, sb;
      if (tb.x == t) { load3(g.V4, qb.x, QB); sb = 1.0; }
      else { load3(g.V4, qb.y, QB); sb = -1.0; }
      pb = sb * g.bfArea[b] / (3.0 * vol);
      cd accv = cmk(0, 0);
      double accr = 0.0;
      for (int i = 0; i < 33; i++) {
        const double *u = c_tcr33 + 4 * i;
        double wt = 6.0 * vol * u[3], x[3];
        for (int c = 0; c < 3; c++) x[c] = V0[c] + u[0] * L[0][c] + u[1] * L[1][c] + u[2] * L[2][c];
        cd E[3][3];
        mat_eval(mat, mex, x, E);
        E[0][0].r -= 1.0; E[1][1].r -= 1.0; E[2][2].r -= 1.0;
        double FA[3], FB[3];
        for (int c = 0; c < 3; c++) { FA[c] = pa * (x[c] - QA[c]); FB[c] = pb * (x[c] - QB[c]); }
        cd v = cmk(0, 0);
        double r = 0.0;
        for (int mu = 0; mu < 3; mu++)
          for (int nu = 0; nu < 3; nu++) {
            v = cadd(v, cscale(E[mu][nu], FA[mu] * FB[nu]));
            r += FA[mu] * E[mu][nu].i * FB[nu];
          }
        accv = cadd(accv, cscale(v, vpre * wt));
        accr += rpre * r * wt;
      }
      if (b == a) {
        vv[0] = cadd(vv[0], accv);
        rv[0] += accr;
      } else {
        double pf = 2.0 * sa * sb * Aa * g.bfArea[b] / (3.0 * vol);
        double xd = XmQ[0] * (QA[0] - QB[0]) + XmQ[1] * (QA[1] - QB[1]) + XmQ[2] * (QA[2] - QB[2]);
        ix[nnz] = b;
        sv[nnz] = pf * (3.0 * XmQ2 / 40.0 + L2s / 120.0 + xd / 8.0);
        vv[nnz] = accv;
        rv[nnz] = accr;
        nnz++;
      }
    }
  }
  for (int i = 0; i < 8; i++) {
    size_t o = 8 * (size_t)a + i;
    idx[o] = i < nnz ? ix[i] : -1;
    S[o] = i < nnz ? sv[i] : 0.0;
    V[o] = i < nnz ? vv[i] : cmk(0, 0);
    R[o] = i < nnz ? rv[i] : 0.0;
  }
  cnt[a] = nnz;
}

int neq_overlaps(bg_geometry *g, double w, int *idx, double *S, void *V, double *R, int *cnt) {
  int st = init_tables();
  if (st) return st;
  if ((st = refresh_materials(g, w, 0.0))) return st;
  k_neq_overlaps<<<(g->N + 127) / 128, 128, 0, stream()>>>(g->dev, w, idx, S, (cd *)V, R, cnt);
  BG_LAUNCHED();
  return BG_OK;
}

// Absorbed power per object by the overlap method with every number kept on
// the device (for captured graphs): partial sums into part (ceil(N/128) x NO
// doubles), then out[o] = sum over blocks, o < NO.
int opft_enqueue(bg_geometry *g, double wr, double wi, const void *dJ, const double *fq, double *part,
                 double *out_dev) {
  if (g->dispersive && fq) { set_error("frequency-dependent materials need a host frequency"); return BG_ERR_ARG; }
  int NO = (int)g->objs.size();
  if (NO > PMAXOBJ) { set_error("PFT supports at most %d objects", PMAXOBJ); return BG_ERR_ARG; }
  PftArgs P{g->dev, (const cd *)dJ, wr, std::sqrt(wr * wr + wi * wi), NO};
  const int nblk = pft_point_blocks(g);
  k_opft<<<nblk, 128, 0, stream()>>>(P, cd{wr, wi}, part, fq);
  BG_LAUNCHED();
  k_opft_reduce<<<NO, 256, 0, stream()>>>(nblk, NO, part, out_dev);
  BG_LAUNCHED();
  return BG_OK;
}

}  // namespace bg
