// Learned form, network side: a graph network over the near-field graph of
// the SWG basis functions (nodes = basis functions, edges = pairs sharing a
// vertex, self pairs included) that predicts the entries of a sparse
// approximate inverse M on that pattern, used as the right preconditioner of
// GMRES (gmres.cu).
//
//   node features f_i (8) and edge features g_e (8) from the assembled
//   matrix (ratios to the diagonal) and the geometry;
//   h^0 = relu(W0 f + b0)                                           (width 64)
//   3 x [ z_e = Wmh h_{j(e)} + Wme g_e + bm         (Wmh h computed per node)
//         agg_i = mean_{e in row i} relu(z_e)
//         h_i <- h_i + relu(Wuh h_i + Wua agg_i + bu) ]
//   edge readout: y_e = relu(Wri h_i + Wrj h_j + Wrg g_e + br)       (64)
//                 o_e = Wo y_e + bo                                 (4)
//                 c = GNN_CMAX (tanh(o0) + i tanh(o1))
//                 s = smax (tanh(o2) + i tanh(o3) / 2)
//   m_ij = [delta_ij + c - [i != j] s A_ij / A_ii] / A_jj
// With s = 1 and c = 0 the off-diagonal term would be the first-order
// Neumann approximation of A^{-1} around its diagonal.  Written D M = I - K
// (D = diag A), M is singular where K has an eigenvalue 1, and a preconditioner
// close to that makes GMRES stall on a few modes that no averaged objective
// sees.  For a constant coefficient K = s K1, K1 the scaled near-field
// off-diagonal part (K1_ij = A_ij / A_jj on the pattern), whose dominant
// eigenvalue is real and positive on these matrices (about 2.2 at N = 8k, 2.6
// at N = 57k); GMRES stalled exactly when s crossed 1 / rho(K1).  So a power
// iteration estimates rho(K1) for the matrix at hand and the coefficient is
// bounded by smax = GNN_SREL / max(GNN_SREL, rho(K1)), with the diagonal
// correction c kept small.  Wo and bo start at zero, so the untrained network
// is the Jacobi (diagonal) inverse.
//
// Training objective (per matrix; p probes z and a right-hand side b with its
// LU solution x):
//   L = |A M Z - Z|_F^2 / (N p) + lambda |M b - x|^2 / |x|^2
// The probes are random, or random vectors pushed k times through the Jacobi
// error map z <- z - A D^{-1} z and rescaled to |z|^2 = 2N: those concentrate
// on the modes where the off-diagonal part dominates, which a Frobenius
// objective over random probes barely sees but which decide how many GMRES
// steps the preconditioned system takes.
// The parameters descend log L (gradient dL / L), which weighs matrices of
// very different conditioning alike.  G = 2 dL/dconj(M) on the pattern,
// hand-written backward kernels, Adam with global gradient-norm clipping.
// FP32 in the network; products with A in FP64.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <vector>

#include "internal.h"

namespace bg {

#define GW 64          // width
#define GF 8           // node features
#define GE 8           // edge features
#define GL 3           // message-passing layers
#define GO 4           // outputs per edge
#define GNN_MAXP 16    // probes per training step
#define GNN_CMAX 0.1f  // bound of the diagonal-term correction c
#define GNN_SREL 0.7   // |Re s| < GNN_SREL / rho(K1)
#define GNN_POWER_ITERS 16

// parameter layout (floats); matrices row-major (out x in)
struct GnnLayout {
  int W0, b0, Wmh[GL], Wme[GL], bm[GL], Wuh[GL], Wua[GL], bu[GL], Wri, Wrj, Wrg, br, Wo, bo, total;
  GnnLayout() {
    int o = 0;
    W0 = o; o += GW * GF;
    b0 = o; o += GW;
    for (int l = 0; l < GL; l++) {
      Wmh[l] = o; o += GW * GW;
      Wme[l] = o; o += GW * GE;
      bm[l] = o; o += GW;
      Wuh[l] = o; o += GW * GW;
      Wua[l] = o; o += GW * GW;
      bu[l] = o; o += GW;
    }
    Wri = o; o += GW * GW;
    Wrj = o; o += GW * GW;
    Wrg = o; o += GW * GE;
    br = o; o += GW;
    Wo = o; o += GO * GW;
    bo = o; o += GO;
    total = o;
  }
};
static const GnnLayout LAY;

struct z2g { double r, i; };

__device__ __forceinline__ z2g zmul(z2g a, z2g b) { return z2g{a.r * b.r - a.i * b.i, a.r * b.i + a.i * b.r}; }
__device__ __forceinline__ z2g zconj(z2g a) { return z2g{a.r, -a.i}; }
__device__ __forceinline__ z2g zdiv(z2g a, z2g b) {
  double d = b.r * b.r + b.i * b.i;
  return z2g{(a.r * b.r + a.i * b.i) / d, (a.i * b.r - a.r * b.i) / d};
}

// ------------------------------------------------------------------ features
// One warp per row i, its lanes over the edges (one thread per row left 30
// blocks of scattered reads at N = 3,822: 590 -> 44 us).  A column-major: A_ij at
// A[j * lda + i].
// node: 1, Re/Im(A_ii)/|A_ii|, omega h, area/h^2, radius/h, degree/100, log10|A_ii|/10
// edge: Re/Im(A_ij/A_ii), Re/Im(A_ji/A_jj), distance of face centroids / h,
//       common vertices / 5, [i == j], |A_ij/A_ii|
__global__ void k_gnn_features(int N, const int *rowptr, const int *col, const z2g *A, size_t lda, DevGeom g,
                               double omega, double h, float *F, float *Ef, z2g *ratio, z2g *dinv) {
  const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (i >= N) return;
  z2g a = A[(size_t)i * lda + i];
  double am = sqrt(a.r * a.r + a.i * a.i);
  float *f = F + (size_t)i * GF;
  int deg = rowptr[i + 1] - rowptr[i];
  if (lane == 0) {
    dinv[i] = zdiv(z2g{1.0, 0.0}, a);
    f[0] = 1.f;
    f[1] = (float)(a.r / am);
    f[2] = (float)(a.i / am);
    f[3] = (float)(omega * h);
    f[4] = (float)(g.bfArea[i] / (h * h));
    f[5] = (float)(g.bfRadius[i] / h);
    f[6] = (float)(deg / 100.0);
    f[7] = (float)(0.1 * log10(am + 1e-300));
  }
  int4 vi = g.bfV[i];
  int2 qi = g.bfQ[i];
  int Vi[5] = {qi.x, vi.x, vi.y, vi.z, qi.y};
  double ci[3] = {0, 0, 0};
  for (int k = 1; k < 4; k++)
    for (int c = 0; c < 3; c++) ci[c] += g.V4[4 * Vi[k] + c] / 3.0;
  for (int e = rowptr[i] + lane; e < rowptr[i + 1]; e += 32) {
    int j = col[e];
    z2g r = zdiv(A[(size_t)j * lda + i], a);
    z2g rt = zdiv(A[(size_t)i * lda + j], A[(size_t)j * lda + j]);
    int4 vj = g.bfV[j];
    int2 qj = g.bfQ[j];
    int Vj[5] = {qj.x, vj.x, vj.y, vj.z, qj.y};
    int ncv = 0;
    for (int p = 0; p < 5; p++)
      for (int q = 0; q < 5; q++) ncv += Vi[p] == Vj[q];
    double cj[3] = {0, 0, 0};
    for (int k = 1; k < 4; k++)
      for (int c = 0; c < 3; c++) cj[c] += g.V4[4 * Vj[k] + c] / 3.0;
    double dist = sqrt((ci[0] - cj[0]) * (ci[0] - cj[0]) + (ci[1] - cj[1]) * (ci[1] - cj[1]) +
                       (ci[2] - cj[2]) * (ci[2] - cj[2]));
    float *ge = Ef + (size_t)e * GE;
    ge[0] = (float)r.r;
    ge[1] = (float)r.i;
    ge[2] = (float)rt.r;
    ge[3] = (float)rt.i;
    ge[4] = (float)(dist / h);
    ge[5] = (float)(ncv / 5.0);
    ge[6] = (i == j) ? 1.f : 0.f;
    ge[7] = (float)sqrt(r.r * r.r + r.i * r.i);
    ratio[e] = r;
  }
}

// ------------------------------------------------------------------ node maps
// Y[n][o] (+)= sum_k X[n][k] w(o, k) (+ bias[o]) for `out` <= 64 outputs and `in`
// <= 64 inputs, w(o, k) = W[o][k] (TRANS false, row length in) or W[k][o] (TRANS
// true, row length out: the gradient with respect to the input).  A block takes
// 64 nodes with the weights and the rows of X in shared memory, a thread 4 x 4
// outputs; every output is one chain of fused multiply-adds over k in order.
// One block per node re-read the weights column by column: 56 -> 11 us a call at
// N = 3,822, 545 -> 21 us at N = 39,150.
#define GLN 64
template <bool TRANS>
__global__ void __launch_bounds__(256) k_gnn_linear(int N, int in, int out, const float *X, int ldx, const float *W,
                                                    const float *bias, float *Y, int ldy, int accumulate) {
  __shared__ __align__(16) float sw[GW][GW + 4];     // sw[k][o]
  __shared__ float sx[GLN][GW + 1];
  const int tid = threadIdx.x, n0 = blockIdx.x * GLN;
  for (int e = tid; e < in * GW; e += 256) {
    const int k = TRANS ? e / GW : e % in, o = TRANS ? e % GW : e / in;
    sw[k][o] = o < out ? W[TRANS ? (size_t)k * out + o : (size_t)o * in + k] : 0.f;
  }
  for (int e = tid; e < GLN * in; e += 256) {
    const int n = e / in, k = e % in;
    sx[n][k] = n0 + n < N ? X[(size_t)(n0 + n) * ldx + k] : 0.f;
  }
  __syncthreads();
  const int o0 = (tid & 15) * 4, r0 = (tid >> 4) * 4;
  float s[4][4];
#pragma unroll
  for (int r = 0; r < 4; r++)
#pragma unroll
    for (int c = 0; c < 4; c++) s[r][c] = bias && o0 + c < out ? bias[o0 + c] : 0.f;
#pragma unroll 4
  for (int k = 0; k < in; k++) {
    const float4 w = *reinterpret_cast<const float4 *>(&sw[k][o0]);
#pragma unroll
    for (int r = 0; r < 4; r++) {
      const float x = sx[r0 + r][k];
      s[r][0] = fmaf(x, w.x, s[r][0]);
      s[r][1] = fmaf(x, w.y, s[r][1]);
      s[r][2] = fmaf(x, w.z, s[r][2]);
      s[r][3] = fmaf(x, w.w, s[r][3]);
    }
  }
#pragma unroll
  for (int r = 0; r < 4; r++)
#pragma unroll
    for (int c = 0; c < 4; c++) {
      if (n0 + r0 + r >= N || o0 + c >= out) continue;
      float *y = Y + (size_t)(n0 + r0 + r) * ldy + o0 + c;
      *y = accumulate ? *y + s[r][c] : s[r][c];
    }
}

__global__ void k_gnn_relu(int n, const float *Z, float *H) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) H[i] = fmaxf(Z[i], 0.f);
}

// messages and mean aggregation over row i: Zm[e] = P[j(e)] + Wme g_e + bm
__global__ void k_gnn_msg(int N, const int *__restrict__ rowptr, const int *__restrict__ col,
                          const float *__restrict__ P, const float *__restrict__ Ef, const float *Wme, const float *bm,
                          float *__restrict__ Zm, float *agg) {
  int i = blockIdx.x, o = threadIdx.x;
  if (i >= N) return;
  float w[GE];
  for (int k = 0; k < GE; k++) w[k] = Wme[o * GE + k];
  float b = bm[o], s = 0.f;
  int e0 = rowptr[i], e1 = rowptr[i + 1];
#pragma unroll 4
  for (int e = e0; e < e1; e++) {
    const float4 g0 = reinterpret_cast<const float4 *>(Ef)[2 * (size_t)e], g1 = reinterpret_cast<const float4 *>(Ef)[2 * (size_t)e + 1];
    const float ge[GE] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
    float z = P[(size_t)col[e] * GW + o] + b;
#pragma unroll
    for (int k = 0; k < GE; k++) z += w[k] * ge[k];
    if (Zm) Zm[(size_t)e * GW + o] = z;
    s += fmaxf(z, 0.f);
  }
  agg[(size_t)i * GW + o] = s / fmaxf(1.f, (float)(e1 - e0));
}

// H_next = H + relu(U)
__global__ void k_gnn_residual(int n, const float *H, const float *U, float *Hn) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) Hn[i] = H[i] + fmaxf(U[i], 0.f);
}

// edge readout, one warp per row, four edges at a time; lane owns hidden units
// lane and lane + 32.  The 16 sums over hidden units (4 edges x 4 outputs) are
// reduced together, each exchange halving the values a lane still carries (31
// shuffles in place of 80), and end one per lane pair, so that the bounded
// outputs of the four edges are evaluated side by side (240 -> 123 us at N =
// 3,822, 1.78 -> 0.89 ms at N = 39,150).
__global__ void __launch_bounds__(128) k_gnn_readout(int N, const int *__restrict__ rowptr, const int *__restrict__ col,
                                                     const float *__restrict__ Pr, const float *__restrict__ Qr,
                                                     const float *__restrict__ Ef, const float *Wrg, const float *br,
                                                     const float *Wo, const float *bo, const z2g *__restrict__ ratio,
                                                     const z2g *__restrict__ dinv, float smax, float *__restrict__ Zr,
                                                     float *__restrict__ Oe, z2g *__restrict__ Mval) {
  int i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  int lane = threadIdx.x & 31;
  if (i >= N) return;
  float wg[2][GE], wo[2][GO], bb[2], pi[2];
  for (int t = 0; t < 2; t++) {
    int o = lane + 32 * t;
    for (int k = 0; k < GE; k++) wg[t][k] = Wrg[o * GE + k];
    for (int k = 0; k < GO; k++) wo[t][k] = Wo[k * GW + o];
    bb[t] = br[o];
    pi[t] = Pr[(size_t)i * GW + o];
  }
  const float bk = bo[(lane >> 1) & 3];
  const int e1 = rowptr[i + 1];
  for (int eb = rowptr[i]; eb < e1; eb += 4) {
    float v[4 * GO];
#pragma unroll
    for (int m = 0; m < 4; m++) {
      const int e = min(eb + m, e1 - 1);
      const float4 g0 = reinterpret_cast<const float4 *>(Ef)[2 * (size_t)e], g1 = reinterpret_cast<const float4 *>(Ef)[2 * (size_t)e + 1];
      const float g[GE] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
      const int j = col[e];
#pragma unroll
      for (int k = 0; k < GO; k++) v[m * GO + k] = 0.f;
#pragma unroll
      for (int t = 0; t < 2; t++) {
        int o = lane + 32 * t;
        float z = pi[t] + Qr[(size_t)j * GW + o] + bb[t];
#pragma unroll
        for (int k = 0; k < GE; k++) z += wg[t][k] * g[k];
        if (Zr && eb + m < e1) Zr[(size_t)e * GW + o] = z;
        float y = fmaxf(z, 0.f);
#pragma unroll
        for (int k = 0; k < GO; k++) v[m * GO + k] += wo[t][k] * y;
      }
    }
#pragma unroll
    for (int h = 8; h > 0; h >>= 1) {      // partner lane ^ 2h; v[0 .. 2h) -> v[0 .. h)
      const bool up = lane & (2 * h);
#pragma unroll
      for (int k = 0; k < h; k++) {
        const float give = up ? v[k] : v[k + h], keep = up ? v[k + h] : v[k];
        v[k] = keep + __shfl_xor_sync(0xffffffffu, give, 2 * h);
      }
    }
    const float o = v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1) + bk;   // edge lane >> 3, output (lane >> 1) & 3
    const int e = eb + (lane >> 3), ec = min(e, e1 - 1);
    if (Oe && e < e1 && !(lane & 1)) Oe[(size_t)e * GO + ((lane >> 1) & 3)] = o;
    const float t0 = tanhf(o), t1 = __shfl_down_sync(0xffffffffu, t0, 2), t2 = __shfl_down_sync(0xffffffffu, t0, 4),
                t3 = __shfl_down_sync(0xffffffffu, t0, 6);
    if (e < e1 && !(lane & 7)) {
      const int j = col[ec];
      z2g c{(i == j ? 1.0 : 0.0) + GNN_CMAX * t0, (double)(GNN_CMAX * t1)};
      if (i != j) {
        z2g sr = zmul(z2g{(double)(smax * t2), (double)(0.5f * smax * t3)}, ratio[ec]);
        c.r -= sr.r;
        c.i -= sr.i;
      }
      Mval[e] = zmul(c, dinv[j]);
    }
  }
}

// W[:, q] = K1 V[:, q] / |V[:, q]|, (K1)_ij = A_ij / A_jj = r_e dinv_j / dinv_i off
// the diagonal, nrm2 holding the squared norms of V; part[block][q] = the
// block's share of |W[:, q]|^2.  Norm and scaling stay on the device, so the
// power iteration runs without a round trip per step.
__global__ void __launch_bounds__(256) k_gnn_k1mv(int N, const int *rowptr, const int *col, const z2g *ratio,
                                                  const z2g *dinv, const z2g *V, const double *nrm2, int nv, z2g *W,
                                                  double *part) {
  // a warp per row (its entries are contiguous), all nv <= 4 vectors per
  // read of the row; lane partial sums combined by a fixed butterfly
  int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, sub = threadIdx.x & 31;
  z2g s[4] = {{0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}};
  if (i < N) {
    int e1 = rowptr[i + 1];
#pragma unroll 2
    for (int e = rowptr[i] + sub; e < e1; e += 32) {
      int j = col[e];
      z2g rj = zmul(ratio[e], dinv[j]);
      if (j == i) rj = z2g{0.0, 0.0};
#pragma unroll
      for (int q = 0; q < 4; q++)
        if (q < nv) {
          z2g t = zmul(rj, V[(size_t)q * N + j]);
          s[q].r += t.r;
          s[q].i += t.i;
        }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int q = 0; q < 4; q++) {
      s[q].r += __shfl_xor_sync(0xffffffffu, s[q].r, o);
      s[q].i += __shfl_xor_sync(0xffffffffu, s[q].i, o);
    }
  __shared__ double red[8][4];     // rows of the block
  if (sub == 0) {
    const z2g ai = i < N ? zdiv(z2g{1.0, 0.0}, dinv[i]) : z2g{0.0, 0.0};
    for (int q = 0; q < 4; q++) {
      double n2 = 0.0;
      if (i < N && q < nv) {
        const double f = nrm2[q] > 0 ? 1.0 / sqrt(nrm2[q]) : 0.0;
        z2g w = zmul(ai, s[q]);
        w.r *= f;
        w.i *= f;
        W[(size_t)q * N + i] = w;
        n2 = w.r * w.r + w.i * w.i;
      }
      red[threadIdx.x >> 5][q] = n2;
    }
  }
  __syncthreads();
  if (threadIdx.x < 4) {
    double t = 0.0;
    for (int r = 0; r < 8; r++) t += red[r][threadIdx.x];
    part[4 * (size_t)blockIdx.x + threadIdx.x] = t;
  }
}

// nrm2[q] = sum of part[0 .. nblk)[q]
__global__ void __launch_bounds__(256) k_gnn_norm4(int nblk, const double *part, double *nrm2) {
  __shared__ double red[64][4];
  const int q = threadIdx.x & 3, l = threadIdx.x >> 2;
  double s = 0.0;
  for (int b = l; b < nblk; b += 64) s += part[4 * (size_t)b + q];
  red[l][q] = s;
  __syncthreads();
  if (threadIdx.x < 4) {
    double t = 0.0;
    for (int r = 0; r < 64; r++) t += red[r][threadIdx.x];
    nrm2[threadIdx.x] = t;
  }
}

// squared norms of columns (one block per column, fixed reduction order)
__global__ void k_gnn_colnorm2(int N, const z2g *V, double *out) {
  const z2g *v = V + (size_t)blockIdx.x * N;
  __shared__ double red[32];
  double s = 0;
  for (int i = threadIdx.x; i < N; i += blockDim.x) s += v[i].r * v[i].r + v[i].i * v[i].i;
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0;
    for (int k = 0; k < (int)(blockDim.x >> 5); k++) t += red[k];
    out[blockIdx.x] = t;
  }
}

// ------------------------------------------------------------------ backward
// output gradients per edge from G = 2 dL/dconj(m):
// t = conj(G) d_j, u = conj(G) r_e d_j ; d(c, s) = (Re t, -Im t, -Re u, Im u)
// (u terms off-diagonal only), then through the bounded tanh maps of o
__global__ void k_gnn_dout(int N, const int *rowptr, const int *col, const z2g *G, double gscale, const z2g *ratio,
                           const z2g *dinv, float smax, const float *Oe, float *dO) {
  // a warp per row, its lanes over the edges
  const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (i >= N) return;
  for (int e = rowptr[i] + lane; e < rowptr[i + 1]; e += 32) {
    int j = col[e];
    z2g t = zmul(zconj(G[e]), dinv[j]);
    t.r *= gscale;
    t.i *= gscale;
    float *d = dO + (size_t)e * GO;
    d[0] = (float)t.r;
    d[1] = (float)(-t.i);
    if (i != j) {
      z2g u = zmul(t, ratio[e]);
      d[2] = (float)(-u.r);
      d[3] = (float)u.i;
    } else {
      d[2] = d[3] = 0.f;
    }
    for (int k = 0; k < GO; k++) {
      float th = tanhf(Oe[(size_t)e * GO + k]);
      d[k] *= (k < 2 ? GNN_CMAX : (k == 2 ? smax : 0.5f * smax)) * (1.f - th * th);
    }
  }
}

// Weight gradients are sums over all nodes or edges.  The blocks of a kernel
// leave partial sums, each over its own rows in a fixed order, and
// k_gnn_reduce adds them in block order: no atomics, results do not depend on
// the schedule.
#define GPB 740                  // blocks (and partial sums) of an edge kernel at most
#define GWB 148                  // and of k_gnn_wgrad
__global__ void __launch_bounds__(256) k_gnn_reduce(int nblk, int stride, const float *part, int off, int n, float *out) {
  __shared__ float sh[16][17];
  const int c = threadIdx.x & 15, g = threadIdx.x >> 4, i = blockIdx.x * 16 + c;
  float s = 0.f;
  if (i < n)
#pragma unroll 8
    for (int b = g; b < nblk; b += 16) s += part[(size_t)b * stride + off + i];
  sh[g][c] = s;
  __syncthreads();
  if (threadIdx.x < 16 && i < n) {
    float t = 0.f;
#pragma unroll
    for (int k = 0; k < 16; k++) t += sh[k][c];
    out[i] += t;
  }
}

// weight gradient of a node map: part[block][o][k] = sum_n dY[n][o] X[n][k] over
// the block's nodes, then part[block][64 * in + o] = sum_n dY[n][o].  64 x in
// outputs as 4 x 4 per thread, 32 nodes at a time in shared memory (64 blocks
// with a 65-element array per thread took 360 us a call at N = 3,822; now 7 us and
// 7 us for the sums over blocks).
__global__ void __launch_bounds__(256) k_gnn_wgrad(int N, int in, const float *dY, int lddy, const float *X, int ldx,
                                                   float *part) {
  __shared__ __align__(16) float sy[32][GW + 4], sx[32][GW + 4];
  const int tid = threadIdx.x, o0 = (tid >> 4) * 4, k0 = (tid & 15) * 4;
  float s[4][4], sb[4];
#pragma unroll
  for (int r = 0; r < 4; r++) {
    sb[r] = 0.f;
#pragma unroll
    for (int c = 0; c < 4; c++) s[r][c] = 0.f;
  }
  for (int n0 = blockIdx.x * 32; n0 < N; n0 += gridDim.x * 32) {
    __syncthreads();
    for (int e = tid; e < 32 * GW; e += 256) {
      const int n = e / GW, k = e % GW;
      sy[n][k] = n0 + n < N ? dY[(size_t)(n0 + n) * lddy + k] : 0.f;
      sx[n][k] = n0 + n < N && k < in ? X[(size_t)(n0 + n) * ldx + k] : 0.f;
    }
    __syncthreads();
#pragma unroll 4
    for (int n = 0; n < 32; n++) {
      const float4 g = *reinterpret_cast<const float4 *>(&sy[n][o0]), x = *reinterpret_cast<const float4 *>(&sx[n][k0]);
      const float gv[4] = {g.x, g.y, g.z, g.w}, xv[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
      for (int r = 0; r < 4; r++) {
        sb[r] += gv[r];
#pragma unroll
        for (int c = 0; c < 4; c++) s[r][c] = fmaf(gv[r], xv[c], s[r][c]);
      }
    }
  }
  float *p = part + (size_t)blockIdx.x * (GW * in + GW);
#pragma unroll
  for (int r = 0; r < 4; r++) {
#pragma unroll
    for (int c = 0; c < 4; c++)
      if (k0 + c < in) p[(o0 + r) * in + k0 + c] = s[r][c];
    if (k0 == 0) p[GW * in + o0 + r] = sb[r];
  }
}

// Edge kernels of the backward pass: four rows at a time per block (64 threads
// each, thread = hidden unit o), rows strided over the grid; sums over edges
// stay in registers until the block's end.  The gradient of the edge maps,
// part[block][o][k] = sum_e dZ[e][o] g_e[k] and [64 * 8 + o] = sum_e dZ[e][o],
// is formed while dZ is at hand instead of in a pass of its own over it (1.24 ms
// a layer at N = 3,822 beside 0.33 ms for dZ; together 0.18).
#define GEP (GW * (GE + 1))
__device__ __forceinline__ void edge_acc(const float *Ef, int e, float d, float (&acc)[GE + 1]) {
  const float4 a = reinterpret_cast<const float4 *>(Ef)[2 * (size_t)e], b = reinterpret_cast<const float4 *>(Ef)[2 * (size_t)e + 1];
  acc[0] = fmaf(d, a.x, acc[0]); acc[1] = fmaf(d, a.y, acc[1]); acc[2] = fmaf(d, a.z, acc[2]); acc[3] = fmaf(d, a.w, acc[3]);
  acc[4] = fmaf(d, b.x, acc[4]); acc[5] = fmaf(d, b.y, acc[5]); acc[6] = fmaf(d, b.z, acc[6]); acc[7] = fmaf(d, b.w, acc[7]);
  acc[GE] += d;
}
// sum of v over the four row groups, in order, by group 0
__device__ __forceinline__ float group_sum(float v, float (*sh)[GW]) {
  const int o = threadIdx.x & (GW - 1), g = threadIdx.x / GW;
  __syncthreads();
  sh[g][o] = v;
  __syncthreads();
  return sh[0][o] + sh[1][o] + sh[2][o] + sh[3][o];
}
__device__ __forceinline__ void edge_acc_out(const float (&acc)[GE + 1], float (*sh)[GW], float *p) {
  const int o = threadIdx.x & (GW - 1);
#pragma unroll
  for (int k = 0; k <= GE; k++) {
    const float v = group_sum(acc[k], sh);
    if (threadIdx.x < GW) p[k < GE ? o * GE + k : GW * GE + o] = v;
  }
}

// message backward: dZm[e] = dagg_i / deg_i [Zm > 0], with the edge-map sums
__global__ void __launch_bounds__(256) k_gnn_msg_back(int N, const int *__restrict__ rowptr, const float *__restrict__ Zm,
                                                      const float *__restrict__ dagg, const float *__restrict__ Ef,
                                                      float *__restrict__ dZm, float *part) {
  __shared__ float sh[4][GW];
  const int o = threadIdx.x & (GW - 1), g = threadIdx.x / GW;
  float acc[GE + 1];
#pragma unroll
  for (int k = 0; k <= GE; k++) acc[k] = 0.f;
  for (int i = blockIdx.x * 4 + g; i < N; i += gridDim.x * 4) {
    const int e0 = rowptr[i], e1 = rowptr[i + 1];
    const float da = dagg[(size_t)i * GW + o] / fmaxf(1.f, (float)(e1 - e0));
#pragma unroll 4
    for (int e = e0; e < e1; e++) {
      const float d = __ldcs(Zm + (size_t)e * GW + o) > 0.f ? da : 0.f;
      dZm[(size_t)e * GW + o] = d;
      edge_acc(Ef, e, d, acc);
    }
  }
  edge_acc_out(acc, sh, part + (size_t)blockIdx.x * GEP);
}

// readout backward: dZr[e][o] = (sum_k Wo[k][o] dO[e][k]) [Zr > 0], its row sums
// dP, and the sums for Wrg, br (as above), Wo[k][o] (+ GEP + k * 64 + o) and
// bo[k] (+ GEP + 4 * 64 + k)
#define GRP (GEP + GO * GW + GO)
__global__ void __launch_bounds__(256) k_gnn_readout_back(int N, const int *__restrict__ rowptr, const float *__restrict__ Zr,
                                                          const float *__restrict__ dO, const float *Wo,
                                                          const float *__restrict__ Ef, float *__restrict__ dZr,
                                                          float *__restrict__ dP, float *part) {
  __shared__ float sh[4][GW];
  const int o = threadIdx.x & (GW - 1), g = threadIdx.x / GW;
  float w[GO], acc[GE + 1], aw[GO] = {0.f, 0.f, 0.f, 0.f}, ab = 0.f;
#pragma unroll
  for (int k = 0; k < GO; k++) w[k] = Wo[k * GW + o];
#pragma unroll
  for (int k = 0; k <= GE; k++) acc[k] = 0.f;
  for (int i = blockIdx.x * 4 + g; i < N; i += gridDim.x * 4) {
    float s = 0.f;
    const int e1 = rowptr[i + 1];
#pragma unroll 4
    for (int e = rowptr[i]; e < e1; e++) {
      const float4 d4 = reinterpret_cast<const float4 *>(dO)[e];
      const float zr = __ldcs(Zr + (size_t)e * GW + o), y = fmaxf(zr, 0.f);
      float da = w[0] * d4.x;
      da = fmaf(w[1], d4.y, da);
      da = fmaf(w[2], d4.z, da);
      da = fmaf(w[3], d4.w, da);
      const float d = zr > 0.f ? da : 0.f;
      dZr[(size_t)e * GW + o] = d;
      s += d;
      edge_acc(Ef, e, d, acc);
      aw[0] = fmaf(d4.x, y, aw[0]); aw[1] = fmaf(d4.y, y, aw[1]); aw[2] = fmaf(d4.z, y, aw[2]); aw[3] = fmaf(d4.w, y, aw[3]);
      ab += o == 0 ? d4.x : o == 1 ? d4.y : o == 2 ? d4.z : d4.w;      // used for o < 4
    }
    dP[(size_t)i * GW + o] = s;
  }
  float *p = part + (size_t)blockIdx.x * GRP;
  edge_acc_out(acc, sh, p);
#pragma unroll
  for (int k = 0; k < GO; k++) {
    const float v = group_sum(aw[k], sh);
    if (threadIdx.x < GW) p[GEP + k * GW + o] = v;
  }
  const float v = group_sum(ab, sh);
  if (threadIdx.x < GO) p[GEP + GO * GW + o] = v;
}

// dP[j] = sum over edges e with col(e) = j of dZ[e]  (= sum over row j of dZ[etr])
__global__ void k_gnn_col_gather(int N, const int *rowptr, const int *etr, const float *dZ, float *dP) {
  int j = blockIdx.x, o = threadIdx.x;
  if (j >= N) return;
  float s = 0.f;
  const int e1 = rowptr[j + 1];
#pragma unroll 8
  for (int e = rowptr[j]; e < e1; e++) s += dZ[(size_t)etr[e] * GW + o];
  dP[(size_t)j * GW + o] = s;
}

__global__ void k_gnn_relu_back(int n, const float *Z, const float *dH, float *dZ) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dZ[i] = Z[i] > 0.f ? dH[i] : 0.f;
}

__global__ void k_gnn_sumsq(int n, const float *g, double *out) {
  double s = 0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) s += (double)g[i] * g[i];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) atomicAdd(out, s);
}

// Adam with the gradient scaled to global norm <= clip
__global__ void k_gnn_adam(int n, float *p, const float *g, float *m, float *v, const double *sumsq, float lr,
                           float b1, float b2, float c1, float c2, float eps, float clip) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double nrm = sqrt(*sumsq);
  float sc = nrm > clip ? (float)(clip / nrm) : 1.f;
  float gi = g[i] * sc;
  float mi = b1 * m[i] + (1 - b1) * gi, vi = b2 * v[i] + (1 - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

// ------------------------------------------------------------------ objective
// G_e = scale sum_q S[i,q] conj(Z[j,q]) + scale2 rb_i conj(b_j)
__global__ void k_gnn_sddmm(int N, const int *rowptr, const int *col, const z2g *S, const z2g *Z, int p,
                            double scale, const z2g *rb, const z2g *b, double scale2, z2g *G) {
  const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;   // a warp per row
  if (i >= N) return;
  for (int e = rowptr[i] + lane; e < rowptr[i + 1]; e += 32) {
    int j = col[e];
    double gr = 0, gi = 0;
    for (int q = 0; q < p; q++) {
      z2g s = S[(size_t)q * N + i], z = Z[(size_t)q * N + j];
      gr += s.r * z.r + s.i * z.i;
      gi += s.i * z.r - s.r * z.i;
    }
    gr *= scale;
    gi *= scale;
    if (rb) {
      z2g r = rb[i], bb = b[j];
      gr += scale2 * (r.r * bb.r + r.i * bb.i);
      gi += scale2 * (r.i * bb.r - r.r * bb.i);
    }
    G[e] = z2g{gr, gi};
  }
}

// S[c, q] = sum_r conj(A[r, c]) R[r, q] for GQ columns q at a time: a block takes
// GAC columns of A, its threads the rows, so that a row of R is read once per
// GAC columns; FP64-pipe bound for 8 probes (one warp per column read R from L2
// for every column: 776 -> 136 us at N = 3,822, 8 probes).
#define GQ 8
#define GAC 4
__global__ void __launch_bounds__(128) k_gnn_ahr(int N, const z2g *A, size_t lda, const z2g *R, int p, z2g *S) {
  const int c0 = blockIdx.x * GAC, q0 = blockIdx.y * GQ, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int nq = min(GQ, p - q0);
  z2g s[GAC][GQ];
#pragma unroll
  for (int c = 0; c < GAC; c++)
#pragma unroll
    for (int q = 0; q < GQ; q++) s[c][q] = z2g{0.0, 0.0};
  for (int r = tid; r < N; r += 128) {
    z2g a[GAC];
#pragma unroll
    for (int c = 0; c < GAC; c++) a[c] = c0 + c < N ? A[(size_t)(c0 + c) * lda + r] : z2g{0.0, 0.0};
#pragma unroll
    for (int q = 0; q < GQ; q++) {
      const z2g x = R[(size_t)(q0 + min(q, nq - 1)) * N + r];   // no branch: eight loads in flight
#pragma unroll
      for (int c = 0; c < GAC; c++) {
        s[c][q].r += a[c].r * x.r + a[c].i * x.i;
        s[c][q].i += a[c].r * x.i - a[c].i * x.r;
      }
    }
  }
  __shared__ z2g red[4][GAC][GQ];
#pragma unroll
  for (int c = 0; c < GAC; c++)
#pragma unroll
    for (int q = 0; q < GQ; q++) {
      for (int o = 16; o > 0; o >>= 1) {
        s[c][q].r += __shfl_xor_sync(0xffffffffu, s[c][q].r, o);
        s[c][q].i += __shfl_xor_sync(0xffffffffu, s[c][q].i, o);
      }
      if (lane == 0) red[wid][c][q] = s[c][q];
    }
  __syncthreads();
  if (tid < GAC * GQ) {
    const int c = tid / GQ, q = tid % GQ;
    if (c0 + c < N && q < nq) {
      z2g t = red[0][c][q];
      for (int w = 1; w < 4; w++) { t.r += red[w][c][q].r; t.i += red[w][c][q].i; }
      S[(size_t)(q0 + q) * N + c0 + c] = t;
    }
  }
}

// part[chunk][q][r] = sum over the chunk's columns c of A[r, c] X[c, q]; then
// k_gnn_mul_sum adds the chunks in order, times sign.  A is read once per GQ
// probes (a 64-column GEMM tile on 8 probes: 190 -> 70 us, and 22 us
// for the chunk sums, at N = 3,822; reading A once takes 36).
__global__ void __launch_bounds__(128) k_gnn_mul(int N, const z2g *__restrict__ A, size_t lda,
                                                 const z2g *__restrict__ X, int p, int chunk, z2g *__restrict__ part) {
  __shared__ z2g xs[32][GQ];
  const int r = blockIdx.x * 256 + threadIdx.x, q0 = blockIdx.z * GQ, nq = min(GQ, p - q0);
  const int ra = min(r, N - 1), rb = min(r + 128, N - 1);
  const int c0 = blockIdx.y * chunk, c1 = min(N, c0 + chunk);
  z2g s[2][GQ];
#pragma unroll
  for (int q = 0; q < GQ; q++) s[0][q] = s[1][q] = z2g{0.0, 0.0};
  for (int cb = c0; cb < c1; cb += 32) {
    __syncthreads();
    for (int e = threadIdx.x; e < 32 * GQ; e += 128) {
      const int c = e & 31, q = e >> 5;
      xs[c][q] = cb + c < c1 && q < nq ? X[(size_t)(q0 + q) * N + cb + c] : z2g{0.0, 0.0};
    }
    __syncthreads();
    const int nc = min(32, c1 - cb);
#pragma unroll 4
    for (int c = 0; c < nc; c++) {
      const z2g *Ac = A + (size_t)(cb + c) * lda;
      const z2g a[2] = {Ac[ra], Ac[rb]};
#pragma unroll
      for (int q = 0; q < GQ; q++) {
        const z2g x = xs[c][q];
#pragma unroll
        for (int t = 0; t < 2; t++) {
          s[t][q].r += a[t].r * x.r - a[t].i * x.i;
          s[t][q].i += a[t].r * x.i + a[t].i * x.r;
        }
      }
    }
  }
#pragma unroll
  for (int t = 0; t < 2; t++)
    if (r + 128 * t < N)
#pragma unroll
      for (int q = 0; q < GQ; q++)
        if (q < nq) part[((size_t)blockIdx.y * p + q0 + q) * N + r + 128 * t] = s[t][q];
}
__global__ void k_gnn_mul_sum(size_t np, int nchunk, const z2g *part, double sign, z2g *Y) {
  const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i >= np) return;
  z2g s{0.0, 0.0};
  for (int k = 0; k < nchunk; k++) {
    const z2g v = part[(size_t)k * np + i];
    s.r += v.r;
    s.i += v.i;
  }
  Y[i] = z2g{sign * s.r, sign * s.i};
}

// Y = D^{-1} Z row-wise (d: 1/A_jj), p columns of length N
__global__ void k_gnn_rowscale(int N, int p, const z2g *d, const z2g *Z, z2g *Y) {
  size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (t >= (size_t)N * p) return;
  Y[t] = zmul(d[t % N], Z[t]);
}

// Z[:, q] += W[:, q] and rescale the column to squared norm 2N (one block per column)
__global__ void k_gnn_probe_update(int N, const z2g *W, z2g *Z) {
  int q = blockIdx.x;
  z2g *z = Z + (size_t)q * N;
  const z2g *w = W + (size_t)q * N;
  __shared__ double red[32];
  double s = 0;
  for (int i = threadIdx.x; i < N; i += blockDim.x) {
    z2g v{z[i].r + w[i].r, z[i].i + w[i].i};
    z[i] = v;
    s += v.r * v.r + v.i * v.i;
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0;
    for (int k = 0; k < (int)(blockDim.x >> 5); k++) t += red[k];
    red[0] = t > 0 ? sqrt(2.0 * N / t) : 1.0;
  }
  __syncthreads();
  double f = red[0];
  for (int i = threadIdx.x; i < N; i += blockDim.x) z[i] = z2g{z[i].r * f, z[i].i * f};
}

__global__ void k_gnn_sub(size_t n, const z2g *A, const z2g *B, z2g *C) {   // C = A - B
  size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i < n) C[i] = z2g{A[i].r - B[i].r, A[i].i - B[i].i};
}

// Y = M X for up to four columns per blockIdx.y, eight lanes per row
__global__ void k_gnn_spmm(int N, const int *rowptr, const int *col, const z2g *val, const z2g *X, int p, z2g *Y) {
  const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 3, sub = threadIdx.x & 7, q0 = 4 * blockIdx.y;
  z2g s[4] = {{0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}};
  if (i < N) {
    const int e1 = rowptr[i + 1];
    for (int e = rowptr[i] + sub; e < e1; e += 8) {
      const z2g m = val[e];
      const int j = col[e];
#pragma unroll
      for (int q = 0; q < 4; q++)
        if (q0 + q < p) {
          const z2g x = X[(size_t)(q0 + q) * N + j];
          s[q].r += m.r * x.r - m.i * x.i;
          s[q].i += m.r * x.i + m.i * x.r;
        }
    }
  }
#pragma unroll
  for (int o = 4; o > 0; o >>= 1)
#pragma unroll
    for (int q = 0; q < 4; q++) {
      s[q].r += __shfl_xor_sync(0xffffffffu, s[q].r, o);
      s[q].i += __shfl_xor_sync(0xffffffffu, s[q].i, o);
    }
  if (i < N && sub == 0)
#pragma unroll
    for (int q = 0; q < 4; q++)
      if (q0 + q < p) Y[(size_t)(q0 + q) * N + i] = s[q];
}

}  // namespace bg

// =============================================================================
// host side
// =============================================================================
struct bg_gnn {
  float *params = nullptr, *grads = nullptr, *m = nullptr, *v = nullptr;
  double *sumsq = nullptr;
  int step = 0;
};

namespace bg {

// per-call activations (the graph itself is cached in the geometry)
struct GnnBufs {
  int N = 0, E = 0;
  double rho_ref = 0;   // estimate of rho(K1)
  float smax = 0;       // bound of the Neumann coefficient
  const int *rowptr = nullptr, *col = nullptr, *etr = nullptr;
  float *F = nullptr, *Ef = nullptr;
  z2g *ratio = nullptr, *dinv = nullptr;
  float *Z0 = nullptr, *H[GL + 1] = {}, *P = nullptr, *Q = nullptr, *agg[GL] = {}, *U[GL] = {};
  float *Zm[GL] = {}, *Zr = nullptr, *Oe = nullptr;
  // backward
  float *dH = nullptr, *dU = nullptr, *dagg = nullptr, *dZ = nullptr, *dP = nullptr, *dQ = nullptr, *dO = nullptr;
  float *part = nullptr;   // partial sums of the weight gradients
  bool pooled = false;     // stream-ordered allocations (a training step's buffers)
  std::vector<void *> owned;
};

static void bufs_free(GnnBufs &B) {
  for (void *p : B.owned) {
    if (B.pooled) cudaFreeAsync(p, stream());
    else cudaFree(p);
  }
  B = GnnBufs();
}

template <typename T>
static int balloc(GnnBufs &B, T **p, size_t count) {
  void *q = nullptr;
  const size_t bytes = sizeof(T) * std::max<size_t>(count, 1);
  cudaError_t e = B.pooled ? cudaMallocAsync(&q, bytes, stream()) : cudaMalloc(&q, bytes);
  if (e != cudaSuccess) {
    set_error("graph network buffers (%zu bytes): %s", sizeof(T) * count, cudaGetErrorString(e));
    return BG_ERR_NOMEM;
  }
  B.owned.push_back(q);
  *p = (T *)q;
  return BG_OK;
}

// Near-field graph from the geometry's near pairs (same object, >= 1 common
// vertex, a <= b): both directions plus self pairs, sorted columns, reverse map.
static int ensure_graph(bg_geometry *g) {
  if (g->graph.rowptr) return BG_OK;
  int st = bg_geometry_precompute(g);
  if (st) return st;
  int N = g->N, np = g->near.npairs;
  std::vector<int2> pairs(np);
  if (np) BG_CUDA_TRY(cudaMemcpy(pairs.data(), g->near.pairs, sizeof(int2) * np, cudaMemcpyDeviceToHost));
  std::vector<int> deg(N, 1);   // self pair
  for (auto &p : pairs)
    if (p.x != p.y) { deg[p.x]++; deg[p.y]++; }
  std::vector<int> rowptr(N + 1, 0);
  for (int i = 0; i < N; i++) rowptr[i + 1] = rowptr[i] + deg[i];
  int E = rowptr[N];
  std::vector<int> col(E), fill(rowptr.begin(), rowptr.end() - 1);
  for (int i = 0; i < N; i++) col[fill[i]++] = i;
  for (auto &p : pairs)
    if (p.x != p.y) { col[fill[p.x]++] = p.y; col[fill[p.y]++] = p.x; }
  for (int i = 0; i < N; i++) {
    std::sort(col.begin() + rowptr[i], col.begin() + rowptr[i + 1]);
    if (std::adjacent_find(col.begin() + rowptr[i], col.begin() + rowptr[i + 1]) != col.begin() + rowptr[i + 1]) {
      set_error("near graph: duplicate basis-function pair");
      return BG_ERR_STATE;
    }
  }
  std::vector<int> etr(E);
  for (int i = 0; i < N; i++)
    for (int e = rowptr[i]; e < rowptr[i + 1]; e++) {
      int j = col[e];
      auto it = std::lower_bound(col.begin() + rowptr[j], col.begin() + rowptr[j + 1], i);
      if (it == col.begin() + rowptr[j + 1] || *it != i) { set_error("near graph: pattern not symmetric"); return BG_ERR_STATE; }
      etr[e] = (int)(it - col.begin());
    }
  double hsum = 0;
  for (auto &o : g->objs)
    for (int a = 0; a < o.nif; a++) hsum += o.F[a].radius;
  NearGraph G;
  G.E = E;
  G.h = hsum / std::max(1, N);
  BG_CUDA_TRY(cudaMalloc(&G.rowptr, sizeof(int) * (N + 1)));
  BG_CUDA_TRY(cudaMalloc(&G.col, sizeof(int) * E));
  BG_CUDA_TRY(cudaMalloc(&G.etr, sizeof(int) * E));
  BG_CUDA_TRY(cudaMemcpy(G.rowptr, rowptr.data(), sizeof(int) * (N + 1), cudaMemcpyHostToDevice));
  BG_CUDA_TRY(cudaMemcpy(G.col, col.data(), sizeof(int) * E, cudaMemcpyHostToDevice));
  BG_CUDA_TRY(cudaMemcpy(G.etr, etr.data(), sizeof(int) * E, cudaMemcpyHostToDevice));
  BG_CUDA_TRY(uploads_done());
  g->graph = G;
  return BG_OK;
}

static int bound_coefficient(GnnBufs &B);

static int bufs_alloc(bg_geometry *g, bool train, GnnBufs &B) {
  int st = ensure_graph(g);
  if (st) return st;
  int N = g->N, E = g->graph.E;
  B.N = N;
  B.E = E;
  B.rowptr = g->graph.rowptr;
  B.col = g->graph.col;
  B.etr = g->graph.etr;
  size_t n64 = (size_t)N * GW, e64 = (size_t)E * GW;
  // a training step allocates and frees about 25 buffers, some of 64 floats per
  // edge: from the stream-ordered pool (with cudaMalloc and cudaFree the step took
  // 34 ms at N = 3,822, its kernels 20)
  B.pooled = train;
  if ((st = balloc(B, &B.F, (size_t)N * GF)) || (st = balloc(B, &B.Ef, (size_t)E * GE)) ||
      (st = balloc(B, &B.ratio, (size_t)E)) || (st = balloc(B, &B.dinv, (size_t)N)) ||
      (st = balloc(B, &B.Z0, n64)) || (st = balloc(B, &B.P, n64)) || (st = balloc(B, &B.Q, n64)))
    return st;
  for (int l = 0; l <= GL; l++)
    if ((st = balloc(B, &B.H[l], n64))) return st;
  for (int l = 0; l < GL; l++)
    if ((st = balloc(B, &B.agg[l], n64)) || (st = balloc(B, &B.U[l], n64))) return st;
  if (train) {
    for (int l = 0; l < GL; l++)
      if ((st = balloc(B, &B.Zm[l], e64))) return st;
    if ((st = balloc(B, &B.Zr, e64)) || (st = balloc(B, &B.dZ, e64)) || (st = balloc(B, &B.dO, (size_t)E * GO)) ||
        (st = balloc(B, &B.Oe, (size_t)E * GO)) ||
        (st = balloc(B, &B.dH, n64)) || (st = balloc(B, &B.dU, n64)) || (st = balloc(B, &B.dagg, n64)) ||
        (st = balloc(B, &B.dP, n64)) || (st = balloc(B, &B.dQ, n64)) ||
        (st = balloc(B, &B.part, std::max((size_t)GPB * GRP, (size_t)GWB * (GW * GW + GW)))))
      return st;
  }
  return BG_OK;
}

static int bound_coefficient(GnnBufs &B);

// per-call part: features of (A, omega) and the coefficient bound
static int bufs_compute(bg_geometry *g, bg_matrix *A, double omega, GnnBufs &B) {
  int N = B.N;
  k_gnn_features<<<(N + 7) / 8, 256, 0, stream()>>>(N, B.rowptr, B.col, (const z2g *)A->d, A->ld, g->dev, omega,
                                                        g->graph.h, B.F, B.Ef, B.ratio, B.dinv);
  BG_LAUNCHED();
  return bound_coefficient(B);
}

static int bufs_init(bg_geometry *g, bg_matrix *A, double omega, bool train, GnnBufs &B) {
  int st = bufs_alloc(g, train, B);
  return st ? st : bufs_compute(g, A, omega, B);
}

// The inference buffers (about 15 node-sized and 2 edge-sized arrays) are kept
// with the geometry and reused by every learned preconditioner built for it,
// so a frequency step allocates no graph-network memory.
static int inference_bufs(bg_geometry *g, GnnBufs *&B) {
  int st = ensure_graph(g);
  if (st) return st;
  GnnBufs *c = static_cast<GnnBufs *>(g->gnn_cache);
  if (c && (c->N != g->N || c->E != g->graph.E)) {
    bufs_free(*c);
    delete c;
    c = nullptr;
    g->gnn_cache = nullptr;
  }
  if (!c) {
    c = new GnnBufs();
    if ((st = bufs_alloc(g, false, *c))) {
      bufs_free(*c);
      delete c;
      return st;
    }
    g->gnn_cache = c;
  }
  B = c;
  return BG_OK;
}

void gnn_cache_free(bg_geometry *g) {
  GnnBufs *c = static_cast<GnnBufs *>(g->gnn_cache);
  if (c) {
    bufs_free(*c);
    delete c;
  }
  g->gnn_cache = nullptr;
}

// Power iteration (four seeded vectors in lockstep, GNN_POWER_ITERS steps)
// for the spectral radius of K1; sets the coefficient bound smax.
static int bound_coefficient(GnnBufs &B) {
  const int nv = 4;
  int N = B.N;
  size_t nn = (size_t)N * nv;
  char *w = nullptr;
  const int nblk = (int)(((size_t)N * 32 + 255) / 256);
  BG_CUDA_TRY(cudaMallocAsync((void **)&w, sizeof(z2g) * 2 * nn + sizeof(double) * (nv + 4 * (size_t)nblk), stream()));
  z2g *V = (z2g *)w, *W = V + nn;
  double *nrm = (double *)(W + nn), *part = nrm + nv;
  std::vector<z2g> h(nn);
  uint64_t s = 0x9e3779b97f4a7c15ull;
  for (auto &v : h) {
    s = s * 6364136223846793005ull + 1442695040888963407ull;
    double a = (double)(s >> 11) / 9007199254740992.0 - 0.5;
    s = s * 6364136223846793005ull + 1442695040888963407ull;
    double b = (double)(s >> 11) / 9007199254740992.0 - 0.5;
    v = z2g{a, b};
  }
  double hn[nv];
  for (int q = 0; q < nv; q++) {
    double t = 0;
    for (int i = 0; i < N; i++) {
      const z2g v = h[(size_t)q * N + i];
      t += v.r * v.r + v.i * v.i;
    }
    hn[q] = t;
  }
  int st = BG_OK;
  cudaError_t e = cudaMemcpyAsync(V, h.data(), sizeof(z2g) * nn, cudaMemcpyHostToDevice, stream());
  if (e == cudaSuccess) e = cudaMemcpyAsync(nrm, hn, sizeof(double) * nv, cudaMemcpyHostToDevice, stream());
  // W = K1 V / |V|: the norm of the last one is the estimate
  for (int it = 0; e == cudaSuccess && it < GNN_POWER_ITERS; it++) {
    k_gnn_k1mv<<<nblk, 256, 0, stream()>>>(N, B.rowptr, B.col, B.ratio, B.dinv, V, nrm, nv, W, part);
    k_gnn_norm4<<<1, 256, 0, stream()>>>(nblk, part, nrm);
    g_launches += 2;
    std::swap(V, W);
    e = cudaGetLastError();
  }
  double rho = 0;
  if (e == cudaSuccess) e = cudaMemcpyAsync(hn, nrm, sizeof(double) * nv, cudaMemcpyDeviceToHost, stream());
  if (e == cudaSuccess) e = cudaStreamSynchronize(stream());
  if (e == cudaSuccess)
    for (int q = 0; q < nv; q++) rho = std::max(rho, std::sqrt(hn[q]));
  if (e != cudaSuccess) { set_error("near-field spectral estimate: %s", cudaGetErrorString(e)); st = BG_ERR_CUDA; }
  if (!st && !std::isfinite(rho)) { set_error("near-field spectral estimate: non-finite"); st = BG_ERR_NUMERIC; }
  cudaFreeAsync(w, stream());
  B.rho_ref = rho;
  B.smax = (float)(GNN_SREL / std::max(rho, GNN_SREL));
  return st;
}

static int forward(const bg_gnn *net, GnnBufs &B, z2g *Mval) {
  const float *W = net->params;
  int N = B.N, n64 = N * GW, nb = (n64 + 255) / 256;
  k_gnn_linear<false><<<(N + GLN - 1) / GLN, 256, 0, stream()>>>(N, GF, GW, B.F, GF, W + LAY.W0, W + LAY.b0, B.Z0, GW, 0);
  BG_LAUNCHED();
  k_gnn_relu<<<nb, 256, 0, stream()>>>(n64, B.Z0, B.H[0]);
  BG_LAUNCHED();
  for (int l = 0; l < GL; l++) {
    k_gnn_linear<false><<<(N + GLN - 1) / GLN, 256, 0, stream()>>>(N, GW, GW, B.H[l], GW, W + LAY.Wmh[l], nullptr, B.P, GW, 0);
    BG_LAUNCHED();
    k_gnn_msg<<<N, GW, 0, stream()>>>(N, B.rowptr, B.col, B.P, B.Ef, W + LAY.Wme[l], W + LAY.bm[l], B.Zm[l],
                                      B.agg[l]);
    BG_LAUNCHED();
    k_gnn_linear<false><<<(N + GLN - 1) / GLN, 256, 0, stream()>>>(N, GW, GW, B.H[l], GW, W + LAY.Wuh[l], W + LAY.bu[l], B.U[l], GW, 0);
    BG_LAUNCHED();
    k_gnn_linear<false><<<(N + GLN - 1) / GLN, 256, 0, stream()>>>(N, GW, GW, B.agg[l], GW, W + LAY.Wua[l], nullptr, B.U[l], GW, 1);
    BG_LAUNCHED();
    k_gnn_residual<<<nb, 256, 0, stream()>>>(n64, B.H[l], B.U[l], B.H[l + 1]);
    BG_LAUNCHED();
  }
  k_gnn_linear<false><<<(N + GLN - 1) / GLN, 256, 0, stream()>>>(N, GW, GW, B.H[GL], GW, W + LAY.Wri, nullptr, B.P, GW, 0);
  BG_LAUNCHED();
  k_gnn_linear<false><<<(N + GLN - 1) / GLN, 256, 0, stream()>>>(N, GW, GW, B.H[GL], GW, W + LAY.Wrj, nullptr, B.Q, GW, 0);
  BG_LAUNCHED();
  k_gnn_readout<<<(N + 3) / 4, 128, 0, stream()>>>(N, B.rowptr, B.col, B.P, B.Q, B.Ef, W + LAY.Wrg, W + LAY.br,
                                                   W + LAY.Wo, W + LAY.bo, B.ratio, B.dinv, B.smax, B.Zr, B.Oe,
                                                   Mval);
  BG_LAUNCHED();
  return BG_OK;
}

// backward from gscale * G, G = 2 dL/dconj(m); accumulates into net->grads (zeroed by the caller)
static int backward(bg_gnn *net, GnnBufs &B, const z2g *G, double gscale) {
  const float *W = net->params;
  float *dW = net->grads;
  int N = B.N, n64 = N * GW, nb = (n64 + 255) / 256, st;
  const int eb = std::min(GPB, (N + 3) / 4);
  auto reduce = [&](int nblk, int stride, int off, int n, float *out) {
    k_gnn_reduce<<<(n + 15) / 16, 256, 0, stream()>>>(nblk, stride, B.part, off, n, out);
    BG_LAUNCHED();
    return BG_OK;
  };
  // dW += dY^T X, db += column sums of dY
  auto wgrad = [&](int in, const float *dY, const float *X, float *dWp, float *dbp) {
    const int blk = std::min(GWB, (N + 31) / 32), stride = GW * in + GW;
    k_gnn_wgrad<<<blk, 256, 0, stream()>>>(N, in, dY, GW, X, in, B.part);
    BG_LAUNCHED();
    int r = reduce(blk, stride, 0, GW * in, dWp);
    if (!r && dbp) r = reduce(blk, stride, GW * in, GW, dbp);
    return r;
  };
  auto dx = [&](const float *dY, const float *Wp, float *dX, int accumulate) {
    k_gnn_linear<true><<<(N + GLN - 1) / GLN, 256, 0, stream()>>>(N, GW, GW, dY, GW, Wp, nullptr, dX, GW, accumulate);
    BG_LAUNCHED();
    return BG_OK;
  };
  k_gnn_dout<<<(N + 7) / 8, 256, 0, stream()>>>(N, B.rowptr, B.col, G, gscale, B.ratio, B.dinv, B.smax, B.Oe, B.dO);
  BG_LAUNCHED();
  k_gnn_readout_back<<<eb, 256, 0, stream()>>>(N, B.rowptr, B.Zr, B.dO, W + LAY.Wo, B.Ef, B.dZ, B.dP, B.part);
  BG_LAUNCHED();
  if ((st = reduce(eb, GRP, 0, GW * GE, dW + LAY.Wrg)) || (st = reduce(eb, GRP, GW * GE, GW, dW + LAY.br)) ||
      (st = reduce(eb, GRP, GEP, GO * GW, dW + LAY.Wo)) || (st = reduce(eb, GRP, GEP + GO * GW, GO, dW + LAY.bo)))
    return st;
  k_gnn_col_gather<<<N, GW, 0, stream()>>>(N, B.rowptr, B.etr, B.dZ, B.dQ);
  BG_LAUNCHED();
  if ((st = wgrad(GW, B.dP, B.H[GL], dW + LAY.Wri, nullptr)) || (st = wgrad(GW, B.dQ, B.H[GL], dW + LAY.Wrj, nullptr)) ||
      (st = dx(B.dP, W + LAY.Wri, B.dH, 0)) || (st = dx(B.dQ, W + LAY.Wrj, B.dH, 1)))
    return st;
  for (int l = GL - 1; l >= 0; l--) {
    // H_{l+1} = H_l + relu(U_l): dU = dH [U > 0]; dH_l = dH + Wuh^T dU + Wmh^T dP; dagg = Wua^T dU
    k_gnn_relu_back<<<nb, 256, 0, stream()>>>(n64, B.U[l], B.dH, B.dU);
    BG_LAUNCHED();
    if ((st = wgrad(GW, B.dU, B.H[l], dW + LAY.Wuh[l], dW + LAY.bu[l])) ||
        (st = wgrad(GW, B.dU, B.agg[l], dW + LAY.Wua[l], nullptr)) || (st = dx(B.dU, W + LAY.Wuh[l], B.dH, 1)) ||
        (st = dx(B.dU, W + LAY.Wua[l], B.dagg, 0)))
      return st;
    k_gnn_msg_back<<<eb, 256, 0, stream()>>>(N, B.rowptr, B.Zm[l], B.dagg, B.Ef, B.dZ, B.part);
    BG_LAUNCHED();
    if ((st = reduce(eb, GEP, 0, GW * GE, dW + LAY.Wme[l])) || (st = reduce(eb, GEP, GW * GE, GW, dW + LAY.bm[l])))
      return st;
    k_gnn_col_gather<<<N, GW, 0, stream()>>>(N, B.rowptr, B.etr, B.dZ, B.dP);
    BG_LAUNCHED();
    if ((st = wgrad(GW, B.dP, B.H[l], dW + LAY.Wmh[l], nullptr)) || (st = dx(B.dP, W + LAY.Wmh[l], B.dH, 1))) return st;
  }
  k_gnn_relu_back<<<nb, 256, 0, stream()>>>(n64, B.Z0, B.dH, B.dU);
  BG_LAUNCHED();
  return wgrad(GF, B.dU, B.F, dW + LAY.W0, dW + LAY.b0);
}

// Y = sign A X for p columns
static int gnn_mul(bg_matrix *A, const z2g *X, int p, double sign, z2g *Y) {
  const int N = A->N, rb = (N + 255) / 256;
  // about eight blocks per SM, at least 32 columns each
  const int want = std::max(1, 8 * 148 / (rb * ((p + GQ - 1) / GQ)));
  const int chunk = std::max(32, (N + want - 1) / want), nchunk = (N + chunk - 1) / chunk;
  const size_t np = (size_t)N * p;
  z2g *part = nullptr;
  BG_CUDA_TRY(cudaMallocAsync((void **)&part, sizeof(z2g) * np * nchunk, stream()));
  k_gnn_mul<<<dim3(rb, nchunk, (p + GQ - 1) / GQ), 128, 0, stream()>>>(N, (const z2g *)A->d, A->ld, X, p, chunk, part);
  BG_LAUNCHED();
  k_gnn_mul_sum<<<(unsigned)((np + 255) / 256), 256, 0, stream()>>>(np, nchunk, part, sign, Y);
  BG_LAUNCHED();
  BG_CUDA_TRY(cudaFreeAsync(part, stream()));
  return BG_OK;
}

// objective and G = 2 dL/dconj(M) on the pattern
static int loss_grad(bg_matrix *A, GnnBufs &B, const z2g *Mval, const z2g *Z, int p, const z2g *b, const z2g *x,
                     double lambda, z2g *G, double *loss_out) {
  int N = B.N;
  size_t np = (size_t)N * p;
  z2g *buf = nullptr;
  // R, the residual Mb - x and x lie one after another: their column norms in one launch
  BG_CUDA_TRY(cudaMallocAsync((void **)&buf, sizeof(z2g) * (4 * np + 3 * (size_t)N) + sizeof(double) * (p + 2), stream()));
  z2g *Y = buf, *S = Y + np, *W = S + np, *R = W + np, *rb = R + np, *xc = rb + N, *Mb = xc + N;
  double *nrm = (double *)(Mb + N), hn[GNN_MAXP + 2];
  int st = BG_OK;
  k_gnn_spmm<<<dim3((8 * N + 255) / 256, (p + 3) / 4), 256, 0, stream()>>>(N, B.rowptr, B.col, Mval, Z, p, Y);
  BG_LAUNCHED();
  // R = A Y - Z; S = A^H R
  if ((st = gnn_mul(A, Y, p, 1.0, W))) { cudaFreeAsync(buf, stream()); return st; }
  k_gnn_sub<<<(np + 255) / 256, 256, 0, stream()>>>(np, W, Z, R);
  BG_LAUNCHED();
  k_gnn_ahr<<<dim3((N + GAC - 1) / GAC, (p + GQ - 1) / GQ), 128, 0, stream()>>>(N, (const z2g *)A->d, A->ld, R, p, S);
  BG_LAUNCHED();
  const bool rhs = b && x && lambda > 0;
  if (rhs) {
    k_gnn_spmm<<<dim3((8 * N + 255) / 256, 1), 256, 0, stream()>>>(N, B.rowptr, B.col, Mval, b, 1, Mb);
    BG_LAUNCHED();
    k_gnn_sub<<<(N + 255) / 256, 256, 0, stream()>>>(N, Mb, x, rb);
    BG_LAUNCHED();
    BG_CUDA_TRY(cudaMemcpyAsync(xc, x, sizeof(z2g) * N, cudaMemcpyDeviceToDevice, stream()));
  }
  k_gnn_colnorm2<<<p + (rhs ? 2 : 0), 512, 0, stream()>>>(N, R, nrm);
  BG_LAUNCHED();
  BG_CUDA_TRY(cudaMemcpyAsync(hn, nrm, sizeof(double) * (p + (rhs ? 2 : 0)), cudaMemcpyDeviceToHost, stream()));
  BG_CUDA_TRY(cudaStreamSynchronize(stream()));
  double scale = 2.0 / ((double)N * p), scale2 = 0.0, l1 = 0.0, l2 = 0.0;
  for (int q = 0; q < p; q++) l1 += hn[q];
  if (rhs) {
    scale2 = 2.0 * lambda / std::max(hn[p + 1], 1e-300);
    l2 = lambda * hn[p] / std::max(hn[p + 1], 1e-300);
  }
  k_gnn_sddmm<<<(N + 7) / 8, 256, 0, stream()>>>(N, B.rowptr, B.col, S, Z, p, scale, scale2 > 0 ? rb : nullptr,
                                                     b, scale2, G);
  BG_LAUNCHED();
  *loss_out = l1 / ((double)N * p) + l2;
  cudaFreeAsync(buf, stream());
  return BG_OK;
}

}  // namespace bg

using namespace bg;

extern "C" {

int bg_gnn_create(unsigned long long seed, bg_gnn **out) {
  if (!out) { set_error("bg_gnn_create: null output"); return BG_ERR_ARG; }
  *out = nullptr;
  int st = ensure_device();
  if (st) return st;
  int n = LAY.total;
  std::vector<float> p(n, 0.f);
  // Glorot-uniform weights from a 64-bit LCG; biases and the output map start at zero
  uint64_t s = seed * 6364136223846793005ull + 1442695040888963407ull;
  auto uni = [&]() {
    s = s * 6364136223846793005ull + 1442695040888963407ull;
    return ((s >> 11) * (1.0 / 9007199254740992.0)) * 2 - 1;
  };
  auto fill = [&](int off, int out_, int in_, double gain) {
    double a = gain * std::sqrt(6.0 / (in_ + out_));
    for (int i = 0; i < out_ * in_; i++) p[off + i] = (float)(a * uni());
  };
  fill(LAY.W0, GW, GF, 1.0);
  for (int l = 0; l < GL; l++) {
    fill(LAY.Wmh[l], GW, GW, 1.0);
    fill(LAY.Wme[l], GW, GE, 1.0);
    fill(LAY.Wuh[l], GW, GW, 0.3);
    fill(LAY.Wua[l], GW, GW, 0.3);
  }
  fill(LAY.Wri, GW, GW, 1.0);
  fill(LAY.Wrj, GW, GW, 1.0);
  fill(LAY.Wrg, GW, GE, 1.0);
  size_t nalloc = 4 * (size_t)n + 2;   // params, grads, Adam moments; then one double (8-byte aligned)
  bg_gnn *net = new bg_gnn();
  cudaError_t e = cudaMalloc(&net->params, sizeof(float) * (nalloc + 2));
  if (e != cudaSuccess) { delete net; set_error("bg_gnn_create: %s", cudaGetErrorString(e)); return BG_ERR_NOMEM; }
  net->grads = net->params + n;
  net->m = net->grads + n;
  net->v = net->m + n;
  net->sumsq = (double *)(net->params + ((4 * (size_t)n + 1) & ~(size_t)1));
  e = cudaMemset(net->params, 0, sizeof(float) * (nalloc + 2));
  if (e == cudaSuccess) e = cudaMemcpy(net->params, p.data(), sizeof(float) * n, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = uploads_done();
  if (e != cudaSuccess) {
    cudaFree(net->params);
    delete net;
    set_error("bg_gnn_create: %s", cudaGetErrorString(e));
    return BG_ERR_CUDA;
  }
  *out = net;
  return BG_OK;
}

void bg_gnn_destroy(bg_gnn *net) {
  if (!net) return;
  if (net->params) cudaFree(net->params);
  delete net;
}

int bg_gnn_num_params(void) { return LAY.total; }

int bg_gnn_get_params(const bg_gnn *net, float *host) {
  if (!net || !host) { set_error("bg_gnn_get_params: bad arguments"); return BG_ERR_ARG; }
  BG_CUDA_TRY(cudaStreamSynchronize(stream()));
  BG_CUDA_TRY(cudaMemcpy(host, net->params, sizeof(float) * LAY.total, cudaMemcpyDeviceToHost));
  return BG_OK;
}

int bg_gnn_set_params(bg_gnn *net, const float *host) {
  if (!net || !host) { set_error("bg_gnn_set_params: bad arguments"); return BG_ERR_ARG; }
  BG_CUDA_TRY(cudaStreamSynchronize(stream()));
  BG_CUDA_TRY(cudaMemcpy(net->params, host, sizeof(float) * LAY.total, cudaMemcpyHostToDevice));
  net->step = 0;
  BG_CUDA_TRY(cudaMemset(net->m, 0, sizeof(float) * 2 * LAY.total));
  BG_CUDA_TRY(uploads_done());
  return BG_OK;
}

int bg_gnn_get_grads(const bg_gnn *net, float *host) {
  if (!net || !host) { set_error("bg_gnn_get_grads: bad arguments"); return BG_ERR_ARG; }
  BG_CUDA_TRY(cudaStreamSynchronize(stream()));
  BG_CUDA_TRY(cudaMemcpy(host, net->grads, sizeof(float) * LAY.total, cudaMemcpyDeviceToHost));
  return BG_OK;
}

int bg_precond_create_learned(bg_geometry *g, bg_matrix *A, double omega, const bg_gnn *net, bg_precond **out) {
  if (!g || !A || !net || !out || A->precision != BG_C128 || A->N != g->N) {
    set_error("bg_precond_create_learned: bad arguments");
    return BG_ERR_ARG;
  }
  *out = nullptr;
  if (A->factored) { set_error("bg_precond_create_learned: matrix holds LU factors"); return BG_ERR_STATE; }
  GnnBufs *Bp = nullptr;
  prof_start(PROF_GNN);
  int st = inference_bufs(g, Bp);
  if (st) {
    prof_stop(PROF_GNN, 0.0);
    return st;
  }
  GnnBufs &B = *Bp;
  st = bufs_compute(g, A, omega, B);
  bg_precond *P = nullptr;
  if (!st) {
    P = new bg_precond();
    P->N = B.N;
    P->nnz = B.E;

    cudaError_t e = cudaMallocAsync((void **)&P->rowptr, sizeof(int) * (B.N + 1), stream());
    if (e == cudaSuccess) e = cudaMallocAsync((void **)&P->col, sizeof(int) * B.E, stream());
    if (e == cudaSuccess) e = cudaMallocAsync((void **)&P->val, sizeof(z2g) * B.E, stream());
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(P->rowptr, B.rowptr, sizeof(int) * (B.N + 1), cudaMemcpyDeviceToDevice, stream());
    if (e == cudaSuccess) e = cudaMemcpyAsync(P->col, B.col, sizeof(int) * B.E, cudaMemcpyDeviceToDevice, stream());
    if (e != cudaSuccess) { set_error("learned preconditioner: %s", cudaGetErrorString(e)); st = BG_ERR_NOMEM; }
  }
  if (!st) st = forward(net, B, (z2g *)P->val);
  if (!st) {
    P->rho = B.rho_ref;
    P->theta = B.smax;
  }
  prof_stop(PROF_GNN, 0.0);
  if (st) {
    bg_precond_destroy(P);
    return st;
  }
  *out = P;
  return BG_OK;
}

// One training step on one matrix: forward, objective, backward of log L, Adam (lr > 0).
int bg_gnn_train_step(bg_gnn *net, bg_geometry *g, bg_matrix *A, double omega, const double *Z_host, int p,
                      int probe_power, const double *b_host, const double *x_host, double lambda, double lr,
                      double *loss_out) {
  if (!net || !g || !A || !Z_host || p <= 0 || p > GNN_MAXP || A->precision != BG_C128 || A->N != g->N || lr < 0 ||
      probe_power < 0 || probe_power > 64) {
    set_error("bg_gnn_train_step: bad arguments (at most %d probes)", GNN_MAXP);
    return BG_ERR_ARG;
  }
  if (A->factored) { set_error("bg_gnn_train_step: matrix holds LU factors"); return BG_ERR_STATE; }
  GnnBufs B;
  int st = bufs_init(g, A, omega, true, B);
  int N = g->N;
  z2g *dbuf = nullptr;
  if (!st) {
    size_t bytes = sizeof(z2g) * (3 * (size_t)N * p + 2 * (size_t)N + 2 * (size_t)B.E);
    cudaError_t e = cudaMallocAsync((void **)&dbuf, bytes, stream());
    if (e != cudaSuccess) { set_error("train step: %s", cudaGetErrorString(e)); st = BG_ERR_NOMEM; }
  }
  bool rhs = b_host && x_host && lambda > 0;
  z2g *Z = dbuf, *b = Z + (size_t)N * p, *x = b + N, *Mval = x + N, *Gg = Mval + B.E, *Y = Gg + B.E,
      *W = Y + (size_t)N * p;
  if (!st) {
    cudaError_t e = cudaMemcpyAsync(Z, Z_host, sizeof(z2g) * (size_t)N * p, cudaMemcpyHostToDevice, stream());
    if (e == cudaSuccess && rhs) e = cudaMemcpyAsync(b, b_host, sizeof(z2g) * N, cudaMemcpyHostToDevice, stream());
    if (e == cudaSuccess && rhs) e = cudaMemcpyAsync(x, x_host, sizeof(z2g) * N, cudaMemcpyHostToDevice, stream());
    if (e != cudaSuccess) { set_error("train step: %s", cudaGetErrorString(e)); st = BG_ERR_CUDA; }
  }
  // probes through the Jacobi error map: Z <- Z - A D^{-1} Z, rescaled
  for (int k = 0; !st && k < probe_power; k++) {
    size_t np = (size_t)N * p;
    k_gnn_rowscale<<<(np + 255) / 256, 256, 0, stream()>>>(N, p, B.dinv, Z, Y);
    g_launches++;
    if ((st = gnn_mul(A, Y, p, -1.0, W))) break;   // W = -A D^{-1} Z
    k_gnn_probe_update<<<p, 512, 0, stream()>>>(N, W, Z);
    g_launches++;
  }
  if (!st) st = forward(net, B, Mval);
  double loss = 0;
  if (!st) st = loss_grad(A, B, Mval, Z, p, rhs ? b : nullptr, rhs ? x : nullptr, lambda, Gg, &loss);
  if (!st) {
    cudaError_t e = cudaMemsetAsync(net->grads, 0, sizeof(float) * LAY.total, stream());
    if (e != cudaSuccess) { set_error("train step: %s", cudaGetErrorString(e)); st = BG_ERR_CUDA; }
  }
  if (!st && !(loss > 0 && std::isfinite(loss))) { set_error("train step: objective %g", loss); st = BG_ERR_NUMERIC; }
  if (!st) st = backward(net, B, Gg, 1.0 / loss);
  if (!st && lr > 0) {
    net->step++;
    const float b1 = 0.9f, b2 = 0.999f;
    float c1 = 1.f - std::pow(b1, (float)net->step), c2 = 1.f - std::pow(b2, (float)net->step);
    cudaError_t e = cudaMemsetAsync(net->sumsq, 0, sizeof(double), stream());
    if (e != cudaSuccess) { set_error("train step: %s", cudaGetErrorString(e)); st = BG_ERR_CUDA; }
    if (!st) {
      k_gnn_sumsq<<<64, 256, 0, stream()>>>(LAY.total, net->grads, net->sumsq);
      g_launches++;
      k_gnn_adam<<<(LAY.total + 255) / 256, 256, 0, stream()>>>(LAY.total, net->params, net->grads, net->m, net->v,
                                                                net->sumsq, (float)lr, b1, b2, c1, c2, 1e-8f, 1.0f);
      g_launches++;
    }
  }
  if (dbuf) cudaFreeAsync(dbuf, stream());
  cudaError_t e2 = cudaStreamSynchronize(stream());
  if (!st && e2 != cudaSuccess) { set_error("train step: %s", cudaGetErrorString(e2)); st = BG_ERR_CUDA; }
  bufs_free(B);
  if (loss_out) *loss_out = loss;
  return st;
}

int bg_precond_bound(const bg_precond *P, double *rho, double *smax) {
  if (!P) { set_error("bg_precond_bound: null"); return BG_ERR_ARG; }
  if (rho) *rho = P->rho;
  if (smax) *smax = P->theta;
  return BG_OK;
}

int bg_precond_download(const bg_precond *P, int *rowptr, int *col, double *val) {
  if (!P) { set_error("bg_precond_download: null"); return BG_ERR_ARG; }
  BG_CUDA_TRY(cudaStreamSynchronize(stream()));
  if (rowptr) BG_CUDA_TRY(cudaMemcpy(rowptr, P->rowptr, sizeof(int) * (P->N + 1), cudaMemcpyDeviceToHost));
  if (col) BG_CUDA_TRY(cudaMemcpy(col, P->col, sizeof(int) * P->nnz, cudaMemcpyDeviceToHost));
  if (val) BG_CUDA_TRY(cudaMemcpy(val, P->val, sizeof(z2g) * P->nnz, cudaMemcpyDeviceToHost));
  return BG_OK;
}

}  // extern "C"
