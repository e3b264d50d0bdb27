// EMT pair sums through tetrahedra (included by kernels.cu).
//
// The EMT power, force and torque are sums over basis-function pairs a <= b of
// Z0 JJ(a, b) times ten integrals of the pair (scat_q / scat_terms).  A pair's
// integrand is bilinear in the two basis functions, and at most four of them
// live on one tetrahedron, so for one quadrature rule the sum over pairs
// collapses to a sum over tetrahedron pairs of the tetrahedra's total
// currents: 1/16 of the kernel values of the pair-by-pair sum.
//
// Within one object every pair quantity is symmetric in (a, b), so with t4 the
// terms by the 4-point rule and t those by the rule the pair asks for
// (4 points far, 16 near, EMTPFT.cc:305-313)
//   sum_{a<=b} t = 1/2 sum_{all a,b} t4  +  sum_{near a<=b} (t - t4)
//                  + 1/2 sum_a t4(a, a),
// where the first sum runs over unordered tetrahedron pairs (k_emt_far,
// k_emt_far_dr), the second over the near tetrahedron pairs (k_emt_near) and
// the third over basis functions (k_emt_self).  Pairs of different objects are
// all far and are summed once, the lower object first.  Valid when no basis
// function reaches the rule switch |omega| R > 5; the general kernels
// (k_pft_far, k_pft_near) serve the other frequencies.
//
// Im(phi) = sin(kr)/(4 pi r) and Im(psi) = (kr cos kr - sin kr)/(4 pi r^3) are
// entire in r^2: up to |k| r = 4 they are Taylor polynomials in r^2 (no square
// root and no sincos; the first omitted terms stay below 2e-17 of the value at
// r = 0).  Below |k| r = 2e-2 both are cut after two terms, as in the
// reference (EMTPFT.cc:236-243).
#pragma once

// Taylor coefficients in r^2, the powers of k^2 folded in: phi = k/(4 pi) *
// sum c[n] r^(2n), psi = k^3/(4 pi) * sum d[n] r^(2n)
#define EMT_MAXT 16
struct EmtKernel {
  double c[EMT_MAXT], d[EMT_MAXT];
  double tiny2;          // (2e-2 / k)^2
  double k, k2;
};

// per quadrature point: x, y, z (relative to the object's origin), Re rho,
// Im rho, Re/Im of the three current components, pad.  rho carries 1/k.
#define EMT_PT 12
struct EmtBlockMap {     // blocks of one object pair: i chunks x j tiles
  int nmap, ic;          // object pairs; points i per block
  int first[10];         // first block
  int oa[10], ob[10];
  int i0[10], i1[10], j0[10], j1[10], nj[10];
};

template <int NT>
__device__ __forceinline__ void emt_phipsi(const EmtKernel &K, double r2, double &phi, double &psi) {
  if (NT > 0) {
    double p = K.c[NT > 0 ? NT - 1 : 0], q = K.d[NT > 0 ? NT - 1 : 0];
#pragma unroll
    for (int n = NT - 2; n >= 0; n--) {
      p = fma(p, r2, K.c[n]);
      q = fma(q, r2, K.d[n]);
    }
    const bool tiny = r2 < K.tiny2;
    phi = tiny ? fma(r2, K.c[1], 1.0) : p;
    psi = tiny ? fma(r2, K.d[1], K.d[0]) : q;
  } else {
    const double r = sqrt(r2), kr = K.k * r;
    if (fabs(kr) < 2.0e-2) {
      phi = fma(r2, K.c[1], 1.0);
      psi = fma(r2, K.d[1], K.d[0]);
    } else {
      double s, c;
      sincos(kr, &s, &c);
      phi = s / kr;
      psi = (kr * c - s) / (kr * kr * kr);
    }
  }
}

// currents of the tetrahedra at the points of the 4-point rule, the weights
// 6 V / 24 folded in (the volumes cancel against the basis functions' 1/3V)
__global__ void k_emt_points(DevGeom g, const cd *J, double invk, double *pts) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= 4 * g.NT) return;
  const int t = e >> 2, i = e & 3;
  const double *x = g.tetP4 + 16 * (size_t)t + 4 * i;
  const double *tc = g.objOrigin + 3 * g.tetObj[t];
  const int4 vi = g.tetVI[t], fi = g.tetFI[t];
  const int v[4] = {vi.x, vi.y, vi.z, vi.w}, f[4] = {fi.x, fi.y, fi.z, fi.w};
  cd A[3] = {cmk(0, 0), cmk(0, 0), cmk(0, 0)}, rho = cmk(0, 0);
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const int a = f[q];
    if (a < 0 || a >= g.N) continue;
    const double s = (g.bfTet[a].x == t ? 1.0 : -1.0) * g.bfArea[a] * (1.0 / 12.0);
    const cd Ja = cscale(J[a], s);
    double Q[3];
    load3(g.V4, v[q], Q);
#pragma unroll
    for (int c = 0; c < 3; c++) A[c] = cadd(A[c], cscale(Ja, x[c] - Q[c]));
    rho = cadd(rho, cscale(Ja, 3.0 * invk));
  }
  double *p = pts + (size_t)EMT_PT * e;
  p[0] = x[0] - tc[0]; p[1] = x[1] - tc[1]; p[2] = x[2] - tc[2];
  p[3] = rho.r; p[4] = rho.i;
#pragma unroll
  for (int c = 0; c < 3; c++) { p[5 + 2 * c] = A[c].r; p[6 + 2 * c] = A[c].i; }
  p[11] = 0.0;
}

// block sum of the ten quantities (128 threads), written by thread 0..9
__device__ __forceinline__ void emt_block_out(const double (&d)[NPQ], double *out) {
  __shared__ double red[4][NPQ];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int n = 0; n < NPQ; n++) {
    const double v = warp_sum(d[n]);
    if (lane == 0) red[wid][n] = v;
  }
  __syncthreads();
  if (threadIdx.x < NPQ) {
    double s = 0.0;
    for (int w = 0; w < 4; w++) s += red[w][threadIdx.x];
    out[threadIdx.x] = s;
  }
}

// Far sum for JJ = conj(J_a) J_b: an N-body sum over the 4 NT quadrature
// points.  A thread keeps one point j, a block walks a chunk of bm.ic points
// i (a multiple of EMT_JT) staged in shared memory; the unordered pairs of one object are the tiles
// i-chunk <= j-tile, with weight 1/2 inside the diagonal (all ordered pairs of
// a diagonal chunk are walked, pairs i > j count 0 through the tile order).
// Per pair of points 27 FP64 operations beside the two polynomials: the
// potentials E = sum phi A_i, V = sum phi rho_i give power and the first
// torque at the end, t = psi Im(P) with P = conj(A_i).A_j - conj(rho_i) rho_j
// gives force (sum t x_i, sum t) and the second torque.  FP64-pipe bound: 335 us
// at N = 4,494 (two objects), against 12,625 us of the pair-by-pair kernel.
#define EMT_JT 128      // points j per block
#define EMT_IS 64       // points i staged at a time
template <int NT>
__global__ void __launch_bounds__(EMT_JT, 4) k_emt_far(DevGeom g, EmtKernel K, EmtBlockMap bm, const double *pts,
                                                       double *part) {
  __shared__ __align__(16) double sp[EMT_IS * EMT_PT];
  int m = 0;
  while (m + 1 < bm.nmap && (int)blockIdx.x >= bm.first[m + 1]) m++;
  const int rel = blockIdx.x - bm.first[m], jt = rel % bm.nj[m], ic = rel / bm.nj[m];
  const int oa = bm.oa[m], ob = bm.ob[m];
  const bool same = oa == ob;
  const int ib = bm.i0[m] + ic * bm.ic, jb = bm.j0[m] + jt * EMT_JT, tid = threadIdx.x;
  double d[NPQ];
#pragma unroll
  for (int n = 0; n < NPQ; n++) d[n] = 0.0;
  // same object: this block owns the points i < jb + EMT_JT of its chunk;
  // [jb, jb + EMT_JT) itself with weight 1/2
  const int iend = min(min(ib + bm.ic, bm.i1[m]), same ? jb + EMT_JT : bm.i1[m]);
  if (ib < iend) {
    const int j = jb + tid;
    const bool live = j < bm.j1[m];
    double P[11];
    {
      const double *p = pts + (size_t)EMT_PT * (live ? j : jb);
#pragma unroll
      for (int c = 0; c < 11; c++) P[c] = p[c];
    }
    // positions are relative to each object's origin; an object pair uses the
    // lower object's origin for both
    if (!same)
#pragma unroll
      for (int c = 0; c < 3; c++) P[c] += g.objOrigin[3 * ob + c] - g.objOrigin[3 * oa + c];
    double E[6] = {0, 0, 0, 0, 0, 0}, V[2] = {0, 0}, T = 0, G[3] = {0, 0, 0};
    for (int i0 = ib; i0 < iend; i0 += EMT_IS) {
      const int n = min(EMT_IS, iend - i0);
      __syncthreads();
      // the diagonal tile starts on a staging boundary (EMT_JT is a multiple
      // of EMT_IS); its weight 1/2 rides on the staged currents
      const double wgt = same && i0 >= jb ? 0.5 : 1.0;
      for (int e = tid; e < n * (EMT_PT / 2); e += EMT_JT) {
        double2 v = ((const double2 *)(pts + (size_t)EMT_PT * i0))[e];
        const int c = e % (EMT_PT / 2);
        if (c >= 2) v.x *= wgt;
        if (c >= 1) v.y *= wgt;
        ((double2 *)sp)[e] = v;
      }
      __syncthreads();
      if (same) {
#pragma unroll 2
        for (int q = 0; q < n; q++) {
          const double *s = sp + EMT_PT * q;
          const double x = s[0], y = s[1], z = s[2];
          const double R0 = x - P[0], R1 = y - P[1], R2 = z - P[2];
          const double r2 = fma(R0, R0, fma(R1, R1, R2 * R2));
          double phi, psi;
          emt_phipsi<NT>(K, r2, phi, psi);
          const double rr = s[3], ri = s[4];
          double im = ri * P[3] - rr * P[4];
          V[0] = fma(phi, rr, V[0]);
          V[1] = fma(phi, ri, V[1]);
#pragma unroll
          for (int c = 0; c < 3; c++) {
            const double ar = s[5 + 2 * c], ai = s[6 + 2 * c];
            E[2 * c] = fma(phi, ar, E[2 * c]);
            E[2 * c + 1] = fma(phi, ai, E[2 * c + 1]);
            im = fma(ar, P[6 + 2 * c], fma(-ai, P[5 + 2 * c], im));
          }
          const double t = psi * im;
          T += t;
          G[0] = fma(t, x, G[0]);
          G[1] = fma(t, y, G[1]);
          G[2] = fma(t, z, G[2]);
        }
      } else {
        // different objects: phi = e^{ikr}/(4 pi r), psi = phi (ikr - 1)/r^2,
        // E = sum phi conj(A_i), V = sum phi conj(rho_i), t = Re(P psi)
        for (int q = 0; q < n; q++) {
          const double *s = sp + EMT_PT * q;
          const double x = s[0], y = s[1], z = s[2];
          const double R0 = x - P[0], R1 = y - P[1], R2 = z - P[2];
          const double r2 = fma(R0, R0, fma(R1, R1, R2 * R2));
          const double ir = rsqrt_fast(r2), kr = K.k * (r2 * ir);
          double sn, cs;
          sincos(kr, &sn, &cs);
          const double ir2 = ir * ir, fr = cs * ir, fi = sn * ir;
          const double gr = (-fr - kr * fi) * ir2, gi = (-fi + kr * fr) * ir2;
          const double rr = s[3], ri = s[4];
          // P = conj(A).B - conj(rho) rho_j
          double pr = -(rr * P[3] + ri * P[4]), im = ri * P[3] - rr * P[4];
          V[0] = fma(fr, rr, fma(fi, ri, V[0]));
          V[1] = fma(fi, rr, fma(-fr, ri, V[1]));
#pragma unroll
          for (int c = 0; c < 3; c++) {
            const double ar = s[5 + 2 * c], ai = s[6 + 2 * c];
            E[2 * c] = fma(fr, ar, fma(fi, ai, E[2 * c]));
            E[2 * c + 1] = fma(fi, ar, fma(-fr, ai, E[2 * c + 1]));
            pr = fma(ar, P[5 + 2 * c], fma(ai, P[6 + 2 * c], pr));
            im = fma(ar, P[6 + 2 * c], fma(-ai, P[5 + 2 * c], im));
          }
          const double t = pr * gr - im * gi;
          T += t;
          G[0] = fma(t, x, G[0]);
          G[1] = fma(t, y, G[1]);
          G[2] = fma(t, z, G[2]);
        }
      }
    }
    if (live) {
      const double Z0 = 376.73031346177, i4p = 0.25 / M_PI;
      const double x[3] = {P[0], P[1], P[2]};
      double pw, tq[3];
      if (same) {
        pw = -(V[0] * P[3] + V[1] * P[4]);
#pragma unroll
        for (int c = 0; c < 3; c++) pw += E[2 * c] * P[5 + 2 * c] + E[2 * c + 1] * P[6 + 2 * c];
        // Im(conj(E) x B)
#pragma unroll
        for (int c = 0; c < 3; c++) {
          const int c1 = (c + 1) % 3, c2 = (c + 2) % 3;
          tq[c] = (E[2 * c1] * P[6 + 2 * c2] - E[2 * c1 + 1] * P[5 + 2 * c2]) -
                  (E[2 * c2] * P[6 + 2 * c1] - E[2 * c2 + 1] * P[5 + 2 * c1]);
        }
        const double fp = Z0 * K.k * i4p, fs = Z0 * TEN_THIRDS * K.k2 * K.k * i4p;
        d[0] = fp * K.k * pw;
#pragma unroll
        for (int c = 0; c < 3; c++) {
          const int c1 = (c + 1) % 3, c2 = (c + 2) % 3;
          d[1 + c] = fs * (G[c] - T * x[c]);
          d[4 + c] = fp * TEN_THIRDS * tq[c];
          d[7 + c] = fs * (x[c1] * G[c2] - x[c2] * G[c1]);
        }
      } else {
        // 1/2 Im and -1/2 Re of the complex sums
        pw = -(V[0] * P[4] + V[1] * P[3]);
#pragma unroll
        for (int c = 0; c < 3; c++) pw += E[2 * c] * P[6 + 2 * c] + E[2 * c + 1] * P[5 + 2 * c];
#pragma unroll
        for (int c = 0; c < 3; c++) {
          const int c1 = (c + 1) % 3, c2 = (c + 2) % 3;
          tq[c] = (E[2 * c1] * P[5 + 2 * c2] - E[2 * c1 + 1] * P[6 + 2 * c2]) -
                  (E[2 * c2] * P[5 + 2 * c1] - E[2 * c2 + 1] * P[6 + 2 * c1]);
        }
        const double h = Z0 * i4p * 0.5;
        d[0] = h * K.k * pw;
#pragma unroll
        for (int c = 0; c < 3; c++) {
          const int c1 = (c + 1) % 3, c2 = (c + 2) % 3;
          d[1 + c] = -h * TEN_THIRDS * (G[c] - T * x[c]);
          d[4 + c] = -h * TEN_THIRDS * tq[c];
          d[7 + c] = -h * TEN_THIRDS * (x[c1] * G[c2] - x[c2] * G[c1]);
        }
      }
    }
  }
  emt_block_out(d, part + (size_t)blockIdx.x * NPQ);
}

// The bilinear form of one tetrahedron pair for general JJ: with D the 4 x 4
// products JJ(a, b) s_a s_b A_a A_b of the faces and centroid-relative points
// and vertices, sum D (x - Q).(y - Q') = s x.y - x.v - w.y + c and
// sum D (x - Q) x (y - Q') = s x cross y - x cross v - w cross y + cc.
struct EmtForm {
  cd s, v[3], w[3], c, cc[3];
};

__device__ __forceinline__ void emt_form_zero(EmtForm &F) {
  F.s = F.c = cmk(0, 0);
  for (int i = 0; i < 3; i++) F.v[i] = F.w[i] = F.cc[i] = cmk(0, 0);
}
__device__ __forceinline__ void emt_form_add(EmtForm &F, cd D, const double *Q, const double *P) {
  F.s = cadd(F.s, D);
  F.c = cadd(F.c, cscale(D, Q[0] * P[0] + Q[1] * P[1] + Q[2] * P[2]));
#pragma unroll
  for (int i = 0; i < 3; i++) {
    const int i1 = (i + 1) % 3, i2 = (i + 2) % 3;
    F.v[i] = cadd(F.v[i], cscale(D, P[i]));
    F.w[i] = cadd(F.w[i], cscale(D, Q[i]));
    F.cc[i] = cadd(F.cc[i], cscale(D, Q[i1] * P[i2] - Q[i2] * P[i1]));
  }
}

// centroid, centroid-relative vertices of a tetrahedron
__device__ __forceinline__ void emt_tet(const DevGeom &g, int t, double *o, double (*Q)[3]) {
  const int4 vi = g.tetVI[t];
  const int v[4] = {vi.x, vi.y, vi.z, vi.w};
#pragma unroll
  for (int q = 0; q < 4; q++) load3(g.V4, v[q], Q[q]);
#pragma unroll
  for (int c = 0; c < 3; c++) o[c] = 0.25 * (Q[0][c] + Q[1][c] + Q[2][c] + Q[3][c]);
#pragma unroll
  for (int q = 0; q < 4; q++)
#pragma unroll
    for (int c = 0; c < 3; c++) Q[q][c] -= o[c];
}

// signed area of the face of basis function a on tetrahedron t
__device__ __forceinline__ double emt_sarea(const DevGeom &g, int a, int t) {
  return (g.bfTet[a].x == t ? 1.0 : -1.0) * g.bfArea[a];
}

// Z0 JJ(a, b) in the orientation (a, b) for any order of a and b: the sums
// take a <= b only, and the quantities' (anti)symmetry makes the reversed
// pair the conjugate.  The imaginary part of a = b is not used by the sums.
template <bool DRM>
__device__ __forceinline__ cd emt_jj(const PftArgs &P, int a, int b) {
  if (DRM) {
    const cd v = a <= b ? P.DR[(size_t)b + (size_t)a * P.ldr] : P.DR[(size_t)a + (size_t)b * P.ldr];
    return cmk(v.r, a == b ? 0.0 : (a < b ? v.i : -v.i));
  }
  const cd Ja = P.J[a], Jb = P.J[b];
  return cmk(Ja.r * Jb.r + Ja.i * Jb.i, a == b ? 0.0 : Ja.r * Jb.i - Ja.i * Jb.r);
}

// Far sum for a dressed Rytov matrix: thread per tetrahedron pair, 4 x 4
// points.  Blocks as in k_emt_far over tetrahedra: EMT_DJ tetrahedra j (one
// per thread) x EMT_DI tetrahedra i, i <= j within one object.
#define EMT_DJ 128
#define EMT_DI 16
template <int NT>
__global__ void __launch_bounds__(EMT_DJ) k_emt_far_dr(PftArgs P, EmtKernel K, EmtBlockMap bm, double *part) {
  const DevGeom &g = P.g;
  __shared__ double sQ[EMT_DI][4][3], sO[EMT_DI][3], sX[EMT_DI][4][3], sA[EMT_DI][4];
  __shared__ int sF[EMT_DI][4];
  int m = 0;
  while (m + 1 < bm.nmap && (int)blockIdx.x >= bm.first[m + 1]) m++;
  const int rel = blockIdx.x - bm.first[m], jt = rel % bm.nj[m], ic = rel / bm.nj[m];
  const int oa = bm.oa[m], ob = bm.ob[m];
  const bool same = oa == ob;
  const int ib = bm.i0[m] + ic * EMT_DI, jb = bm.j0[m] + jt * EMT_DJ, tid = threadIdx.x;
  const int iend = min(ib + EMT_DI, bm.i1[m]);
  double d[NPQ];
#pragma unroll
  for (int n = 0; n < NPQ; n++) d[n] = 0.0;
  if (!same || ib < jb + EMT_DJ) {
    if (tid < EMT_DI && ib + tid < iend) {
      const int t = ib + tid;
      double Q[4][3], o[3];
      emt_tet(g, t, o, Q);
      const int4 fi = g.tetFI[t];
      const int f[4] = {fi.x, fi.y, fi.z, fi.w};
      for (int q = 0; q < 4; q++) {
        const bool in = f[q] >= 0 && f[q] < g.N;
        sF[tid][q] = in ? f[q] : -1;
        sA[tid][q] = in ? emt_sarea(g, f[q], t) : 0.0;
        for (int c = 0; c < 3; c++) {
          sQ[tid][q][c] = Q[q][c];
          sX[tid][q][c] = g.tetP4[16 * (size_t)t + 4 * q + c] - o[c];
        }
      }
      for (int c = 0; c < 3; c++) sO[tid][c] = o[c] - g.objOrigin[3 * oa + c];
    }
    __syncthreads();
    const int j = jb + tid;
    if (j < bm.j1[m]) {
      double Q2[4][3], o2[3], y[4][3], A2[4];
      int F2[4];
      emt_tet(g, j, o2, Q2);
      {
        const int4 fi = g.tetFI[j];
        const int f[4] = {fi.x, fi.y, fi.z, fi.w};
#pragma unroll
        for (int q = 0; q < 4; q++) {
          const bool in = f[q] >= 0 && f[q] < g.N;
          F2[q] = in ? f[q] : -1;
          A2[q] = in ? emt_sarea(g, f[q], j) : 0.0;
#pragma unroll
          for (int c = 0; c < 3; c++) y[q][c] = g.tetP4[16 * (size_t)j + 4 * q + c] - o2[c];
        }
      }
#pragma unroll
      for (int c = 0; c < 3; c++) o2[c] -= g.objOrigin[3 * oa + c];
      for (int i = ib; i < iend; i++) {
        if (same && i > j) break;
        const int li = i - ib;
        EmtForm F;
        emt_form_zero(F);
        for (int p = 0; p < 4; p++) {
          const int a = sF[li][p];
          if (a < 0) continue;
#pragma unroll
          for (int q = 0; q < 4; q++) {
            if (F2[q] < 0) continue;
            emt_form_add(F, cscale(emt_jj<true>(P, a, F2[q]), sA[li][p] * A2[q]), sQ[li][p], Q2[q]);
          }
        }
        const double wgt = same && i == j ? 0.5 : 1.0;
        const double ox[3] = {sO[li][0], sO[li][1], sO[li][2]};
        const double nine_k2 = 9.0 / K.k2;
        cd pw = cmk(0, 0);
        double X0[3] = {0, 0, 0}, tq[3] = {0, 0, 0}, t2[3] = {0, 0, 0};
        for (int p = 0; p < 4; p++) {
          const double x0 = sX[li][p][0], x1 = sX[li][p][1], x2 = sX[li][p][2];
          // P = al.y + be; first torque: Im(al) cross y + ga
          const cd al[3] = {csub(cscale(F.s, x0), F.w[0]), csub(cscale(F.s, x1), F.w[1]), csub(cscale(F.s, x2), F.w[2])};
          const cd be = csub(csub(F.c, cadd(cadd(cscale(F.v[0], x0), cscale(F.v[1], x1)), cscale(F.v[2], x2))),
                             cscale(F.s, nine_k2));
          const cd ga[3] = {csub(F.cc[0], csub(cscale(F.v[2], x1), cscale(F.v[1], x2))),
                            csub(F.cc[1], csub(cscale(F.v[0], x2), cscale(F.v[2], x0))),
                            csub(F.cc[2], csub(cscale(F.v[1], x0), cscale(F.v[0], x1)))};
          const double xa0 = x0 + ox[0], xa1 = x1 + ox[1], xa2 = x2 + ox[2];
          double Ph = 0, Ys[3] = {0, 0, 0}, T = 0, H[3] = {0, 0, 0};
          cd Phc = cmk(0, 0), Yc[3] = {cmk(0, 0), cmk(0, 0), cmk(0, 0)};
#pragma unroll
          for (int q = 0; q < 4; q++) {
            const double R0 = xa0 - (o2[0] + y[q][0]), R1 = xa1 - (o2[1] + y[q][1]), R2 = xa2 - (o2[2] + y[q][2]);
            const double r2 = fma(R0, R0, fma(R1, R1, R2 * R2));
            if (same) {
              double phi, psi;
              emt_phipsi<NT>(K, r2, phi, psi);
              Ph += phi;
              const double im = fma(al[0].i, y[q][0], fma(al[1].i, y[q][1], fma(al[2].i, y[q][2], be.i)));
              const double t = psi * im;
              T += t;
#pragma unroll
              for (int c = 0; c < 3; c++) {
                Ys[c] = fma(phi, y[q][c], Ys[c]);
                H[c] = fma(t, y[q][c], H[c]);
              }
            } else {
              const double ir = rsqrt_fast(r2), kr = K.k * (r2 * ir);
              double sn, cs;
              sincos(kr, &sn, &cs);
              const cd phi = cmk(cs * ir, sn * ir), psi = cscale(cmul(phi, cmk(-1.0, kr)), ir * ir);
              const cd pp = cadd(cadd(cadd(cscale(al[0], y[q][0]), cscale(al[1], y[q][1])), cscale(al[2], y[q][2])), be);
              const double t = pp.r * psi.r - pp.i * psi.i;
              T += t;
              Phc = cadd(Phc, phi);
#pragma unroll
              for (int c = 0; c < 3; c++) {
                Yc[c] = cadd(Yc[c], cscale(phi, y[q][c]));
                H[c] = fma(t, y[q][c], H[c]);
              }
            }
          }
          // force sum t (xa - xb), second torque sum t (xb cross xa)
          const double xa[3] = {xa0, xa1, xa2};
          double xb[3];
#pragma unroll
          for (int c = 0; c < 3; c++) {
            xb[c] = fma(T, o2[c], H[c]);        // sum t xb
            X0[c] += fma(T, xa[c], -xb[c]);
          }
#pragma unroll
          for (int c = 0; c < 3; c++) {
            const int c1 = (c + 1) % 3, c2 = (c + 2) % 3;
            t2[c] += xb[c1] * xa[c2] - xb[c2] * xa[c1];
          }
          if (same) {
            pw.r += fma(al[0].r, Ys[0], fma(al[1].r, Ys[1], fma(al[2].r, Ys[2], be.r * Ph)));
#pragma unroll
            for (int c = 0; c < 3; c++) {
              const int c1 = (c + 1) % 3, c2 = (c + 2) % 3;
              tq[c] += al[c1].i * Ys[c2] - al[c2].i * Ys[c1] + ga[c].i * Ph;
            }
          } else {
            const cd e = cadd(cadd(cadd(cmul(al[0], Yc[0]), cmul(al[1], Yc[1])), cmul(al[2], Yc[2])), cmul(be, Phc));
            pw = cadd(pw, e);
#pragma unroll
            for (int c = 0; c < 3; c++) {
              const int c1 = (c + 1) % 3, c2 = (c + 2) % 3;
              tq[c] += csub(cmul(al[c1], Yc[c2]), cmul(al[c2], Yc[c1])).r + cmul(ga[c], Phc).r;
            }
          }
        }
        const double Z0 = 376.73031346177, i4p = 0.25 / M_PI, w2 = wgt * Z0 * i4p / 144.0;
        double f0, f1, f2;
        if (same) { f0 = w2 * K.k2 * pw.r; f1 = w2 * TEN_THIRDS * K.k2 * K.k; f2 = w2 * TEN_THIRDS * K.k; }
        else { f0 = 0.5 * w2 * K.k * pw.i; f1 = f2 = -0.5 * w2 * TEN_THIRDS; }
        d[0] += f0;
#pragma unroll
        for (int c = 0; c < 3; c++) {
          d[1 + c] = fma(f1, X0[c], d[1 + c]);
          d[4 + c] = fma(f2, tq[c], d[4 + c]);
          d[7 + c] = fma(f1, t2[c], d[7 + c]);
        }
      }
    }
  }
  emt_block_out(d, part + (size_t)blockIdx.x * NPQ);
}

// Near pairs: for every ordered tetrahedron pair that feeds a near pair
// (a <= b) the 16-point rule minus the 4-point rule, 16 lanes per tetrahedron
// pair.  Lane (f1, f2) forms one product of the 4 x 4 form, a shuffle tree
// sums them; then lane i holds point i of the row tetrahedron and walks the 16
// points of the column tetrahedron.  Each half warp takes a contiguous run of
// pairs (their objects change rarely) and keeps its sums in registers.  550 us at
// N = 4,494 against 8,817 us for one warp per basis-function pair.
#define EMT_NG 8         // half warps per block
template <int NT, bool DRM>
__global__ void __launch_bounds__(EMT_NG * 16) k_emt_near(PftArgs P, NearData nd, EmtKernel K, int per, double *part) {
  const DevGeom &g = P.g;
  __shared__ double sy[EMT_NG][16 * 4 + 2];      // column points and weights of each group
  __shared__ double acc[EMT_NG][PMAXOBJ][NPQ];
  const int tid = threadIdx.x, l = tid & 15, grp = tid >> 4, lane = tid & 31;
  const unsigned mask = 0xffffu << (lane & 16);
  for (int e = tid; e < EMT_NG * PMAXOBJ * NPQ; e += EMT_NG * 16) (&acc[0][0][0])[e] = 0.0;
  __syncthreads();
  const double ub[4] = {c_tcr16[4 * l], c_tcr16[4 * l + 1], c_tcr16[4 * l + 2], c_tcr16[4 * l + 3]};
  const double lam0 = 1.0 - ub[0] - ub[1] - ub[2];
  const double qa = 0.13819660112501051, qb = 0.58541019662496850;
  const int f1 = l >> 2, f2 = l & 3;
  const double Z0 = 376.73031346177, i4p = 0.25 / M_PI;
  const double fp = Z0 * K.k * i4p, fs = Z0 * TEN_THIRDS * K.k2 * K.k * i4p, nine_k2 = 9.0 / K.k2;
  double d[NPQ];
#pragma unroll
  for (int n = 0; n < NPQ; n++) d[n] = 0.0;
  const long long p0 = ((long long)blockIdx.x * EMT_NG + grp) * per;
  const int beg = (int)min((long long)nd.ntp, p0), end = (int)min((long long)nd.ntp, p0 + per);
  int obj = -1;
  for (int p = beg; p < end; p++) {
    const int4 tp = nd.tp[p];
    const int to = g.tetObj[tp.x];
    if (to != obj) {
      if (obj >= 0)
        for (int n = 0; n < NPQ; n++) {
          double s = d[n];
          for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(mask, s, o);
          if (l == 0) acc[grp][obj][n] += s;
          d[n] = 0.0;
        }
      obj = to;
    }
    const int4 fa = g.tetFI[tp.x], fb = g.tetFI[tp.y];
    double Q1[4][3], Q2[4][3], o1[3], o2[3];
    emt_tet(g, tp.x, o1, Q1);
    emt_tet(g, tp.y, o2, Q2);
    // this lane's entry of the form
    const int a = f1 == 0 ? fa.x : f1 == 1 ? fa.y : f1 == 2 ? fa.z : fa.w;
    const int b = f2 == 0 ? fb.x : f2 == 1 ? fb.y : f2 == 2 ? fb.z : fb.w;
    cd D = cmk(0, 0);
    if (a >= 0 && a < g.N && b >= 0 && b < g.N && a <= b) {
      const int4 va = g.bfV[a], vb = g.bfV[b];
      const int2 ea = g.bfQ[a], eb = g.bfQ[b];
      const int A5[5] = {ea.x, va.x, va.y, va.z, ea.y}, B5[5] = {eb.x, vb.x, vb.y, vb.z, eb.y};
      int ncv = 0;
#pragma unroll
      for (int i = 0; i < 5; i++)
#pragma unroll
        for (int j = 0; j < 5; j++) ncv += A5[i] == B5[j];
      if (ncv) D = cscale(emt_jj<DRM>(P, a, b), emt_sarea(g, a, tp.x) * emt_sarea(g, b, tp.y));
    }
    EmtForm F;
    emt_form_zero(F);
    {
      double qq1[3], qq2[3];
#pragma unroll
      for (int c = 0; c < 3; c++) {
        qq1[c] = f1 == 0 ? Q1[0][c] : f1 == 1 ? Q1[1][c] : f1 == 2 ? Q1[2][c] : Q1[3][c];
        qq2[c] = f2 == 0 ? Q2[0][c] : f2 == 1 ? Q2[1][c] : f2 == 2 ? Q2[2][c] : Q2[3][c];
      }
      emt_form_add(F, D, qq1, qq2);
    }
    auto sum16 = [&](double x) {
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) x += __shfl_xor_sync(mask, x, o);
      return x;
    };
    F.s.r = sum16(F.s.r); F.s.i = sum16(F.s.i);
    F.c.r = sum16(F.c.r); F.c.i = sum16(F.c.i);
#pragma unroll
    for (int c = 0; c < 3; c++) {
      F.v[c].r = sum16(F.v[c].r); F.v[c].i = sum16(F.v[c].i);
      F.w[c].r = sum16(F.w[c].r); F.w[c].i = sum16(F.w[c].i);
      F.cc[c].i = sum16(F.cc[c].i);
    }
    double x[3], y[3];
#pragma unroll
    for (int c = 0; c < 3; c++) {
      x[c] = lam0 * Q1[0][c] + ub[0] * Q1[1][c] + ub[1] * Q1[2][c] + ub[2] * Q1[3][c];
      y[c] = lam0 * Q2[0][c] + ub[0] * Q2[1][c] + ub[1] * Q2[2][c] + ub[2] * Q2[3][c];
    }
    __syncwarp(mask);
    sy[grp][4 * l] = y[0]; sy[grp][4 * l + 1] = y[1]; sy[grp][4 * l + 2] = y[2]; sy[grp][4 * l + 3] = ub[3];
    __syncwarp(mask);
    const double oo[3] = {o1[0] - o2[0], o1[1] - o2[1], o1[2] - o2[2]};
    const double *tc = g.objOrigin + 3 * to;
    const double c2[3] = {o2[0] - tc[0], o2[1] - tc[1], o2[2] - tc[2]};
    // pass 0: this lane's row point against the 16 column points, weight +;
    // pass 1: one point pair of the 4-point rule, weight -
#pragma unroll 1
    for (int pass = 0; pass < 2; pass++) {
      double wx = 2.0 * ub[3];
      double yq[3];
      if (pass) {
        wx = -2.0 / 24.0;
#pragma unroll
        for (int c = 0; c < 3; c++) {
          // centroid-relative vertices sum to zero: qa sum + (qb - qa) Q
          x[c] = (qb - qa) * (f1 == 0 ? Q1[0][c] : f1 == 1 ? Q1[1][c] : f1 == 2 ? Q1[2][c] : Q1[3][c]);
          yq[c] = (qb - qa) * (f2 == 0 ? Q2[0][c] : f2 == 1 ? Q2[1][c] : f2 == 2 ? Q2[2][c] : Q2[3][c]);
        }
      }
      const cd al[3] = {csub(cscale(F.s, x[0]), F.w[0]), csub(cscale(F.s, x[1]), F.w[1]), csub(cscale(F.s, x[2]), F.w[2])};
      const cd be = csub(csub(F.c, cadd(cadd(cscale(F.v[0], x[0]), cscale(F.v[1], x[1])), cscale(F.v[2], x[2]))),
                         cscale(F.s, nine_k2));
      const double ga[3] = {F.cc[0].i - (x[1] * F.v[2].i - x[2] * F.v[1].i),
                            F.cc[1].i - (x[2] * F.v[0].i - x[0] * F.v[2].i),
                            F.cc[2].i - (x[0] * F.v[1].i - x[1] * F.v[0].i)};
      const double xr[3] = {x[0] + oo[0], x[1] + oo[1], x[2] + oo[2]};
      double Ph = 0, Ys[3] = {0, 0, 0}, T = 0, H[3] = {0, 0, 0};
      const int nq = pass ? 1 : 16;
#pragma unroll 1
      for (int q = 0; q < nq; q++) {
        double wy = 2.0 / 24.0;
        if (!pass) {
          yq[0] = sy[grp][4 * q]; yq[1] = sy[grp][4 * q + 1]; yq[2] = sy[grp][4 * q + 2];
          wy = 2.0 * sy[grp][4 * q + 3];
        }
        const double R0 = xr[0] - yq[0], R1 = xr[1] - yq[1], R2 = xr[2] - yq[2];
        const double r2 = fma(R0, R0, fma(R1, R1, R2 * R2));
        double phi, psi;
        emt_phipsi<NT>(K, r2, phi, psi);
        phi *= wy;
        const double im = fma(al[0].i, yq[0], fma(al[1].i, yq[1], fma(al[2].i, yq[2], be.i)));
        const double t = wy * psi * im;
        Ph += phi;
        T += t;
#pragma unroll
        for (int c = 0; c < 3; c++) {
          Ys[c] = fma(phi, yq[c], Ys[c]);
          H[c] = fma(t, yq[c], H[c]);
        }
      }
      double xb[3], xa[3];
#pragma unroll
      for (int c = 0; c < 3; c++) {
        xb[c] = fma(T, c2[c], H[c]);
        xa[c] = xr[c] + c2[c];
      }
      const double pw = fma(al[0].r, Ys[0], fma(al[1].r, Ys[1], fma(al[2].r, Ys[2], be.r * Ph)));
      d[0] = fma(wx * fp * K.k, pw, d[0]);
#pragma unroll
      for (int c = 0; c < 3; c++) {
        const int c1 = (c + 1) % 3, cc2 = (c + 2) % 3;
        d[1 + c] = fma(wx * fs, fma(T, xa[c], -xb[c]), d[1 + c]);
        d[4 + c] = fma(wx * fp * TEN_THIRDS, al[c1].i * Ys[cc2] - al[cc2].i * Ys[c1] + ga[c] * Ph, d[4 + c]);
        d[7 + c] = fma(wx * fs, xb[c1] * xa[cc2] - xb[cc2] * xa[c1], d[7 + c]);
      }
    }
  }
  if (obj >= 0)
    for (int n = 0; n < NPQ; n++) {
      double s = d[n];
      for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(mask, s, o);
      if (l == 0) acc[grp][obj][n] += s;
    }
  __syncthreads();
  for (int e = tid; e < P.nobj * NPQ; e += EMT_NG * 16) {
    double s = 0.0;
    for (int q = 0; q < EMT_NG; q++) s += acc[q][e / NPQ][e % NPQ];
    part[(size_t)blockIdx.x * P.nobj * NPQ + e] = s;
  }
}

// 1/2 sum_a t4(a, a), power only: part[block][object]
__global__ void k_emt_self(PftArgs P, double *part) {
  const int a = (blockIdx.x * blockDim.x + threadIdx.x) >> 4, l = threadIdx.x & 15;
  __shared__ double red[8][PMAXOBJ];
  double v = 0.0;
  int obj = 0;
  if (a < P.g.N) {
    obj = P.g.bfV[a].w;
    cd q[NPQ];
    scat_q(P, a, a, 4, true, l, 16, q);
    const double Z0 = 376.73031346177;
    double u;
    if (P.DR) u = P.DR[(size_t)a + (size_t)a * P.ldr].r;
    else u = P.J[a].r * P.J[a].r + P.J[a].i * P.J[a].i;
    v = 0.5 * Z0 * u * q[0].i;
  }
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int o = 0; o < P.nobj; o++) {
    const double s = warp_sum(o == obj ? v : 0.0);
    if (lane == 0) red[wid][o] = s;
  }
  __syncthreads();
  if (threadIdx.x < P.nobj) {
    double s = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) s += red[w][threadIdx.x];
    part[(size_t)blockIdx.x * P.nobj + threadIdx.x] = s;
  }
}

// Fixed-order sums of block partials: block b of the grid sums the rows
// [row0, row1) of an array of `width` columns into out[0..width), column by
// column (threads stride the rows, then a shared-memory tree).
struct EmtReduce {
  int n, wmax;
  const double *src[16];
  long long rows[16];
  int width[16];
  double *dst[16];
};
__global__ void __launch_bounds__(256) k_emt_reduce(EmtReduce R) {
  const int job = blockIdx.x;
  __shared__ double red[8];
  const double *s = R.src[job];
  const long long rows = R.rows[job];
  const int w = R.width[job], c = blockIdx.y;
  if (c >= w) return;
  double v = 0.0;
  for (long long r = threadIdx.x; r < rows; r += 256) v += s[r * w + c];
  v = warp_sum(v);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int i = 0; i < 8; i++) t += red[i];
    R.dst[job][c] = t;
  }
}
