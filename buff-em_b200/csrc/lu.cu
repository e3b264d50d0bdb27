// Dense complex128 LU with partial pivoting and the triangular solves on
// sm_100a: replaces HMatrix::LUFactorize / LUSolve (LAPACK zgetrf / zgetrs,
// call sites buff-scatter.cc:285,314).
//
// Factorisation: recursive right-looking LU over column halves down to blocks of
// 128 columns, which are factored in panels of 32 with the panel's rows in
// registers (one cluster, or the whole grid for tall panels).  Row interchanges
// are applied to every other column (LAPACK ipiv semantics: ipiv[i] is the
// 1-based row swapped with row i, applied in order).  Off-diagonal blocks use a
// unit-lower TRSM (128-row leaf + GEMM recursion).  The Schur complements go to
// the INT8 tensor cores (gemm_i8.cu) where they are large enough, else to the
// FP64 tensor path (mma.sync f64), 4M complex product, cp.async pipelines.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <mutex>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "internal.h"

namespace cg = cooperative_groups;

namespace bg {

struct cdl { double r, i; };
struct cfl { float r, i; };
// The kernels of the factorisation's chain follow one another within a few
// microseconds of work: each is launched while its predecessor still runs
// (programmatic dependent launch) and starts with pdl_enter, which lets its own
// successor launch and then waits until the predecessor has finished and its
// writes are visible.  Factor and solve 18.6 -> 17.9 ms at N = 4,092, small body
// of N = 1,350 4.87 -> 4.79 ms.  Only where one factorisation has the device to
// itself (t_pdl): CTAs that wait take room from the other streams of a batched
// sweep (217 -> 246 ms).
static thread_local bool t_pdl = false;
__device__ __forceinline__ void pdl_enter() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
template <class... P, class... A>
static cudaError_t pdl_launch(void (*kern)(P...), dim3 grid, int threads, size_t smem, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream();
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = t_pdl;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, P(args)...);
}

template <class C> struct CxT;
template <> struct CxT<cdl> { typedef double R; };
template <> struct CxT<cfl> { typedef float R; };

// tensor-core complex-FP32 GEMM (gemm_tc.cu)
size_t zgemm_i8_bytes(int M, int N, int K);
int zgemm_i8(int M, int N, int K, const void *A, size_t lda, const void *B, size_t ldb, void *C, size_t ldc, void *work,
             size_t bytes, int *err);
int cgemm_sub_tf32(int M, int N, int K, const void *A, size_t lda, const void *B, size_t ldb, void *C, size_t ldc,
                   float *At, int *err);

// =========================================================================
// complex GEMM  C(MxN) -= A(MxK) * B(KxN), column-major, complex128, on the
// FP64 tensor cores with mma.sync m16n8k16 f64 (the sm_90+/sm_100 DMMA shape:
// 2048 FMAs per instruction).  Warp tile 32x32 complex (2 x m16, 4 x n8),
// CTA tile BM x BN, K chunk BK, STAGES-deep cp.async pipeline.  Shared tiles
// are complex-interleaved (one 16-byte load gives re and im); row strides are
// padded so every fragment load phase hits 32 distinct banks.
//   Cr += Ar Br + Ai (-Bi),   Ci += Ar Bi + Ai Br        (4M product)
// Fragment layouts (m16n8k16, lane = 4*t1 + t0):
//   A: a[v] = A[t1 + 8(v&1)][t0 + 4(v>>1)], v = 0..7
//   B: b[v] = B[t0 + 4v][t1],               v = 0..3
//   C: c[v] = C[t1 + 8(v>>1)][2 t0 + (v&1)]
// =========================================================================
__device__ __forceinline__ void dmma16(double (&d)[4], const double (&a)[8], const double (&b)[4]) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7,%8,%9,%10,%11}, "
      "{%12,%13,%14,%15}, {%0,%1,%2,%3};\n"
      : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
      : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(a[4]), "d"(a[5]), "d"(a[6]), "d"(a[7]), "d"(b[0]),
        "d"(b[1]), "d"(b[2]), "d"(b[3]));
}

// one access per entry of an aligned shared array
__device__ __forceinline__ cdl lds_c(const cdl *p) {
  const double2 v = *reinterpret_cast<const double2 *>(p);
  return cdl{v.x, v.y};
}
__device__ __forceinline__ cfl lds_c(const cfl *p) {
  const float2 v = *reinterpret_cast<const float2 *>(p);
  return cfl{v.x, v.y};
}
__device__ __forceinline__ void sts_c(cdl *p, cdl v) { *reinterpret_cast<double2 *>(p) = make_double2(v.r, v.i); }
__device__ __forceinline__ void sts_c(cfl *p, cfl v) { *reinterpret_cast<float2 *>(p) = make_float2(v.r, v.i); }

__device__ __forceinline__ void cp16(void *smem, const void *gmem, bool pred) {
  unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  int n = pred ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(n));
}
// one matrix entry, zero when !pred
__device__ __forceinline__ void cp_entry(cdl *smem, const cdl *gmem, bool pred) { cp16(smem, gmem, pred); }
__device__ __forceinline__ void cp_entry(cfl *smem, const cfl *gmem, bool pred) {
  unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  int n = pred ? 8 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(s), "l"(gmem), "r"(n));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

template <int BM, int BN, int BK, int STAGES>
struct GemmCfg {
  static constexpr int WM = BM / 32, WN = BN / 32, THREADS = WM * WN * 32;
  static constexpr int AP = BM + 2;   // As[k][m] stride (complex), = 2 mod 8
  static constexpr int BP = BK + 4;   // Bs[n][k] stride (complex), = 4 mod 8
  static constexpr int SMEM = STAGES * (BK * AP + BN * BP) * 16;
};

template <int BM, int BN, int BK, int STAGES>
__global__ void __launch_bounds__(GemmCfg<BM, BN, BK, STAGES>::THREADS)
    k_zgemm_sub(int M, int N, int K, const cdl *__restrict__ A, size_t lda, const cdl *__restrict__ B, size_t ldb,
                cdl *C, size_t ldc) {
  pdl_enter();
  using Cfg = GemmCfg<BM, BN, BK, STAGES>;
  constexpr int T = Cfg::THREADS, AP = Cfg::AP, BP = Cfg::BP;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cdl *As = (cdl *)smem_raw;              // [STAGES][BK][AP]
  cdl *Bs = As + STAGES * BK * AP;        // [STAGES][BN][BP]
  const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = warp % Cfg::WM, wn = warp / Cfg::WM;
  const int t0 = lane & 3, t1 = lane >> 2;
  double cr[2][4][4], ci[2][4][4];
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int j = 0; j < 4; j++)
#pragma unroll
      for (int v = 0; v < 4; v++) cr[i][j][v] = ci[i][j][v] = 0.0;
  const int nchunks = (K + BK - 1) / BK;
  auto load_chunk = [&](int chunk, int stage) {
    const int k0 = chunk * BK;
    cdl *as = As + stage * BK * AP;
    cdl *bs = Bs + stage * BN * BP;
#pragma unroll
    for (int it = 0; it < (BM * BK) / T; it++) {
      int e = tid + it * T;
      int r = e % BM, kk = e / BM;
      int gr = m0 + r, gk = k0 + kk;
      bool ok = gr < M && gk < K;
      cp16(as + kk * AP + r, ok ? A + (size_t)gk * lda + gr : A, ok);
    }
#pragma unroll
    for (int it = 0; it < (BK * BN) / T; it++) {
      int e = tid + it * T;
      int kb = e % BK, nb = e / BK;
      int gk = k0 + kb, gn = n0 + nb;
      bool ok = gk < K && gn < N;
      cp16(bs + nb * BP + kb, ok ? B + (size_t)gn * ldb + gk : B, ok);
    }
  };
#pragma unroll
  for (int s = 0; s < STAGES - 1; s++) {
    if (s < nchunks) load_chunk(s, s);
    cp_commit();
  }
  for (int chunk = 0; chunk < nchunks; chunk++) {
    cp_wait<STAGES - 2>();
    __syncthreads();
    int nxt = chunk + STAGES - 1;
    if (nxt < nchunks) load_chunk(nxt, nxt % STAGES);
    cp_commit();
    const cdl *as = As + (chunk % STAGES) * BK * AP + wm * 32 + t1;
    const cdl *bs = Bs + (chunk % STAGES) * BN * BP + (wn * 32 + t1) * BP + t0;
#pragma unroll
    for (int ks = 0; ks < BK / 16; ks++) {
      double ar[2][8], ai[2][8];
#pragma unroll
      for (int mt = 0; mt < 2; mt++)
#pragma unroll
        for (int v = 0; v < 8; v++) {
          cdl x = as[(ks * 16 + t0 + 4 * (v >> 1)) * AP + mt * 16 + 8 * (v & 1)];
          ar[mt][v] = x.r;
          ai[mt][v] = x.i;
        }
#pragma unroll
      for (int nt = 0; nt < 4; nt++) {
        double br[4], bi[4], nbi[4];
#pragma unroll
        for (int v = 0; v < 4; v++) {
          cdl x = bs[nt * 8 * BP + ks * 16 + 4 * v];
          br[v] = x.r;
          bi[v] = x.i;
          nbi[v] = -x.i;
        }
#pragma unroll
        for (int mt = 0; mt < 2; mt++) {
          dmma16(cr[mt][nt], ar[mt], br);
          dmma16(cr[mt][nt], ai[mt], nbi);
          dmma16(ci[mt][nt], ar[mt], bi);
          dmma16(ci[mt][nt], ai[mt], br);
        }
      }
    }
  }
  cp_wait<0>();
  // C -= accumulators, eight entries at a time: the loads of a group are
  // issued together before its stores (one memory round trip per group
  // instead of one per entry)
#pragma unroll
  for (int nt = 0; nt < 4; nt++) {
    cdl x[2][4];
#pragma unroll
    for (int mt = 0; mt < 2; mt++)
#pragma unroll
      for (int v = 0; v < 4; v++) {
        const int row = m0 + wm * 32 + mt * 16 + t1 + 8 * (v >> 1);
        const int col = n0 + wn * 32 + nt * 8 + 2 * t0 + (v & 1);
        x[mt][v] = (row < M && col < N) ? C[(size_t)col * ldc + row] : cdl{0.0, 0.0};
      }
#pragma unroll
    for (int mt = 0; mt < 2; mt++)
#pragma unroll
      for (int v = 0; v < 4; v++) {
        const int row = m0 + wm * 32 + mt * 16 + t1 + 8 * (v >> 1);
        const int col = n0 + wn * 32 + nt * 8 + 2 * t0 + (v & 1);
        if (row < M && col < N) {
          cdl y = x[mt][v];
          y.r -= cr[mt][nt][v];
          y.i -= ci[mt][nt][v];
          C[(size_t)col * ldc + row] = y;
        }
      }
  }
}

// The same product with 32 x 32 tiles and the K loop split over the four warps
// of a CTA (warp q takes rows 8 q .. 8 q + 7 of every 32-deep chunk; the four
// partial tiles are summed in shared memory in warp order).  A 64 x 64 tile
// occupies its SM for 17 us at K = 128 whatever the grid; where a product has
// too few of them for the 148 SMs this form has four times the tiles, a quarter
// of the time each: 128 x 128 x 128 27.9 -> 10.5 us, 512^3 90 -> 43 us,
// 256 x 2048 x 256 49 -> 45 us.  It reads twice the operand bytes per flop and
// loses from about 230 tiles on (3840 x 256 x 256, 240 tiles: 83 against 87 us).
__device__ __forceinline__ void dmma8(double (&d)[4], const double (&a)[4], const double (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
      : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}
#define ZG_SMALL 220             // 64 x 64 tiles up to which the small tiles are taken
#define ZS_ST 3
#define ZS_AP 34                 // As[k][m] stride, = 2 mod 8
#define ZS_BP 36                 // Bs[n][k] stride, = 4 mod 8
#define ZS_STAGE (32 * ZS_AP + 32 * ZS_BP)
#define ZS_SMEM (ZS_ST * ZS_STAGE * 16)
__device__ __forceinline__ void zgemm_small_tile(cdl *sm, int m0, int n0, int M, int N, int K, const cdl *__restrict__ A,
                                                 size_t lda, const cdl *__restrict__ B, size_t ldb, cdl *C, size_t ldc) {
  const int tid = threadIdx.x, lane = tid & 31, wk = tid >> 5, t0 = lane & 3, t1 = lane >> 2;
  double cr[2][4][4], ci[2][4][4];
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int j = 0; j < 4; j++)
#pragma unroll
      for (int v = 0; v < 4; v++) cr[i][j][v] = ci[i][j][v] = 0.0;
  const int nchunks = (K + 31) / 32;
  auto load_chunk = [&](int chunk) {
    const int k0 = chunk * 32;
    cdl *as = sm + (chunk % ZS_ST) * ZS_STAGE, *bs = as + 32 * ZS_AP;
#pragma unroll
    for (int it = 0; it < 8; it++) {
      const int kk = wk + 4 * it;
      const bool oka = m0 + lane < M && k0 + kk < K, okb = k0 + lane < K && n0 + kk < N;
      cp16(as + kk * ZS_AP + lane, oka ? A + (size_t)(k0 + kk) * lda + m0 + lane : A, oka);
      cp16(bs + kk * ZS_BP + lane, okb ? B + (size_t)(n0 + kk) * ldb + k0 + lane : B, okb);
    }
  };
#pragma unroll
  for (int s = 0; s < ZS_ST - 1; s++) {
    if (s < nchunks) load_chunk(s);
    cp_commit();
  }
  // this thread's entries of C (the rows 8 wk .. of the tile), read early
  cdl x[8];
#pragma unroll
  for (int e = 0; e < 8; e++) {
    const int col = n0 + wk * 8 + e;
    x[e] = (m0 + lane < M && col < N) ? C[(size_t)col * ldc + m0 + lane] : cdl{0.0, 0.0};
  }
  for (int chunk = 0; chunk < nchunks; chunk++) {
    cp_wait<ZS_ST - 2>();
    __syncthreads();
    if (chunk + ZS_ST - 1 < nchunks) load_chunk(chunk + ZS_ST - 1);
    cp_commit();
    const cdl *as = sm + (chunk % ZS_ST) * ZS_STAGE + (8 * wk + t0) * ZS_AP + t1;
    const cdl *bs = sm + (chunk % ZS_ST) * ZS_STAGE + 32 * ZS_AP + t1 * ZS_BP + 8 * wk + t0;
    double ar[2][4], ai[2][4];
#pragma unroll
    for (int mt = 0; mt < 2; mt++)
#pragma unroll
      for (int v = 0; v < 4; v++) {
        const cdl z = lds_c(as + 4 * (v >> 1) * ZS_AP + mt * 16 + 8 * (v & 1));
        ar[mt][v] = z.r;
        ai[mt][v] = z.i;
      }
#pragma unroll
    for (int nt = 0; nt < 4; nt++) {
      double br[2], bi[2], nbi[2];
#pragma unroll
      for (int v = 0; v < 2; v++) {
        const cdl z = lds_c(bs + nt * 8 * ZS_BP + 4 * v);
        br[v] = z.r;
        bi[v] = z.i;
        nbi[v] = -z.i;
      }
#pragma unroll
      for (int mt = 0; mt < 2; mt++) {
        dmma8(cr[mt][nt], ar[mt], br);
        dmma8(cr[mt][nt], ai[mt], nbi);
        dmma8(ci[mt][nt], ar[mt], bi);
        dmma8(ci[mt][nt], ai[mt], br);
      }
    }
  }
  cp_wait<0>();
  __syncthreads();
  // partial tiles [warp][col][row], then C -= their sum
#pragma unroll
  for (int mt = 0; mt < 2; mt++)
#pragma unroll
    for (int nt = 0; nt < 4; nt++)
#pragma unroll
      for (int v = 0; v < 4; v++)
        sts_c(sm + wk * 32 * 33 + (nt * 8 + 2 * t0 + (v & 1)) * 33 + mt * 16 + t1 + 8 * (v >> 1),
              cdl{cr[mt][nt][v], ci[mt][nt][v]});
  __syncthreads();
#pragma unroll
  for (int e = 0; e < 8; e++) {
    const int c = wk * 8 + e, col = n0 + c;
    cdl s{0.0, 0.0};
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const cdl z = lds_c(sm + q * 32 * 33 + c * 33 + lane);
      s.r += z.r;
      s.i += z.i;
    }
    if (m0 + lane < M && col < N) C[(size_t)col * ldc + m0 + lane] = cdl{x[e].r - s.r, x[e].i - s.i};
  }
}
__global__ void __launch_bounds__(128) k_zgemm_small(int M, int N, int K, const cdl *__restrict__ A, size_t lda,
                                                      const cdl *__restrict__ B, size_t ldb, cdl *C, size_t ldc) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pdl_enter();
  zgemm_small_tile((cdl *)smem_raw, blockIdx.x * 32, blockIdx.y * 32, M, N, K, A, lda, B, ldb, C, ldc);
}
// The parts of C that the INT8 path leaves out: 128 x 64 tiles with a flag (tile (tm, tn)
// at tn * ntm + tm), eight 32 x 32 tiles each, so that the CTAs share few of them evenly
// (a CTA per 128 x 64 tile: one of K = 2,048 takes 0.54 ms).  With no flag 3 us.
#define ZF_MAX 2048              // flags of one launch at most
__global__ void __launch_bounds__(128) k_zgemm_flagged(int M, int N, int K, const cdl *__restrict__ A, size_t lda,
                                                        const cdl *__restrict__ B, size_t ldb, cdl *C, size_t ldc,
                                                        const unsigned char *flag, int ntm, int ntiles) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ unsigned short list[ZF_MAX];
  __shared__ int wsum[4];
  pdl_enter();
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  int n = 0, total = 0;
  for (int i = 0; i < ZF_MAX / 128; i++) {
    const int t = tid * (ZF_MAX / 128) + i;
    n += t < ntiles && flag[t] != 0;
  }
  if (!__syncthreads_or(n)) return;
  int x = n;
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) wsum[wid] = x;
  __syncthreads();
  x -= n;
  for (int w = 0; w < 4; w++) {
    if (w < wid) x += wsum[w];
    total += wsum[w];
  }
  for (int i = 0; i < ZF_MAX / 128; i++) {
    const int t = tid * (ZF_MAX / 128) + i;
    if (t < ntiles && flag[t]) list[x++] = (unsigned short)t;
  }
  for (int u = blockIdx.x; u < 8 * total; u += gridDim.x) {
    __syncthreads();
    const int t = list[u >> 3], m0 = t % ntm * 128 + (u & 3) * 32, n0 = t / ntm * 64 + ((u >> 2) & 1) * 32;
    if (m0 < M && n0 < N) zgemm_small_tile((cdl *)smem_raw, m0, n0, M, N, K, A, lda, B, ldb, C, ldc);
  }
}
static int zgemm_small(int M, int N, int K, const cdl *A, size_t lda, const cdl *B, size_t ldb, cdl *C, size_t ldc) {
  static bool attr = false;
  if (!attr) {
    BG_CUDA_TRY(cudaFuncSetAttribute(k_zgemm_small, cudaFuncAttributeMaxDynamicSharedMemorySize, ZS_SMEM));
    attr = true;
  }
  BG_CUDA_TRY(pdl_launch(k_zgemm_small, dim3((M + 31) / 32, (N + 31) / 32), 128, ZS_SMEM, M, N, K, A, lda, B, ldb, C, ldc));
  BG_LAUNCHED();
  return BG_OK;
}

// CTA tile of the complex128 GEMM, chosen at run time (the batching form's
// autotuner times them per size class): 0 = 64 x 64, 1 = 128 x 64,
// 2 = 64 x 128 complex outputs; warps always own 32 x 32.
static int zg_tile = 0;
void lu_set_gemm_tile(int t) { zg_tile = (t >= 0 && t <= 2) ? t : 0; }
int lu_get_gemm_tile() { return zg_tile; }

template <int BM, int BN>
static int zgemm_launch(int M, int N, int K, const cdl *A, size_t lda, const cdl *B, size_t ldb, cdl *C, size_t ldc) {
  using Cfg = GemmCfg<BM, BN, 16, 3>;
  auto kern = k_zgemm_sub<BM, BN, 16, 3>;
  static bool attr = false;
  if (!attr) {
    BG_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM));
    attr = true;
  }
  dim3 grid((M + BM - 1) / BM, (N + BN - 1) / BN);
  if (grid.y > 65535) { set_error("zgemm: N too large"); return BG_ERR_ARG; }
  BG_CUDA_TRY(pdl_launch(kern, grid, Cfg::THREADS, Cfg::SMEM, M, N, K, A, lda, B, ldb, C, ldc));
  BG_LAUNCHED();
  return BG_OK;
}
// the tiles with a flag (gemm_i8.cu: at most 4,096 x 4,096)
int zgemm_flagged(int M, int N, int K, const void *A, size_t lda, const void *B, size_t ldb, void *C, size_t ldc,
                  const unsigned char *flag) {
  static bool attr = false;
  if (!attr) {
    BG_CUDA_TRY(cudaFuncSetAttribute(k_zgemm_flagged, cudaFuncAttributeMaxDynamicSharedMemorySize, ZS_SMEM));
    attr = true;
  }
  const int ntm = (M + 127) / 128, ntiles = ntm * ((N + 63) / 64);
  if (ntiles > ZF_MAX) { set_error("zgemm: too many tiles"); return BG_ERR_ARG; }
  BG_CUDA_TRY(pdl_launch(k_zgemm_flagged, dim3(std::min(8 * ntiles, 2 * 148)), 128, ZS_SMEM, M, N, K, (const cdl *)A, lda,
                         (const cdl *)B, ldb, (cdl *)C, ldc, flag, ntm, ntiles));
  BG_LAUNCHED();
  return BG_OK;
}

// scratch of the INT8 path, set around the calls that may take it
struct I8Scratch {
  void *p;
  size_t bytes;
  int *err;
};
static thread_local I8Scratch *t_i8 = nullptr;
// Which products go there, from measured times in us: 128 x 64 tiles in waves of
// 148 at 0.117 us per column of K and 8.9 us for the two combinations, 36 us of
// launches and of the guard, exponents and splitting at 96 bytes per element of A and B and
// 5 TB/s; the FP64 tiles at 28 TFLOP/s.  Measured INT8 / FP64, calls one by one:
// 2048 x 512 x 512 140 / 157 us, 1350 x 672 x 672 162 / 203, 4096 x 4096 x 128
// 443 / 641, 1024^3 210 / 304, 9936 x 9936 x 1024 12.0 / 24.9 ms; 2048 x 1024 x 128
// 113 / 89 us.
static bool i8_takes(int M, int N, int K) {
  if (M <= 0 || N <= 0 || K <= 0) return false;
  const double tiles = std::ceil((double)M / 128) * std::ceil((double)N / 64);
  const double split = 36.0 + ((double)M + N) * K * (96 / 5e6);
  const double i8 = std::ceil(tiles / 148) * (0.117 * K + 8.9) + split, fp64 = 8.0 * M * (double)N * K / 28e6;
  return i8 < 0.95 * fp64;
}

static int zgemm_sub(int M, int N, int K, const cdl *A, size_t lda, const cdl *B, size_t ldb, cdl *C, size_t ldc) {
  if (M <= 0 || N <= 0 || K <= 0) return BG_OK;
  prof_start(PROF_GEMM);
  if (t_i8 && i8_takes(M, N, K) && zgemm_i8_bytes(M, N, K) <= t_i8->bytes) {
    int st = zgemm_i8(M, N, K, A, lda, B, ldb, C, ldc, t_i8->p, t_i8->bytes, t_i8->err);
    prof_stop(PROF_GEMM, 8.0 * M * (double)N * K);
    return st;
  }
  // few 64 x 64 tiles leave SMs without work (both sides measured, see k_zgemm_small)
  const long tiles = (long)((M + 63) / 64) * ((N + 63) / 64);
  int st = tiles <= ZG_SMALL ? zgemm_small(M, N, K, A, lda, B, ldb, C, ldc)
         : zg_tile == 1 ? zgemm_launch<128, 64>(M, N, K, A, lda, B, ldb, C, ldc)
         : zg_tile == 2 ? zgemm_launch<64, 128>(M, N, K, A, lda, B, ldb, C, ldc)
                        : zgemm_launch<64, 64>(M, N, K, A, lda, B, ldb, C, ldc);
  prof_stop(PROF_GEMM, 8.0 * M * (double)N * K);
  return st;
}

// a - l u with one rounding of the size of a per part (two fused operations
// on a would round twice; over a factorisation that is 1.5 times the error)
template <class C>
__device__ __forceinline__ C cfms(C a, C l, C u) {
  return C{a.r - fma(l.r, u.r, -(l.i * u.i)), a.i - fma(l.r, u.i, l.i * u.r)};
}
// s + a b
template <class C>
__device__ __forceinline__ C cmac(C s, C a, C b) {
  return C{fma(a.r, b.r, fma(-a.i, b.i, s.r)), fma(a.r, b.i, fma(a.i, b.r, s.i))};
}
template <class C>
__device__ __forceinline__ C cshfl(C v, int src) {
  return C{__shfl_sync(0xffffffffu, v.r, src), __shfl_sync(0xffffffffu, v.i, src)};
}

// =========================================================================
// leaf triangular solves (n <= 128 rows).  The triangle is staged in shared
// memory once per CTA, as the 32 x 32 blocks on and below (above) the
// diagonal, column-major; a warp solves CPW right-hand-side columns, lane l
// holding rows l, l + 32, l + 64, l + 96 of each in registers.  Step i
// broadcasts the solved entry of every column with shuffles and updates all
// later rows, those of the following blocks included, so the off-diagonal
// products need no further pass where a 64-row leaf left them to GEMM launches
// of 64 rows.  TRSM class of one factorisation: 5.2 -> 1.5 ms at N = 4,092,
// 41 -> 23 ms at N = 19,872 (complex64 32 -> 13 ms).  CPW is the smallest of
// 1, 2, 4 with which all CTAs run at once.
// =========================================================================
#define TRS_WARPS 8
#define TRS_MAX 128
template <class C>
constexpr int trsm_smem() { return 10 * 32 * 32 * (int)sizeof(C) + TRS_MAX * (int)sizeof(C); }
// block (br, bc) of the staged triangle: lower br >= bc, upper br <= bc
__device__ __forceinline__ int trs_block(int br, int bc, bool upper) {
  const int hi = upper ? bc : br, lo = upper ? br : bc;
  return (hi * (hi + 1) / 2 + lo) * 1024;
}
template <class C, int CPW, bool UPPER>
__global__ void __launch_bounds__(TRS_WARPS * 32) k_trsm_leaf(int n, int m, const C *T, size_t ldt, C *B, size_t ldb) {
  pdl_enter();
  typedef typename CxT<C>::R R;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C *Ts = (C *)smem_raw;
  C *dinv = Ts + 10 * 1024;      // upper: conj(u) / |u|^2 of the diagonal
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nb = (n + 31) / 32;
  const int cbase = (blockIdx.x * TRS_WARPS + warp) * CPW;
  C b[4][CPW];
#pragma unroll
  for (int q = 0; q < 4; q++)
#pragma unroll
    for (int j = 0; j < CPW; j++) {
      const int r = 32 * q + lane, col = cbase + j;
      b[q][j] = (r < n && col < m) ? B[(size_t)col * ldb + r] : C{0, 0};
    }
  // one column of one block per warp and copy, all of them in flight together
  for (int br = 0; br < nb; br++)
    for (int bc = UPPER ? br : 0; bc < (UPPER ? nb : br + 1); bc++) {
      C *dst = Ts + trs_block(br, bc, UPPER);
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const int r = 32 * br + lane, c = 32 * bc + warp + TRS_WARPS * u;
        const bool ok = r < n && c < n;
        cp_entry(dst + (warp + TRS_WARPS * u) * 32 + lane, ok ? T + (size_t)c * ldt + r : T, ok);
      }
    }
  cp_commit();
  if (UPPER && tid < n) {
    const C u = T[(size_t)tid * ldt + tid];
    const R d = u.r * u.r + u.i * u.i;
    dinv[tid] = C{u.r / d, -u.i / d};
  }
  cp_wait<0>();
  __syncthreads();
  if (cbase >= m) return;
  if (!UPPER) {
#pragma unroll
    for (int q = 0; q < 4; q++) {
      if (q >= nb) break;
      const int ni = min(32, n - 32 * q);
      const C *t0 = Ts + trs_block(q, q, false) + lane;
      C sum[4][CPW];       // products for the following blocks, subtracted once
#pragma unroll
      for (int s = 0; s < 4; s++)
#pragma unroll
        for (int j = 0; j < CPW; j++) sum[s][j] = C{0, 0};
#pragma unroll 4
      for (int i = 0; i < ni; i++) {
        C x[CPW];
#pragma unroll
        for (int j = 0; j < CPW; j++) x[j] = cshfl(b[q][j], i);
        const C l0 = lane > i ? lds_c(t0 + i * 32) : C{0, 0};
#pragma unroll
        for (int j = 0; j < CPW; j++) b[q][j] = cfms(b[q][j], l0, x[j]);
#pragma unroll
        for (int s = q + 1; s < 4; s++)
          if (s < nb) {
            const C l = lds_c(Ts + trs_block(s, q, false) + i * 32 + lane);
#pragma unroll
            for (int j = 0; j < CPW; j++) sum[s][j] = cmac(sum[s][j], l, x[j]);
          }
      }
#pragma unroll
      for (int s = q + 1; s < 4; s++)
#pragma unroll
        for (int j = 0; j < CPW; j++) b[s][j] = C{b[s][j].r - sum[s][j].r, b[s][j].i - sum[s][j].i};
    }
  } else {
#pragma unroll
    for (int q = 3; q >= 0; q--) {
      if (q >= nb) continue;
      const int ni = min(32, n - 32 * q);
      const C *t0 = Ts + trs_block(q, q, true) + lane;
      C sum[4][CPW];
#pragma unroll
      for (int s = 0; s < 4; s++)
#pragma unroll
        for (int j = 0; j < CPW; j++) sum[s][j] = C{0, 0};
#pragma unroll 4
      for (int i = ni - 1; i >= 0; i--) {
        const C iu = lds_c(dinv + 32 * q + i);
        C x[CPW];
#pragma unroll
        for (int j = 0; j < CPW; j++) {
          const C v = cshfl(b[q][j], i);
          x[j] = C{v.r * iu.r - v.i * iu.i, v.r * iu.i + v.i * iu.r};
          if (lane == i) b[q][j] = x[j];
        }
        const C l0 = lane < i ? lds_c(t0 + i * 32) : C{0, 0};
#pragma unroll
        for (int j = 0; j < CPW; j++) b[q][j] = cfms(b[q][j], l0, x[j]);
#pragma unroll
        for (int s = 0; s < q; s++) {
          const C l = lds_c(Ts + trs_block(s, q, true) + i * 32 + lane);
#pragma unroll
          for (int j = 0; j < CPW; j++) sum[s][j] = cmac(sum[s][j], l, x[j]);
        }
      }
#pragma unroll
      for (int s = 0; s < q; s++)
#pragma unroll
        for (int j = 0; j < CPW; j++) b[s][j] = C{b[s][j].r - sum[s][j].r, b[s][j].i - sum[s][j].i};
    }
  }
#pragma unroll
  for (int q = 0; q < 4; q++)
#pragma unroll
    for (int j = 0; j < CPW; j++) {
      const int r = 32 * q + lane, col = cbase + j;
      if (r < n && col < m) B[(size_t)col * ldb + r] = b[q][j];
    }
}

template <class C, int CPW, bool UPPER>
static int trsm_launch(int n, int m, const C *T, size_t ldt, C *B, size_t ldb) {
  static bool attr = false;
  if (!attr) {
    BG_CUDA_TRY(cudaFuncSetAttribute(k_trsm_leaf<C, CPW, UPPER>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     trsm_smem<C>()));
    attr = true;
  }
  const int cols = TRS_WARPS * CPW;
  prof_start(PROF_TRSM);
  BG_CUDA_TRY(pdl_launch(k_trsm_leaf<C, CPW, UPPER>, dim3((m + cols - 1) / cols), TRS_WARPS * 32, trsm_smem<C>(), n, m, T,
                         ldt, B, ldb));
  BG_LAUNCHED();
  prof_stop(PROF_TRSM, 4.0 * n * (double)n * m);
  return BG_OK;
}

// small-N complex64 GEMM (C -= A B, N <= 16): one thread per row, used where
// a tensor-core tile would be mostly padding (few right-hand sides)
__global__ void k_cgemm_small(int M, int N, int K, const cfl *A, size_t lda, const cfl *B, size_t ldb, cfl *Cm,
                              size_t ldc) {
  int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= M) return;
  float ar[16], ai[16];
  for (int n = 0; n < N; n++) ar[n] = ai[n] = 0.f;
  for (int k = 0; k < K; k++) {
    cfl a = A[(size_t)k * lda + m];
#pragma unroll 4
    for (int n = 0; n < N; n++) {
      cfl b = B[(size_t)n * ldb + k];
      ar[n] += a.r * b.r - a.i * b.i;
      ai[n] += a.r * b.i + a.i * b.r;
    }
  }
  for (int n = 0; n < N; n++) {
    cfl *p = Cm + (size_t)n * ldc + m;
    p->r -= ar[n];
    p->i -= ai[n];
  }
}

// per-matrix scratch for the tensor-core path
struct TcScratch {
  float *At = nullptr;
  size_t at_floats = 0;
  int *err = nullptr;
};
static thread_local TcScratch *t_tc = nullptr;
#define TC_MCHUNK 8192

static int gemm_sub(int M, int N, int K, const cdl *A, size_t lda, const cdl *B, size_t ldb, cdl *C, size_t ldc) {
  return zgemm_sub(M, N, K, A, lda, B, ldb, C, ldc);
}
static int gemm_sub(int M, int N, int K, const cfl *A, size_t lda, const cfl *B, size_t ldb, cfl *C, size_t ldc) {
  if (M <= 0 || N <= 0 || K <= 0) return BG_OK;
  if (N <= 16 || !t_tc) {
    if (N > 16) { set_error("complex64 GEMM needs the tensor-core scratch"); return BG_ERR_STATE; }
    k_cgemm_small<<<(M + 127) / 128, 128, 0, stream()>>>(M, N, K, A, lda, B, ldb, C, ldc);
    BG_LAUNCHED();
    return BG_OK;
  }
  size_t lda2 = ((size_t)2 * K + 31) / 32 * 32;
  size_t cap = std::min<size_t>(t_tc->at_floats / (2 * lda2), TC_MCHUNK);
  int mch = (int)std::min<size_t>((size_t)M, cap);
  if (mch < M) mch = mch / 64 * 64;   // chunked: whole 64-row tiles per chunk
  if (mch <= 0) { set_error("tensor-core scratch too small"); return BG_ERR_STATE; }
  for (int m0 = 0; m0 < M; m0 += mch) {
    int mm = std::min(mch, M - m0);
    int st = cgemm_sub_tf32(mm, N, K, A + m0, lda, B, ldb, C + m0, ldc, t_tc->At, t_tc->err);
    if (st) return st;
  }
  return BG_OK;
}

// X = L^{-1} B (unit lower, upper=0) or U^{-1} B (upper=1), L/U n x n at T
template <class C>
static int trsm(int n, int m, const C *T, size_t ldt, C *B, size_t ldb, int upper) {
  if (n <= 0 || m <= 0) return BG_OK;
  if (n <= TRS_MAX) {
    const int cap = 148 * (sizeof(C) == 16 ? 1 : 2);      // CTAs the shared memory lets run at once
    const int cpw = m <= cap * TRS_WARPS ? 1 : m <= 2 * cap * TRS_WARPS ? 2 : 4;
    if (upper)
      return cpw == 4   ? trsm_launch<C, 4, true>(n, m, T, ldt, B, ldb)
             : cpw == 2 ? trsm_launch<C, 2, true>(n, m, T, ldt, B, ldb)
                        : trsm_launch<C, 1, true>(n, m, T, ldt, B, ldb);
    return cpw == 4   ? trsm_launch<C, 4, false>(n, m, T, ldt, B, ldb)
           : cpw == 2 ? trsm_launch<C, 2, false>(n, m, T, ldt, B, ldb)
                      : trsm_launch<C, 1, false>(n, m, T, ldt, B, ldb);
  }
  int n1 = (n / 2 + TRS_MAX - 1) / TRS_MAX * TRS_MAX;   // multiples of the leaf (n > TRS_MAX, so n1 < n)
  int n2 = n - n1;
  int st;
  if (!upper) {
    if ((st = trsm(n1, m, T, ldt, B, ldb, 0))) return st;
    if ((st = gemm_sub(n2, m, n1, T + n1, ldt, B, ldb, B + n1, ldb))) return st;
    return trsm(n2, m, T + n1 + (size_t)n1 * ldt, ldt, B + n1, ldb, 0);
  }
  if ((st = trsm(n2, m, T + n1 + (size_t)n1 * ldt, ldt, B + n1, ldb, 1))) return st;
  if ((st = gemm_sub(n1, m, n2, T + (size_t)n1 * ldt, ldt, B + n1, ldb, B, ldb))) return st;
  return trsm(n1, m, T, ldt, B, ldb, 1);
}

// =========================================================================
// cooperative panel factorisation of A[k0:Nr, k0:k0+w] (w <= 32) for panels too
// tall for the register form below (more than 37,888 rows).  Each CTA
// holds a slice of rows_per rows in shared memory, column-major (column c at
// S + c * rows_per): the pivot scan and the rank-1 update walk a column with
// consecutive threads on consecutive rows, free of bank conflicts.  One grid
// barrier per column exchanges the CTAs' pivot candidates.
// =========================================================================
static constexpr int panel_max_grid = 148;   // CTAs of a grid-wide panel at most
template <class C>
struct PanelArgs {
  C *A;
  size_t ld;
  int Nr;          // number of rows of the full matrix
  int k0, w;
  int rows_per;    // rows owned per CTA
  int *ipiv;       // global, 1-based
  int *info;       // device int (0 = ok)
  double *cval;    // [2][grid] candidate |re|+|im|
  int *cidx;       // [2][grid] candidate row
  C *crow;         // [2][grid][32] candidate row values
  C *jrow;         // [2][32] values of row k0+j before the swap
  unsigned long long *slots;   // k_panel_rf over the grid: tagged candidate messages
};

__device__ __forceinline__ bool better(double v, int i, double bv, int bi) {
  return v > bv || (v == bv && i < bi);
}

template <class C>
__global__ void __launch_bounds__(256) k_panel(PanelArgs<C> P) {
  typedef typename CxT<C>::R R;
  cg::grid_group grid = cg::this_grid();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C *S = (C *)smem_raw;                     // [w][rows_per]: column c at S + c * rows_per
  __shared__ double rv[8];
  __shared__ int ri[8];
  __shared__ int s_piv;
  __shared__ C prow[32];
  const int w = P.w, G = gridDim.x, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int r0 = P.k0 + blockIdx.x * P.rows_per;
  const int r1 = min(P.Nr, r0 + P.rows_per);
  const int nr = max(0, r1 - r0), lds = P.rows_per;
  // slice staged with eight loads per thread in flight
  for (int e0 = 0; e0 < nr * w; e0 += 8 * 256) {
    C v[8];
#pragma unroll
    for (int u = 0; u < 8; u++) {
      const int e = e0 + u * 256 + tid;
      v[u] = e < nr * w ? P.A[(size_t)(P.k0 + e / nr) * P.ld + r0 + e % nr] : C{0, 0};
    }
#pragma unroll
    for (int u = 0; u < 8; u++) {
      const int e = e0 + u * 256 + tid;
      if (e < nr * w) S[(e / nr) * lds + e % nr] = v[u];
    }
  }
  __syncthreads();
  for (int j = 0; j < w; j++) {
    const int gj = P.k0 + j, buf = j & 1;
    // 1. local pivot candidate (i[cz]amax: max |re|+|im|, first index on ties)
    double bv = -1.0;
    int bi = 0x7fffffff;
    for (int r = tid; r < nr; r += 256) {
      int gr = r0 + r;
      if (gr < gj) continue;
      C v = S[j * lds + r];
      double a = (double)(fabs(v.r) + fabs(v.i));
      if (better(a, gr, bv, bi)) { bv = a; bi = gr; }
    }
    for (int o = 16; o > 0; o >>= 1) {
      double ov = __shfl_xor_sync(0xffffffffu, bv, o);
      int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (better(ov, oi, bv, bi)) { bv = ov; bi = oi; }
    }
    if (lane == 0) { rv[wid] = bv; ri[wid] = bi; }
    __syncthreads();
    if (tid == 0) {
      for (int k = 1; k < 8; k++)
        if (better(rv[k], ri[k], rv[0], ri[0])) { rv[0] = rv[k]; ri[0] = ri[k]; }
      P.cval[buf * G + blockIdx.x] = rv[0];
      P.cidx[buf * G + blockIdx.x] = ri[0];
    }
    __syncthreads();
    int myc = ri[0];
    if (rv[0] >= 0.0 && tid < w) P.crow[((size_t)buf * G + blockIdx.x) * 32 + tid] = S[tid * lds + myc - r0];
    if (gj >= r0 && gj < r1 && tid < w) P.jrow[buf * 32 + tid] = S[tid * lds + gj - r0];
    grid.sync();
    // 2. global pivot
    if (tid < 32) {
      double v = -1.0;
      int i = 0x7fffffff, b = 0;
      for (int k = lane; k < G; k += 32) {
        double cv = P.cval[buf * G + k];
        int ci = P.cidx[buf * G + k];
        if (better(cv, ci, v, i)) { v = cv; i = ci; b = k; }
      }
      for (int o = 16; o > 0; o >>= 1) {
        double ov = __shfl_xor_sync(0xffffffffu, v, o);
        int oi = __shfl_xor_sync(0xffffffffu, i, o);
        int ob = __shfl_xor_sync(0xffffffffu, b, o);
        if (better(ov, oi, v, i)) { v = ov; i = oi; b = ob; }
      }
      // a column of NaNs has no candidate and takes its own row
      const bool none = i == 0x7fffffff;
      if (lane < w) prow[lane] = none ? P.jrow[buf * 32 + lane] : P.crow[((size_t)buf * G + b) * 32 + lane];
      if (lane == 0) s_piv = none ? gj : i;
    }
    __syncthreads();
    const int piv = s_piv;
    if (blockIdx.x == 0 && tid == 0) P.ipiv[gj] = piv + 1;
    // 3. swap rows gj and piv inside the panel
    if (piv != gj) {
      if (piv >= r0 && piv < r1 && tid < w) S[tid * lds + piv - r0] = P.jrow[buf * 32 + tid];
      if (gj >= r0 && gj < r1 && tid < w) S[tid * lds + gj - r0] = prow[tid];
    }
    __syncthreads();
    // 4. scale the column below the pivot and update the rest of the panel
    C p = prow[j];
    R d = p.r * p.r + p.i * p.i;
    if (d == (R)0) {
      if (blockIdx.x == 0 && tid == 0) atomicCAS(P.info, 0, gj + 1);
    } else {
      C inv{p.r / d, -p.i / d};
      int ncol = w - j - 1;
      for (int r = tid; r < nr; r += 256) {
        int gr = r0 + r;
        if (gr <= gj) continue;
        C v = S[j * lds + r];
        C l{v.r * inv.r - v.i * inv.i, v.r * inv.i + v.i * inv.r};
        S[j * lds + r] = l;
        for (int c = 1; c <= ncol; c++) {
          C u = prow[j + c];
          C &t = S[(j + c) * lds + r];
          t.r -= l.r * u.r - l.i * u.i;
          t.i -= l.r * u.i + l.i * u.r;
        }
      }
    }
    __syncthreads();
  }
  for (int e = tid; e < nr * w; e += 256) {
    const int r = e % nr, c = e / nr;
    P.A[(size_t)(P.k0 + c) * P.ld + r0 + r] = S[c * lds + r];
  }
}

template <class C>
__device__ __forceinline__ C ldcg_c(const C *p);
template <>
__device__ __forceinline__ cdl ldcg_c<cdl>(const cdl *p) {
  double2 v = __ldcg((const double2 *)p);
  return cdl{v.x, v.y};
}
template <>
__device__ __forceinline__ cfl ldcg_c<cfl>(const cfl *p) {
  float2 v = __ldcg((const float2 *)p);
  return cfl{v.x, v.y};
}

// -------------------------------------------------------------------------
// The panel with its rows in registers, on one cluster.  A thread owns one row
// of the panel in registers, so the rank-1 update reads and writes registers
// only; finished columns go to shared memory (Ls[c][row]), from where the whole
// slice is written out once.  Columns are updated in fixed groups of eight
// that end past column j: the finished columns among them compute on
// leftovers that nothing reads.  The
// shared-memory form above moves 32 bytes of shared memory per updated entry
// and is bound by that and by its barriers: 3.3-3.9 us a column.
//
// One column costs two block barriers and one exchange.  Every warp finds its
// pivot candidate with redux on the bits of |re| + |im| (non-negative, so they
// order as integers) and the candidate's thread copies its row to shared
// memory; after the barrier every warp knows the CTA's candidate, and warp q
// pushes its row to CTAs q, q + warps, ... with st.async, which counts its
// bytes on the receiver's mbarrier.  An extra warp pushes the candidate's key
// and the reciprocal of its pivot.  When the mbarrier completes, a CTA has
// every candidate in its own shared memory: no remote loads, no cluster
// barrier.  The other row of the interchange, k0 + j, is in every CTA as
// well: the extra warp keeps a copy of the w top rows and updates it like its
// own.  The next column is updated first, so that the search for its pivot
// runs while the other columns are updated.  What bounds a column is the
// number of instructions a warp issues between two exchanges (8 cycles each
// with two or three warps per scheduler): registers keep their columns (moving
// them down by one place per step cost two moves per register), offsets are
// constants of the unrolled code, column j + 1 is picked by a jump, and the
// division is left to the extra warp.
// Two buffers by column parity: a CTA sends column j + 2 after it has received
// every candidate of column j + 1, which each CTA sends only after all its
// warps have finished with column j.  Waits are bounded; one that runs out is
// reported through info, and the CTA goes on so that the cluster ends.
//
// GRID: panels taller than one cluster.  The same CTAs over the whole grid (a
// cooperative launch), one row a thread, and the exchange through L2: a CTA
// stores its candidate as 64-bit words that carry a 32-bit tag (launch count
// and column) beside 32 bits of data, so no fence and no flag orders them; one
// warp per CTA polls all keys, finds the winner and fetches its row and
// reciprocal, which arrive by the same tags.  Two block barriers a column
// instead of a grid barrier; three trips through L2 (keys out, keys in, row in)
// set the time: panels of one factorisation at N = 19,872 77 -> 71 ms, complex64
// 64 -> 53 ms.
//
// Pivot choice (first index on ties), interchanges and arithmetic are those of
// k_panel.  A NaN never wins; a column of NaNs takes its own row.
// -------------------------------------------------------------------------
#define PRF_MAXCL 16
#define PRF_SPIN (1 << 17)
// Rows per CTA at most: T0 while that is enough (256 / 512 threads with the
// extra warp, so that a thread may use 255 / 128 registers and the eight
// loads of a group are in flight together), T1 for the tallest panels
template <class C> struct PrfCfg;
template <> struct PrfCfg<cdl> { static constexpr int T0 = 224, T1 = 256; };   // 32 columns = 128 registers a row
template <> struct PrfCfg<cfl> { static constexpr int T0 = 480, T1 = 512; };

template <class C>
struct alignas(16) PrfMsg {        // st.async writes 16 bytes at a time
  C row[32];
  unsigned long long key;
  long long idx;
  C inv;                            // reciprocal of the candidate
};
template <class C>
struct alignas(16) PrfSmem {
  static constexpr int NW = PrfCfg<C>::T1 / 32;
  PrfMsg<C> msg[2][PRF_MAXCL];
  alignas(16) C wrow[2][NW][32];    // candidate rows of the warps, columns >= j
  alignas(16) C jrow[2][32];                    // row k0 + j before the interchange, columns >= j
  alignas(16) C Lt[32][32];                // Lt[c][i]: finished columns of the copy of row k0 + i
  unsigned long long wkey[2][NW];
  int widx[2][NW];
  unsigned long long bar[2];
};
__device__ __forceinline__ unsigned long long pivot_key(cdl v) {
  const double a = fabs(v.r) + fabs(v.i);
  return a == a ? (unsigned long long)__double_as_longlong(a) : 0ull;
}
__device__ __forceinline__ unsigned long long pivot_key(cfl v) {
  const float a = fabsf(v.r) + fabsf(v.i);
  return a == a ? (unsigned long long)__float_as_uint(a) << 32 : 0ull;
}
// lane of the first maximum of key over the lanes with ok (-1: none), key of
// it; mh: the warp's maximum of the high words (of the lanes with ok, else 0).
// Equal high words are rare, so the low words are compared only then.
__device__ __forceinline__ unsigned key_hi(unsigned long long key, bool ok) { return ok ? (unsigned)(key >> 32) : 0u; }
template <class C>
__device__ __forceinline__ int warp_first_max(unsigned long long &key, bool ok, unsigned mh) {
  bool c = ok && (unsigned)(key >> 32) == mh;
  unsigned b = __ballot_sync(0xffffffffu, c);
  if (sizeof(C) == 16 && (b & (b - 1))) {
    const unsigned lo = c ? (unsigned)key : 0u, ml = __reduce_max_sync(0xffffffffu, lo);
    c = c && lo == ml;
    b = __ballot_sync(0xffffffffu, c);
  }
  const int src = b ? __ffs(b) - 1 : -1;
  key = __shfl_sync(0xffffffffu, key, src < 0 ? 0 : src);
  return src;
}
__device__ __forceinline__ unsigned smem_addr(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned map_cta(unsigned a, int rank) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
__device__ __forceinline__ void st_async16(unsigned dst, unsigned long long x, unsigned long long y, unsigned bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];" ::"r"(dst),
               "l"(x), "l"(y), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void st_async8(unsigned dst, unsigned long long x, unsigned bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(dst), "l"(x), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void push_c(unsigned dst, cdl v, unsigned bar) {
  st_async16(dst, (unsigned long long)__double_as_longlong(v.r), (unsigned long long)__double_as_longlong(v.i), bar);
}
__device__ __forceinline__ void push_c(unsigned dst, cfl v, unsigned bar) {
  st_async8(dst, (unsigned long long)__float_as_uint(v.i) << 32 | __float_as_uint(v.r), bar);
}

// tagged words: 32 bits of data each.  A complex entry takes 4 (complex128) or
// 2 (complex64) of them.
#define PRG_STRIDE 136            // words per CTA and buffer: key (3, pad to 4), inv (4), row (32 x 4)
template <class C> struct PrgWords { static constexpr int N = sizeof(C) / 4; };
__device__ __forceinline__ void prg_split(cdl v, unsigned (&x)[4]) {
  x[0] = (unsigned)__double2loint(v.r); x[1] = (unsigned)__double2hiint(v.r);
  x[2] = (unsigned)__double2loint(v.i); x[3] = (unsigned)__double2hiint(v.i);
}
__device__ __forceinline__ void prg_split(cfl v, unsigned (&x)[2]) { x[0] = __float_as_uint(v.r); x[1] = __float_as_uint(v.i); }
__device__ __forceinline__ void prg_join(const unsigned (&x)[4], cdl &v) {
  v = cdl{__hiloint2double((int)x[1], (int)x[0]), __hiloint2double((int)x[3], (int)x[2])};
}
__device__ __forceinline__ void prg_join(const unsigned (&x)[2], cfl &v) { v = cfl{__uint_as_float(x[0]), __uint_as_float(x[1])}; }
__device__ __forceinline__ void st_word(unsigned long long *p, unsigned tag, unsigned v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"((unsigned long long)tag << 32 | v) : "memory");
}
__device__ __forceinline__ unsigned long long ld_word(const unsigned long long *p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
template <class C>
__device__ __forceinline__ void prg_put(unsigned long long *p, unsigned tag, C v) {
  unsigned x[PrgWords<C>::N];
  prg_split(v, x);
#pragma unroll
  for (int k = 0; k < PrgWords<C>::N; k++) st_word(p + k, tag, x[k]);
}
// one entry once its tags have arrived; false when the wait runs out
template <class C>
__device__ __forceinline__ bool prg_get(const unsigned long long *p, unsigned tag, int limit, C &v) {
  unsigned x[PrgWords<C>::N];
  for (int it = 0; it < limit; it++) {
    bool ok = true;
#pragma unroll
    for (int k = 0; k < PrgWords<C>::N; k++) {
      const unsigned long long q = ld_word(p + k);
      ok = ok && (unsigned)(q >> 32) == tag;
      x[k] = (unsigned)q;
    }
    if (ok) {
      prg_join(x, v);
      return true;
    }
  }
  v = C{0, 0};
  return false;
}

template <class C, int TMAX, bool GRID>
__global__ void __launch_bounds__(TMAX + 32) k_panel_rf(PanelArgs<C> P) {
  typedef typename CxT<C>::R R;
  constexpr int T = TMAX + 1;      // column stride of Ls: a row's columns fall into different banks
  extern __shared__ __align__(16) unsigned char smem_raw[];
  PrfSmem<C> &S = *reinterpret_cast<PrfSmem<C> *>(smem_raw);
  C *Ls = reinterpret_cast<C *>(smem_raw + sizeof(PrfSmem<C>));   // [32][T]
  cg::cluster_group cl = cg::this_cluster();
  const int w = P.w, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nw = (int)(blockDim.x >> 5) - 1;
  const int rank = GRID ? (int)blockIdx.x : (int)cl.block_rank(), G = GRID ? (int)gridDim.x : (int)cl.num_blocks();
  const int r0 = P.k0 + rank * P.rows_per, nr = max(0, min(P.rows_per, P.Nr - r0));
  const bool top = wid == nw;                      // the copy of the top rows
  const int row = top ? P.k0 + lane : r0 + tid;
  const bool mine = !top && tid < nr, held = mine || (top && lane < w);
  // finished columns of this thread's row: column c at Lrow[c * Lstep]
  C *Lrow = top ? &S.Lt[0][lane] : Ls + tid;
  const int Lstep = top ? 32 : T;
  pdl_enter();
  C a[32];
#pragma unroll
  for (int c = 0; c < 32; c++) a[c] = (held && c < w) ? P.A[(size_t)(P.k0 + c) * P.ld + row] : C{0, 0};
  const unsigned base = smem_addr(&S);
  const unsigned bar0 = smem_addr(&S.bar[0]);
  // GRID: launch count at ctr[0] (the last CTA of a launch raises it), tickets
  // of finished CTAs at ctr[1]
  unsigned long long *ctr = P.slots + 2 * (size_t)panel_max_grid * PRG_STRIDE;
  unsigned tag0 = 0;
  __shared__ int s_piv;
  if (GRID) {
    tag0 = (unsigned)ld_word(ctr) * 64u + 1u;
  } else if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar0) : "memory");
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar0 + 8) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (!GRID) cl.sync();   // barriers of every CTA are ready
  const unsigned bytes = (unsigned)(G * (33 * sizeof(C) + 16));
  int limit = PRF_SPIN;
  // search state of the coming column: this row's entry, its key, the warp's maximum
  C cur = a[0];
  unsigned long long key = pivot_key(cur);
  unsigned mh = __reduce_max_sync(0xffffffffu, key_hi(key, mine));
  for (int j = 0; j < w; j++) {
    const int gj = P.k0 + j, buf = j & 1;
    const unsigned bar = bar0 + 8 * buf;
    if (!GRID && tid == 0)
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
    // 1. candidate of every warp; its row, and row gj from the top copy
    int src = j;
    C *keep = S.jrow[buf];
    if (!top) {
      src = warp_first_max<C>(key, mine && row >= gj, mh);
      if (lane == 0) {
        S.wkey[buf][wid] = key;
        S.widx[buf][wid] = src < 0 ? 0x7fffffff : r0 + wid * 32 + src;
      }
      keep = S.wrow[buf][wid];
    }
    if (lane == src)
#pragma unroll
      for (int c0 = 0; c0 < 32; c0 += 8)
        if (c0 + 7 >= j)
#pragma unroll
          for (int c = c0; c < c0 + 8; c++) sts_c(keep + c, a[c]);
    __syncthreads();
    int b = 0, piv = gj;
    if (GRID) {
      // 2. the CTA's candidate: key and row by the first warp, the reciprocal
      // of its pivot by the extra warp
      const unsigned tag = tag0 + j;
      unsigned long long *slot = P.slots + ((size_t)buf * panel_max_grid + rank) * PRG_STRIDE;
      if (wid == 0 || top) {
        unsigned long long k2 = lane < nw ? S.wkey[buf][lane] : 0ull;
        const int idx = lane < nw ? S.widx[buf][lane] : 0x7fffffff;
        const bool ok = idx != 0x7fffffff;
        const int bw = warp_first_max<C>(k2, ok, __reduce_max_sync(0xffffffffu, key_hi(k2, ok)));
        const int bi = __shfl_sync(0xffffffffu, idx, bw < 0 ? 0 : bw);
        if (top) {
          C iv = C{0, 0};
          if (bw >= 0) {
            const C p = lds_c(&S.wrow[buf][bw][j]);
            const R d = p.r * p.r + p.i * p.i;
            iv = C{p.r / d, -p.i / d};
          }
          if (lane == 0) prg_put(slot + 4, tag, iv);
        } else {
          if (lane < 3) st_word(slot + lane, tag, lane == 0 ? (unsigned)(k2 >> 32) : lane == 1 ? (unsigned)k2 : (unsigned)(bw < 0 ? 0x7fffffff : bi));
          C v = C{0, 0};
          if (bw >= 0 && lane < w) v = lds_c(lane < j ? &Ls[lane * T + (bi - r0)] : &S.wrow[buf][bw][lane]);
          prg_put(slot + 8 + lane * PrgWords<C>::N, tag, v);
        }
      }
      // 3. the first warp polls every key, then fetches the winner's row
      if (wid == 0) {
        unsigned long long bk = 0;
        int bidx = 0x7fffffff;
        // the lane's up to five CTAs together where the registers allow it
        // (complex64: 67 -> 64 us a panel; complex128 keeps 128 registers of rows
        // and spills: 71 -> 92 ms of panels at N = 19,872)
        constexpr int NQ = sizeof(C) == 8 ? (panel_max_grid + 31) / 32 : 1;
        bool fine = true;
        for (int q0 = lane; q0 < G; q0 += 32 * NQ) {
          unsigned long long x[NQ][3];
          bool in = false;
          for (int it = 0; it < limit && !in; it++) {
            in = true;
#pragma unroll
            for (int u = 0; u < NQ; u++) {
              const int q = q0 + 32 * u;
              const unsigned long long *ps = P.slots + ((size_t)buf * panel_max_grid + (q < G ? q : q0)) * PRG_STRIDE;
              x[u][0] = ld_word(ps);
              x[u][1] = ld_word(ps + 1);
              x[u][2] = ld_word(ps + 2);
            }
#pragma unroll
            for (int u = 0; u < NQ; u++)
              in = in && (unsigned)(x[u][0] >> 32) == tag && (unsigned)(x[u][1] >> 32) == tag && (unsigned)(x[u][2] >> 32) == tag;
          }
          fine = fine && in;
#pragma unroll
          for (int u = 0; u < NQ; u++) {
            const unsigned long long k = x[u][0] << 32 | (unsigned)x[u][1];
            const int id = (int)(unsigned)x[u][2];
            // the lane's CTAs come in row order: the first of equal keys stays
            if (in && q0 + 32 * u < G && id != 0x7fffffff && (bidx == 0x7fffffff || k > bk)) { bk = k; bidx = id; }
          }
        }
        const bool has = bidx != 0x7fffffff;
        const unsigned mh2 = __reduce_max_sync(0xffffffffu, has ? (unsigned)(bk >> 32) : 0u);
        bool c = has && (unsigned)(bk >> 32) == mh2;
        const unsigned ml2 = __reduce_max_sync(0xffffffffu, c ? (unsigned)bk : 0u);
        c = c && (unsigned)bk == ml2;
        piv = (int)__reduce_min_sync(0xffffffffu, c ? (unsigned)bidx : 0x7fffffffu);
        if (piv < gj || piv >= P.Nr) piv = gj;
        const int wq = min((piv - P.k0) / P.rows_per, G - 1);
        const unsigned long long *ps = P.slots + ((size_t)buf * panel_max_grid + wq) * PRG_STRIDE;
        C v, iv = C{0, 0};
        fine = prg_get(ps + 8 + lane * PrgWords<C>::N, tag, limit, v) && fine;
        if (lane == 0) fine = prg_get(ps + 4, tag, limit, iv) && fine;
        sts_c(&S.msg[buf][0].row[lane], v);
        if (lane == 0) {
          sts_c(&S.msg[buf][0].inv, iv);
          s_piv = piv;
        }
        if (!fine) { limit = 1; atomicExch(P.info, 0x7fffffff); atomicExch(P.info + 1, 300); }
      }
      __syncthreads();
      piv = s_piv;
    } else {
      // 2. the CTA's candidate, pushed to every CTA: its row by warp q to CTAs
      // q, q + nw, ..., key and reciprocal by the extra warp, lane q to CTA q
      {
        unsigned long long k2 = lane < nw ? S.wkey[buf][lane] : 0ull;
        const int idx = lane < nw ? S.widx[buf][lane] : 0x7fffffff;
        const bool ok = idx != 0x7fffffff;
        const int bw = warp_first_max<C>(k2, ok, __reduce_max_sync(0xffffffffu, key_hi(k2, ok)));
        const unsigned msg = smem_addr(&S.msg[buf][rank]) - base;
        if (top) {
          const int bi = __shfl_sync(0xffffffffu, idx, bw < 0 ? 0 : bw);
          if (lane < G) {
            const unsigned rbase = map_cta(base, lane), rb = rbase + (bar - base);
            st_async16(rbase + msg + 32 * (unsigned)sizeof(C), k2, (unsigned long long)(bw < 0 ? -1ll : (long long)bi), rb);
            C iv = C{0, 0};
            if (bw >= 0) {
              const C p = lds_c(&S.wrow[buf][bw][j]);
              const R d = p.r * p.r + p.i * p.i;
              iv = C{p.r / d, -p.i / d};
            }
            push_c(rbase + msg + 32 * (unsigned)sizeof(C) + 16, iv, rb);
          }
        } else {
          const int bi = __shfl_sync(0xffffffffu, idx, bw < 0 ? 0 : bw);
          C v = C{0, 0};
          if (bw >= 0 && lane < w) v = lds_c(lane < j ? &Ls[lane * T + (bi - r0)] : &S.wrow[buf][bw][lane]);
          const unsigned dst = msg + lane * (unsigned)sizeof(C);
          for (int q = wid; q < G; q += nw) {
            const unsigned rbase = map_cta(base, q);
            push_c(rbase + dst, v, rbase + (bar - base));
          }
        }
      }
      // 3. everyone's candidates
      {
        unsigned done = 0;
        for (int it = 0; it < limit && !done; it++)
          asm volatile(
              "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
              " selp.u32 %0, 1, 0, p;\n}\n"
              : "=r"(done)
              : "r"(bar), "r"((unsigned)((j >> 1) & 1))
              : "memory");
        if (!done) { limit = 1; atomicExch(P.info, 0x7fffffff); atomicExch(P.info + 1, 300); }
      }
      const int ql = lane < G ? lane : 0;
      unsigned long long k3 = S.msg[buf][ql].key;
      const int idx = (int)S.msg[buf][ql].idx;
      const bool ok = lane < G && idx >= 0;
      b = warp_first_max<C>(k3, ok, __reduce_max_sync(0xffffffffu, key_hi(k3, ok)));
      if (b < 0) b = 0;
      piv = __shfl_sync(0xffffffffu, idx, b);
      if (piv < gj || piv >= P.Nr) piv = gj;   // no candidate, or a wait ran out
    }
    const PrfMsg<C> &W = S.msg[buf][b];
    const C p = lds_c(&W.row[j]), pinv = lds_c(&W.inv);
    if (!GRID) __syncthreads();   // every warp has read the rows it pushes (Ls changes below)
    // 4. interchange: row gj is final and goes to Ls (a warp of rank 0); the
    // pivot's place takes over the old row gj
    if (rank == 0) {
      if (tid == 0) P.ipiv[gj] = piv + 1;
      if (wid == nw - 1 && lane < w) sts_c(&Ls[lane * T + j], lds_c(&W.row[lane]));
    }
    if (piv != gj && held && row == piv) {
#pragma unroll
      for (int c0 = 0; c0 < 32; c0 += 8)
        if (c0 + 7 >= j)
#pragma unroll
          for (int c = c0; c < c0 + 8; c++) a[c] = lds_c(&S.jrow[buf][c]);
      cur = lds_c(&S.jrow[buf][j]);
#pragma unroll 8
      for (int c = 0; c < j; c++) sts_c(&Lrow[c * Lstep], lds_c(&S.Lt[c][j]));
    }
    // 5. scale and update
    const R d = p.r * p.r + p.i * p.i;
    const bool zero = d == (R)0, below = held && row > gj;
    C l = cur;
    if (zero) {
      if (rank == 0 && tid == 0) atomicCAS(P.info, 0, gj + 1);
    } else {
      l = C{cur.r * pinv.r - cur.i * pinv.i, cur.r * pinv.i + cur.i * pinv.r};
    }
    if (below) sts_c(&Lrow[j * Lstep], l);
    if (j + 1 == w) break;
    switch (j + 1) {
#define PRF_PICK(c) case c: cur = a[c]; break;
      PRF_PICK(1) PRF_PICK(2) PRF_PICK(3) PRF_PICK(4) PRF_PICK(5) PRF_PICK(6) PRF_PICK(7) PRF_PICK(8) PRF_PICK(9)
      PRF_PICK(10) PRF_PICK(11) PRF_PICK(12) PRF_PICK(13) PRF_PICK(14) PRF_PICK(15) PRF_PICK(16) PRF_PICK(17)
      PRF_PICK(18) PRF_PICK(19) PRF_PICK(20) PRF_PICK(21) PRF_PICK(22) PRF_PICK(23) PRF_PICK(24) PRF_PICK(25)
      PRF_PICK(26) PRF_PICK(27) PRF_PICK(28) PRF_PICK(29) PRF_PICK(30) PRF_PICK(31)
#undef PRF_PICK
    }
    if (!zero) cur = cfms(cur, l, lds_c(&W.row[j + 1]));
    key = pivot_key(cur);
    mh = __reduce_max_sync(0xffffffffu, key_hi(key, mine && row > gj));
    if (!zero) {
#pragma unroll
      for (int c0 = 0; c0 < 32; c0 += 8)
        if (c0 + 7 > j)
#pragma unroll
          for (int c = c0; c < c0 + 8; c++) a[c] = cfms(a[c], l, lds_c(&W.row[c]));
    }
  }
  __syncthreads();
  // rows k0 .. k0 + w - 1 hold U (and the L of their interchanges), written
  // to Ls by step 4; the others hold their L
  if (mine)
    for (int c = 0; c < w; c++) P.A[(size_t)(P.k0 + c) * P.ld + row] = lds_c(&Ls[c * T + tid]);
  if (GRID) {
    // every CTA has read the launch count before any CTA can finish
    if (tid == 0 && atomicAdd(ctr + 1, 1ull) == (unsigned long long)(G - 1)) {
      ctr[1] = 0;
      ctr[0] = ctr[0] + 1;
    }
  } else {
    cl.sync();   // no CTA leaves while messages for it may be in flight
  }
}

// Row interchanges ipiv[k0..k0+w) on the columns [0, ncols) outside
// [skip0, skip1), one warp per column.  The w interchanges are one
// permutation of at most 2 w rows: the w top rows (lane l holds row k0 + l)
// and the pivot rows below them (lane l holds the row that interchange l is
// the first to name).  The source of each place is found once per block by
// walking the w interchanges on row numbers; each lane then loads two
// entries and stores two, independent of one another.  Walking the
// interchanges on the data, one thread per column, was a chain of w dependent
// round trips (27 us for scattered pivots at N = 4,092).
#define LSW_WARPS 8
// On the columns [sol0, sol1) the warp also solves with the unit lower
// triangle of the panel (lane l holds row k0 + l): the rows of U beside the
// panel inside its block.
template <class C>
__global__ void __launch_bounds__(LSW_WARPS * 32) k_laswp(C *A, size_t ld, const int *ipiv, int k0, int w, int ncols,
                                                           int skip0, int skip1, int sol0, int sol1) {
  __shared__ int src[64], slot[32], rowof[64];
  __shared__ __align__(16) C L[32][32];   // L[c][r]
  pdl_enter();
  const int tid = threadIdx.x, lane = tid & 31;
  if (tid < 32) {
    const int p = lane < w ? ipiv[k0 + lane] - 1 : -1 - lane;
    const unsigned same = __match_any_sync(0xffffffffu, p);
    const bool below = p >= k0 + w;
    slot[lane] = lane < w ? (below ? 32 + __ffs(same) - 1 : p - k0) : 0;
    rowof[lane] = lane < w ? k0 + lane : -1;
    rowof[32 + lane] = lane < w && below && __ffs(same) - 1 == lane ? p : -1;
    src[lane] = lane;
    src[32 + lane] = 32 + lane;
    __syncwarp();
    if (lane == 0)
      for (int i = 0; i < w; i++) {
        const int q = slot[i], x = src[i], y = src[q];
        src[i] = y;
        src[q] = x;
      }
  }
  // the block's columns are blockIdx.x * LSW_WARPS + warp (+ whole grids)
  bool solves = false;
  for (int c = blockIdx.x * LSW_WARPS; c < ncols; c += gridDim.x * LSW_WARPS)
    solves |= c < sol1 && c + LSW_WARPS > sol0;
  if (solves) {
    for (int e = tid; e < w * 32; e += LSW_WARPS * 32)
      L[e >> 5][lane] = lane > (e >> 5) && lane < w ? A[(size_t)(k0 + (e >> 5)) * ld + k0 + lane] : C{0, 0};
  }
  __syncthreads();
  // place s takes the entry that was at place src[s]
  const int d0 = rowof[lane], d1 = rowof[32 + lane];
  const int s0 = d0 >= 0 ? rowof[src[lane]] : -1, s1 = d1 >= 0 ? rowof[src[32 + lane]] : -1;
  const bool m0 = d0 >= 0 && s0 != d0, m1 = d1 >= 0 && s1 != d1;
  for (int c = blockIdx.x * LSW_WARPS + (tid >> 5); c < ncols; c += gridDim.x * LSW_WARPS) {
    if (c >= skip0 && c < skip1) continue;
    const bool sol = c >= sol0 && c < sol1;
    C *cp = A + (size_t)c * ld;
    C v0 = (m0 || (sol && d0 >= 0)) ? cp[s0] : C{0, 0};
    const C v1 = m1 ? cp[s1] : C{0, 0};
    __syncwarp();   // every load of the column before its stores
    if (sol) {
      for (int i = 0; i < w; i++) v0 = cfms(v0, lds_c(&L[i][lane]), cshfl(v0, i));
      if (d0 >= 0) cp[d0] = v0;
    } else if (m0) {
      cp[d0] = v0;
    }
    if (m1) cp[d1] = v1;
  }
}

template <class C>
static int laswp(bg_matrix *m, int k0, int w, int blk_end) {
  const int blocks = std::min((m->N + LSW_WARPS - 1) / LSW_WARPS, 148 * 8);
  prof_start(PROF_LASWP);
  BG_CUDA_TRY(pdl_launch(k_laswp<C>, dim3(blocks), LSW_WARPS * 32, 0, (C *)m->d, m->ld, m->d_ipiv, k0, w, m->N, k0,
                         k0 + w, k0 + w, blk_end));
  BG_LAUNCHED();
  prof_stop(PROF_LASWP, 0.0);
  return BG_OK;
}

// -------------------------------------------------------------------------
// Update inside a block of LU_BLOCK columns after one of its panels:
// C (M x nc, nc <= LU_BLOCK - 32) -= L (M x K) U (K x nc), K <= 32, on the
// FP64 (FP32) pipe, whose rate is that of the FP64 tensor path.  A CTA takes
// 32 rows, a warp 1/4 of the columns (lane = row): L by rows and U by
// broadcasts from shared memory, accumulators in registers, C read while the
// operands are staged with cp.async.  Tensor-core tiles of this shape (K = 32,
// at most 96 columns) were one launch per level of a deeper recursion.
// -------------------------------------------------------------------------
#define LU_BLOCK 128
template <class C, int NC>
__global__ void __launch_bounds__(128) k_blk_update(int M, int nc, int K, const C *L, const C *U, C *Cm, size_t ld) {
  __shared__ __align__(16) C Ls[32][32];   // Ls[k][r]
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C *Us = (C *)smem_raw;                   // Us[c * 32 + k]
  pdl_enter();
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int r = blockIdx.x * 32 + lane, c0 = wid * NC;
#pragma unroll
  for (int q = 0; q < 8; q++) {
    const int k = wid + 4 * q;
    const bool ok = r < M && k < K;
    cp_entry(&Ls[k][lane], ok ? L + (size_t)k * ld + r : L, ok);
  }
#pragma unroll
  for (int q = 0; q < NC; q++) {
    const int c = wid + 4 * q;
    const bool ok = lane < K && c < nc;
    cp_entry(Us + c * 32 + lane, ok ? U + (size_t)c * ld + lane : U, ok);
  }
  cp_commit();
  // the products are summed first and subtracted from C once
  C acc[NC], old[NC];
#pragma unroll
  for (int c = 0; c < NC; c++) {
    acc[c] = C{0, 0};
    old[c] = (r < M && c0 + c < nc) ? Cm[(size_t)(c0 + c) * ld + r] : C{0, 0};
  }
  cp_wait<0>();
  __syncthreads();
#pragma unroll 2
  for (int k = 0; k < 32; k++) {
    const C l = lds_c(&Ls[k][lane]);
#pragma unroll
    for (int c = 0; c < NC; c++) acc[c] = cmac(acc[c], l, lds_c(Us + (c0 + c) * 32 + k));
  }
#pragma unroll
  for (int c = 0; c < NC; c++)
    if (r < M && c0 + c < nc) Cm[(size_t)(c0 + c) * ld + r] = C{old[c].r - acc[c].r, old[c].i - acc[c].i};
}
template <class C, int NC>
static int blk_update_launch(int M, int nc, int K, const C *L, const C *U, C *Cm, size_t ld) {
  const int smem = 32 * 4 * NC * (int)sizeof(C);
  static bool attr = false;
  if (!attr) {
    BG_CUDA_TRY(cudaFuncSetAttribute(k_blk_update<C, NC>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    attr = true;
  }
  prof_start(PROF_GEMM);
  BG_CUDA_TRY(pdl_launch(k_blk_update<C, NC>, dim3((M + 31) / 32), 128, smem, M, nc, K, L, U, Cm, ld));
  BG_LAUNCHED();
  prof_stop(PROF_GEMM, 8.0 * M * (double)nc * K);
  return BG_OK;
}
template <class C>
static int blk_update(int M, int nc, int K, const C *L, const C *U, C *Cm, size_t ld) {
  if (M <= 0 || nc <= 0) return BG_OK;
  return nc > 64   ? blk_update_launch<C, 24>(M, nc, K, L, U, Cm, ld)
         : nc > 32 ? blk_update_launch<C, 16>(M, nc, K, L, U, Cm, ld)
                   : blk_update_launch<C, 8>(M, nc, K, L, U, Cm, ld);
}

struct LUWork {
  double *cval;
  int *cidx;
  void *crow, *jrow;
  int *info;
  unsigned long long *slots;
};

static int panel_grid = 0, panel_smem_max = 0, panel_rows_target = 32;

template <class C, int TMAX>
constexpr int panel_rf_smem() { return (int)sizeof(PrfSmem<C>) + 32 * (TMAX + 1) * (int)sizeof(C); }

// CTAs per cluster of k_panel_rf that this device can place (16, 8 or 0)
template <class C, int TMAX>
static int panel_rf_cluster() {
  static int cs = -1;
  if (cs >= 0) return cs;
  cs = 0;
  const int smem = panel_rf_smem<C, TMAX>();
  if (cudaFuncSetAttribute(k_panel_rf<C, TMAX, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess ||
      cudaFuncSetAttribute(k_panel_rf<C, TMAX, false>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
    cudaGetLastError();
    return cs;
  }
  for (int want = PRF_MAXCL; want >= 8 && !cs; want /= 2) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    cfg.gridDim = dim3(want);
    cfg.blockDim = dim3(TMAX + 32);
    cfg.dynamicSmemBytes = smem;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = want;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, (void *)k_panel_rf<C, TMAX, false>, &cfg) == cudaSuccess && n >= 1) cs = want;
  }
  cudaGetLastError();
  return cs;
}

// the panel on one cluster with its rows in registers; *done = false: too tall
template <class C, int TMAX>
static int panel_rf(bg_matrix *m, const LUWork &W, int k0, int w, int blk_end, bool *done) {
  const int N = m->N, Mp = N - k0, RS = panel_rf_cluster<C, TMAX>();
  *done = RS && Mp <= RS * TMAX;
  if (!*done) return BG_OK;
  // 128 rows per CTA, one warp per scheduler, until the cluster is full (rank 0
  // owns the w rows of the diagonal block); 192 inside a batched sweep, where
  // clusters of fewer SMs start sooner beside the other streams' work (64 jobs of
  // N about 2,650 and 2,000: 212 -> 207 ms, 224 rows 212)
  const int per = t_pdl ? 128 : 192;
  const int G = std::min(RS, std::max(1, (Mp + per - 1) / per));
  const int rows = (Mp + G - 1) / G, threads = (rows + 31) / 32 * 32 + 32;
  PanelArgs<C> P{(C *)m->d, m->ld, N, k0, w, rows, m->d_ipiv, W.info, W.cval, W.cidx, (C *)W.crow, (C *)W.jrow, W.slots};
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(G);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = panel_rf_smem<C, TMAX>();
  cfg.stream = stream();
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = G;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = t_pdl;
  cfg.attrs = at;
  cfg.numAttrs = 2;
  prof_start(PROF_PANEL);
  BG_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_panel_rf<C, TMAX, false>, P));
  BG_LAUNCHED();
  prof_stop(PROF_PANEL, 8.0 * Mp * (double)w * w / 2);
  return laswp<C>(m, k0, w, blk_end);
}

// the same panel over the grid, through L2
#define PRG_T 256
#define PRG_ROWS 192     // rows per CTA until the grid is full
template <class C>
static int panel_rg(bg_matrix *m, const LUWork &W, int k0, int w, int blk_end, bool *done) {
  const int N = m->N, Mp = N - k0;
  const int maxg = std::min(panel_max_grid, panel_grid);
  *done = Mp <= maxg * PRG_T;
  if (!*done) return BG_OK;
  static bool attr = false;
  if (!attr) {
    BG_CUDA_TRY(cudaFuncSetAttribute(k_panel_rf<C, PRG_T, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     panel_rf_smem<C, PRG_T>()));
    attr = true;
  }
  const int G = std::min(maxg, (Mp + PRG_ROWS - 1) / PRG_ROWS);
  const int rows = (Mp + G - 1) / G, threads = (rows + 31) / 32 * 32 + 32;
  PanelArgs<C> P{(C *)m->d, m->ld, N, k0, w, rows, m->d_ipiv, W.info, W.cval, W.cidx, (C *)W.crow, (C *)W.jrow, W.slots};
  void *args[] = {&P};
  prof_start(PROF_PANEL);
  BG_CUDA_TRY(cudaLaunchCooperativeKernel((void *)k_panel_rf<C, PRG_T, true>, dim3(G), dim3(threads), args,
                                          (size_t)panel_rf_smem<C, PRG_T>(), stream()));
  BG_LAUNCHED();
  prof_stop(PROF_PANEL, 8.0 * Mp * (double)w * w / 2);
  return laswp<C>(m, k0, w, blk_end);
}

template <class C>
static int panel_leaf(bg_matrix *m, const LUWork &W, int k0, int w, int blk_end) {
  int N = m->N;
  int Mp = N - k0;
  // rows in the registers of one cluster, while they fit (a row per thread:
  // 4,096 rows of complex128, 8,192 of complex64 with 16 CTAs)
  bool done = false;
  int st = panel_rf<C, PrfCfg<C>::T0>(m, W, k0, w, blk_end, &done);
  if (!st && !done) st = panel_rf<C, PrfCfg<C>::T1>(m, W, k0, w, blk_end, &done);
  if (!st && !done) st = panel_rg<C>(m, W, k0, w, blk_end, &done);
  if (st || done) return st;
  // still taller (more than 37,888 rows): slices in shared memory
  int G = std::min(panel_grid, std::max(1, (Mp + panel_rows_target - 1) / panel_rows_target));
  while (G < panel_grid && (size_t)((Mp + G - 1) / G) * w * sizeof(C) > (size_t)panel_smem_max) G++;
  int rows = (Mp + G - 1) / G;
  size_t smem = (size_t)rows * w * sizeof(C);
  if ((int)smem > panel_smem_max) {
    set_error("panel slice of %zu bytes exceeds shared memory (N=%d too large for this build)", smem, N);
    return BG_ERR_ARG;
  }
  static bool attr = false;
  if (!attr) {
    BG_CUDA_TRY(cudaFuncSetAttribute(k_panel<C>, cudaFuncAttributeMaxDynamicSharedMemorySize, panel_smem_max));
    attr = true;
  }
  PanelArgs<C> P{(C *)m->d, m->ld, N, k0, w, rows, m->d_ipiv, W.info, W.cval, W.cidx, (C *)W.crow, (C *)W.jrow, W.slots};
  void *args[] = {&P};
  prof_start(PROF_PANEL);
  BG_CUDA_TRY(cudaLaunchCooperativeKernel((void *)k_panel<C>, dim3(G), dim3(256), args, smem, stream()));
  BG_LAUNCHED();
  prof_stop(PROF_PANEL, 8.0 * Mp * (double)w * w / 2);
  return laswp<C>(m, k0, w, blk_end);
}

// factor columns [k0, k0+n) (rows k0..N-1); interchanges applied to all columns.
// Blocks of LU_BLOCK columns are factored right-looking in panels of 32 (three
// launches a panel: panel, interchanges with the panel's triangular solve
// inside the block, update of the rest of the block); above them the recursion
// over column halves keeps the Schur complements large.
template <class C>
static int getrf_rec(bg_matrix *m, const LUWork &W, int k0, int n) {
  int st;
  C *A = (C *)m->d;
  size_t ld = m->ld;
  int N = m->N;
  if (n <= LU_BLOCK) {
    for (int p = k0; p < k0 + n; p += 32) {
      const int w = std::min(32, k0 + n - p), nc = k0 + n - p - w;
      if ((st = panel_leaf<C>(m, W, p, w, k0 + n))) return st;
      if ((st = blk_update<C>(N - p - w, nc, w, A + (p + w) + (size_t)p * ld, A + p + (size_t)(p + w) * ld,
                              A + (p + w) + (size_t)(p + w) * ld, ld)))
        return st;
    }
    return BG_OK;
  }
  int n1 = (n / 2 + LU_BLOCK - 1) / LU_BLOCK * LU_BLOCK;   // < n, as n > LU_BLOCK
  int n2 = n - n1;
  if ((st = getrf_rec<C>(m, W, k0, n1))) return st;
  C *A11 = A + k0 + (size_t)k0 * ld;
  C *A12 = A + k0 + (size_t)(k0 + n1) * ld;
  C *A21 = A + (k0 + n1) + (size_t)k0 * ld;
  C *A22 = A + (k0 + n1) + (size_t)(k0 + n1) * ld;
  if ((st = trsm<C>(n1, n2, A11, ld, A12, ld, 0))) return st;
  if ((st = gemm_sub(N - k0 - n1, n2, n1, A21, ld, A12, ld, A22, ld))) return st;
  return getrf_rec<C>(m, W, k0 + n1, n2);
}

static int build_perm(bg_matrix *m);

static int panel_init() {
  if (panel_grid) return BG_OK;
  int dev = 0, sms = 0, smemopt = 0;
  BG_CUDA_TRY(cudaGetDevice(&dev));
  BG_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  BG_CUDA_TRY(cudaDeviceGetAttribute(&smemopt, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  panel_smem_max = smemopt - 2048;
  panel_grid = sms;  // at most one CTA per SM (cooperative residency)
  if (const char *e = std::getenv("BG_PANEL_ROWS")) panel_rows_target = std::max(8, std::atoi(e));
  return BG_OK;
}

#define PRG_BYTES (sizeof(unsigned long long) * (2 * (size_t)panel_max_grid * PRG_STRIDE + 2))   // slots, launch count, tickets
static size_t lu_work_bytes(bg_matrix *m) {
  const size_t csz = m->precision == BG_C128 ? sizeof(cdl) : sizeof(cfl);
  return PRG_BYTES + csz * 2 * panel_grid * 32 + csz * 64 + sizeof(double) * 2 * panel_grid +
         sizeof(int) * 2 * panel_grid + 256;
}
static int lu_work_alloc(bg_matrix *m, size_t need) {
  if (m->work_bytes >= need) return BG_OK;
  if (m->d_work) cudaFree(m->d_work);
  m->d_work = nullptr;
  m->work_bytes = 0;
  BG_CUDA_TRY(cudaMalloc(&m->d_work, need));
  m->work_bytes = need;
  // tags, launch count and tickets of the grid-wide panel start at zero
  BG_CUDA_TRY(cudaMemsetAsync(m->d_work, 0, PRG_BYTES, stream()));
  return BG_OK;
}

// the products (M, N, K) of a triangular solve and of a factorisation, as trsm and getrf_rec form them
template <class F>
static void trsm_products(int n, int m, F &&f) {
  if (n <= TRS_MAX) return;
  const int n1 = (n / 2 + TRS_MAX - 1) / TRS_MAX * TRS_MAX;
  trsm_products(n1, m, f);
  f(n - n1, m, n1);
  trsm_products(n - n1, m, f);
}
template <class F>
static void getrf_products(int N, int k0, int n, F &&f) {
  if (n <= LU_BLOCK) return;
  const int n1 = (n / 2 + LU_BLOCK - 1) / LU_BLOCK * LU_BLOCK;
  getrf_products(N, k0, n1, f);
  trsm_products(n1, n - n1, f);
  f(N - k0 - n1, n - n1, n1);
  getrf_products(N, k0 + n1, n - n1, f);
}

// scratch of the INT8 products of a factorisation (0: every product is too small for them)
static size_t i8_factor_bytes(int N) {
  size_t b = 0;
  getrf_products(N, 0, N, [&](int m, int n, int k) {
    if (i8_takes(m, n, k)) b = std::max(b, zgemm_i8_bytes(m, n, k));
  });
  return b;
}

// whether a factorisation in complex128 depends on the settings that a batched sweep tunes:
// rows per CTA of the shared-memory panel, CTA tile of the FP64 products
bool lu_uses_panel_rows(int N) { return N > std::min(panel_max_grid, panel_grid ? panel_grid : panel_max_grid) * PRG_T; }
bool lu_uses_gemm_tile(int N) {
  bool used = false;
  getrf_products(N, 0, N, [&](int m, int n, int k) {
    used |= !i8_takes(m, n, k) && (long)((m + 63) / 64) * ((n + 63) / 64) > ZG_SMALL;
  });
  return used;
}

int lu_factor(bg_matrix *m) {
  int st = ensure_device();
  if (!st) st = panel_init();
  if (st) return st;
  int N = m->N;
  const size_t csz = m->precision == BG_C128 ? sizeof(cdl) : sizeof(cfl);
  // workspace: candidate rows, j-rows, candidate values/indices, info, error
  // flag, and (complex64) the expanded-A scratch of the tensor-core GEMM
  size_t at_floats = 0;
  if (m->precision == BG_C64) at_floats = (size_t)2 * TC_MCHUNK * (((size_t)2 * N + 31) / 32 * 32);
  size_t need = lu_work_bytes(m) + sizeof(float) * at_floats;
  if ((st = lu_work_alloc(m, need))) return st;
  char *w = (char *)m->d_work;
  LUWork W;
  W.slots = (unsigned long long *)w; w += PRG_BYTES;
  W.crow = (void *)w; w += csz * 2 * panel_grid * 32;
  W.jrow = (void *)w; w += csz * 64;
  W.cval = (double *)w; w += sizeof(double) * 2 * panel_grid;
  W.cidx = (int *)w; w += sizeof(int) * 2 * panel_grid;
  W.info = (int *)w;
  int *tcerr = W.info + 1;
  w += 256;
  BG_CUDA_TRY(cudaMemsetAsync(W.info, 0, 2 * sizeof(int), stream()));
  t_pdl = true;
  if (m->precision == BG_C128) {
    I8Scratch sc{nullptr, i8_factor_bytes(N), W.info + 1};
    if (sc.bytes && cudaMallocAsync(&sc.p, sc.bytes, stream()) != cudaSuccess) {
      cudaGetLastError();      // no room: the FP64 tiles need no scratch
      sc.p = nullptr;
    }
    t_i8 = sc.p ? &sc : nullptr;
    st = getrf_rec<cdl>(m, W, 0, N);
    t_i8 = nullptr;
    t_pdl = false;
    if (sc.p) cudaFreeAsync(sc.p, stream());
    if (st) return st;
  } else {
    TcScratch sc;
    sc.At = (float *)w;
    sc.at_floats = at_floats;
    sc.err = tcerr;
    t_tc = &sc;
    st = getrf_rec<cfl>(m, W, 0, N);
    t_tc = nullptr;
    t_pdl = false;
    if (st) return st;
  }
  int info[2] = {0, 0};
  BG_CUDA_TRY(cudaMemcpyAsync(info, W.info, 2 * sizeof(int), cudaMemcpyDeviceToHost, stream()));
  BG_CUDA_TRY(cudaStreamSynchronize(stream()));
  if (info[1]) {
    set_error("factorisation: a %s wait timed out (code %d)", info[1] == 300 ? "panel" : "tensor-core GEMM", info[1]);
    return BG_ERR_CUDA;
  }
  if ((st = build_perm(m))) return st;
  return info[0];
}

// by FP64 whatever the size, without a synchronisation: buff-neq's products with S^-1,
// whose entries fall off so fast that most of their tiles would be left out of the digits
// (flux of two bodies, N = 2,022: 12.6 -> 12.4 ms, 5,172: 122 -> 119)
int zgemm_fp64_device(int M, int N, int K, const void *A, int lda, const void *B, int ldb, void *C, int ldc) {
  int st = ensure_device();
  return st ? st : zgemm_sub(M, N, K, (const cdl *)A, (size_t)lda, (const cdl *)B, (size_t)ldb, (cdl *)C, (size_t)ldc);
}

int zgemm_sub_device(int M, int N, int K, const void *A, int lda, const void *B, int ldb, void *C, int ldc) {
  int st = ensure_device();
  if (st) return st;
  I8Scratch sc{nullptr, 0, nullptr};
  if (M > 0 && N > 0 && K > 0 && i8_takes(M, N, K)) {
    sc.bytes = zgemm_i8_bytes(M, N, K);
    if (cudaMallocAsync(&sc.p, sc.bytes + 256, stream()) != cudaSuccess) {
      cudaGetLastError();      // no scratch: the FP64 tiles need none
      sc.p = nullptr;
    }
  }
  if (!sc.p) return zgemm_sub(M, N, K, (const cdl *)A, (size_t)lda, (const cdl *)B, (size_t)ldb, (cdl *)C, (size_t)ldc);
  sc.err = (int *)((char *)sc.p + sc.bytes);
  cudaError_t e = cudaMemsetAsync(sc.err, 0, sizeof(int), stream());
  t_i8 = &sc;
  st = zgemm_sub(M, N, K, (const cdl *)A, (size_t)lda, (const cdl *)B, (size_t)ldb, (cdl *)C, (size_t)ldc);
  t_i8 = nullptr;
  int h = 0;
  if (e == cudaSuccess) e = cudaMemcpyAsync(&h, sc.err, sizeof(int), cudaMemcpyDeviceToHost, stream());
  if (e == cudaSuccess) e = cudaStreamSynchronize(stream());
  cudaFreeAsync(sc.p, stream());
  if (!st && e != cudaSuccess) { set_error("zgemm: %s", cudaGetErrorString(e)); st = BG_ERR_CUDA; }
  if (!st && h) { set_error("zgemm: a tensor-core wait timed out (code %d)", h); st = BG_ERR_CUDA; }
  return st;
}

// =========================================================================
// few-right-hand-side solves: B <- U^{-1} L^{-1} P B in one gather and two
// single-pass triangular sweeps.  In a sweep each CTA takes the next 64-row
// block in dependency order from a ticket counter, accumulates the products
// with already-solved blocks as their ready flags appear (flag == epoch),
// solves its diagonal block (one warp per right-hand side), publishes the
// block and raises its flag.  A CTA only ever waits on blocks with smaller
// tickets, which are already running, so the sweep always makes progress;
// every wait is bounded and a timeout is recorded in the error word, which
// also makes the other CTAs give up early.
// The chain from block to block sets the time: flag and data through L2, one
// 64 x 64 product, the diagonal solve.  The 16 x 16 diagonal blocks are
// inverted while the CTA waits, so the solve of one is three 16-wide products
// (x = T^{-1} b, r = b - T x, x += T^{-1} r) instead of 16 dependent substitutions
// with a shuffle each; every thread polls the flag and fetches its own entry of the
// solved block (one barrier a block).  The correction makes the residual that of
// substitution, a few units in the last place of |T||x|: x = T^{-1} b alone leaves
// cond(T) times that (componentwise backward error of a solve at N = 4,092, 48 systems:
// 6.2e-16 with substitution, 8.7e-16 without the correction, 6.6e-16 with it).  One
// correction squares cond(T) eps, so blocks beyond TrsvCond are solved by substitution.
// Solve of one right-hand side: 1.10 ms by substitution throughout, 0.73 ms now (0.51
// without the correction) at N = 4,092; complex64 at N = 19,872 3.9 and 2.7 ms (1.9).
// =========================================================================
#define TV_B 64
#define TV_MAXRHS 4
#define TV_SPIN (1 << 22)

template <class C>
__global__ void k_gather_rows(int N, int nrhs, const int *perm, const C *src, size_t lds, C *dst, size_t ldd) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  int j = blockIdx.y;
  if (i < N && j < nrhs) dst[(size_t)j * ldd + i] = src[(size_t)j * lds + perm[i]];
}

// 1-norm condition of a 16 x 16 block up to which it is solved by its inverse: 16 cond eps
// squared stays below eps
template <class C> struct TrsvCond;
template <> struct TrsvCond<cdl> { static constexpr double MAX = 1e6; };
template <> struct TrsvCond<cfl> { static constexpr float MAX = 200.f; };
template <class C>
constexpr int trsv_smem() {
  return TV_B * (TV_B + 1) * (int)sizeof(C) + 4 * TV_B * TV_MAXRHS * (int)sizeof(C) + TV_B * 17 * (int)sizeof(C);
}

__device__ __forceinline__ int ld_acquire(const int *p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release(int *p, int v) {
  asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

template <class C, bool UPPER>
__global__ void __launch_bounds__(128) k_trsv(int N, const C *A, size_t ld, C *X, size_t ldx, int nrhs, int *flags,
                                              int epoch, int *ticket, int *err) {
  typedef typename CxT<C>::R R;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C(*D)[TV_B + 1] = (C(*)[TV_B + 1])smem_raw;   // diagonal block, the other triangle of its 16 x 16 diagonal blocks zero
  C(*part)[TV_MAXRHS] = (C(*)[TV_MAXRHS])(smem_raw + TV_B * (TV_B + 1) * sizeof(C));   // part[row][rhs]
  C(*xs)[TV_B][TV_MAXRHS] = (C(*)[TV_B][TV_MAXRHS])(part + TV_B);                     // solved blocks, two buffers
  C(*sol)[TV_MAXRHS] = (C(*)[TV_MAXRHS])(xs + 2);                                    // solution and residual of a diagonal block
  C(*Iv)[17] = (C(*)[17])(sol + TV_B);                                               // inverses of the four diagonal blocks
  __shared__ int s_blk, s_abort, s_subst;                                            // s_subst: blocks to solve by substitution
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nb = (N + TV_B - 1) / TV_B;
  if (tid == 0) { s_blk = atomicAdd(ticket, 1); s_abort = s_subst = 0; }
  __syncthreads();
  const int lb = s_blk;
  const int bi = UPPER ? nb - 1 - lb : lb;
  const int r0 = bi * TV_B, rows = min(TV_B, N - r0);
  const int row = tid & (TV_B - 1), half = tid >> 6;
  // this block's right-hand-side rows (written by no other CTA), read now
  // so that the final combine does not wait for memory
  C bx[TV_MAXRHS];
#pragma unroll
  for (int j = 0; j < TV_MAXRHS; j++)
    bx[j] = (half == 0 && row < rows && j < nrhs) ? X[(size_t)j * ldx + r0 + row] : C{0, 0};
  // stage the diagonal block, eight loads per thread in flight; rows and
  // columns past the matrix are those of the identity
  for (int e0 = 0; e0 < TV_B * TV_B; e0 += 8 * 128) {
    C v[8];
#pragma unroll
    for (int u = 0; u < 8; u++) {
      const int e = e0 + u * 128 + tid, c = e / TV_B, r = e % TV_B;
      v[u] = (r < rows && c < rows) ? A[(size_t)(r0 + c) * ld + r0 + r] : C{(R)(r == c ? 1 : 0), 0};
    }
#pragma unroll
    for (int u = 0; u < 8; u++) {
      const int e = e0 + u * 128 + tid, r = e % TV_B, c = e / TV_B;
      if (r / 16 == c / 16) {
        if (UPPER ? r > c : r < c) v[u] = C{0, 0};
        if (!UPPER && r == c) v[u] = C{1, 0};
      }
      D[r][c] = v[u];
    }
  }
  __syncthreads();
  {
    // column c of the inverse of 16 x 16 block s, by substitution
    C v[16];
    const int s = tid >> 4, c = tid & 15, o = 16 * s;
    if (tid < TV_B) {
      if (!UPPER) {
#pragma unroll
        for (int i = 0; i < 16; i++) {
          C t{(R)(i == c ? 1 : 0), 0};
#pragma unroll
          for (int k = 0; k < i; k++) t = cfms(t, D[o + i][o + k], v[k]);
          v[i] = i < c ? C{0, 0} : t;
        }
      } else {
#pragma unroll
        for (int i = 15; i >= 0; i--) {
          C t{(R)(i == c ? 1 : 0), 0};
#pragma unroll
          for (int k = 15; k > i; k--) t = cfms(t, D[o + i][o + k], v[k]);
          const C u = D[o + i][o + i];
          const R d = u.r * u.r + u.i * u.i;
          v[i] = i > c ? C{0, 0} : C{(t.r * u.r + t.i * u.i) / d, (t.i * u.r - t.r * u.i) / d};
        }
      }
    }
    if (tid < TV_B) {
      R si = 0, st = 0;      // column sums of the inverse and of the block
#pragma unroll
      for (int i = 0; i < 16; i++) {
        Iv[o + i][c] = v[i];
        const C t = D[o + i][o + c];
        si += fabs(v[i].r) + fabs(v[i].i);
        st += fabs(t.r) + fabs(t.i);
      }
      R mt = st;
#pragma unroll
      for (int k = 8; k > 0; k >>= 1) mt = max(mt, __shfl_xor_sync(0xffffffffu, mt, k));
      if (!(si * mt <= TrsvCond<C>::MAX && st == st)) atomicOr(&s_subst, 1 << s);
    }
  }
  C acc[TV_MAXRHS];
#pragma unroll
  for (int j = 0; j < TV_MAXRHS; j++) acc[j] = C{0, 0};
  for (int q = 0; q < lb; q++) {
    const int bj = UPPER ? nb - 1 - q : q;
    const int c0 = bj * TV_B, cols = min(TV_B, N - c0);
    // this thread's row of block (bi, bj) over its half of the columns:
    // A does not depend on x, so it is read before waiting for block bj
    C a[32];
    {
      const C *ap = A + (size_t)(c0 + half * 32) * ld + r0 + row;
#pragma unroll
      for (int u = 0; u < 32; u++)
        a[u] = (row < rows && half * 32 + u < cols) ? ap[(size_t)u * ld] : C{0, 0};
    }
    // every thread waits for the block and fetches its entries of x (at most 2)
    {
      const int *f = flags + bj;
      int it = 0;
      while (ld_acquire(f) != epoch) {
        if (*(volatile int *)err || ++it > TV_SPIN) {
          if (it > TV_SPIN) atomicCAS(err, 0, 100 + (UPPER ? 1 : 0));
          s_abort = 1;
          break;
        }
        if (lb - q > 4) __nanosleep(64);   // not next in the chain
      }
      C v[2];
#pragma unroll
      for (int u = 0; u < 2; u++) {
        const int e = u * 128 + tid;
        v[u] = e < TV_B * nrhs && (e & (TV_B - 1)) < cols ? ldcg_c(X + (size_t)(e / TV_B) * ldx + c0 + (e & (TV_B - 1)))
                                                          : C{0, 0};
      }
#pragma unroll
      for (int u = 0; u < 2; u++) {
        const int e = u * 128 + tid;
        if (e < TV_B * nrhs) xs[q & 1][e & (TV_B - 1)][e / TV_B] = v[u];
      }
    }
    __syncthreads();
    if (s_abort) return;
    // the buffer of this block is rewritten two blocks on, behind the next barrier
    const C(*x)[TV_MAXRHS] = xs[q & 1] + half * 32;
#pragma unroll
    for (int u = 0; u < 32; u++) {
#pragma unroll
      for (int j = 0; j < TV_MAXRHS; j++)
        if (j < nrhs) acc[j] = cmac(acc[j], a[u], x[u][j]);
    }
  }
  if (half == 1)
#pragma unroll
    for (int j = 0; j < TV_MAXRHS; j++)
      if (j < nrhs) part[row][j] = acc[j];
  __syncthreads();
  if (half == 0)
#pragma unroll
    for (int j = 0; j < TV_MAXRHS; j++)
      if (j < nrhs) {
        const C b = bx[j];
        C p = part[row][j];
        part[row][j] = row < rows ? C{b.r - acc[j].r - p.r, b.i - acc[j].i - p.i} : C{0, 0};
      }
  __syncthreads();
  // diagonal solve: warp j handles right-hand side j
  if (warp < nrhs) {
    const int j = warp, r = lane & 15, h = lane >> 4;
#pragma unroll
    for (int t = 0; t < 4; t++) {
      const int o = 16 * (UPPER ? 3 - t : t);
      // row r of M v, columns 8 h .. 8 h + 7 by each half of the warp
      auto times = [&](const C *M, const C(*v)[TV_MAXRHS]) {
        C y[4] = {{0, 0}, {0, 0}, {0, 0}, {0, 0}};
#pragma unroll
        for (int k = 0; k < 8; k++) y[k & 3] = cmac(y[k & 3], M[8 * h + k], v[8 * h + k][j]);
        C w{(y[0].r + y[1].r) + (y[2].r + y[3].r), (y[0].i + y[1].i) + (y[2].i + y[3].i)};
        w.r += __shfl_xor_sync(0xffffffffu, w.r, 16);
        w.i += __shfl_xor_sync(0xffffffffu, w.i, 16);
        return w;
      };
      C y;
      if (!(s_subst >> (o / 16) & 1)) {
        y = times(Iv[o + r], part + o);
        if (h == 0) sol[o + r][j] = y;
        __syncwarp();
        const C t = times(&D[o + r][o], sol + o), b = part[o + r][j];
        __syncwarp();
        if (h == 0) sol[o + r][j] = C{b.r - t.r, b.i - t.i};
        __syncwarp();
        const C d = times(Iv[o + r], sol + o);
        y.r += d.r;
        y.i += d.i;
      } else {
        y = part[o + r][j];
        for (int n = 0; n < 16; n++) {
          const int i = UPPER ? 15 - n : n;
          C x = cshfl(y, i);
          if (UPPER) {
            const C u = D[o + i][o + i];
            const R d = u.r * u.r + u.i * u.i;
            const C iu{u.r / d, -u.i / d};
            x = C{x.r * iu.r - x.i * iu.i, x.r * iu.i + x.i * iu.r};
          }
          if (r == i) y = x;
          else if (UPPER ? r < i : r > i) y = cfms(y, D[o + r][o + i], x);
        }
      }
      __syncwarp();
      if (h == 0) {
        part[o + r][j] = y;
        if (o + r < rows) X[(size_t)j * ldx + r0 + o + r] = y;
      }
      __syncwarp();
      // the rows still to solve
      if (t < 3) {
        const int left = 16 * (3 - t), base = UPPER ? 0 : o + 16;
        for (int q = lane; q < left; q += 32) {
          C s[4] = {{0, 0}, {0, 0}, {0, 0}, {0, 0}};
#pragma unroll
          for (int k = 0; k < 16; k++) s[k & 3] = cmac(s[k & 3], D[base + q][o + k], part[o + k][j]);
          C p = part[base + q][j];
          p.r -= (s[0].r + s[1].r) + (s[2].r + s[3].r);
          p.i -= (s[0].i + s[1].i) + (s[2].i + s[3].i);
          part[base + q][j] = p;
        }
        __syncwarp();
      }
    }
  }
  __syncthreads();
  if (tid == 0) st_release(flags + bi, epoch);   // after every thread's stores (the barrier above)
}

// host: permutation from LAPACK interchanges, kept beside the factors
static int build_perm(bg_matrix *m) {
  int N = m->N;
  std::vector<int> ipiv(N), perm(N);
  BG_CUDA_TRY(cudaMemcpyAsync(ipiv.data(), m->d_ipiv, sizeof(int) * N, cudaMemcpyDeviceToHost, stream()));
  BG_CUDA_TRY(cudaStreamSynchronize(stream()));
  for (int i = 0; i < N; i++) perm[i] = i;
  for (int i = 0; i < N; i++) std::swap(perm[i], perm[ipiv[i] - 1]);
  if (!m->d_perm) BG_CUDA_TRY(cudaMalloc(&m->d_perm, sizeof(int) * (N + 2 * ((N + TV_B - 1) / TV_B) + 8)));
  BG_CUDA_TRY(cudaMemcpyAsync(m->d_perm, perm.data(), sizeof(int) * N, cudaMemcpyHostToDevice, stream()));
  // ready flags of both sweeps + tickets + error word, zeroed once
  BG_CUDA_TRY(cudaMemsetAsync(m->d_perm + N, 0, sizeof(int) * (2 * ((N + TV_B - 1) / TV_B) + 8), stream()));
  BG_CUDA_TRY(cudaStreamSynchronize(stream()));
  return BG_OK;
}

template <class C>
static int getrs(bg_matrix *m, C *B, size_t ldb, int nrhs) {
  int N = m->N;
  const C *A = (const C *)m->d;
  const int nb = (N + TV_B - 1) / TV_B;
  int *flagsL = m->d_perm + N, *flagsU = flagsL + nb, *tick = flagsU + nb, *err = tick + 2;
  const int smem = trsv_smem<C>();
  static bool attr = false;
  if (!attr) {
    BG_CUDA_TRY(cudaFuncSetAttribute(k_trsv<C, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    BG_CUDA_TRY(cudaFuncSetAttribute(k_trsv<C, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    attr = true;
  }
  for (int r0 = 0; r0 < nrhs; r0 += TV_MAXRHS) {
    int nr = std::min(TV_MAXRHS, nrhs - r0);
    C *Bp = B + (size_t)r0 * ldb;
    C *T = nullptr;
    BG_CUDA_TRY(cudaMallocAsync((void **)&T, sizeof(C) * (size_t)N * nr, stream()));
    k_gather_rows<C><<<dim3((N + 255) / 256, nr), 256, 0, stream()>>>(N, nr, m->d_perm, Bp, ldb, T, N);
    BG_LAUNCHED();
    int epoch = ++m->solve_epoch;
    BG_CUDA_TRY(cudaMemsetAsync(tick, 0, 2 * sizeof(int), stream()));
    prof_start(PROF_TRSV);
    k_trsv<C, false><<<nb, 128, smem, stream()>>>(N, A, m->ld, T, N, nr, flagsL, epoch, tick, err);
    BG_LAUNCHED();
    k_trsv<C, true><<<nb, 128, smem, stream()>>>(N, A, m->ld, T, N, nr, flagsU, epoch, tick + 1, err);
    BG_LAUNCHED();
    // bytes of the two triangles read once
    prof_stop(PROF_TRSV, (double)sizeof(C) * (double)N * N);
    BG_CUDA_TRY(cudaMemcpy2DAsync(Bp, sizeof(C) * ldb, T, sizeof(C) * N, sizeof(C) * N, nr, cudaMemcpyDeviceToDevice,
                                  stream()));
    BG_CUDA_TRY(cudaFreeAsync(T, stream()));
  }
  return BG_OK;
}

// Many right-hand sides (N-column blocks of the buff-neq chain): one row
// gather by the factor permutation, then the recursive GEMM-based triangular
// solves used inside the factorisation (unit L, then U), in column chunks so
// the scratch stays bounded.
int lu_solve_many(bg_matrix *m, void *dB, size_t ldb, int nrhs) {
  if (!m->d_perm) { set_error("solve: factorization state missing"); return BG_ERR_STATE; }
  if (m->precision != BG_C128) { set_error("lu_solve_many: complex128 only"); return BG_ERR_ARG; }
  int N = m->N;
  const cdl *A = (const cdl *)m->d;
  cdl *B = (cdl *)dB;
  const int chunk = 4096;
  cdl *T = nullptr;
  int w = std::min(chunk, nrhs);
  if (w <= 0) return BG_OK;
  BG_CUDA_TRY(cudaMallocAsync((void **)&T, sizeof(cdl) * (size_t)N * w, stream()));
  // scratch of the INT8 products, where some are large enough for them (the products
  // of the upper solve have rows and inner index exchanged)
  I8Scratch sc{nullptr, 0, nullptr};
  trsm_products(N, w, [&](int m, int n, int k) {
    if (i8_takes(m, n, k)) sc.bytes = std::max(sc.bytes, zgemm_i8_bytes(m, n, k));
    if (i8_takes(k, n, m)) sc.bytes = std::max(sc.bytes, zgemm_i8_bytes(k, n, m));
  });
  if (sc.bytes && cudaMallocAsync(&sc.p, sc.bytes + 256, stream()) != cudaSuccess) {
    cudaGetLastError();
    sc.p = nullptr;
  }
  int st = BG_OK, tcerr = 0;
  if (sc.p) {
    sc.err = (int *)((char *)sc.p + sc.bytes);
    if (cudaMemsetAsync(sc.err, 0, sizeof(int), stream()) != cudaSuccess) { cudaGetLastError(); st = BG_ERR_CUDA; }
    t_i8 = &sc;
  }
  t_pdl = true;
  for (int r0 = 0; r0 < nrhs && !st; r0 += chunk) {
    int nr = std::min(chunk, nrhs - r0);
    cdl *Bp = B + (size_t)r0 * ldb;
    k_gather_rows<cdl><<<dim3((N + 255) / 256, nr), 256, 0, stream()>>>(N, nr, m->d_perm, Bp, ldb, T, N);
    if (cudaGetLastError() != cudaSuccess) { set_error("lu_solve_many: launch failed"); st = BG_ERR_CUDA; break; }
    g_launches++;
    if ((st = trsm<cdl>(N, nr, A, m->ld, T, N, 0))) break;
    if ((st = trsm<cdl>(N, nr, A, m->ld, T, N, 1))) break;
    cudaError_t e = cudaMemcpy2DAsync(Bp, sizeof(cdl) * ldb, T, sizeof(cdl) * N, sizeof(cdl) * N, nr,
                                      cudaMemcpyDeviceToDevice, stream());
    if (e != cudaSuccess) { set_error("lu_solve_many: %s", cudaGetErrorString(e)); st = BG_ERR_CUDA; }
  }
  t_pdl = false;
  t_i8 = nullptr;
  if (sc.p) {
    cudaError_t e = cudaMemcpyAsync(&tcerr, sc.err, sizeof(int), cudaMemcpyDeviceToHost, stream());
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream());
    cudaFreeAsync(sc.p, stream());
    if (!st && e != cudaSuccess) { set_error("lu_solve_many: %s", cudaGetErrorString(e)); st = BG_ERR_CUDA; }
    if (!st && tcerr) { set_error("lu_solve_many: a tensor-core wait timed out (code %d)", tcerr); st = BG_ERR_CUDA; }
  }
  cudaFreeAsync(T, stream());
  return st;
}

int lu_solve(bg_matrix *m, void *dB, int ldb, int nrhs) {
  if (!m->d_perm) { set_error("solve: factorization state missing"); return BG_ERR_STATE; }
  if (m->precision == BG_C128) return getrs<cdl>(m, (cdl *)dB, (size_t)ldb, nrhs);
  return getrs<cfl>(m, (cfl *)dB, (size_t)ldb, nrhs);
}

// error word of the triangular sweeps (0 = ok)
int lu_solve_status(bg_matrix *m) {
  if (!m->d_perm) return BG_OK;
  int N = m->N, nb = (N + TV_B - 1) / TV_B, e = 0;
  BG_CUDA_TRY(cudaMemcpyAsync(&e, m->d_perm + N + 2 * nb + 2, sizeof(int), cudaMemcpyDeviceToHost, stream()));
  BG_CUDA_TRY(cudaStreamSynchronize(stream()));
  if (e) { set_error("triangular solve timed out waiting for a block (code %d)", e); return BG_ERR_CUDA; }
  return BG_OK;
}


// =========================================================================
// Allocation-free variant of the device solve.
//
// Some callers cannot allocate GPU memory at solve time: a host application
// whose framework has already reserved the device memory for its own pool,
// or a time-critical loop that cannot accept an allocation's possible failure
// or implicit synchronisation.  For them the gather buffer of the solve lives
// in this fixed device array instead of a stream-ordered allocation.  The
// array (NOALLOC_BYTES) is held by every GPU that loads the library until the
// process exits.  All calls share it: it keeps the last call's contents, and
// two calls whose work overlaps on the GPU would race on it (calls through
// this library are ordered on its single stream).  The gather overwrites the
// part of the array a call uses before it is read, so nothing in it has to
// start at zero; the sweep tickets that must start at zero live beside the
// factors and are cleared by every call.
// =========================================================================
#define NOALLOC_BYTES (4u << 20)
static __device__ __align__(256) unsigned char g_noalloc_scratch[NOALLOC_BYTES];
static void *s_noalloc_ptr[64];
static std::mutex s_noalloc_mu;

// once per device, with that device current: the array's device address (the
// host-side symbol is only a stand-in and must never be passed to a kernel)
static int noalloc_setup(void **ptr) {
  int dev = 0;
  BG_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) { set_error("device ordinal %d out of range", dev); return BG_ERR_CUDA; }
  std::lock_guard<std::mutex> lock(s_noalloc_mu);
  if (!s_noalloc_ptr[dev]) {
    void *p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess || !p) {
      set_error("cudaGetSymbolAddress of the solve scratch failed: %s", cudaGetErrorString(e));
      return BG_ERR_CUDA;
    }
    s_noalloc_ptr[dev] = p;
  }
  *ptr = s_noalloc_ptr[dev];
  return BG_OK;
}

template <class C>
static int getrs_noalloc(bg_matrix *m, C *B, size_t ldb, int nrhs, void *scratch) {
  int N = m->N;
  const C *A = (const C *)m->d;
  const int nb = (N + TV_B - 1) / TV_B;
  int *flagsL = m->d_perm + N, *flagsU = flagsL + nb, *tick = flagsU + nb, *err = tick + 2;
  const int smem = trsv_smem<C>();
  BG_CUDA_TRY(cudaFuncSetAttribute(k_trsv<C, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  BG_CUDA_TRY(cudaFuncSetAttribute(k_trsv<C, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  C *T = (C *)scratch;
  k_gather_rows<C><<<dim3((N + 255) / 256, nrhs), 256, 0, stream()>>>(N, nrhs, m->d_perm, B, ldb, T, N);
  BG_LAUNCHED();
  int epoch = ++m->solve_epoch;
  BG_CUDA_TRY(cudaMemsetAsync(tick, 0, 2 * sizeof(int), stream()));
  k_trsv<C, false><<<nb, 128, smem, stream()>>>(N, A, m->ld, T, N, nrhs, flagsL, epoch, tick, err);
  BG_LAUNCHED();
  k_trsv<C, true><<<nb, 128, smem, stream()>>>(N, A, m->ld, T, N, nrhs, flagsU, epoch, tick + 1, err);
  BG_LAUNCHED();
  BG_CUDA_TRY(cudaMemcpy2DAsync(B, sizeof(C) * ldb, T, sizeof(C) * N, sizeof(C) * N, nrhs, cudaMemcpyDeviceToDevice,
                                stream()));
  return BG_OK;
}

int lu_noalloc_check(const bg_matrix *m, int nrhs) {
  size_t esz = m->precision == BG_C128 ? sizeof(cdl) : sizeof(cfl);
  if (nrhs > TV_MAXRHS) {
    set_error("allocation-free solve: at most %d right-hand sides per call (got %d)", TV_MAXRHS, nrhs);
    return BG_ERR_ARG;
  }
  if ((size_t)m->N * nrhs * esz > NOALLOC_BYTES) {
    set_error("allocation-free solve: N*nrhs*%zu = %zu bytes exceeds its fixed %u-byte scratch", esz,
              (size_t)m->N * nrhs * esz, NOALLOC_BYTES);
    return BG_ERR_ARG;
  }
  return BG_OK;
}

int lu_solve_noalloc(bg_matrix *m, void *dB, int ldb, int nrhs) {
  int st0 = lu_noalloc_check(m, nrhs);
  if (st0) return st0;
  if (!m->d_perm) { set_error("solve: factorization state missing"); return BG_ERR_STATE; }
  void *scratch = nullptr;
  int st = noalloc_setup(&scratch);
  if (st) return st;
  if (m->precision == BG_C128) st = getrs_noalloc<cdl>(m, (cdl *)dB, (size_t)ldb, nrhs, scratch);
  else st = getrs_noalloc<cfl>(m, (cfl *)dB, (size_t)ldb, nrhs, scratch);
  if (!st) st = lu_solve_status(m);
  return st;
}

// =========================================================================
// Capture-safe factor and solve for the batched frequency sweeps: no host
// synchronisation and no allocation between lu_capture_prepare() and the
// end of the solve, so the whole sequence can be recorded into a CUDA graph
// and replayed.  The pivot permutation is built on the device, the
// factorisation status stays in the workspace (lu_capture_info), and the
// solve clears its ready flags itself on every replay (epoch 1).
// =========================================================================

// perm = composition of the interchanges ipiv (1-based), one block; the
// sequential swaps run in shared memory when 8 N bytes fit, else in global
__global__ void k_build_perm(int N, const int *ipiv, int *perm, int use_smem) {
  extern __shared__ int sp[];
  int *p = use_smem ? sp : perm;
  const int *iv = ipiv;
  int *ivs = use_smem ? sp + N : nullptr;
  for (int i = threadIdx.x; i < N; i += blockDim.x) {
    p[i] = i;
    if (use_smem) ivs[i] = ipiv[i];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const int *q = use_smem ? ivs : iv;
    for (int i = 0; i < N; i++) {
      int j = q[i] - 1, t = p[i];
      p[i] = p[j];
      p[j] = t;
    }
  }
  __syncthreads();
  if (use_smem)
    for (int i = threadIdx.x; i < N; i += blockDim.x) perm[i] = p[i];
}

// allocates everything the captured factor/solve touch (complex128 only)
int lu_capture_prepare(bg_matrix *m) {
  int st = ensure_device();
  if (!st) st = panel_init();
  if (st) return st;
  if (m->precision != BG_C128) { set_error("batched sweeps factor complex128 matrices"); return BG_ERR_ARG; }
  int N = m->N;
  if (lu_work_alloc(m, lu_work_bytes(m) + i8_factor_bytes(N)) != BG_OK) {
    cudaGetLastError();        // no room for the INT8 products' scratch: without
    if ((st = lu_work_alloc(m, lu_work_bytes(m)))) return st;
  }
  if (!m->d_perm) BG_CUDA_TRY(cudaMalloc(&m->d_perm, sizeof(int) * (N + 2 * ((N + TV_B - 1) / TV_B) + 8)));
  BG_CUDA_TRY(cudaMemsetAsync(m->d_perm + N, 0, sizeof(int) * (2 * ((N + TV_B - 1) / TV_B) + 8), stream()));
  BG_CUDA_TRY(cudaStreamSynchronize(stream()));
  static bool attr = false;
  if (!attr) {
    BG_CUDA_TRY(cudaFuncSetAttribute(k_build_perm, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    attr = true;
  }
  return BG_OK;
}

void lu_set_panel_rows(int rows) { panel_rows_target = std::max(8, rows); }
int lu_get_panel_rows() { return panel_rows_target; }

int lu_factor_enqueue(bg_matrix *m) {
  int N = m->N;
  char *w = (char *)m->d_work;
  LUWork W;
  W.slots = (unsigned long long *)w; w += PRG_BYTES;
  W.crow = (void *)w; w += sizeof(cdl) * 2 * panel_grid * 32;
  W.jrow = (void *)w; w += sizeof(cdl) * 64;
  W.cval = (double *)w; w += sizeof(double) * 2 * panel_grid;
  W.cidx = (int *)w; w += sizeof(int) * 2 * panel_grid;
  W.info = (int *)w;
  w += 256;
  BG_CUDA_TRY(cudaMemsetAsync(W.info, 0, 2 * sizeof(int), stream()));
  I8Scratch sc{w, i8_factor_bytes(N), W.info + 1};
  if (sc.bytes && m->work_bytes >= lu_work_bytes(m) + sc.bytes) t_i8 = &sc;
  int st = getrf_rec<cdl>(m, W, 0, N);
  t_i8 = nullptr;
  if (st) return st;
  int use_smem = (size_t)8 * N <= 200 * 1024;
  k_build_perm<<<1, 1024, use_smem ? 8 * (size_t)N : 0, stream()>>>(N, m->d_ipiv, m->d_perm, use_smem);
  BG_LAUNCHED();
  m->factored = true;
  return BG_OK;
}

// device address of the factorisation status of the last captured factor
// (LAPACK info; 0 = ok) and of the triangular sweeps' sticky error word
int *lu_capture_info_ptr(bg_matrix *m) {
  char *w = (char *)m->d_work + PRG_BYTES + sizeof(cdl) * 2 * panel_grid * 32 + sizeof(cdl) * 64 +
            sizeof(double) * 2 * panel_grid + sizeof(int) * 2 * panel_grid;
  return (int *)w;
}
int *lu_capture_solve_err_ptr(bg_matrix *m) {
  int nb = (m->N + TV_B - 1) / TV_B;
  return m->d_perm + m->N + 2 * nb + 2;
}

// B (N x nrhs, nrhs <= TV_MAXRHS) <- A^{-1} B with T an N x nrhs device scratch
int lu_solve_enqueue(bg_matrix *m, void *dB, int ldb, int nrhs, void *dT) {
  int N = m->N;
  if (nrhs > TV_MAXRHS) { set_error("captured solve: at most %d right-hand sides", TV_MAXRHS); return BG_ERR_ARG; }
  const cdl *A = (const cdl *)m->d;
  cdl *B = (cdl *)dB, *T = (cdl *)dT;
  const int nb = (N + TV_B - 1) / TV_B;
  int *flagsL = m->d_perm + N, *flagsU = flagsL + nb, *tick = flagsU + nb, *err = tick + 2;
  const int smem = trsv_smem<cdl>();
  static bool attr = false;
  if (!attr) {
    BG_CUDA_TRY(cudaFuncSetAttribute(k_trsv<cdl, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    BG_CUDA_TRY(cudaFuncSetAttribute(k_trsv<cdl, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    attr = true;
  }
  BG_CUDA_TRY(cudaMemsetAsync(flagsL, 0, sizeof(int) * (2 * nb + 2), stream()));
  k_gather_rows<cdl><<<dim3((N + 255) / 256, nrhs), 256, 0, stream()>>>(N, nrhs, m->d_perm, B, ldb, T, N);
  BG_LAUNCHED();
  k_trsv<cdl, false><<<nb, 128, smem, stream()>>>(N, A, m->ld, T, N, nrhs, flagsL, 1, tick, err);
  BG_LAUNCHED();
  k_trsv<cdl, true><<<nb, 128, smem, stream()>>>(N, A, m->ld, T, N, nrhs, flagsU, 1, tick + 1, err);
  BG_LAUNCHED();
  BG_CUDA_TRY(cudaMemcpy2DAsync(B, sizeof(cdl) * ldb, T, sizeof(cdl) * N, sizeof(cdl) * N, nrhs,
                                cudaMemcpyDeviceToDevice, stream()));
  return BG_OK;
}

}  // namespace bg
