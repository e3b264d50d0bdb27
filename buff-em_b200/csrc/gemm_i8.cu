// C <- C - A B, complex128, on the INT8 tensor cores (tcgen05, kind::i8).
//
// The update of a factorisation is FP64-pipe bound (37 TFLOP/s); the INT8 path
// is about 120 times faster, so each operand is split exactly into I8_S = 8
// signed bytes (method: K. Ozaki, T. Ogita, S. Oishi, S. Rump, "Error-free
// transformations of matrix multiplication by using fast routines of matrix
// multiplication and its applications", Numer. Algorithms 59, 2012; its integer
// form: H. Ootomo, K. Ozaki, R. Yokota, 2024).  Row m of A is scaled by the
// power of two above its largest part, X = rint(a 2^(62 - e)) is a 63-bit
// integer, and with balanced base-256 digits a = 2^e sum_i a_i 2^(2 - 8 i),
// a_i in [-128, 127]; the same for the columns of B.  Products of digits are
// summed exactly in 32-bit integers, all products with i + j = d in one
// accumulator, d = 2 .. 9; products with i + j > 9 are below 2^-60 of the
// largest product of the row and the column and are left out.  The eight sums
// are added in FP64 from the smallest up, in two halves, so C is rounded twice per
// call and 2,048 columns of K, where a chain of fused multiply-adds rounds it K
// times.
//
// Real embedding: A as M x 2K (re, im interleaved along K), B as 2K x 2N with
// columns (br, -bi) and (bi, br), so that columns 2n, 2n + 1 of the product are
// the two parts of column n.
//
// Kernel: persistent, tiles of 128 rows x 128 real columns in two passes over K:
// first the digit products with d = 6 .. 9, then (half of the digits) d = 2 .. 5,
// four accumulators of 128 columns = all 512 TMEM columns each time.  Stages of
// 32 bytes of K of all 16 slices (64 KB, two contiguous copies; half of it in the
// second pass), three deep; warp 0 loads, warp 1 issues the 26 or 10 MMAs of a
// stage, warps 2-17 combine and update C.  Every wait is bounded; on a timeout
// the error word is set, copies in flight are waited for and TMEM is freed.
//
// What bounds it: shared memory, 8 KB of operands read per 128 x 128 x 32 MMA and
// 96 KB written per 36 of them, 85 cycles an MMA at 128 bytes where the arithmetic
// takes 64, and the combinations, which no second set of accumulators can hide
// (8.9 us a tile).  All eight sums of a 64-column tile at once took less of C's
// traffic but 57 cycles per half as large an MMA (a 64-column MMA alone runs at
// 3.04 of 4.56 POP/s): 12.9 ms for 9936 x 9936 x 1024; a CTA pair (256 rows, half
// of B in each) 14.9.  Now 11.0 (73 TFLOP/s; 84 at 4096^3), FP64 tiles 24.9 (32.5);
// 1024^3: 0.304 -> 0.163 ms.  Factorisation of N = 19,872: products 660 -> 315 ms.  Error
// of 1024 x 1024 x 2048 products against 80-bit sums: rms 2.1e-17 of the largest
// entry (FP64 tiles 3.7e-16 at 512 x 512 x 2048).
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstdio>

#include "internal.h"
#include "tcgen05.cuh"

namespace bg {

struct z2i { double r, i; };

#define I8_S 8                    // digits per number
#define I8_BM 128                 // rows of a tile
#define I8_BN 128                 // real columns of a tile (64 complex)
#define I8_BK 32                  // bytes of K per stage: one MMA deep, one 32-byte swizzle row
#define I8_STAGES 3
#define I8_GROUP 16               // row blocks per raster group
#define I8_THREADS 576
#define I8_A_BYTES (I8_S * I8_BM * I8_BK)
#define I8_B_BYTES (I8_S * I8_BN * I8_BK)
#define I8_STAGE (I8_A_BYTES + I8_B_BYTES)
#define I8_SMEM (I8_STAGES * I8_STAGE + 1024 + 256)

struct I8Args {
  int M, N, nk;                   // rows, complex columns, K blocks
  const int8_t *A, *B;            // digit blocks
  z2i *C;
  size_t ldc;
  const double *sa, *sb;          // scale of each row of A and column of B
  int *err;
  int ntm, ntn;
};

__device__ __forceinline__ void i8_tile(const I8Args &P, int t, int &tm, int &tn) {
  const int per = I8_GROUP * P.ntn;
  const int g = t / per, w = t - g * per;
  const int gm = min(I8_GROUP, P.ntm - g * I8_GROUP);
  tn = w / gm;
  tm = g * I8_GROUP + (w - tn * gm);
}

// a 256 + b as a double, exactly (|a|, |b| < 2^31)
__device__ __forceinline__ double pair_to_double(int a, int b) {
  const long long y = (long long)a * 256 + b;
  return __longlong_as_double(y + 0x4338000000000000ll) - 6755399441055744.0;   // 1.5 2^52
}

__global__ void __launch_bounds__(I8_THREADS, 1)
    k_zgemm_i8(const I8Args P) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char *ring = (unsigned char *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t *full = (uint64_t *)(ring + I8_STAGES * I8_STAGE);
  uint64_t *empty = full + I8_STAGES;
  uint64_t *acc_full = empty + I8_STAGES, *acc_empty = acc_full + 1, *mma_done = acc_empty + 1;
  uint32_t *tmem_slot = (uint32_t *)(mma_done + 1);
  __shared__ volatile int s_fail;
  __shared__ int s_issued, s_consumed;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nk = P.nk;
  const int ntiles = P.ntm * P.ntn;

  if (threadIdx.x == 0) {
    for (int s = 0; s < I8_STAGES; s++) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    mbar_init(acc_full, 1);
    mbar_init(acc_empty, 16);
    mbar_init(mma_done, 1);
    s_fail = 0;
    s_issued = 0;
    s_consumed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      int kc = 0;
      for (int t = blockIdx.x; t < ntiles && !s_fail; t += gridDim.x) {
        int tm, tn;
        i8_tile(P, t, tm, tn);
        for (int it = 0; it < 2 * nk; it++, kc++) {
          const int s = kc % I8_STAGES, kb = it < nk ? it : it - nk, half = it < nk ? 1 : 2;   // pass 1: digits 0 .. 3
          if (kc >= I8_STAGES && !mbar_wait(&empty[s], ((kc / I8_STAGES) - 1) & 1)) { s_fail = 1; break; }
          unsigned char *sa = ring + s * I8_STAGE;
          mbar_expect_tx(&full[s], I8_STAGE / half);
          bulk_load(sa, P.A + ((size_t)tm * nk + kb) * I8_A_BYTES, I8_A_BYTES / half, &full[s]);
          bulk_load(sa + I8_A_BYTES, P.B + ((size_t)tn * nk + kb) * I8_B_BYTES, I8_B_BYTES / half, &full[s]);
          s_issued = kc + 1;
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      // instruction descriptor, kind::i8: D s32 (2 at bits 4-5), A and B signed
      // 8-bit (1 at bits 7-9 and 10-12), both K-major, N>>3 at 17-22, M>>4 at 24-28
      const uint32_t idesc = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(I8_BN >> 3) << 17) |
                             ((uint32_t)(I8_BM >> 4) << 24);
      auto mma = [&](uint32_t d, uint64_t da, uint64_t db, uint32_t acc) {
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}"
            ::"r"(d), "l"(da), "l"(db), "r"(idesc), "r"(acc));
      };
      int kc = 0, i = 0;      // i: passes of this CTA so far
      for (int t = blockIdx.x; t < ntiles && !s_fail; t += gridDim.x) {
#pragma unroll
        for (int pass = 0; pass < 2; pass++, i++) {
          if (s_fail) break;
          if (i >= 1 && !mbar_wait(acc_empty, (i - 1) & 1)) { s_fail = 4; break; }
          asm volatile("tcgen05.fence::after_thread_sync;");
          for (int kb = 0; kb < nk; kb++, kc++) {
            const int s = kc % I8_STAGES;
            if (!mbar_wait(&full[s], (kc / I8_STAGES) & 1)) { s_fail = 2; break; }
            asm volatile("tcgen05.fence::after_thread_sync;");
            const uint32_t sa = smem_u32(ring + s * I8_STAGE);
            const uint64_t da0 = sw32_desc(sa), db0 = sw32_desc(sa + I8_A_BYTES);
            // pass 0: a + b = 4 .. 7, pass 1: a + b = 0 .. 3, each group first met at a = 0
#pragma unroll
            for (int a = 0; a < (pass ? 4 : I8_S); a++)
#pragma unroll
              for (int b = 0; b < I8_S; b++) {
                const int g = a + b - (pass ? 0 : 4);
                if (g < 0 || g > 3) continue;
                mma(tmem + (uint32_t)(g * I8_BN), da0 + ((a * I8_BM * I8_BK) >> 4), db0 + ((b * I8_BN * I8_BK) >> 4),
                    (kb > 0 || a > 0) ? 1u : 0u);
              }
            mma_commit(&empty[s]);
            s_consumed = kc + 1;
          }
          if (s_fail) break;
          mma_commit(acc_full);
        }
      }
      // no MMA may still run when the TMEM is freed, whichever way the loop ended
      mma_commit(mma_done);
      if (!mbar_wait(mma_done, 0) && !s_fail) s_fail = 5;
    }
  } else {
    // warps 2 .. 17: TMEM lanes 32 (warp % 4) .. + 31, 16 complex columns each
    const int q = warp & 3, h = (warp - 2) >> 2;
    int i = 0;
    for (int t = blockIdx.x; t < ntiles && !s_fail; t += gridDim.x) {
      int tm, tn;
      i8_tile(P, t, tm, tn);
      const int row = tm * I8_BM + q * 32 + lane, col0 = tn * (I8_BN / 2) + 16 * h;
      z2i *pc = P.C + (size_t)col0 * P.ldc + row;
      double sa = row < P.M ? P.sa[row] * 0x1p-32 : 0.0;      // the second pass's groups weigh 2^32 more
#pragma unroll 1
      for (int pass = 0; pass < 2; pass++, i++) {
        // eight columns of C ahead: the first before the accumulators are ready
        z2i cv[8];
#pragma unroll
        for (int j = 0; j < 8; j++)
          cv[j] = row < P.M && col0 + j < P.N ? pc[(size_t)j * P.ldc] : z2i{0.0, 0.0};
        if (!mbar_wait(acc_full, i & 1)) { s_fail = 3; break; }
        asm volatile("tcgen05.fence::after_thread_sync;");
#pragma unroll
        for (int c = 0; c < 16; c += 2) {      // two complex = four real columns at a time
          uint32_t r[4][4];
          const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(32 * h + 2 * c);
#pragma unroll
          for (int g = 0; g < 4; g++)
            asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                         : "=r"(r[g][0]), "=r"(r[g][1]), "=r"(r[g][2]), "=r"(r[g][3])
                         : "r"(taddr + (uint32_t)(g * I8_BN)));
          asm volatile("tcgen05.wait::ld.sync.aligned;");
          double v[4];
#pragma unroll
          for (int x = 0; x < 4; x++)
            v[x] = fma(pair_to_double((int)r[2][x], (int)r[3][x]), 0x1p-16, pair_to_double((int)r[0][x], (int)r[1][x])) * sa;
#pragma unroll
          for (int j = 0; j < 2; j++)
            if (row < P.M && col0 + c + j < P.N) {
              const double sb = P.sb[col0 + c + j];
              z2i &x = cv[(c + j) & 7];
              pc[(size_t)(c + j) * P.ldc] = z2i{fma(-v[2 * j], sb, x.r), fma(-v[2 * j + 1], sb, x.i)};
              if (c < 8 && col0 + c + j + 8 < P.N) x = pc[(size_t)(c + j + 8) * P.ldc];
            }
        }
        sa *= 0x1p+32;
        asm volatile("tcgen05.fence::before_thread_sync;");
        __syncwarp();
        if (lane == 0) mbar_arrive(acc_empty);
      }
    }
  }
  __syncthreads();
  if (s_fail && threadIdx.x == 0) {
    atomicExch(P.err, s_fail);
    for (int c = s_consumed; c < s_issued; c++) mbar_wait(&full[c % I8_STAGES], (c / I8_STAGES) & 1);
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
}

// ------------------------------------------------------------------ splitting
// largest |part| as ordered bits; NaN and infinity lie above every number
__device__ __forceinline__ unsigned long long abs_bits(double x) {
  return (unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffull;
}
// e with |x| < 2^e for the largest part (bits mx); zeros and denormals: -1022
__device__ __forceinline__ int top_exp(unsigned long long mx) { return (int)(mx >> 52) - 1022; }
__device__ __forceinline__ double pow2(int e) {   // -1022 <= e <= 1023
  return __longlong_as_double((long long)(e + 1023) << 52);
}
// 2^(e - 10): the two scales carry the 2^-20 of the digit weights; not a number
// where the row or column holds one (every product with it then is none)
__device__ __forceinline__ double digit_scale(unsigned long long mx) {
  if (mx >= 0x7ff0000000000000ull) return __longlong_as_double(0x7ff8000000000000ll);
  const int e = top_exp(mx);
  return pow2(e / 2) * pow2(e - e / 2 - 10);
}
// digits of x: byte 7 the leading one
struct DigitScale { double f, g; };
__device__ __forceinline__ DigitScale split_scale(unsigned long long mx) {
  const int e = 62 - top_exp(mx), h = e / 2;
  return DigitScale{pow2(h), pow2(e - h)};
}
__device__ __forceinline__ unsigned long long digits(long long X) {
  return ((unsigned long long)X + 0x0080808080808080ull) ^ 0x0080808080808080ull;
}
__device__ __forceinline__ long long to_int(double x, DigitScale s) { return __double2ll_rn(x * s.f * s.g); }

// byte b of four numbers as one word, for the eight b: w[0] the leading digit
__device__ __forceinline__ void transpose8(const unsigned long long (&d)[4], uint32_t (&w)[8]) {
#pragma unroll
  for (int half = 0; half < 2; half++) {
    uint32_t x[4];
#pragma unroll
    for (int i = 0; i < 4; i++) x[i] = half ? (uint32_t)d[i] : (uint32_t)(d[i] >> 32);
    const uint32_t a = __byte_perm(x[0], x[1], 0x5140), b = __byte_perm(x[2], x[3], 0x5140);   // bytes 0, 1
    const uint32_t c = __byte_perm(x[0], x[1], 0x7362), e = __byte_perm(x[2], x[3], 0x7362);   // bytes 2, 3
    w[4 * half + 3] = __byte_perm(a, b, 0x5410);
    w[4 * half + 2] = __byte_perm(a, b, 0x7632);
    w[4 * half + 1] = __byte_perm(c, e, 0x5410);
    w[4 * half + 0] = __byte_perm(c, e, 0x7632);
  }
}

__global__ void __launch_bounds__(128) k_i8_rowmax(int M, int K, const z2i *A, size_t lda, unsigned long long *mx) {
  const int m = blockIdx.x * 128 + threadIdx.x, k0 = blockIdx.y * 32, k1 = min(K, k0 + 32);
  if (m >= M) return;
  unsigned long long x = 0;
#pragma unroll 8
  for (int k = k0; k < k1; k++) {
    const z2i a = A[(size_t)k * lda + m];
    x = max(x, max(abs_bits(a.r), abs_bits(a.i)));
  }
  atomicMax(mx + m, x);
}

// Digit blocks: 32 bytes of K (16 columns, re and im interleaved) of 128 rows of
// A or 128 rows of B, [digit][row][32 bytes], one contiguous piece per block in the
// order the stages read them, the two 16-byte halves of a row exchanged where
// bit 2 of the row is set (the tensor core's 32-byte swizzle).  Loads are then
// whole lines; as planes of rows, a stage read half a line per row.
__device__ __forceinline__ size_t digit_row(int row, int kb, int nk, int rows) {
  return ((size_t)(row / rows) * nk + kb) * (I8_S * rows * I8_BK) + (row % rows) * I8_BK;
}

// a thread takes one row and 16 columns
__global__ void __launch_bounds__(128) k_i8_slice_a(int M, int K, const z2i *A, size_t lda,
                                                    const unsigned long long *mx, int8_t *S, int nk, double *sa) {
  const int m = blockIdx.x * 128 + threadIdx.x, k0 = blockIdx.y * 16;
  if (m >= M) return;
  const unsigned long long top = mx[m];
  const DigitScale sc = split_scale(top);
  if (blockIdx.y == 0) sa[m] = digit_scale(top);
  int8_t *p = S + digit_row(m, blockIdx.y, nk, I8_BM);
#pragma unroll
  for (int h = 0; h < 2; h++) {
    uint32_t w[4][8];
    z2i a[8];
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const int k = k0 + 8 * h + i;
      a[i] = k < K ? A[(size_t)k * lda + m] : z2i{0.0, 0.0};
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const unsigned long long d[4] = {digits(to_int(a[2 * i].r, sc)), digits(to_int(a[2 * i].i, sc)),
                                       digits(to_int(a[2 * i + 1].r, sc)), digits(to_int(a[2 * i + 1].i, sc))};
      transpose8(d, w[i]);
    }
    const int o = 16 * (h ^ ((m >> 2) & 1));
#pragma unroll
    for (int s = 0; s < I8_S; s++)
      *(uint4 *)(p + s * (I8_BM * I8_BK) + o) = make_uint4(w[0][s], w[1][s], w[2][s], w[3][s]);
  }
}

// slices of B, K <= I8_KC: a block takes a column; rows 2n: (br, -bi), 2n + 1: (bi, br)
#define I8_KC 2048
__global__ void __launch_bounds__(I8_KC / 8) k_i8_slice_b(int K, const z2i *B, size_t ldb, int8_t *S, int nk, double *sb) {
  const int n = blockIdx.x, t = threadIdx.x;
  const z2i *b = B + (size_t)n * ldb;
  z2i v[4][2];
  unsigned long long x = 0;
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int k = 2 * t + I8_KC / 4 * i + h;
      v[i][h] = k < K ? b[k] : z2i{0.0, 0.0};
      x = max(x, max(abs_bits(v[i][h].r), abs_bits(v[i][h].i)));
    }
  __shared__ unsigned long long red[I8_KC / 256];
  for (int o = 16; o > 0; o >>= 1) x = max(x, __shfl_xor_sync(0xffffffffu, x, o));
  if ((t & 31) == 0) red[t >> 5] = x;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < I8_KC / 256; i++) x = max(x, red[i]);
  const DigitScale sc = split_scale(x);
  if (t == 0) sb[n] = digit_scale(x);
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int k = 2 * t + I8_KC / 4 * i;
    if (k / 16 >= nk) continue;
    long long r[2], m[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
      r[h] = to_int(v[i][h].r, sc);
      m[h] = to_int(v[i][h].i, sc);
    }
    uint32_t w0[8], w1[8];
    const unsigned long long d0[4] = {digits(r[0]), digits(-m[0]), digits(r[1]), digits(-m[1])};
    const unsigned long long d1[4] = {digits(m[0]), digits(r[0]), digits(m[1]), digits(r[1])};
    transpose8(d0, w0);
    transpose8(d1, w1);
    int8_t *p = S + digit_row(2 * n, k / 16, nk, I8_BN);
    const int o = 2 * (k % 16) ^ (((2 * n) >> 2) & 1) * 16;      // rows 2n and 2n + 1: the same half
#pragma unroll
    for (int s = 0; s < I8_S; s++) {
      *(uint32_t *)(p + s * (I8_BN * I8_BK) + o) = w0[s];
      *(uint32_t *)(p + s * (I8_BN * I8_BK) + I8_BK + o) = w1[s];
    }
  }
}

// ------------------------------------------------------------------ host side
#define I8_MC 4096                // rows of A and complex columns of B sliced at a time at most
#define I8_NC 4096

static size_t up256(size_t x) { return (x + 255) & ~(size_t)255; }

// digits of r rows (in whole blocks) and k columns
static size_t digit_bytes(int r, int rows, int k) {
  return up256((size_t)((r + rows - 1) / rows) * ((k + 15) / 16) * (I8_S * rows * I8_BK));
}
// scratch for products of at most M x N x K
size_t zgemm_i8_bytes(int M, int N, int K) {
  const int mc = std::min(M, I8_MC), nc = std::min(N, I8_NC), kc = std::min(K, I8_KC);
  return digit_bytes(mc, I8_BM, kc) + digit_bytes(2 * nc, I8_BN, kc) + up256(8 * mc) * 2 + up256(8 * nc);
}

// C -= A B with the scratch `work` of `bytes`; err: device int, nonzero after a failed wait
int zgemm_i8(int M, int N, int K, const void *Av, size_t lda, const void *Bv, size_t ldb, void *Cv, size_t ldc,
             void *work, size_t bytes, int *err) {
  static int sms = 0;
  if (!sms) {
    int dev = 0;
    BG_CUDA_TRY(cudaGetDevice(&dev));
    BG_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    BG_CUDA_TRY(cudaFuncSetAttribute(k_zgemm_i8, cudaFuncAttributeMaxDynamicSharedMemorySize, I8_SMEM));
  }
  if (zgemm_i8_bytes(M, N, K) > bytes) { set_error("zgemm: scratch too small"); return BG_ERR_STATE; }
  const z2i *A = (const z2i *)Av, *B = (const z2i *)Bv;
  z2i *C = (z2i *)Cv;
  const int mc = std::min(M, I8_MC), nc = std::min(N, I8_NC), kc = std::min(K, I8_KC);
  char *w = (char *)work;
  int8_t *Sa = (int8_t *)w; w += digit_bytes(mc, I8_BM, kc);
  int8_t *Sb = (int8_t *)w; w += digit_bytes(2 * nc, I8_BN, kc);
  unsigned long long *mx = (unsigned long long *)w; w += up256(8 * mc);
  double *sa = (double *)w; w += up256(8 * mc);
  double *sb = (double *)w;
  for (int k0 = 0; k0 < K; k0 += kc) {
    const int kk = std::min(kc, K - k0), nk = (kk + 15) / 16;
    for (int n0 = 0; n0 < N; n0 += nc) {
      const int nn = std::min(nc, N - n0);
      k_i8_slice_b<<<nn, I8_KC / 8, 0, stream()>>>(kk, B + k0 + (size_t)n0 * ldb, ldb, Sb, nk, sb);
      BG_LAUNCHED();
      for (int m0 = 0; m0 < M; m0 += mc) {
        const int mm = std::min(mc, M - m0);
        const z2i *Am = A + m0 + (size_t)k0 * lda;
        BG_CUDA_TRY(cudaMemsetAsync(mx, 0, 8 * (size_t)mm, stream()));
        k_i8_rowmax<<<dim3((mm + 127) / 128, (kk + 31) / 32), 128, 0, stream()>>>(mm, kk, Am, lda, mx);
        BG_LAUNCHED();
        k_i8_slice_a<<<dim3((mm + 127) / 128, nk), 128, 0, stream()>>>(mm, kk, Am, lda, mx, Sa, nk, sa);
        BG_LAUNCHED();
        I8Args P{mm, nn, nk, Sa, Sb, C + m0 + (size_t)n0 * ldc, ldc, sa, sb, err,
                 (mm + I8_BM - 1) / I8_BM, (2 * nn + I8_BN - 1) / I8_BN};
        k_zgemm_i8<<<std::min(P.ntm * P.ntn, sms), I8_THREADS, I8_SMEM, stream()>>>(P);
        BG_LAUNCHED();
      }
    }
  }
  return BG_OK;
}

}  // namespace bg
