// C <- C - A B, complex128, on the INT8 tensor cores (tcgen05, kind::i8).
//
// The update of a factorisation is FP64-pipe bound (37 TFLOP/s); the INT8 path
// is about 120 times faster, so each operand is split into I8_S = 8
// signed bytes (method: K. Ozaki, T. Ogita, S. Oishi, S. Rump, "Error-free
// transformations of matrix multiplication by using fast routines of matrix
// multiplication and its applications", Numer. Algorithms 59, 2012; its integer
// form: H. Ootomo, K. Ozaki, R. Yokota, 2024).
//
// Real embedding: A as M x 2K (re, im interleaved along K), B as 2K x 2N with
// columns (br, -bi) and (bi, br), so that columns 2n, 2n + 1 of the product are
// the two parts of column n.
//
// Digits.  Row m of A is scaled by a power of two 2^-e above its largest part,
// X = rint(a 2^(62 - e)) is a 63-bit integer, and with balanced base-256 digits
// a = 2^e sum_i a_i 2^(2 - 8 i), a_i in [-128, 127]; the same for every real
// column of B (scale 2^f).  Products of digits are summed exactly in 32-bit
// integers, all products with i + j = d in one accumulator, d = 2 .. 9.  The
// eight sums are added in FP64 from the smallest up, in two halves, so C is
// rounded twice per call and 2,048 columns of K, where a chain of fused
// multiply-adds rounds it K times.
//
// What the digits lose is relative to the row's and the column's largest part,
// not to the entry.  Rounding the operands to 2^-63 of their scales costs up to
// 2^-62 2^(e + f) per real term, the products left out (seven with i + j = 10, each
// at most 2^-62, and smaller ones) up to 7.03 2^-62: at most K 2^-58 2^(e + f) if
// every digit were extreme, 2^-62 sqrt(2K) 2^(e + f) rms.  A chain of FP64 operations is
// bounded by K 2^-52 S, S = sum |a| |b| over the 2K real terms.  Two things keep the first
// below the second:
//  * the inner index is scaled as well, exactly: real index (k, part) by 2^p in A
//    and 2^-p in B, p = (y - x) / 2 + max(d / 2, d - 6), with x the exponent of column k
//    of A, x - d that of this part of it, y that of row k of B.  Rows or columns
//    of any size, and any diagonal matrix between A and B, then leave the digits as
//    they are (bodies or cells of different size, imaginary parts far below the
//    real ones at low frequency).  Tiles of a factorisation with an entry of S below
//    2^-6 2^(e + f): 13 % at omega = 1, N = 8,262 (with d in full 34 %), 19 % for a
//    lossless body at omega = 0.01 (with d / 2 alone 93 %); without scaling 23 % and 100 %.
//  * a tile is taken only if every entry has S >= 2^-7 2^(e + f) (k_i8_guard); the others
//    go to FP64, as does a product whose operands hold an infinity or a NaN and rows or
//    columns beyond 2^+-900.
// Factors of bodies of N = 4,494, 5,760 and 8,262, entry by entry and part by part
// against 80-bit sums, in units of 2^-53 |L||U|: rms 0.35-0.89, largest 4.3-11; FP64
// products 0.85-2.1 and 9-28; digits without the two 0.8-12 and 29-880.
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
// of B in each) 14.9.  Now 11.4, with the inner scales and the guard 12.0 (67 TFLOP/s),
// FP64 tiles 24.9 (32.5); 1024^3 0.210 ms, FP64 0.304.  Where tiles go to FP64 the product
// takes longer: factorisation of N = 19,872 (omega = 1) 409 -> 469 ms.  Error of
// 1151 x 1000 x 2100 products against 80-bit sums: rms 0.015 of 2^-53 S, FP64 tiles 0.34.
#include <cuda.h>
#include <cuda_fp16.h>
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
  const double *sa, *sb;          // scale of each row of A and real column of B (0: no part, NaN: not in range)
  unsigned char *flag;            // per tile (tn * ntm + tm): left to FP64
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
        if (P.flag[tn * P.ntm + tm]) continue;
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
        int tm, tn;
        i8_tile(P, t, tm, tn);
        if (P.flag[tn * P.ntm + tm]) continue;
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
      if (kc > 0) {      // no MMA may still run when the TMEM is freed, whichever way the loop ended
        mma_commit(mma_done);
        if (!mbar_wait(mma_done, 0) && !s_fail) s_fail = 5;
      }
    }
  } else {
    // warps 2 .. 17: TMEM lanes 32 (warp % 4) .. + 31, 16 complex columns each
    const int q = warp & 3, h = (warp - 2) >> 2;
    int i = 0;
    for (int t = blockIdx.x; t < ntiles && !s_fail; t += gridDim.x) {
      int tm, tn;
      i8_tile(P, t, tm, tn);
      if (P.flag[tn * P.ntm + tm]) continue;
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
              const double2 sb = ((const double2 *)P.sb)[col0 + c + j];
              z2i &x = cv[(c + j) & 7];
              pc[(size_t)(c + j) * P.ldc] = z2i{fma(-v[2 * j], sb.x, x.r), fma(-v[2 * j + 1], sb.y, x.i)};
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

// ------------------------------------------------------------------ guard
// S of every entry of a tile, from below: sums of |a'| |b'| with the scaled parts
// truncated to e5m2 (kind::f8f6f4, FP32 accumulation; a part of 2^15 is the row's
// scale), 128 bytes of K per stage; a tile with an entry below the line (and neither
// its row nor its column zero) is flagged.  1/36 of the digit products' work,
// bound by the stages' copies and the start of each tile; two CTAs per SM so
// that one reads its accumulator while the other loads.  4096 x 4096 x 128:
// 15 us (a pass over 16 columns at a time, every one compared: 36), 2560 x 1536 x 1536: 25.
#define GD_STAGES 3
#define GD_ROWS (128 * 128)       // bytes of 128 rows of a stage
#define GD_STAGE (2 * GD_ROWS)
#define GD_SMEM (GD_STAGES * GD_STAGE + 1024 + 256)
#define GD_THREADS 192
#define GD_LINE 8388608.f         // 2^23 = 2^-7 of 2^15 2^15
struct I8Guard {
  int M, N2, nk;                  // rows, real columns, blocks of 128 bytes of K
  const uint8_t *A, *B;
  const double *sa, *sb;
  unsigned char *flag;
  int *err;
  int ntm, ntn;
};

__global__ void __launch_bounds__(GD_THREADS, 2) k_i8_guard(const I8Guard P) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char *ring = (unsigned char *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t *full = (uint64_t *)(ring + GD_STAGES * GD_STAGE);
  uint64_t *empty = full + GD_STAGES;
  uint64_t *acc_full = empty + GD_STAGES, *acc_empty = acc_full + 1, *mma_done = acc_empty + 1;
  uint32_t *tmem_slot = (uint32_t *)(mma_done + 1);
  __shared__ volatile int s_fail;
  __shared__ int s_issued, s_consumed;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nk = P.nk, ntiles = P.ntm * P.ntn;
  if (threadIdx.x == 0) {
    for (int s = 0; s < GD_STAGES; s++) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    mbar_init(acc_full, 1);
    mbar_init(acc_empty, 4);
    mbar_init(mma_done, 1);
    s_fail = 0;
    s_issued = 0;
    s_consumed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(I8_BN));
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
        const int tm = t % P.ntm, tn = t / P.ntm;
        for (int kb = 0; kb < nk; kb++, kc++) {
          const int s = kc % GD_STAGES;
          if (kc >= GD_STAGES && !mbar_wait(&empty[s], ((kc / GD_STAGES) - 1) & 1)) { s_fail = 1; break; }
          unsigned char *st = ring + s * GD_STAGE;
          mbar_expect_tx(&full[s], GD_STAGE);
          bulk_load(st, P.A + ((size_t)tm * nk + kb) * GD_ROWS, GD_ROWS, &full[s]);
          bulk_load(st + GD_ROWS, P.B + ((size_t)tn * nk + kb) * GD_ROWS, GD_ROWS, &full[s]);
          s_issued = kc + 1;
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      // instruction descriptor, kind::f8f6f4: D f32 (1 at bits 4-5), A and B e5m2 (1 at
      // bits 7-9 and 10-12), both K-major, N>>3 at 17-22, M>>4 at 24-28
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(I8_BN >> 3) << 17) |
                             ((uint32_t)(I8_BM >> 4) << 24);
      int kc = 0, i = 0;
      for (int t = blockIdx.x; t < ntiles && !s_fail; t += gridDim.x, i++) {
        if (i >= 1 && !mbar_wait(acc_empty, (i - 1) & 1)) { s_fail = 4; break; }
        asm volatile("tcgen05.fence::after_thread_sync;");
        for (int kb = 0; kb < nk; kb++, kc++) {
          const int s = kc % GD_STAGES;
          if (!mbar_wait(&full[s], (kc / GD_STAGES) & 1)) { s_fail = 2; break; }
          asm volatile("tcgen05.fence::after_thread_sync;");
          const uint32_t st = smem_u32(ring + s * GD_STAGE);
#pragma unroll
          for (int k = 0; k < 4; k++)
            asm volatile(
                "{\n\t.reg .pred p;\n\t"
                "setp.ne.b32 p, %4, 0;\n\t"
                "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}"
                ::"r"(tmem), "l"(sw128_desc(st + k * 32)), "l"(sw128_desc(st + GD_ROWS + k * 32)), "r"(idesc),
                  "r"((kb > 0 || k > 0) ? 1u : 0u));
          mma_commit(&empty[s]);
          s_consumed = kc + 1;
        }
        if (s_fail) break;
        mma_commit(acc_full);
      }
      if (kc > 0) {      // no MMA may still run when the TMEM is freed, whichever way the loop ended
        mma_commit(mma_done);
        if (!mbar_wait(mma_done, 0) && !s_fail) s_fail = 5;
      }
    }
  } else {
    // warps 2 .. 5: TMEM lanes 32 (warp % 4) .. + 31
    const int q = warp & 3;
    int i = 0;
    for (int t = blockIdx.x; t < ntiles && !s_fail; t += gridDim.x, i++) {
      const int tm = t % P.ntm, tn = t / P.ntm, row = tm * I8_BM + q * 32 + lane;
      const double sa = row < P.M ? P.sa[row] : 0.0;
      bool bad = false;
      if (!mbar_wait(acc_full, i & 1)) { s_fail = 3; break; }
      asm volatile("tcgen05.fence::after_thread_sync;");
#pragma unroll 1
      for (int c0 = 0; c0 < I8_BN; c0 += 32) {
        uint32_t r[32];
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
            "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
              "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
              "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]),
              "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]),
              "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
            : "r"(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)c0));
        asm volatile("tcgen05.wait::ld.sync.aligned;");
        // sums of non-negative terms: their bits order as they do
        uint32_t least = r[0];
#pragma unroll
        for (int j = 1; j < 32; j++) least = min(least, r[j]);
        if (least < __float_as_uint(GD_LINE) && row < P.M) {
#pragma unroll
          for (int j = 0; j < 32; j++) {
            const int col = tn * I8_BN + c0 + j;
            if (r[j] < __float_as_uint(GD_LINE) && col < P.N2) {
              const double sb = P.sb[col];      // an entry with a zero row or column is exact
              bad |= !((sa == 0.0 || sb == 0.0) && sa == sa && sb == sb);
            }
          }
        }
        __syncwarp();
      }
      asm volatile("tcgen05.fence::before_thread_sync;");
      const bool any = __any_sync(0xffffffffu, bad);
      if (lane == 0) {
        mbar_arrive(acc_empty);
        if (any) P.flag[tn * P.ntm + tm] = 1;
      }
    }
  }
  __syncthreads();
  if (s_fail && threadIdx.x == 0) {
    atomicExch(P.err, 10 + s_fail);
    for (int c = s_consumed; c < s_issued; c++) mbar_wait(&full[c % GD_STAGES], (c / GD_STAGES) & 1);
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(I8_BN));
}

// ------------------------------------------------------------------ splitting
// Exponents are integers throughout: e with |x| < 2^e; I8_NONE (what a memset to
// 0x80 leaves) for "no part", I8_OVER for an infinity or a NaN
#define I8_NONE (-2139062144)
#define I8_OVER (1 << 20)
#define I8_RANGE 900              // row and column scales beyond 2^+-900 are left to FP64
__device__ __forceinline__ unsigned long long abs_bits(double x) {
  return (unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffull;
}
__device__ __forceinline__ int exp_of(double x) {      // denormals: -1022
  const unsigned long long b = abs_bits(x);
  return b == 0 ? I8_NONE : b >= 0x7ff0000000000000ull ? I8_OVER : (int)(b >> 52) - 1022;
}
// exponent of x 2^p; p = I8_NONE: the part meets no other (infinities and NaN count all the same)
__device__ __forceinline__ int exp_of(double x, int p) {
  const int e = exp_of(x);
  return e == I8_OVER ? I8_OVER : e == I8_NONE || p == I8_NONE ? I8_NONE : e + p;
}
__device__ __forceinline__ double pow2(int e) {   // -1022 <= e <= 1023
  return __longlong_as_double((long long)(e + 1023) << 52);
}

// Exponents of the inner index: ia[2k + part] of the real columns of A, ib[k] of row k of B
struct I8Inner { const int *ia, *ib; };
// shifts of the two parts of index k (added in A, subtracted in B); I8_NONE: one of
// the operands has no part there and the products with it are zero
__device__ __forceinline__ int2 inner_shift(const I8Inner &I, int k) {
  const int2 a = ((const int2 *)I.ia)[k];
  const int b = I.ib[k], x = max(a.x, a.y);
  if (x == I8_NONE || b == I8_NONE) return make_int2(I8_NONE, I8_NONE);
  const int g = (b - x) >> 1;
  auto part = [&](int a) { return a == I8_NONE ? I8_NONE : g + max((x - a) >> 1, x - a - 6); };
  return make_int2(part(a.x), part(a.y));
}

// 2^(e - 10): the two scales carry the 2^-20 of the digit weights
__device__ __forceinline__ double digit_scale(int e) {
  if (e == I8_NONE) return 0.0;
  return e < -I8_RANGE || e > I8_RANGE ? __longlong_as_double(0x7ff8000000000000ll) : pow2(e - 10);
}
__device__ __forceinline__ bool in_range(int e) { return e >= -I8_RANGE && e <= I8_RANGE; }
// rint(x 2^(62 - e)) of a part x 2^p in a row of scale 2^e
__device__ __forceinline__ long long to_int(double x, int e, int p) {
  const int s = max(-2044, min(2046, 62 - e + p)), h = s / 2;      // |x| 2^s <= 2^62; beyond the limits x is 0 or vanishes
  return __double2ll_rn(x * pow2(h) * pow2(s - h));
}
// digits of X: byte 7 the leading one
__device__ __forceinline__ unsigned long long digits(long long X) {
  return ((unsigned long long)X + 0x0080808080808080ull) ^ 0x0080808080808080ull;
}
// |X| 2^-47 <= 2^15 truncated to e5m2, the upper byte of an FP16 number
__device__ __forceinline__ uint32_t size_of(long long X) {
  const float f = __ull2float_rz((unsigned long long)(X < 0 ? -X : X)) * 0x1p-47f;
  return (uint32_t)__half_as_ushort(__float2half_rz(f)) >> 8;
}

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

// Exponents of the inner index over all of A and B: blocks [0, nA) take a column of
// 2,048 rows of A, the others 64 rows x 64 columns of B
#define I8_INNER_A 2048
__global__ void __launch_bounds__(256) k_i8_inner(int M, int N, int K, const z2i *A, size_t lda, const z2i *B, size_t ldb,
                                                  int nA, int *ia, int *ib) {
  const int tid = threadIdx.x;
  if ((int)blockIdx.x < nA) {
    const int k = blockIdx.x % K, m0 = blockIdx.x / K * I8_INNER_A, m1 = min(M, m0 + I8_INNER_A);
    int er = I8_NONE, ei = I8_NONE;
#pragma unroll 4
    for (int m = m0 + tid; m < m1; m += 256) {
      const z2i a = A[(size_t)k * lda + m];
      er = max(er, exp_of(a.r));
      ei = max(ei, exp_of(a.i));
    }
    er = __reduce_max_sync(0xffffffffu, er);
    ei = __reduce_max_sync(0xffffffffu, ei);
    if ((tid & 31) == 0) {
      atomicMax(ia + 2 * k, er);
      atomicMax(ia + 2 * k + 1, ei);
    }
    return;
  }
  __shared__ int red[4][64];
  const int b = blockIdx.x - nA, nkb = (K + 63) / 64, kl = tid & 63, g = tid >> 6;
  const int k = (b % nkb) * 64 + kl, n0 = (b / nkb) * 64;
  int e = I8_NONE;
  if (k < K)
#pragma unroll 4
    for (int n = n0 + g; n < min(N, n0 + 64); n += 4) {
      const z2i v = B[(size_t)n * ldb + k];
      e = max(e, max(exp_of(v.r), exp_of(v.i)));
    }
  red[g][kl] = e;
  __syncthreads();
  if (g == 0 && k < K) atomicMax(ib + k, max(max(red[0][kl], red[1][kl]), max(red[2][kl], red[3][kl])));
}

// row exponents of A with the inner shifts, 32 columns per block
__global__ void __launch_bounds__(128) k_i8_rowmax(int M, int K, const z2i *A, size_t lda, I8Inner I, int *em) {
  __shared__ int2 sp[32];
  const int m = blockIdx.x * 128 + threadIdx.x, k0 = blockIdx.y * 32;
  if (threadIdx.x < 32)
    sp[threadIdx.x] = k0 + threadIdx.x < K ? inner_shift(I, k0 + threadIdx.x) : make_int2(I8_NONE, I8_NONE);
  __syncthreads();
  if (m >= M) return;
  int e = I8_NONE;
#pragma unroll
  for (int q = 0; q < 4; q++) {
    z2i a[8];
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const int k = k0 + 8 * q + i;
      a[i] = k < K ? A[(size_t)k * lda + m] : z2i{0.0, 0.0};
    }
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const int2 p = sp[8 * q + i];
      e = max(e, max(exp_of(a[i].r, p.x), exp_of(a[i].i, p.y)));
    }
  }
  atomicMax(em + m, e);
}

// Digit blocks: 32 bytes of K (16 columns, re and im interleaved) of 128 rows of
// A or 128 rows of B, [digit][row][32 bytes], one contiguous piece per block in the
// order the stages read them, the two 16-byte halves of a row exchanged where
// bit 2 of the row is set (the tensor core's 32-byte swizzle).  Loads are then
// whole lines; as planes of rows, a stage read half a line per row.
__device__ __forceinline__ size_t digit_row(int row, int kb, int nk, int rows) {
  return ((size_t)(row / rows) * nk + kb) * (I8_S * rows * I8_BK) + (row % rows) * I8_BK;
}
// Sizes for the guard: 128 bytes of K of 128 rows per block, [row][128 bytes], 16-byte
// pieces in the tensor core's 128-byte swizzle; byte o of K of a row
__device__ __forceinline__ size_t size_byte(int row, int o, int nk) {
  return ((size_t)(row / 128) * nk + o / 128) * GD_ROWS + (row % 128) * 128 + (((o / 16) ^ row) & 7) * 16 + o % 16;
}

// a thread takes one row and 16 columns; blocks past the last one of digits clear
// the rest of the 128-byte blocks of sizes, the first one the tiles' flags
__global__ void __launch_bounds__(128) k_i8_slice_a(int M, int K, const z2i *A, size_t lda, I8Inner I, const int *em,
                                                    int8_t *S, uint8_t *Z, int nk, double *sa, unsigned char *flag,
                                                    int nflag) {
  if (blockIdx.x == 0 && blockIdx.y == 0)
    for (int i = threadIdx.x; i < nflag; i += 128) flag[i] = 0;
  const int m = blockIdx.x * 128 + threadIdx.x, kb = blockIdx.y, k0 = kb * 16, nz = (nk + 3) / 4;
  if (m >= M) return;
  if (kb >= nk) {
#pragma unroll
    for (int h = 0; h < 2; h++) *(uint4 *)(Z + size_byte(m, 32 * kb + 16 * h, nz)) = make_uint4(0, 0, 0, 0);
    return;
  }
  const int e = em[m];
  const bool on = in_range(e);
  if (kb == 0) sa[m] = digit_scale(e);
  int8_t *p = S + digit_row(m, kb, nk, I8_BM);
#pragma unroll
  for (int h = 0; h < 2; h++) {
    uint32_t w[4][8], z[4];
    z2i a[8];
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const int k = k0 + 8 * h + i;
      a[i] = k < K ? A[(size_t)k * lda + m] : z2i{0.0, 0.0};
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
      unsigned long long d[4];
      z[i] = 0;
#pragma unroll
      for (int j = 0; j < 2; j++) {
        const int k = k0 + 8 * h + 2 * i + j;
        const int2 s = on && k < K ? inner_shift(I, k) : make_int2(I8_NONE, I8_NONE);
        const long long xr = s.x == I8_NONE ? 0 : to_int(a[2 * i + j].r, e, s.x);
        const long long xi = s.y == I8_NONE ? 0 : to_int(a[2 * i + j].i, e, s.y);
        d[2 * j] = digits(xr);
        d[2 * j + 1] = digits(xi);
        z[i] |= (size_of(xr) | size_of(xi) << 8) << (16 * j);
      }
      transpose8(d, w[i]);
    }
    const int o = 16 * (h ^ ((m >> 2) & 1));
#pragma unroll
    for (int s = 0; s < I8_S; s++)
      *(uint4 *)(p + s * (I8_BM * I8_BK) + o) = make_uint4(w[0][s], w[1][s], w[2][s], w[3][s]);
    *(uint4 *)(Z + size_byte(m, 32 * kb + 16 * h, nz)) = make_uint4(z[0], z[1], z[2], z[3]);
  }
}

// slices of B, K <= I8_KC: a block takes a column; rows 2n: (br, -bi), 2n + 1: (bi, br),
// each with its own scale
#define I8_KC 2048
__global__ void __launch_bounds__(I8_KC / 8) k_i8_slice_b(int K, const z2i *B, size_t ldb, I8Inner I, int8_t *S, uint8_t *Z,
                                                          int nk, double *sb) {
  const int n = blockIdx.x, t = threadIdx.x, nz = (nk + 3) / 4;
  const z2i *b = B + (size_t)n * ldb;
  z2i v[4][2];
  int f0 = I8_NONE, f1 = I8_NONE;
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int k = 2 * t + I8_KC / 4 * i + h;
      v[i][h] = k < K ? b[k] : z2i{0.0, 0.0};
      if (k >= K) continue;
      const int2 p = inner_shift(I, k);
      const int nx = p.x == I8_NONE ? I8_NONE : -p.x, ny = p.y == I8_NONE ? I8_NONE : -p.y;
      f0 = max(f0, max(exp_of(v[i][h].r, nx), exp_of(v[i][h].i, ny)));
      f1 = max(f1, max(exp_of(v[i][h].i, nx), exp_of(v[i][h].r, ny)));
    }
  __shared__ int red[2][I8_KC / 256];
  f0 = __reduce_max_sync(0xffffffffu, f0);
  f1 = __reduce_max_sync(0xffffffffu, f1);
  if ((t & 31) == 0) { red[0][t >> 5] = f0; red[1][t >> 5] = f1; }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < I8_KC / 256; i++) { f0 = max(f0, red[0][i]); f1 = max(f1, red[1][i]); }
  if (t == 0) ((double2 *)sb)[n] = make_double2(digit_scale(f0), digit_scale(f1));
  const bool on0 = in_range(f0), on1 = in_range(f1);
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int k = 2 * t + I8_KC / 4 * i;
    if (k / 64 >= nz) continue;
    unsigned long long d0[4], d1[4];
    uint32_t z0 = 0, z1 = 0;
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int2 p = k + h < K ? inner_shift(I, k + h) : make_int2(I8_NONE, I8_NONE);
      const z2i x = v[i][h];
      const bool re = p.x != I8_NONE, im = p.y != I8_NONE;
      const long long a0 = on0 && re ? to_int(x.r, f0, -p.x) : 0, a1 = on0 && im ? -to_int(x.i, f0, -p.y) : 0;
      const long long c0 = on1 && re ? to_int(x.i, f1, -p.x) : 0, c1 = on1 && im ? to_int(x.r, f1, -p.y) : 0;
      d0[2 * h] = digits(a0);
      d0[2 * h + 1] = digits(a1);
      d1[2 * h] = digits(c0);
      d1[2 * h + 1] = digits(c1);
      z0 |= (size_of(a0) | size_of(a1) << 8) << (16 * h);
      z1 |= (size_of(c0) | size_of(c1) << 8) << (16 * h);
    }
    *(uint32_t *)(Z + size_byte(2 * n, 2 * k, nz)) = z0;
    *(uint32_t *)(Z + size_byte(2 * n + 1, 2 * k, nz)) = z1;
    if (k / 16 >= nk) continue;
    uint32_t w0[8], w1[8];
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

// scratch of products of at most M x N x K, as offsets into it
struct I8Layout {
  int mc, nc, kc;
  size_t Sa, Sb, Za, Zb, sa, sb, flag, ia, bytes;   // at ia: 2 kc + kc + M exponents
  I8Layout(int M, int N, int K) : mc(std::min(M, I8_MC)), nc(std::min(N, I8_NC)), kc(std::min(K, I8_KC)) {
    const size_t rb = (mc + I8_BM - 1) / I8_BM, cb = (2 * nc + I8_BN - 1) / I8_BN, kb = (kc + 15) / 16, kz = (kb + 3) / 4;
    size_t o = 0;
    auto take = [&](size_t n) { const size_t at = o; o += up256(n); return at; };
    Sa = take(rb * kb * I8_A_BYTES);
    Sb = take(cb * kb * I8_B_BYTES);
    Za = take(rb * kz * GD_ROWS);
    Zb = take(cb * kz * GD_ROWS);
    sa = take(8 * (size_t)mc);
    sb = take(16 * (size_t)nc);
    flag = take(rb * cb);
    ia = take(4 * (3 * (size_t)kc + M));
    bytes = o;
  }
};
size_t zgemm_i8_bytes(int M, int N, int K) { return I8Layout(M, N, K).bytes; }

// the tiles with a flag by FP64 (lu.cu)
int zgemm_flagged(int M, int N, int K, const void *A, size_t lda, const void *B, size_t ldb, void *C, size_t ldc,
                  const unsigned char *flag);

// C -= A B with the scratch `work` of `bytes`; err: device int, nonzero after a failed wait
int zgemm_i8(int M, int N, int K, const void *Av, size_t lda, const void *Bv, size_t ldb, void *Cv, size_t ldc,
             void *work, size_t bytes, int *err) {
  static int sms = 0;
  if (!sms) {
    int dev = 0, n = 0;
    BG_CUDA_TRY(cudaGetDevice(&dev));
    BG_CUDA_TRY(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev));
    BG_CUDA_TRY(cudaFuncSetAttribute(k_zgemm_i8, cudaFuncAttributeMaxDynamicSharedMemorySize, I8_SMEM));
    BG_CUDA_TRY(cudaFuncSetAttribute(k_i8_guard, cudaFuncAttributeMaxDynamicSharedMemorySize, GD_SMEM));
    sms = n;
  }
  const I8Layout L(M, N, K);
  if (L.bytes > bytes) { set_error("zgemm: scratch too small"); return BG_ERR_STATE; }
  const z2i *A = (const z2i *)Av, *B = (const z2i *)Bv;
  z2i *C = (z2i *)Cv;
  char *w = (char *)work;
  int8_t *Sa = (int8_t *)(w + L.Sa), *Sb = (int8_t *)(w + L.Sb);
  uint8_t *Za = (uint8_t *)(w + L.Za), *Zb = (uint8_t *)(w + L.Zb);
  double *sa = (double *)(w + L.sa), *sb = (double *)(w + L.sb);
  unsigned char *flag = (unsigned char *)(w + L.flag);
  int *ia = (int *)(w + L.ia), *ib = ia + 2 * L.kc, *em = ib + L.kc;
  for (int k0 = 0; k0 < K; k0 += L.kc) {
    const int kk = std::min(L.kc, K - k0), nk = (kk + 15) / 16, nz = (nk + 3) / 4;
    const I8Inner I{ia, ib};
    BG_CUDA_TRY(cudaMemsetAsync(ia, 0x80, 4 * (3 * (size_t)L.kc + M), stream()));
    const int nA = kk * ((M + I8_INNER_A - 1) / I8_INNER_A), nB = ((kk + 63) / 64) * ((N + 63) / 64);
    k_i8_inner<<<nA + nB, 256, 0, stream()>>>(M, N, kk, A + (size_t)k0 * lda, lda, B + k0, ldb, nA, ia, ib);
    BG_LAUNCHED();
    k_i8_rowmax<<<dim3((M + 127) / 128, (kk + 31) / 32), 128, 0, stream()>>>(M, kk, A + (size_t)k0 * lda, lda, I, em);
    BG_LAUNCHED();
    for (int n0 = 0; n0 < N; n0 += L.nc) {
      const int nn = std::min(L.nc, N - n0);
      const z2i *Bn = B + k0 + (size_t)n0 * ldb;
      k_i8_slice_b<<<nn, I8_KC / 8, 0, stream()>>>(kk, Bn, ldb, I, Sb, Zb, nk, sb);
      BG_LAUNCHED();
      for (int m0 = 0; m0 < M; m0 += L.mc) {
        const int mm = std::min(L.mc, M - m0), ntm = (mm + I8_BM - 1) / I8_BM, ntn = (2 * nn + I8_BN - 1) / I8_BN;
        const z2i *Am = A + m0 + (size_t)k0 * lda;
        z2i *Cm = C + m0 + (size_t)n0 * ldc;
        k_i8_slice_a<<<dim3(ntm, 4 * nz), 128, 0, stream()>>>(mm, kk, Am, lda, I, em + m0, Sa, Za, nk, sa, flag,
                                                                  ntm * ntn);
        BG_LAUNCHED();
        const I8Guard G{mm, 2 * nn, nz, Za, Zb, sa, sb, flag, err, ntm, ntn};
        k_i8_guard<<<std::min(ntm * ntn, 2 * sms), GD_THREADS, GD_SMEM, stream()>>>(G);
        BG_LAUNCHED();
        const I8Args P{mm, nn, nk, Sa, Sb, Cm, ldc, sa, sb, flag, err, ntm, ntn};
        k_zgemm_i8<<<std::min(ntm * ntn, sms), I8_THREADS, I8_SMEM, stream()>>>(P);
        BG_LAUNCHED();
        int st = zgemm_flagged(mm, nn, kk, Am, lda, Bn, ldb, Cm, ldc, flag);
        if (st) return st;
      }
    }
  }
  return BG_OK;
}

}  // namespace bg
