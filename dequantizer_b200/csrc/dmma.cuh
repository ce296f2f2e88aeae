// FP64 tensor-core tiles (mma.sync m8n8k4, FP64 operands and accumulators) for
// small complex products on padded shared-memory slabs.
//
// On sm_100a the FP64 tensor and vector pipes have the same peak (measured
// here: m8n8k4 36.5 TFLOP/s, DFMA chains 34.8), but one m8n8k4 does 256
// multiply-adds from two operand registers per lane, so a product needs a
// sixth of the shared-memory loads and an eighth of the issue slots of
// register-tiled FMAs, which is what held those at 40% of the peak. Every
// product is an IEEE FP64 fused multiply-add.
//
// Fragments of one m8n8k4 (lane = 4 * row + q): A[row][k = q], B[k = q][col =
// row], C[row][2 q], C[row][2 q + 1]. A contraction may take its index in any
// order, so all loads here let step i of an 8-wide block read index
// 8 block + 2 q + i: this is the column an accumulator fragment holds, hence a
// finished tile is the A operand of the next product without leaving the
// registers, and with odd strides every 16-byte access of a quarter warp falls
// in eight different banks for rows and columns alike.
#pragma once

#include "common.cuh"

namespace dqz {

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
      : "+d"(c[0]), "+d"(c[1])
      : "d"(a), "d"(b));
}

// A (8 TM) x (8 TN) complex tile: row 8 r + (lane >> 2), columns
// 8 n + 2 (lane & 3) + {0, 1}.
template <int TM, int TN>
struct CTile {
  double re[TM][TN][2], im[TM][TN][2];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int r = 0; r < TM; ++r)
#pragma unroll
      for (int n = 0; n < TN; ++n) re[r][n][0] = re[r][n][1] = im[r][n][0] = im[r][n][1] = 0.0;
  }
};

// One k step: c += a b, a conjugated when CA, b when CB.
template <bool CA, bool CB, int TM, int TN>
__device__ __forceinline__ void cstep(CTile<TM, TN> &c, const cd (&a)[TM], const cd (&b)[TN]) {
#pragma unroll
  for (int r = 0; r < TM; ++r) {
    const double ai = CA ? -a[r].y : a[r].y;
#pragma unroll
    for (int n = 0; n < TN; ++n) {
      const double bi = CB ? -b[n].y : b[n].y;
      dmma(c.re[r][n], a[r].x, b[n].x);
      dmma(c.im[r][n], a[r].x, bi);
      dmma(c.re[r][n], -ai, bi);
      dmma(c.im[r][n], ai, b[n].x);
    }
  }
}

// c += A B over k < 8 KB; la(row, k) and lb(k, column) load one entry.
template <bool CA, bool CB, int KB, int TM, int TN, typename LA, typename LB>
__device__ __forceinline__ void cgemm(CTile<TM, TN> &c, LA la, LB lb) {
  const int row = (threadIdx.x & 31) >> 2, q = threadIdx.x & 3;
#pragma unroll
  for (int t = 0; t < KB; ++t)
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int k = 8 * t + 2 * q + i;
      cd a[TM], b[TN];
#pragma unroll
      for (int r = 0; r < TM; ++r) a[r] = la(8 * r + row, k);
#pragma unroll
      for (int n = 0; n < TN; ++n) b[n] = lb(k, 8 * n + row);
      cstep<CA, CB>(c, a, b);
    }
}

// c += X B with X a finished tile (its columns are the contracted index).
template <bool CX, bool CB, int TM, int TK, int TN, typename LB>
__device__ __forceinline__ void cgemm_regs(CTile<TM, TN> &c, const CTile<TM, TK> &x, LB lb) {
  const int row = (threadIdx.x & 31) >> 2, q = threadIdx.x & 3;
#pragma unroll
  for (int t = 0; t < TK; ++t)
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int k = 8 * t + 2 * q + i;
      cd a[TM], b[TN];
#pragma unroll
      for (int r = 0; r < TM; ++r) a[r] = mk(x.re[r][t][i], x.im[r][t][i]);
#pragma unroll
      for (int n = 0; n < TN; ++n) b[n] = lb(k, 8 * n + row);
      cstep<CX, CB>(c, a, b);
    }
}

// put(row, column, value) for every entry this lane holds.
template <int TM, int TN, typename Put>
__device__ __forceinline__ void ctile_each(const CTile<TM, TN> &c, Put put) {
  const int row = (threadIdx.x & 31) >> 2, q = threadIdx.x & 3;
#pragma unroll
  for (int r = 0; r < TM; ++r)
#pragma unroll
    for (int n = 0; n < TN; ++n)
#pragma unroll
      for (int i = 0; i < 2; ++i) put(8 * r + row, 8 * n + 2 * q + i, mk(c.re[r][n][i], c.im[r][n][i]));
}

__device__ __forceinline__ void cp_async16(void *dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async16_or_zero(void *dst, const void *src, bool in) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(in ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

}  // namespace dqz
