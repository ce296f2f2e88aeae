// Trace norm of a Hermitian matrix up to 16 x 16 by one warp: Householder
// reduction to a real tridiagonal matrix in registers (lane (half, r) holds the
// columns of parity `half` of row r), then every eigenvalue at once by
// trisection with Sturm counts, two lanes per eigenvalue.
//
// Only the sum of |eigenvalues| is wanted, to rounding of the matrix norm. The
// Jacobi iteration this replaces needs six to eight sweeps of dependent
// rotations for it (about 0.6 M cycles of one warp at n = 16); the reduction is 14
// steps and the counts 34 passes over the tridiagonal, whose chain is one
// fused multiply-add per row: p_i = (d_i - x) p_(i-1) - e_i^2 p_(i-2) (no division
// as in the quotient form; sign changes count eigenvalues below x). The matrix
// is scaled to norm 1 and e^2 kept above 1e-36 (a shift of the eigenvalues by
// 1e-18 at most), so a zero p_i never stands beside another and 16 rows neither
// overflow nor underflow.
#pragma once

#include "linalg.cuh"

namespace dqz {

struct TraceNormSmem {
  cd v[16], w[16];
  double d[16], e[16];
};

__device__ __forceinline__ double row_sum(double v) {  // over the 16 rows (each half alike)
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// A: n x n, row-major, leading dimension lda, n <= 16, in shared memory (kept).
// NaN for a non-finite matrix.
static __device__ double warp_trace_norm(const cd *A, int lda, int n, TraceNormSmem &S) {
  const int lane = threadIdx.x & 31, r = lane & 15, half = lane >> 4;
  cd a[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int c = 2 * k + half;
    a[k] = r < n && c < n ? A[r * lda + c] : czero();
  }
  if (lane < 16) S.e[lane] = 0.0;
  __syncwarp();
#pragma unroll
  for (int k = 0; k < 14; ++k) {
    if (k + 2 < n) {
      const int from = r + 16 * (k & 1);
      const cd x = mk(__shfl_sync(0xffffffffu, a[k >> 1].x, from), __shfl_sync(0xffffffffu, a[k >> 1].y, from));
      const cd al = mk(__shfl_sync(0xffffffffu, x.x, k + 1), __shfl_sync(0xffffffffu, x.y, k + 1));
      const double xn2 = row_sum(r >= k + 2 ? cabs2(x) : 0.0);
      if (xn2 == 0.0 && al.y == 0.0) {
        if (lane == 0) S.e[k] = al.x;
      } else {
        double beta;
        cd tau, sc;
        householder_scalars(al, xn2, beta, tau, sc);
        const cd v = r == k + 1 ? mk(1.0, 0.0) : (r > k + 1 ? cmul(x, sc) : czero());
        if (half == 0) S.v[r] = v;
        if (lane == 0) S.e[k] = beta;
        __syncwarp();
        cd p = czero();
#pragma unroll
        for (int j = k / 2; j < 8; ++j) cfma(p, a[j], S.v[2 * j + half]);
        p.x += __shfl_xor_sync(0xffffffffu, p.x, 16);
        p.y += __shfl_xor_sync(0xffffffffu, p.y, 16);
        p = r > k ? cmul(tau, p) : czero();
        cd s = cmulc(v, p);
        s = mk(row_sum(s.x), row_sum(s.y));
        const cd w = csub(p, cmul(cmul(mk(0.5 * tau.x, -0.5 * tau.y), s), v));
        if (half == 0) S.w[r] = w;
        __syncwarp();
#pragma unroll
        for (int j = k / 2; j < 8; ++j) {
          const int c = 2 * j + half;
          if (c > k) a[j] = csub(a[j], cadd(cmul(w, cconj(S.v[c])), cmul(v, cconj(S.w[c]))));
        }
        __syncwarp();
      }
    }
  }
  double dr = 0.0;
  cd last = czero();
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int c = 2 * j + half;
    if (c == r) dr = a[j].x;
    if (c == n - 2) last = a[j];
  }
  if (half == (r & 1)) S.d[r] = dr;
  if (n >= 2 && r == n - 1 && half == (n & 1)) S.e[n - 2] = sqrt(cabs2(last));
  __syncwarp();
  const double d0 = fabs(r < n ? S.d[r] : 0.0), e0 = fabs(r + 1 < n ? S.e[r] : 0.0),
               em = fabs(r > 0 && r < n ? S.e[r - 1] : 0.0);
  double span = d0 + e0 + em;  // Gershgorin: |eigenvalues| <= the largest
  const double total = row_sum(span);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) span = fmax(span, __shfl_xor_sync(0xffffffffu, span, o));
  if (!(total < 1.7e308)) return __longlong_as_double(0x7ff8000000000000ll);
  if (span == 0.0) return 0.0;
  const double inv = 1.0 / span;
  double d[16], e2[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    d[i] = i < n ? S.d[i] * inv : 0.0;
    const double e = i > 0 && i < n ? S.e[i - 1] * inv : 0.0;
    e2[i] = fmax(e * e, 1e-36);
  }
  double lo = -1.0000000000000009, hi = 1.0000000000000009;
#pragma unroll 1
  for (int it = 0; it < 34; ++it) {  // 2 * 3^-34 = 1.2e-16
    const double third = (hi - lo) * (1.0 / 3.0);
    const double x1 = lo + third, x2 = hi - third, x = half ? x2 : x1;
    double p0 = 1.0, p1 = d[0] - x;
    bool neg = p1 <= 0.0;
    int count = neg ? 1 : 0;
#pragma unroll
    for (int i = 1; i < 16; ++i) {
      if (i < n) {
        const double p = fma(d[i] - x, p1, -e2[i] * p0);
        const bool now = p < 0.0 || (p == 0.0 && !neg);
        count += now != neg ? 1 : 0;
        neg = now;
        p0 = p1;
        p1 = p;
      }
    }
    const int other = __shfl_xor_sync(0xffffffffu, count, 16);
    const int c1 = half ? other : count, c2 = half ? count : other;
    if (c1 > r) {
      hi = x1;
    } else if (c2 > r) {
      lo = x1;
      hi = x2;
    } else {
      lo = x2;
    }
  }
  return row_sum(r < n ? fabs(0.5 * (lo + hi)) : 0.0) * span;
}

// The same up to 32 x 32 by the first two warps of a CTA (all its threads call):
// lane r of warp `half` holds the columns of parity `half` of row r; a column and
// the half sums of A v pass through shared memory (two barriers of the two warps a
// step), all else is computed by both alike. The eigenvalues by bisection on one
// warp, the recurrence rescaled after 16 rows (a power of two, exact).
struct TraceNorm32Smem {
  cd col[32], v[2][32], w[2][32], p[2][32];
  double d[32], e[32], out;
};

static __device__ double cta_trace_norm32(const cd *A, int lda, int n, TraceNorm32Smem &S) {
  const int r = threadIdx.x & 31, half = threadIdx.x >> 5;
  __syncthreads();
  if (half < 2) {
    const auto pair_sync = [] { asm volatile("bar.sync 1, 64;" ::: "memory"); };
    cd a[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      const int c = 2 * k + half;
      a[k] = r < n && c < n ? A[r * lda + c] : czero();
    }
    if (half == 0) S.e[r] = 0.0;
#pragma unroll
    for (int k = 0; k < 30; ++k) {
      if (k + 2 < n) {
        if (half == (k & 1)) S.col[r] = a[k >> 1];
        pair_sync();
        const cd x = S.col[r], al = S.col[k + 1];
        const double xn2 = warp_sum(r >= k + 2 ? cabs2(x) : 0.0);
        if (xn2 == 0.0 && al.y == 0.0) {
          if (threadIdx.x == 0) S.e[k] = al.x;
          pair_sync();  // the column is read
        } else {
          double beta;
          cd tau, sc;
          householder_scalars(al, xn2, beta, tau, sc);
          const cd v = r == k + 1 ? mk(1.0, 0.0) : (r > k + 1 ? cmul(x, sc) : czero());
          S.v[half][r] = v;
          if (threadIdx.x == 0) S.e[k] = beta;
          __syncwarp();
          cd p = czero(), q = czero();
#pragma unroll
          for (int j = k / 2; j < 16; j += 2) {
            cfma(p, a[j], S.v[half][2 * j + half]);
            if (j + 1 < 16) cfma(q, a[j + 1], S.v[half][2 * j + 2 + half]);
          }
          S.p[half][r] = cadd(p, q);
          pair_sync();
          p = r > k ? cmul(tau, cadd(S.p[0][r], S.p[1][r])) : czero();
          cd s = cmulc(v, p);
          s = mk(warp_sum(s.x), warp_sum(s.y));
          const cd w = csub(p, cmul(cmul(mk(0.5 * tau.x, -0.5 * tau.y), s), v));
          S.w[half][r] = w;
          __syncwarp();
#pragma unroll
          for (int j = k / 2; j < 16; ++j) {
            const int c = 2 * j + half;
            if (c > k) a[j] = csub(a[j], cadd(cmul(w, cconj(S.v[half][c])), cmul(v, cconj(S.w[half][c]))));
          }
          __syncwarp();
        }
      }
    }
    double dr = 0.0;
    cd last = czero();
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const int c = 2 * j + half;
      if (c == r) dr = a[j].x;
      if (c == n - 2) last = a[j];
    }
    if (half == (r & 1)) S.d[r] = dr;
    if (n >= 2 && r == n - 1 && half == (n & 1)) S.e[n - 2] = sqrt(cabs2(last));
    pair_sync();
  }
  if (half == 0) {
    const double d0 = fabs(r < n ? S.d[r] : 0.0), e0 = fabs(r + 1 < n ? S.e[r] : 0.0),
                 em = fabs(r > 0 && r < n ? S.e[r - 1] : 0.0);
    double span = d0 + e0 + em;
    const double total = warp_sum(span);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) span = fmax(span, __shfl_xor_sync(0xffffffffu, span, o));
    double t = total < 1.7e308 ? 0.0 : __longlong_as_double(0x7ff8000000000000ll);
    if (total < 1.7e308 && span > 0.0) {
      const double inv = 1.0 / span, em1 = r > 0 && r < n ? S.e[r - 1] * inv : 0.0;
      __syncwarp();
      S.d[r] = r < n ? S.d[r] * inv : 0.0;
      __syncwarp();
      S.e[r] = fmax(em1 * em1, 1e-36);  // e^2 between rows r - 1 and r
      __syncwarp();
      double lo = -1.0000000000000018, hi = 1.0000000000000018;
#pragma unroll 1
      for (int it = 0; it < 54; ++it) {  // 2^-53
        const double x = 0.5 * (lo + hi);
        double p0 = 1.0, p1 = S.d[0] - x;
        bool neg = p1 <= 0.0;
        int count = neg ? 1 : 0;
#pragma unroll
        for (int i = 1; i < 32; ++i) {
          if (i < n) {
            const double p = fma(S.d[i] - x, p1, -S.e[i] * p0);
            const bool now = p < 0.0 || (p == 0.0 && !neg);
            count += now != neg ? 1 : 0;
            neg = now;
            p0 = p1;
            p1 = p;
            if (i == 16) {
              const int ex = __double2hiint(fmax(fabs(p0), fabs(p1))) >> 20;
              const double f = __hiloint2double((2046 - (ex < 1 ? 1 : ex)) << 20, 0);
              p0 *= f;
              p1 *= f;
            }
          }
        }
        if (count > r)
          hi = x;
        else
          lo = x;
      }
      t = warp_sum(r < n ? fabs(0.5 * (lo + hi)) : 0.0) * span;
    }
    if (r == 0) S.out = t;
  }
  __syncthreads();
  return S.out;
}

}  // namespace dqz
