// CTA-cooperative FP64 linear algebra with the matrix in registers: warp w of W
// owns the columns c with c % W == w (CPW of them), lane l the rows l + 32 t (ROWS
// of them). Conventions as in linalg.cuh (LAPACK Householder vectors, one-sided
// Jacobi with the same tolerances); the matrices of the simple update (up to 256
// x 32 a side, cores up to 32 x 32) fit the register file of one CTA, where the
// shared- or global-memory forms spent their time on loads, stores and
// barriers: only the reflector of a column crosses warps.
#pragma once

#include <type_traits>

#include "linalg.cuh"

namespace dqz {

// Sums of N (a power of two up to 16) doubles over the warp, all lanes getting
// all: halves are exchanged until a lane holds one partial sum, then gathered
// (17 64-bit shuffles for N = 8, where one butterfly per value takes 40).
template <int N>
__device__ __forceinline__ void warp_sum_all(double (&v)[N]) {
  const int lane = threadIdx.x & 31;
  int o = 16;
#pragma unroll
  for (int n = N; n > 1; n >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < n / 2; ++i) {
      const double give = up ? v[i] : v[i + n / 2], own = up ? v[i + n / 2] : v[i];
      v[i] = own + __shfl_xor_sync(0xffffffffu, give, o);
    }
    o >>= 1;
  }
  double x = v[0];
  for (int s = o; s > 0; s >>= 1) x += __shfl_xor_sync(0xffffffffu, x, s);
  // value i sits in the lanes whose top log2(N) bits, most significant first, are i's
#pragma unroll
  for (int i = 0; i < N; ++i) v[i] = __shfl_sync(0xffffffffu, x, i * (32 / N));
}

// a -= v (f conj(v)^T a) style update of C0..CPW-1 columns: a_c -= v * (t * sum
// conj(v) a_c); t = conj(tau) applies H^H, t = tau applies H.
template <int C0, int CPW, int ROWS>
__device__ __forceinline__ void reg_reflect(cd (&a)[CPW][ROWS], const cd (&v)[ROWS], cd t) {
  constexpr int NC = CPW - C0;
  constexpr int N2 = NC <= 1 ? 2 : (NC <= 2 ? 4 : (NC <= 4 ? 8 : 16));
  static_assert(NC <= 8, "at most eight columns a warp");
  double s[N2];
#pragma unroll
  for (int i = 0; i < N2; ++i) s[i] = 0.0;
#pragma unroll
  for (int c = C0; c < CPW; ++c) {
    double xx = 0.0, yy = 0.0, xy = 0.0, yx = 0.0;
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      xx = fma(v[r].x, a[c][r].x, xx);
      yy = fma(v[r].y, a[c][r].y, yy);
      xy = fma(v[r].x, a[c][r].y, xy);
      yx = fma(v[r].y, a[c][r].x, yx);
    }
    s[2 * (c - C0)] = xx + yy;
    s[2 * (c - C0) + 1] = xy - yx;
  }
  warp_sum_all<N2>(s);
#pragma unroll
  for (int c = C0; c < CPW; ++c) {
    const cd f = cmul(t, mk(s[2 * (c - C0)], s[2 * (c - C0) + 1]));
    const cd nf = mk(-f.x, -f.y);
#pragma unroll
    for (int r = 0; r < ROWS; ++r) cfma(a[c][r], v[r], nf);
  }
}

// Reflector j < 32 from column x (rows >= j), published in v (zero above j, 1 at
// j) and kept in x (R above, beta at j, the vector below).
template <int ROWS>
__device__ __forceinline__ void reg_make_reflector(cd (&x)[ROWS], int j, cd *v, cd *tau) {
  const int lane = threadIdx.x & 31;
  double s0 = 0.0, s1 = 0.0;
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
    const bool below = r > 0 || lane > j;  // j < 32
    s0 = below ? fma(x[r].x, x[r].x, s0) : s0;
    s1 = below ? fma(x[r].y, x[r].y, s1) : s1;
  }
  const double s = warp_sum(s0 + s1);
  const cd alpha = mk(__shfl_sync(0xffffffffu, x[0].x, j), __shfl_sync(0xffffffffu, x[0].y, j));
  cd t = czero(), sc = mk(1.0, 0.0);
  double beta = alpha.x;
  const bool live = !(s == 0.0 && alpha.y == 0.0);
  if (live) householder_scalars(alpha, s, beta, t, sc);
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
    const int row = lane + 32 * r;
    cd out = czero();
    if (row > j) {
      if (live) x[r] = cmul(x[r], sc);
      out = x[r];
    } else if (row == j) {
      if (live) x[r] = mk(beta, 0.0);
      out = mk(1.0, 0.0);
    }
    v[row] = out;
  }
  if (lane == 0) tau[j] = t;
}

// Column j's reflector is published through named barrier 1 + j % 4: its owner
// arrives and goes on to its other columns, the other warps wait there before
// they use it. The next owner's chain (its column's update, norm, scalars) thus
// runs while everyone's trailing columns are still being updated. Four vectors in
// rotation: barrier j + 3 completes only after every warp has read vector j.
template <int W>
__device__ __forceinline__ void reg_barrier_arrive(int j) {
  __syncwarp();
  asm volatile("bar.arrive %0, %1;" ::"r"(1 + (j & 3)), "n"(32 * W) : "memory");
}
template <int W>
__device__ __forceinline__ void reg_barrier_wait(int j) {
  __syncwarp();
  asm volatile("bar.sync %0, %1;" ::"r"(1 + (j & 3)), "n"(32 * W) : "memory");
}

// The steps of columns J W .. J W + W - 1 of reg_qr, then the following blocks.
template <int W, int CPW, int ROWS, int J>
__device__ __forceinline__ void reg_qr_block(cd (&a)[CPW][ROWS], int kk, cd *vbuf, cd *tau) {
  constexpr int LEN = 32 * ROWS;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  // the owner of column j + 1 (its column C0) brings it up to date and builds
  // reflector j + 1 before its other trailing columns (from C0 + 1)
  auto own_next = [&](auto c0, const cd(&v)[ROWS], cd tc, int next) {
    constexpr int C0 = decltype(c0)::value;
    cd one[1][ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) one[0][r] = a[C0][r];
    reg_reflect<0, 1, ROWS>(one, v, tc);
#pragma unroll
    for (int r = 0; r < ROWS; ++r) a[C0][r] = one[0][r];
    reg_make_reflector<ROWS>(a[C0], next, vbuf + (next & 3) * LEN, tau);
    reg_barrier_arrive<W>(next);
    if constexpr (C0 + 1 < CPW) reg_reflect<C0 + 1, CPW, ROWS>(a, v, tc);
  };
#pragma unroll 1
  for (int ow = 0; ow < W; ++ow) {
    const int j = J * W + ow, next = j + 1;
    if (j >= kk) return;  // uniform over the CTA
    if (w != ow) reg_barrier_wait<W>(j);
    else __syncwarp();
    const cd tj = tau[j];
    const cd tc = mk(tj.x, -tj.y);
    cd v[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) v[r] = vbuf[(j & 3) * LEN + lane + 32 * r];
    if (w > ow) {  // column J W + w is still trailing
      if (w == ow + 1 && next < kk)
        own_next(std::integral_constant<int, J>(), v, tc, next);
      else
        reg_reflect<J, CPW, ROWS>(a, v, tc);
    } else if constexpr (J + 1 < CPW) {
      if (ow == W - 1 && w == 0 && next < kk)
        own_next(std::integral_constant<int, J + 1>(), v, tc, next);
      else
        reg_reflect<J + 1, CPW, ROWS>(a, v, tc);
    }
  }
  if constexpr (J + 1 < CPW) reg_qr_block<W, CPW, ROWS, J + 1>(a, kk, vbuf, tau);
}

// Householder QR of the M x K matrix in registers (rows from M on are zero, K <=
// 32) by a CTA of W warps. vbuf: four vectors of 32 ROWS entries; tau: min(M, K).
// Begins and ends with a barrier.
template <int W, int CPW, int ROWS>
__device__ __forceinline__ void reg_qr(cd (&a)[CPW][ROWS], int M, int K, cd *vbuf, cd *tau) {
  const int kk = M < K ? M : K;
  __syncthreads();
  if ((threadIdx.x >> 5) == 0 && kk > 0) {
    reg_make_reflector<ROWS>(a[0], 0, vbuf, tau);
    reg_barrier_arrive<W>(0);
  }
  reg_qr_block<W, CPW, ROWS, 0>(a, kk, vbuf, tau);
  __syncthreads();
}

// x <- H_0 ... H_(kk-1) x for the CPW columns of this warp; the packed reflectors
// are columns of V (ld ldv, 1 on the diagonal implied). No barrier.
template <int CPW, int ROWS>
__device__ __forceinline__ void reg_apply_q(cd (&x)[CPW][ROWS], const cd *__restrict__ V, int ldv, int M, int kk,
                                            const cd *__restrict__ tau) {
  const int lane = threadIdx.x & 31;
  cd v[ROWS];
  auto load = [&](int j, cd (&d)[ROWS]) {
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      const int row = lane + 32 * r;
      d[r] = row > j && row < M ? V[(long long)j * ldv + row] : (row == j ? mk(1.0, 0.0) : czero());
    }
  };
  if (kk > 0) load(kk - 1, v);
#pragma unroll 1
  for (int j = kk - 1; j >= 0; --j) {
    const cd t = tau[j];
    cd nx[ROWS];
    if (j > 0) load(j - 1, nx);
    reg_reflect<0, CPW, ROWS>(x, v, t);
#pragma unroll
    for (int r = 0; r < ROWS; ++r) v[r] = nx[r];
  }
}

// One-sided Jacobi SVD (hestenes) of an n x n matrix, n <= 32, by a CTA of 256
// threads, X and V in shared memory (column-major, ld). The first four warps
// rotate X: eight lanes a pair of columns (rows sub + 8 i). The other four apply
// the rotations of the round before to V, off the chain scalar products ->
// rotation -> columns that bounds a round. On entry X holds the matrix; on
// return its columns are u_j (zero for a numerically null one, s_j = 0) and V
// holds the right singular vectors.
// A sweep whose rotated pairs all had |cos| below 1e-9 and turned by less than
// 1e-8 ends the iteration: a rotation gives back at most sin |cos| of what others
// removed, so 2 n of them leave less than 64e-17, below the tolerance, and a further
// sweep would only confirm. The angle matters: columns of equal norm turn by up to
// 45 degrees however small their |cos| (with the first rule alone the gauge of a
// message 1 + 1e-11 H was off by 2e-11).
// Measured on the simple update's 32 x 32 cores: columns in registers moved from
// seat to seat by shuffles (64 of about 9 cycles a round) 2,300 cycles a round and
// 380 us for a launch of one core; this form 210 us.
constexpr int RJ_THREADS = 256, RJ_MAX = 32;
struct JacobiSmem {
  double ph[2][16][2], cs[2][16], sn[2][16];  // [parity][pair]; sn = 0 with cs = 1 for no rotation
  double fro[4];
};

__device__ __forceinline__ double oct_sum(double v) {
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  v += __shfl_xor_sync(0xffffffffu, v, 2);
  return v + __shfl_xor_sync(0xffffffffu, v, 4);
}

// This lane's four rows of conj(x)^T y, |x|^2 and |y|^2, short chains
__device__ __forceinline__ void pair_products(const cd (&x)[4], const cd (&y)[4], cd &ga, double &al, double &be) {
  double re[4], im[4], xx[4], yy[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    re[i] = fma(x[i].x, y[i].x, x[i].y * y[i].y);
    im[i] = fma(x[i].x, y[i].y, -(x[i].y * y[i].x));
    xx[i] = cabs2(x[i]);
    yy[i] = cabs2(y[i]);
  }
  ga = mk((re[0] + re[1]) + (re[2] + re[3]), (im[0] + im[1]) + (im[2] + im[3]));
  al = (xx[0] + xx[1]) + (xx[2] + xx[3]);
  be = (yy[0] + yy[1]) + (yy[2] + yy[3]);
}

// The rotation of pair `grp` applied to columns p, q of V (rows sub + 8 i).
__device__ __forceinline__ void cta_jacobi_v(cd *V, int ld, int n, int p, int q, int sub, const JacobiSmem &E, int par,
                                             int grp) {
  const double sn = E.sn[par][grp], cs = E.cs[par][grp];
  if (sn == 0.0 && cs == 1.0 && E.ph[par][grp][0] == 1.0) return;  // no rotation
  const cd ph = mk(E.ph[par][grp][0], E.ph[par][grp][1]);
  cd *cx = V + p * ld + sub, *cy = V + q * ld + sub;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (sub + 8 * i >= n) continue;
    const cd t = cmul(cx[8 * i], ph), y = cy[8 * i];
    cx[8 * i] = mk(cs * t.x - sn * y.x, cs * t.y - sn * y.y);
    cy[8 * i] = mk(sn * t.x + cs * y.x, sn * t.y + cs * y.y);
  }
}

// Barrier of this Jacobi's RJ_THREADS threads: the CTA's (id 0), or a named one
// where a CTA runs two at once (its warps 8 .. 15 the second).
__device__ __forceinline__ void jacobi_sync(int bar) {
  if (bar == 0)
    __syncthreads();
  else
    asm volatile("bar.sync %0, 256;" ::"r"(bar) : "memory");
}
__device__ __forceinline__ int jacobi_any(int bar, int v) {
  if (bar == 0) return __syncthreads_or(v);
  int r;
  asm volatile(
      "{\n .reg .pred p, q;\n setp.ne.s32 p, %1, 0;\n bar.red.or.pred q, %2, 256, p;\n selp.s32 %0, 1, 0, q;\n}"
      : "=r"(r)
      : "r"(v), "r"(bar)
      : "memory");
  return r;
}

// Called by all RJ_THREADS threads of the barrier `bar`.
static __device__ void cta_jacobi(cd *X, cd *V, int ld, int n, double *s, JacobiSmem &E, int bar = 0) {
  static_assert(RJ_THREADS == 256, "the named barrier's threads");
  const int tid = threadIdx.x % RJ_THREADS, lane = tid & 31, w = tid >> 5;
  const int grp = (tid & 127) >> 3, sub = tid & 7;
  const int np = n + (n & 1), npairs = np / 2;
  const bool main = tid < 128, seat = grp < npairs;
  const double tol = 1.1e-16 * sqrt((double)n) * 2.0;
  for (int i = tid; i < n * n; i += RJ_THREADS) V[(i / n) * ld + i % n] = i / n == i % n ? mk(1.0, 0.0) : czero();
  if (main) {
    double f = 0.0;
    for (int i = tid; i < n * n; i += 128) f += cabs2(X[(i / n) * ld + i % n]);
    f = warp_sum(f);
    if (lane == 0) E.fro[w] = f;
  }
  jacobi_sync(bar);
  const double null_thr = hestenes_null_scale(n) * (((E.fro[0] + E.fro[1]) + E.fro[2]) + E.fro[3]);
  int done = 0;  // rounds of all sweeps so far, for the parity of the rotations
  int pp = 0, pq = n;  // V's pair: the round before
  for (int sweep = 0; sweep < 60 && n > 1; ++sweep) {
    int more = 0;
    for (int round = 0; round < np - 1; ++round, ++done) {
      const int par = done & 1;
      int p = 0, q = n;
      if (seat) rr_pair(round, grp, np, p, q);
      if (main) {
        const bool live = seat && q < n;
        cd *cx = X + p * ld + sub, *cy = X + (live ? q : p) * ld + sub;
        cd x[4], y[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const bool in = live && sub + 8 * i < n;
          x[i] = in ? cx[8 * i] : czero();
          y[i] = in ? cy[8 * i] : czero();
        }
        cd ga;
        double al, be;
        pair_products(x, y, ga, al, be);
        ga = mk(oct_sum(ga.x), oct_sum(ga.y));
        al = oct_sum(al);
        be = oct_sum(be);
        const double g2 = cabs2(ga), ab = al * be;
        PhaseRot R;
        const bool rot = live && al > null_thr && be > null_thr && g2 > tol * tol * ab && phase_rot(al, be, ga, R);
        if (rot) {
          more |= g2 > 1e-18 * ab || fabs(R.t) > 1e-8;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const cd t = cmul(x[i], R.ph);
            if (sub + 8 * i < n) {
              cx[8 * i] = mk(R.cs * t.x - R.sn * y[i].x, R.cs * t.y - R.sn * y[i].y);
              cy[8 * i] = mk(R.sn * t.x + R.cs * y[i].x, R.sn * t.y + R.cs * y[i].y);
            }
          }
        }
        if (sub == 0) {
          E.ph[par][grp][0] = rot ? R.ph.x : 1.0;
          E.ph[par][grp][1] = rot ? R.ph.y : 0.0;
          E.cs[par][grp] = rot ? R.cs : 1.0;
          E.sn[par][grp] = rot ? R.sn : 0.0;
        }
      } else {
        if (done > 0 && seat && pq < n) cta_jacobi_v(V, ld, n, pp, pq, sub, E, par ^ 1, grp);
        pp = p;
        pq = q;
      }
      jacobi_sync(bar);
    }
    if (!jacobi_any(bar, more)) break;
  }
  if (!main && done > 0 && seat && pq < n) cta_jacobi_v(V, ld, n, pp, pq, sub, E, (done - 1) & 1, grp);
  if (main)
    for (int j0 = 0; j0 < n; j0 += 16) {  // whole warps: the sums below are over full warps
      const int j = j0 + grp;
      const bool in = j < n;
      cd *col = X + (in ? j : 0) * ld + sub;
      double t = 0.0;
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (in && sub + 8 * i < n) t += cabs2(col[8 * i]);
      t = oct_sum(t);
      const double sj = t > null_thr ? sqrt(t) : 0.0, inv = sj > 0.0 ? 1.0 / sj : 0.0;
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (in && sub + 8 * i < n) col[8 * i] = cscale(col[8 * i], inv);
      if (in && sub == 0) s[j] = sj;
    }
  jacobi_sync(bar);
}

}  // namespace dqz
