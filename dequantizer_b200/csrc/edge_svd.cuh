// Vidal orthogonalisers of one edge (tensor_ops.py:108-130, edge_svd) without
// message square roots, one warp per edge, bonds up to 16.
//
// The reference takes C = sqrt(m_f) sqrt(m_b)^T = U S V^H and the orthogonalisers
// sqrt(m_f)^-1 U, sqrt(m_b)^-1 conj(V). For positive definite messages any factor
// m = L L^H serves, since sqrt(m) = L W with W unitary: with Cholesky factors,
//   C' = L_f^H conj(L_b) = U' S V'^H   (the same S),
//   G_f = sqrt(m_f)^-1 U = L_f^-H U',  G_b = sqrt(m_b)^-1 conj(V) = L_b^-H conj(V'),
// so two Hermitian eigendecompositions drop out, leaving two 16-step
// factorisations, two triangular solves and a one-sided Jacobi iteration on the
// columns of C'. Both U' (columns orthogonal to the Jacobi tolerance relative to
// their own norms) and V' (a product of rotations) are unitary to rounding,
// also for small singular values. conj(L_f U') S^-1 equals G_b too, without V',
// but its columns carry the rounding of C' over their own singular value, eps
// s_max / s_j: with it the Vidal distance of the gauge (4-regular graph of 26
// nodes, bond 2, lambdas down to 1.4e-6) was off by 3e-12 relative.
//
// The reference drops message eigenvalues up to eps. The factored form is exact
// only when none are: |G_f|_F^2 = sum 1 / (eigenvalues of m_f) (and the same for
// b), so both norms below 1 / (2 eps) prove every eigenvalue above 2 eps. Other
// edges (also those with a pivot up to eps, a null singular value or non-finite
// entries) are marked and left to the kernel with the eigendecompositions.
//
// In the Jacobi rounds four lanes hold a pair of columns of C' in registers (rows
// sub + 4 i), which move to their next seats by shuffles. The columns of V' stay in
// shared memory, where C' is no longer needed: moving them along by shuffles too
// took 207 us against 189 us for 1,536 edges of bond 16 (148 without V').
#pragma once

#include "dmma.cuh"
#include "reg_linalg.cuh"

namespace dqz {

const double F32_MAX = 3.4028234663852886e38;

__device__ __forceinline__ double safe_inverse(double l, double eps) { return 1.0 / ((l < eps ? F32_MAX : 0.0) + l); }
__device__ __forceinline__ double safe_truncate(double l, double eps) { return l > eps ? l : 0.0; }

constexpr int ES_MAX = 16, ES_LD = 17;
constexpr unsigned long long ES_MARK = 0x7ff80000000000e5ull;  // in lambda[0]: edge left to the other kernel

struct EdgeSmem {
  cd L[2][ES_MAX * ES_LD];  // Cholesky factors, row-major, zero above the diagonal and from bond c on
  cd X[ES_MAX * ES_LD];     // C', the unit left singular vectors, then the right ones, column-major
  double dinv[2][ES_MAX], s[ES_MAX];
  int perm[ES_MAX];
};

__device__ __forceinline__ double quad_sum(double v) {
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  return v + __shfl_xor_sync(0xffffffffu, v, 2);
}
__device__ __forceinline__ cd shfl_cd(cd v, int src) {
  return mk(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src));
}

// L L^H = (m + m^H) / 2 of both messages at once (lanes 0-15: rows of f, 16-31:
// rows of b). False when a pivot is not above eps.
__device__ __forceinline__ bool edge_cholesky(EdgeSmem &S, const cd *mf, const cd *mb, int c, double eps) {
  const int lane = threadIdx.x & 31, side = lane >> 4, r = lane & 15;
  for (int i = lane; i < ES_MAX * ES_MAX; i += 32) {
    const int row = i >> 4, col = i & 15;
    const bool in = row < c && col < c;
    S.L[0][row * ES_LD + col] = in ? mf[row * c + col] : czero();
    S.L[1][row * ES_LD + col] = in ? mb[row * c + col] : czero();
  }
  __syncwarp();
  cd *L = S.L[side];
  cd A[ES_MAX];
#pragma unroll
  for (int k = 0; k < ES_MAX; ++k) {
    const cd u = L[r * ES_LD + k], l = L[k * ES_LD + r];
    A[k] = mk(0.5 * (u.x + l.x), 0.5 * (u.y - l.y));
  }
  __syncwarp();
  bool ok = true;
#pragma unroll
  for (int j = 0; j < ES_MAX; ++j) {
    if (j < c) {
      const double piv = __shfl_sync(0xffffffffu, A[j].x, (lane & 16) + j);
      ok = ok && piv > eps;
      const double inv = fast_rsqrt(piv);  // piv > eps, or the edge is given up
      const cd l = r > j ? cscale(A[j], inv) : (r == j ? mk(piv * inv, 0.0) : czero());
      if (r == j) S.dinv[side][j] = inv;
      L[r * ES_LD + j] = r < c ? l : czero();
      __syncwarp();
#pragma unroll
      for (int k = j + 1; k < ES_MAX; ++k) {
        const cd lk = cconj(L[k * ES_LD + j]);
        A[k] = csub(A[k], cmul(l, lk));
      }
    } else {
      L[r * ES_LD + j] = czero();
    }
  }
  __syncwarp();
  return __all_sync(0xffffffffu, ok);
}

// One rotation of the columns x, y by this lane's rows.
__device__ __forceinline__ void rotate_pair(cd (&x)[4], cd (&y)[4], const PhaseRot &R) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const cd p = cmul(x[i], R.ph), q = y[i];
    x[i] = mk(R.cs * p.x - R.sn * q.x, R.cs * p.y - R.sn * q.y);
    y[i] = mk(R.sn * p.x + R.cs * q.x, R.sn * p.y + R.cs * q.y);
  }
}

// This lane's two seats in the Jacobi rounds: columns of the matrix, rows sub + 4 i.
struct EdgeSeat {
  int grp, sub, ct, cb;
  bool seat, last, has_x, has_y;
  __device__ __forceinline__ EdgeSeat(int c) {
    const int lane = threadIdx.x & 31, np = c + (c & 1), npairs = np / 2;
    grp = lane >> 2;
    sub = lane & 3;
    seat = grp < npairs;
    last = grp == npairs - 1;
    ct = grp == 0 ? 0 : grp + 1;  // rr_pair's step 0
    cb = grp == 0 ? 1 : np - grp;
    has_x = seat && ct < c;
    has_y = seat && cb < c;
  }
  __device__ __forceinline__ void store(cd *X, const cd (&x)[4], const cd (&y)[4], double fx, double fy) const {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (has_x) X[ct * ES_LD + sub + 4 * i] = cscale(x[i], fx);
      if (has_y) X[cb * ES_LD + sub + 4 * i] = cscale(y[i], fy);
    }
  }
  // upper columns one seat down (seat 1's to seat 0's lower place), lower ones one up
  __device__ __forceinline__ void move(cd (&x)[4], cd (&y)[4]) const {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const cd nx = shfl_cd(x[i], (lane + 4) & 31), ny = shfl_cd(y[i], (lane - 4) & 31), ky = y[i];
      y[i] = grp == 0 ? nx : ny;
      if (grp > 0) x[i] = last ? ky : nx;
    }
  }
  __device__ __forceinline__ void move(int &x, int &y) const {
    const int lane = threadIdx.x & 31;
    const int nx = __shfl_sync(0xffffffffu, x, (lane + 4) & 31), ny = __shfl_sync(0xffffffffu, y, (lane - 4) & 31),
              ky = y;
    y = grp == 0 ? nx : ny;
    if (grp > 0) x = last ? ky : nx;
  }
};

// One-sided Jacobi on the columns of S.X (c x c): on return S.X holds the unit
// left singular vectors, S.s the singular values and vx, vy the right singular
// vectors of this lane's seats. False when a value is numerically null
// (hestenes' rule).
__device__ __forceinline__ bool edge_jacobi(EdgeSmem &S, int c, const EdgeSeat &E, cd (&vx)[4], cd (&vy)[4]) {
  const int sub = E.sub, ct = E.ct, cb = E.cb;
  const int np = c + (c & 1), npairs = np / 2;
  const double tol = 1.1e-16 * sqrt((double)c) * 2.0;
  const bool seat = E.seat, has_x = E.has_x, has_y = E.has_y;
  cd x[4], y[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    x[i] = has_x ? S.X[ct * ES_LD + sub + 4 * i] : czero();
    y[i] = has_y ? S.X[cb * ES_LD + sub + 4 * i] : czero();
  }
  __syncwarp();
  for (int i = threadIdx.x & 31; i < ES_MAX * ES_MAX; i += 32)
    S.X[(i >> 4) * ES_LD + (i & 15)] = mk(i >> 4 == (i & 15) ? 1.0 : 0.0, 0.0);
  __syncwarp();
  int px = ct, py = cb;  // the columns in this lane's seats
  double al, be;
  cd ga;
  pair_products(x, y, ga, al, be);
  const double null_thr = hestenes_null_scale(c) * warp_sum(al + be);
  for (int sweep = 0; sweep < 60; ++sweep) {
    bool rotated = false;
    for (int round = 0; round < np - 1; ++round) {
      pair_products(x, y, ga, al, be);
      ga = mk(quad_sum(ga.x), quad_sum(ga.y));
      al = quad_sum(al);
      be = quad_sum(be);
      const bool rot = seat && al > null_thr && be > null_thr && cabs2(ga) > tol * tol * al * be;
      PhaseRot R;
      if (rot && phase_rot(al, be, ga, R)) {
        rotated = true;
        rotate_pair(x, y, R);
        cd *vp = S.X + px * ES_LD + sub, *vq = S.X + py * ES_LD + sub;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          vx[i] = vp[4 * i];
          vy[i] = vq[4 * i];
        }
        rotate_pair(vx, vy, R);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          vp[4 * i] = vx[i];
          vq[4 * i] = vy[i];
        }
      }
      if (npairs > 1) {
        E.move(x, y);
        E.move(px, py);
      }
      __syncwarp();  // the pairs' columns of V change lanes
    }
    if (!__any_sync(0xffffffffu, rotated)) break;
  }
  pair_products(x, y, ga, al, be);
  al = quad_sum(al);
  be = quad_sum(be);
  const double sa = sqrt(al), sb = sqrt(be), ia = 1.0 / sa, ib = 1.0 / sb;
#pragma unroll
  for (int i = 0; i < 4; ++i) {  // a whole number of sweeps: every column is back in its first seat
    vx[i] = S.X[ct * ES_LD + sub + 4 * i];
    vy[i] = has_y ? S.X[cb * ES_LD + sub + 4 * i] : czero();
  }
  __syncwarp();
  E.store(S.X, x, y, ia, ib);
  if (sub == 0) {
    if (has_x) S.s[ct] = sa;
    if (has_y) S.s[cb] = sb;
  }
  __syncwarp();
  return __all_sync(0xffffffffu, (!has_x || al > null_thr) && (!has_y || be > null_thr));
}

// G = L^-H B diag(scale where mask, else 0) with B = S.X's columns in descending
// order, conjugated for the b side; the squared norm of L^-H B over the warp. Lane
// (half, j) holds the rows of parity `half` of column j.
__device__ __forceinline__ double edge_solve(const EdgeSmem &S, int side, int c, unsigned mask, double scale, cd *G) {
  const int lane = threadIdx.x & 31, j = lane & 15, half = lane >> 4;
  const cd *L = S.L[side];
  const double *dinv = S.dinv[side];
  cd u[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    u[k] = j < c ? S.X[S.perm[j] * ES_LD + 2 * k + half] : czero();
    if (side) u[k] = cconj(u[k]);
  }
#pragma unroll
  for (int i = ES_MAX - 1; i >= 0; --i) {
    if (i < c) {
      const cd xi = cscale(shfl_cd(u[i >> 1], j + 16 * (i & 1)), dinv[i]);
      if (half == (i & 1)) u[i >> 1] = xi;
#pragma unroll
      for (int k = 0; k < (i + 1) / 2; ++k) {
        const int row = 2 * k + half;
        const cd l = row < i ? L[i * ES_LD + row] : czero();
        u[k] = csub(u[k], cmulc(l, xi));
      }
    }
  }
  double n = 0.0;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int row = 2 * k + half;
    if (j < c && row < c) {
      n += cabs2(u[k]);
      G[row * c + j] = (mask >> j) & 1u ? cscale(u[k], scale) : czero();
    }
  }
  return warp_sum(n);
}

// One edge by the factored form; false (nothing written but possibly
// orthogonalisers, which the other kernel overwrites) when it does not apply.
__device__ __forceinline__ bool edge_svd_factored(EdgeSmem &S, const cd *mf, const cd *mb, int c, double eps, cd *Gf,
                                                  cd *Gb, double *lam) {
  const int lane = threadIdx.x & 31;
  if (!edge_cholesky(S, mf, mb, c, eps)) return false;
  CTile<2, 2> t;
  t.clear();
  cgemm<true, true, 2>(
      t, [&](int i, int k) { return S.L[0][k * ES_LD + i]; }, [&](int k, int j) { return S.L[1][k * ES_LD + j]; });
  ctile_each(t, [&](int i, int j, cd v) { S.X[j * ES_LD + i] = v; });
  __syncwarp();
  const EdgeSeat seats(c);
  cd vx[4], vy[4];
  if (!edge_jacobi(S, c, seats, vx, vy)) return false;
  warp_sort_desc(S.s, c, S.perm);
  const double sj = lane < c ? S.s[S.perm[lane]] : 0.0;
  const double l0 = sj / sqrt(warp_sum(sj * sj));
  const double kept = l0 > eps ? l0 : 0.0;
  const unsigned mask = __ballot_sync(0xffffffffu, lane < c && kept > eps);
  const double scale = 1.0 / sqrt((double)__popc(mask));
  const double nf = edge_solve(S, 0, c, mask, scale, Gf);
  __syncwarp();
  seats.store(S.X, vx, vy, 1.0, 1.0);
  __syncwarp();
  const double nb = edge_solve(S, 1, c, mask, scale, Gb);
  const double limit = 0.5 / eps;
  if (!(nf < limit) || !(nb < limit)) return false;
  if (lane < c) lam[lane] = kept;
  return true;
}

// Bonds from 17 to 32, one CTA per edge: eigendecompositions of both messages and
// the SVD, each a one-sided Jacobi iteration of 16 warps' halves or of one half.
// For a positive semidefinite message m = U S V^H is V S V^H, so its columns'
// Jacobi gives eigenvalues and eigenvectors; f runs on the first 256 threads, b on
// the others. In the eigenvector bases C is diag(w_f) V_f^H conj(V_b) diag(w_b),
// w = sqrt(eigenvalue), = U'' S V''^H, and
//   G_f = V_f diag(1 / w_f) U'',  G_b = V_b diag(1 / w_b) conj(V''),
// which takes three products on the FP64 tensor cores instead of seven sums over
// the bond per entry. Eigenvalues up to eps are dropped as the reference does, so
// rank-deficient messages (leaves of a graph) are no special case. The Jacobi of a
// matrix with a negative eigenvalue may mix it with a positive one of the same
// size: where a column above rounding has no positive U^H V, and for non-finite
// entries, the edge is marked and left to the kernel with two-sided rotations.
struct EdgeCtaSmem {
  static constexpr int LD = RJ_MAX + 1;
  cd X[2][RJ_MAX * LD], V[2][RJ_MAX * LD];  // column-major: f, b
  double w[2][RJ_MAX], wi[2][RJ_MAX], s[RJ_MAX];
  int perm[RJ_MAX];
  unsigned mask;
  double scale;
  JacobiSmem E[2];
};
constexpr int EC_THREADS = 2 * RJ_THREADS;

// As edge_svd_factored, for c up to 32 and a whole CTA of EC_THREADS.
static __device__ bool edge_svd_cta(EdgeCtaSmem &S, const cd *mf, const cd *mb, int c, double eps, cd *Gf, cd *Gb,
                                    double *lam) {
  constexpr int LD = EdgeCtaSmem::LD;
  const int side = threadIdx.x / RJ_THREADS, tid = threadIdx.x % RJ_THREADS, lane = tid & 31, w = threadIdx.x >> 5;
  const cd *m = side ? mb : mf;
  cd *X = S.X[side], *V = S.V[side];
  __syncthreads();  // the previous edge's reads
  for (int i = tid; i < RJ_MAX * RJ_MAX; i += RJ_THREADS) {
    const int row = i / RJ_MAX, col = i % RJ_MAX;
    X[row * LD + col] = row < c && col < c ? m[row * c + col] : czero();
    V[row * LD + col] = czero();
  }
  jacobi_sync(1 + side);
  cd sym[RJ_MAX * RJ_MAX / RJ_THREADS];  // (m + m^H) / 2
#pragma unroll
  for (int j = 0; j < RJ_MAX * RJ_MAX / RJ_THREADS; ++j) {
    const int i = tid + j * RJ_THREADS, row = i / RJ_MAX, col = i % RJ_MAX;
    const cd u = X[row * LD + col], l = X[col * LD + row];
    sym[j] = mk(0.5 * (u.x + l.x), 0.5 * (u.y - l.y));
  }
  jacobi_sync(1 + side);
#pragma unroll
  for (int j = 0; j < RJ_MAX * RJ_MAX / RJ_THREADS; ++j) {
    const int i = tid + j * RJ_THREADS;
    X[(i % RJ_MAX) * LD + i / RJ_MAX] = sym[j];
  }
  jacobi_sync(1 + side);
  cta_jacobi(X, V, LD, c, S.w[side], S.E[side], 1 + side);
  int bad = 0;
  if (tid < 32) {
    const double s = lane < c ? S.w[side][lane] : 0.0;
    double dot = 0.0;
    if (lane < c)
      for (int i = 0; i < c; ++i) {
        const cd u = X[lane * LD + i], v = V[lane * LD + i];
        dot += u.x * v.x + u.y * v.y;
      }
    double top = s;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) top = fmax(top, __shfl_xor_sync(0xffffffffu, top, o));
    bad = s > 1e-13 * top && !(dot > 0.5);
    bad |= !(top > 0.0 && top < 1e300);  // zero, or not finite (no column was above the null threshold)
    const double l = dot < 0.0 ? -s : s;
    __syncwarp();
    if (lane < c) {
      S.w[side][lane] = sqrt(safe_truncate(l, eps));
      S.wi[side][lane] = sqrt(safe_inverse(l, eps));
    } else {
      S.w[side][lane] = S.wi[side][lane] = 0.0;
    }
  }
  if (__syncthreads_or(bad)) return false;
  // C'' in the first 256 threads' buffer: warps 0-15 take 8 x 8 tiles
  const int r0 = 8 * (w >> 2), c0 = 8 * (w & 3);
  CTile<1, 1> t;
  t.clear();
  cgemm<true, true, 4>(
      t, [&](int i, int k) { return S.V[0][(r0 + i) * LD + k]; }, [&](int k, int j) { return S.V[1][(c0 + j) * LD + k]; });
  ctile_each(t, [&](int i, int j, cd v) { S.X[0][(c0 + j) * LD + r0 + i] = cscale(v, S.w[0][r0 + i] * S.w[1][c0 + j]); });
  for (int i = threadIdx.x; i < RJ_MAX * LD; i += EC_THREADS) S.X[1][i] = czero();
  __syncthreads();
  if (side == 0) cta_jacobi(S.X[0], S.X[1], LD, c, S.s, S.E[0], 1);
  __syncthreads();
  if (w == 0) {
    warp_sort_desc(S.s, c, S.perm);
    const double sj = lane < c ? S.s[S.perm[lane]] : 0.0;
    const double l0 = sj / sqrt(warp_sum(sj * sj));
    const double kept = l0 > eps ? l0 : 0.0;
    const unsigned mask = __ballot_sync(0xffffffffu, lane < c && kept > eps);
    if (lane == 0) {
      S.mask = mask;
      S.scale = 1.0 / sqrt((double)__popc(mask));
    }
    if (lane < c) lam[lane] = kept;
    else S.perm[lane] = 0;
  }
  __syncthreads();
  // the two products: rows r0 .., columns c0 .. in descending order
  const unsigned mask = S.mask;
  const double scale = S.scale;
#pragma unroll
  for (int f = 0; f < 2; ++f) {
    const double *wi = S.wi[f];
    const cd *Vf = S.V[f], *B = S.X[f];
    t.clear();
    const auto la = [&](int i, int k) { return Vf[k * LD + r0 + i]; };
    const auto lb = [&](int k, int j) { return cscale(B[S.perm[c0 + j] * LD + k], wi[k]); };
    if (f == 0)
      cgemm<false, false, 4>(t, la, lb);
    else
      cgemm<false, true, 4>(t, la, lb);
    cd *G = f ? Gb : Gf;
    ctile_each(t, [&](int i, int j, cd v) {
      if (r0 + i < c && c0 + j < c) G[(r0 + i) * c + c0 + j] = (mask >> (c0 + j)) & 1u ? cscale(v, scale) : czero();
    });
  }
  return true;
}

}  // namespace dqz
