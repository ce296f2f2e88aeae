// Simple update (tensor_ops.py:265-389) of jobs whose factors fit the registers
// of a CTA: up to 256 rows of other bonds and 32 columns a side (bonds up to 16
// between degree-3 nodes with a rank-2 gate, and everything smaller). Three
// launches, each with its own shape of parallelism:
//  1. a CTA per side of a job: B = Q_B R_B (the lambda-weighted node tensor),
//     S = R_B h = Q_S R_S, both Householder QRs on columns held in registers
//     (reg_linalg.cuh); reflectors and R_S go to a workspace slice of the job;
//  2. a CTA per job: core R_u diag(lambda) R_v^T, its QR-preconditioned one-sided
//     Jacobi SVD (cta_jacobi), truncation, entropy and error; the kept singular
//     vectors go to the workspace, lambda and the bond dimension to their tables;
//  3. a CTA per side: Gamma = (Q_B x I) Q_S [U; 0] / lambda, the reflectors applied
//     to columns in registers, each warp on its own (no barrier).
// The algebra is that of the cluster form in gates.cu (two-step QR, same
// conventions and tolerances). That form ran one job per pair of SMs through all
// phases, with the matrices in shared memory or L2 and the SVD repeated in both
// CTAs; here the QRs fill the registers, the SVDs run several to an SM, and the
// workspace crosses L2 twice.
//
// Bound: the chain of dependent columns (QR: one barrier per column) and Jacobi
// rounds, not the FP64 pipe. Measured at bond 16: one wave 98 + 210 + 57 us; a
// layer of 1,500 gates in 11 node-disjoint levels 9.1 ms with its host part
// (19.5-20 ms on the cluster forms, 33.9 ms on the one-CTA kernel), 3,600 gates
// 16.4 ms (34.9, 55.9); at bond 8 1,500 gates 3.5 ms (4.2).
//
// Jobs outside these limits are left unmarked for the other kernels. The tables a
// job reads (bond dimensions, the other bonds' lambdas) are not those any job of
// the batch writes (node-disjoint edges), except its own edge's, which launch 3
// therefore takes from the job's slice.
#include "reg_linalg.cuh"
#include "su.cuh"

using namespace dqz;

namespace {

constexpr int SR_ROWS = 256, SR_COLS = 32, SR_SROWS = 64;
constexpr int SR_SIDE_THREADS = 256, SR_LD = 33;

struct SrDesc {  // a side of a job, as it was before the update
  SufDims D;
  int node, slot, k, d, ce, r, rank, mu;
  int dims[DQZ_MAX_DEGREE];
};

// Workspace slice of a job, in complex entries: per side B's and S's reflectors
// with R, their taus, the kept singular vectors, the descriptor.
struct SrSlice {
  long long vb, s, taub, taus, x, desc, side;
};
__host__ __device__ inline SrSlice sr_slice(int max_rows) {
  const int rows = max_rows < SR_ROWS ? max_rows : SR_ROWS;
  SrSlice o;
  o.vb = 0;
  o.s = o.vb + (long long)rows * SR_COLS;
  o.taub = o.s + SR_SROWS * SR_COLS;
  o.taus = o.taub + SR_COLS;
  o.x = o.taus + SR_COLS;
  o.desc = o.x + SR_COLS * SR_COLS;
  o.side = o.desc + (sizeof(SrDesc) + sizeof(cd) - 1) / sizeof(cd);
  return o;
}

__device__ __forceinline__ bool sr_fits(const SUSide &S, const SufDims &D) {
  return D.MB <= SR_ROWS && D.KB <= SR_COLS && D.KS <= SR_COLS && D.MS <= SR_SROWS;
}

// Offset (without the updated bond and the physical index, strides st) and weight
// of row b of the other bonds.
// lam: the bonds' lambdas (or their safe inverses) in shared memory, DQZ_MAX_CHI a bond.
__device__ __forceinline__ void sr_row(const SrDesc &S, const double *lam, const long long *st, int b, int &off,
                                       double &wt) {
  unsigned rem = (unsigned)b;
  long long o = 0;
  wt = 1.0;
  for (int f = S.k - 1; f >= 0; --f) {
    if (f == S.slot) continue;
    const unsigned df = (unsigned)S.dims[f], q = rem / df;
    const int a = (int)(rem - q * df);
    rem = q;
    o += a * st[f];
    wt *= lam[f * DQZ_MAX_CHI + a];
  }
  off = (int)o;
}

struct SideSmem {
  cd v[4 * SR_ROWS];
  cd R[SR_COLS * SR_LD];  // R_B, column-major
  cd tau[SR_COLS];
  double red[48], lam[DQZ_MAX_DEGREE * DQZ_MAX_CHI];
  long long st[DQZ_MAX_DEGREE];
};

template <int ROWS>
__device__ __forceinline__ void sr_side(const SrDesc &S, const cd *__restrict__ T, const cd *__restrict__ H, cd *ws,
                                        const SrSlice &o, SideSmem &sm) {
  constexpr int W = SR_SIDE_THREADS / 32, CPW = SR_COLS / W;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const SufDims &D = S.D;
  const int d = S.d;
  {  // B[b, (a, i)] = wt(b) T[.., a, .., i]
    cd a[CPW][ROWS];
    int off[ROWS];
    double wt[ROWS];
#pragma unroll
    for (int t = 0; t < ROWS; ++t) {
      off[t] = 0;
      wt[t] = 0.0;
      if (lane + 32 * t < D.MB) sr_row(S, sm.lam, sm.st, lane + 32 * t, off[t], wt[t]);
    }
#pragma unroll
    for (int ci = 0; ci < CPW; ++ci) {
      const int c = w + W * ci;
      const long long base = (c / d) * sm.st[S.slot] + c % d;
#pragma unroll
      for (int t = 0; t < ROWS; ++t)
        a[ci][t] = c < D.KB && lane + 32 * t < D.MB ? cscale(T[off[t] + base], wt[t]) : czero();
    }
    reg_qr<W, CPW, ROWS>(a, D.MB, D.KB, sm.v, sm.tau);
#pragma unroll
    for (int ci = 0; ci < CPW; ++ci) {
      const int c = w + W * ci;
      if (c >= D.KB) continue;
#pragma unroll
      for (int t = 0; t < ROWS; ++t)
        if (lane + 32 * t < D.MB) ws[o.vb + (long long)c * D.MB + lane + 32 * t] = a[ci][t];
      sm.R[c * SR_LD + lane] = lane <= c && lane < D.muB ? a[ci][0] : czero();
    }
    if (tid < D.muB) ws[o.taub + tid] = sm.tau[tid];
    __syncthreads();
  }
  {  // S[(c, o), (a, rho)] = sum_i R_B[c, (a, i)] h[rho][o][i], normalised
    cd s[CPW][2];
    double n2 = 0.0;
#pragma unroll
    for (int ci = 0; ci < CPW; ++ci) {
      const int C = w + W * ci, a = C / S.r, rho = C % S.r;
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        const int row = lane + 32 * t, c = row / d, oo = row % d;
        cd x = czero();
        if (C < D.KS && row < D.MS)
          for (int i = 0; i < d; ++i) {
            const int cb = a * d + i;
            if (cb >= c) cfma(x, sm.R[cb * SR_LD + c], H[(rho * d + oo) * d + i]);
          }
        s[ci][t] = x;
        n2 += cabs2(x);
      }
    }
    n2 = block_sum(n2, sm.red);
    const double inv = 1.0 / sqrt(n2);
#pragma unroll
    for (int ci = 0; ci < CPW; ++ci)
#pragma unroll
      for (int t = 0; t < 2; ++t) s[ci][t] = cscale(s[ci][t], inv);
    reg_qr<W, CPW, 2>(s, D.MS, D.KS, sm.v, sm.tau);
#pragma unroll
    for (int ci = 0; ci < CPW; ++ci) {
      const int c = w + W * ci;
      if (c >= D.KS) continue;
#pragma unroll
      for (int t = 0; t < 2; ++t)
        if (lane + 32 * t < D.MS) ws[o.s + (long long)c * D.MS + lane + 32 * t] = s[ci][t];
    }
    if (tid < D.muS) ws[o.taus + tid] = sm.tau[tid];
  }
}

__global__ void __launch_bounds__(SR_SIDE_THREADS) su_side_kernel(dqz_graph_t g, const cd *Tall, const double *lambdas,
                                                                  const int32_t *edges, const uint8_t *ctrl_first,
                                                                  const cd *halves, const int32_t *ranks, int first_job,
                                                                  int max_rank, int max_rows, uint8_t *done, cd *gws) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  SideSmem &sm = *reinterpret_cast<SideSmem *>(smem_raw);
  __shared__ SrDesc desc;
  __shared__ const double *lam[DQZ_MAX_DEGREE];
  __shared__ int fits_sh;
  const int j = first_job + (int)(blockIdx.x >> 1), side = (int)(blockIdx.x & 1);
  if (threadIdx.x == 0) {
    const int e = edges[j];
    const bool first = ctrl_first[j] != 0;
    SUSide S[2];
    SufDims D[2];
    const int r = ranks[j];
    bool fits = true;
    for (int q = 0; q < 2; ++q) {
      su_load_side(g, lambdas, g.edge_half[2 * e + ((q == 0) == first ? 0 : 1)], S[q]);
      suf_dims(S[q], r, D[q]);
      fits = fits && S[q].M <= max_rows && sr_fits(S[q], D[q]);
    }
    if (side == 0) done[j] = fits ? 1 : 0;
    fits_sh = fits;
    const SUSide &X = S[side];
    const int kk = D[0].muS < D[1].muS ? D[0].muS : D[1].muS;
    desc.D = D[side];
    desc.node = X.node;
    desc.slot = X.slot;
    desc.k = X.k;
    desc.d = X.d;
    desc.ce = X.dims[X.slot];
    desc.r = r;
    desc.mu = D[side].muS;
    desc.rank = (max_rank > 0 && max_rank < kk) ? max_rank : kk;
    for (int f = 0; f < X.k; ++f) {
      desc.dims[f] = X.dims[f];
      lam[f] = X.lam[f];
      sm.st[f] = X.stride[f];
    }
  }
  __syncthreads();
  if (!fits_sh) return;
  const SrSlice o = sr_slice(max_rows);
  cd *ws = gws + (long long)blockIdx.x * o.side;
  const cd *T = Tall + g.node_off[desc.node];
  const cd *H = halves + ((long long)j * 2 + side) * SU_HALF_STRIDE;
  for (int i = threadIdx.x; i < desc.k * DQZ_MAX_CHI; i += SR_SIDE_THREADS)
    if (i % DQZ_MAX_CHI < desc.dims[i / DQZ_MAX_CHI]) sm.lam[i] = lam[i / DQZ_MAX_CHI][i % DQZ_MAX_CHI];
  __syncthreads();
  if (desc.D.MB <= 64)
    sr_side<2>(desc, T, H, ws, o, sm);
  else
    sr_side<8>(desc, T, H, ws, o, sm);
  if (threadIdx.x == 0) *reinterpret_cast<SrDesc *>(ws + o.desc) = desc;
}

struct CoreSmem {
  cd A[2][SR_COLS * SR_LD];  // R_u, R_v; then the core's reflectors, and R^H -> left vectors
  cd V[SR_COLS * SR_LD];
  cd v[4 * 32], tau[SR_COLS];
  JacobiSmem E;
  double red[48], sv[SR_COLS], lam[SR_COLS], lam_k[SR_COLS];  // lam_k: lambda x 1_r
  int perm[SR_COLS], acc[SR_COLS];
};

__global__ void __launch_bounds__(RJ_THREADS, 2) su_core_kernel(dqz_graph_t g, double *lambdas, const int32_t *edges,
                                                             int first_job, double eps, int max_rows,
                                                             const uint8_t *done, cd *gws, double *err_out,
                                                             double *ent_out) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  CoreSmem &sm = *reinterpret_cast<CoreSmem *>(smem_raw);
  constexpr int W = RJ_THREADS / 32, CPW = SR_COLS / W;
  const int j = first_job + (int)blockIdx.x;
  if (!done[j]) return;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const SrSlice o = sr_slice(max_rows);
  cd *wu = gws + 2ll * blockIdx.x * o.side, *wv = wu + o.side;
  const SrDesc &du = *reinterpret_cast<const SrDesc *>(wu + o.desc), &dv = *reinterpret_cast<const SrDesc *>(wv + o.desc);
  const int e = edges[j];
  const int K = du.D.KS, mu = du.mu, mv = dv.mu, r = du.r, rank = du.rank;
  const int msu = du.D.MS, msv = dv.D.MS;
  cd *Ru = sm.A[0], *Rv = sm.A[1];  // row-major: R[i * LD + c]
#pragma unroll
  for (int t = 0; t < SR_COLS * SR_COLS / RJ_THREADS; ++t) {
    const int x = tid + t * RJ_THREADS;
    const int c = x / SR_COLS, i = x % SR_COLS;
    Ru[i * SR_LD + c] = i < mu && c < K && c >= i ? wu[o.s + (long long)c * msu + i] : czero();
    Rv[i * SR_LD + c] = i < mv && c < K && c >= i ? wv[o.s + (long long)c * msv + i] : czero();
  }
  double *lam_e = lambdas + g.edge_lam_off[e];
  for (int c = tid; c < K; c += RJ_THREADS) sm.lam_k[c] = lam_e[c / r];
  __syncthreads();
  // Z = core (tall) or core^H, zr x kk, core = R_u diag(lambda x 1_r) R_v^T
  const bool tall = mu >= mv;
  const int kk = tall ? mv : mu, zr = tall ? mu : mv;
  cd z[CPW][1];
#pragma unroll
  for (int ci = 0; ci < CPW; ++ci) {
    const int col = w + W * ci;
    cd x = czero();
    if (lane < zr && col < kk) {
      const cd *a = Ru + (tall ? lane : col) * SR_LD, *b = Rv + (tall ? col : lane) * SR_LD;
      for (int c = lane > col ? lane : col; c < K; ++c) cfma(x, cscale(a[c], sm.lam_k[c]), b[c]);
      if (!tall) x = cconj(x);
    }
    z[ci][0] = x;
  }
  reg_qr<W, CPW, 1>(z, zr, kk, sm.v, sm.tau);  // its barriers order the reads of R_u, R_v before the writes below
  cd *Zq = sm.A[0], *X = sm.A[1];  // reflectors (column-major), R^H (column-major)
#pragma unroll
  for (int ci = 0; ci < CPW; ++ci) {
    const int col = w + W * ci;
    if (col >= kk) continue;
    Zq[col * SR_LD + lane] = z[ci][0];
    if (lane < kk) X[lane * SR_LD + col] = lane <= col ? cconj(z[ci][0]) : czero();
  }
  __syncthreads();
  cta_jacobi(X, sm.V, SR_LD, kk, sm.sv, sm.E);
  sort_desc(sm.sv, kk, sm.perm);
  double n2 = 0.0;
  for (int c = tid; c < kk; c += RJ_THREADS) {
    const double l = su_safe_truncate(sm.sv[sm.perm[c]], eps);
    sm.lam[c] = l;
    n2 += l * l;
    // null columns among the kept ones are completed below; the others are never read
    sm.acc[sm.perm[c]] = (sm.sv[sm.perm[c]] > 0.0 || c >= rank) ? 1 : 0;
  }
  n2 = block_sum(n2, sm.red);
  if (w == 0) {  // kk <= 32: a lane per value
    const double p = lane < kk ? sm.lam[lane] * sm.lam[lane] / n2 : 0.0;
    const double ent = warp_sum(p > 0.0 ? -p * log(p) : 0.0), er = warp_sum(lane >= rank ? p : 0.0);
    if (lane == 0) {
      err_out[j] = sqrt(er);
      ent_out[j] = ent;
    }
  }
  complete_orthonormal(X, SR_LD, kk, kk, sm.acc);
  // left vectors of Z: Q [V_x; 0] (orthonormal also for null singular values); right ones: the columns of X
  cd q[CPW][1];
#pragma unroll
  for (int ci = 0; ci < CPW; ++ci) {
    const int p = w + W * ci;
    q[ci][0] = p < rank && lane < kk ? sm.V[sm.perm[p] * SR_LD + lane] : czero();
  }
  reg_apply_q<CPW, 1>(q, Zq, SR_LD, zr, kk, sm.tau);
  cd *xu = wu + o.x, *xv = wv + o.x;  // [p * 32 + row]; the controlled side takes conj of the right vectors
#pragma unroll
  for (int ci = 0; ci < CPW; ++ci) {
    const int p = w + W * ci;
    if (p >= rank) continue;
    const cd other = lane < kk ? X[sm.perm[p] * SR_LD + lane] : czero();
    const cd mine = lane < zr ? q[ci][0] : czero();
    xu[p * SR_COLS + lane] = tall ? mine : other;
    xv[p * SR_COLS + lane] = cconj(tall ? other : mine);
  }
  for (int c = tid; c < rank; c += RJ_THREADS) lam_e[c] = sm.lam[c];
  if (tid == 0) g.edge_chi[e] = rank;
}

template <int ROWS>
__device__ __forceinline__ void sr_write(const SrDesc &S, const double *lam, const cd *ws, const SrSlice &o,
                                         const cd *xs, int ldx, cd *T) {
  constexpr int W = SR_SIDE_THREADS / 32, CPW = SR_COLS / W;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const SufDims &D = S.D;
  const int d = S.d, p = d * S.rank;
  long long nst[DQZ_MAX_DEGREE], st = d;
  for (int f = S.k - 1; f >= 0; --f) {
    nst[f] = st;
    st *= f == S.slot ? S.rank : S.dims[f];
  }
  for (int q0 = 0; q0 < p; q0 += SR_COLS) {
    cd z[CPW][ROWS];
#pragma unroll
    for (int ci = 0; ci < CPW; ++ci) {
      const int q = q0 + w + W * ci, col = q / d, oo = q % d;
#pragma unroll
      for (int t = 0; t < ROWS; ++t)
        z[ci][t] = t == 0 && q < p && lane < D.muB ? xs[col * ldx + lane * d + oo] : czero();
    }
    reg_apply_q<CPW, ROWS>(z, ws + o.vb, D.MB, D.MB, D.muB, ws + o.taub);
#pragma unroll
    for (int t = 0; t < ROWS; ++t) {
      const int b = lane + 32 * t;
      if (b >= D.MB) continue;
      int off;
      double wt;
      sr_row(S, lam, nst, b, off, wt);
#pragma unroll
      for (int ci = 0; ci < CPW; ++ci) {
        const int q = q0 + w + W * ci;
        if (q < p) T[off + (q / d) * nst[S.slot] + q % d] = cscale(z[ci][t], wt);
      }
    }
  }
}

__global__ void __launch_bounds__(SR_SIDE_THREADS) su_write_kernel(dqz_graph_t g, cd *Tall, const double *lambdas,
                                                                   int first_job, double eps, int max_rows,
                                                                   const uint8_t *done, const cd *gws) {
  constexpr int W = SR_SIDE_THREADS / 32, CPW = SR_COLS / W, LDX = SR_SROWS + 1;
  __shared__ cd xs[SR_COLS * LDX];
  __shared__ double lam[DQZ_MAX_DEGREE * DQZ_MAX_CHI];  // safe inverses
  const int j = first_job + (int)(blockIdx.x >> 1);
  if (!done[j]) return;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const SrSlice o = sr_slice(max_rows);
  const cd *ws = gws + (long long)blockIdx.x * o.side;
  const SrDesc &S = *reinterpret_cast<const SrDesc *>(ws + o.desc);
  const int h0 = g.node_half[S.node];
  for (int i = threadIdx.x; i < S.k * DQZ_MAX_CHI; i += SR_SIDE_THREADS) {
    const int f = i / DQZ_MAX_CHI, a = i % DQZ_MAX_CHI;
    if (f != S.slot && a < S.dims[f]) lam[i] = su_safe_inverse(lambdas[g.edge_lam_off[g.half_edge[h0 + f]] + a], eps);
  }
  // X = Q_S [U; 0]
  cd x[CPW][2];
#pragma unroll
  for (int ci = 0; ci < CPW; ++ci) {
    const int p = w + W * ci;
    x[ci][0] = p < S.rank && lane < S.mu ? ws[o.x + p * SR_COLS + lane] : czero();
    x[ci][1] = czero();
  }
  reg_apply_q<CPW, 2>(x, ws + o.s, S.D.MS, S.D.MS, S.D.muS, ws + o.taus);
#pragma unroll
  for (int ci = 0; ci < CPW; ++ci) {
    const int p = w + W * ci;
#pragma unroll
    for (int t = 0; t < 2; ++t) xs[p * LDX + lane + 32 * t] = x[ci][t];
  }
  __syncthreads();
  cd *T = Tall + g.node_off[S.node];
  if (S.D.MB <= 64)
    sr_write<2>(S, lam, ws, o, xs, LDX, T);
  else
    sr_write<8>(S, lam, ws, o, xs, LDX, T);
}

constexpr int SR_CHUNK = 592;  // jobs in flight: four per SM, the workspace of a chunk (214 MB at most) stays bounded

}  // namespace

namespace dqz {

size_t su_reg_scratch_bytes(int n, int max_rows) {
  return (size_t)(n < SR_CHUNK ? n : SR_CHUNK) * 2 * (size_t)sr_slice(max_rows).side * sizeof(cd);
}

int su_reg(const dqz_graph_t *g, void *tensors, double *lambdas, const int32_t *edges, const uint8_t *ctrl_is_first,
           const void *halves, const int32_t *ranks, int n, double eps, int max_rank, int max_rows, double *err,
           double *entropy, uint8_t *done, void *ws, size_t ws_bytes, cudaStream_t stream) {
  DQZ_SMEM_ATTR_ONCE(su_core_kernel, sizeof(CoreSmem));
  DQZ_SMEM_ATTR_ONCE(su_side_kernel, sizeof(SideSmem));
  const size_t fit = ws_bytes / su_reg_scratch_bytes(1, max_rows);
  if (fit == 0) return DQZ_ERR_ARG;
  const int chunk = fit < (size_t)SR_CHUNK ? (int)fit : SR_CHUNK;
  for (int first = 0; first < n; first += chunk) {
    const int m = n - first < chunk ? n - first : chunk;
    su_side_kernel<<<2 * m, SR_SIDE_THREADS, sizeof(SideSmem), stream>>>(*g, (const cd *)tensors, lambdas, edges, ctrl_is_first,
                                                          (const cd *)halves, ranks, first, max_rank, max_rows, done,
                                                          (cd *)ws);
    DQZ_CHECK_LAUNCH();
    su_core_kernel<<<m, RJ_THREADS, sizeof(CoreSmem), stream>>>(*g, lambdas, edges, first, eps, max_rows, done,
                                                                (cd *)ws, err, entropy);
    DQZ_CHECK_LAUNCH();
    su_write_kernel<<<2 * m, SR_SIDE_THREADS, 0, stream>>>(*g, (cd *)tensors, lambdas, first, eps, max_rows, done,
                                                           (const cd *)ws);
    DQZ_CHECK_LAUNCH();
  }
  return DQZ_OK;
}

}  // namespace dqz
