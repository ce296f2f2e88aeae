// Shared by the simple-update kernels (tensor_ops.py:265-389): a side of a job
// and its matrix dimensions.
#pragma once

#include "common.cuh"

namespace dqz {

constexpr int SU_HALF_STRIDE = 4 * DQZ_MAX_PHYS * DQZ_MAX_PHYS;  // complex entries per gate half

__device__ __forceinline__ double su_safe_inverse(double l, double eps) {
  return 1.0 / ((l < eps ? 3.4028234663852886e38 : 0.0) + l);
}
__device__ __forceinline__ double su_safe_truncate(double l, double eps) { return l > eps ? l : 0.0; }

struct SUSide {
  int node, slot, k, d, half0;
  int dims[DQZ_MAX_DEGREE];
  long long stride[DQZ_MAX_DEGREE];
  const double *lam[DQZ_MAX_DEGREE];
  int M;  // rows: d * prod_{f != slot} dims
};

__device__ __forceinline__ void su_load_side(const dqz_graph_t &g, const double *lambdas, int h, SUSide &S) {
  S.node = g.half_node[h];
  NodeShape s;
  load_shape(g, S.node, s);
  S.k = s.k;
  S.d = s.d;
  S.half0 = s.half0;
  S.slot = h - s.half0;
  for (int f = 0; f < s.k; ++f) {
    S.dims[f] = s.dims[f];
    S.stride[f] = s.stride[f];
    S.lam[f] = lambdas + g.edge_lam_off[g.half_edge[s.half0 + f]];
  }
  S.M = (int)(s.size / s.dims[S.slot]);
}

// Dimensions of one side of a job in the two-step QR forms:
//   B = lambda-weighted node tensor, rows b (the other bonds), columns (a, i)
//       (updated bond, physical index): MB x KB;
//   S = R_B with the half gate applied, rows (c, o), columns (a, rho): MS x KS;
//   muB / muS = min(rows, columns): reflector counts, rows of R.
struct SufDims {
  int MB, KB, muB, MS, KS, muS;
};

__device__ __forceinline__ void suf_dims(const SUSide &S, int r, SufDims &D) {
  const int ce = S.dims[S.slot];
  D.MB = S.M / S.d;
  D.KB = ce * S.d;
  D.muB = D.MB < D.KB ? D.MB : D.KB;
  D.MS = D.muB * S.d;
  D.KS = ce * r;
  D.muS = D.MS < D.KS ? D.MS : D.KS;
}

// Largest kept rank of a job: max_rank when it cuts below K = KS, else K.
__host__ __device__ __forceinline__ int suf_rank_bound(int K, int max_rank) {
  return (max_rank > 0 && max_rank < K) ? max_rank : K;
}

}  // namespace dqz
