// Shared pieces of the degree-3 FP64 tensor-core kernels: slab geometry, an
// item's table entries, slab and message loads.
//
// FULL: every node has degree 3, physical dimension 2 and three bonds of
// dimension CHI (compile-time strides). Otherwise the nodes' bonds, up to CHI,
// are zero-padded to CHI^3 slabs and the physical dimension is any.
#pragma once

#include "dmma.cuh"

namespace dqz {

template <int CHI>
struct K3Cfg {
  static constexpr int WARPS = CHI == 16 ? 8 : 4;
  static constexpr int THREADS = 32 * WARPS;
  static constexpr int TN = CHI / 8;
  static constexpr int S2 = CHI * CHI, S3 = CHI * S2;
  static constexpr int SB = CHI + 1;        // slab strides, odd: see dmma.cuh
  static constexpr int SA = CHI * SB + 1;
  static constexpr int SLAB = CHI * SA;
  static constexpr int MS = CHI + 1;        // message row stride
  static constexpr size_t SMEM = (3 * (size_t)SLAB + 3 * (size_t)CHI * MS) * sizeof(cd);
  static constexpr int MIN_BLOCKS = CHI == 16 ? 1 : 5;
  static constexpr int MPT = (S2 + THREADS - 1) / THREADS;  // message entries per thread
};

// A node's table entries.
struct K3Item {
  int ok, mask;         // supported shape; outputs to compute, bit e
  int d, q[3];          // physical dimension, bonds
  long long toff;       // node tensor
  long long hoff[3];    // messages of the node's half-edges
  const cd *msg[3];     // incoming messages
  long long twoff[3];   // messages of the far ends' half-edges, -1 without one
  int new_edge[3];      // the far end reads this sweep's message (edge pass)
};

// Physical slice s of the item's tensor into a padded slab (asynchronous copies,
// one commit group).
template <int CHI, bool FULL>
__device__ __forceinline__ void k3_load_slab(const cd *__restrict__ T, const K3Item &m, int s, cd *dst) {
  typedef K3Cfg<CHI> C;
  const cd *src = T + m.toff + s;
  if (FULL) {
#pragma unroll 4
    for (int i = threadIdx.x; i < C::S3; i += C::THREADS)
      cp_async16(dst + (i / C::S2) * C::SA + ((i / CHI) % CHI) * C::SB + i % CHI, src + 2 * i);
  } else {
    const int q0 = m.q[0], q1 = m.q[1], q2 = m.q[2], d = m.d;
#pragma unroll 4
    for (int i = threadIdx.x; i < C::S3; i += C::THREADS) {
      const int a = i / C::S2, b = (i / CHI) % CHI, c = i % CHI;
      const bool in = a < q0 && b < q1 && c < q2;
      cp_async16_or_zero(dst + a * C::SA + b * C::SB + c, in ? src + ((a * q1 + b) * q2 + c) * (long long)d : src, in);
    }
  }
  cp_async_commit();
}

// This thread's entries (row r, column c of a CHI x CHI block) of the three
// bonds' matrices, get(f, r, c) inside the bond and zero in the padding.
template <int CHI, bool FULL, typename Get>
__device__ __forceinline__ void k3_load_blocks(const K3Item &m, cd (&x)[3][K3Cfg<CHI>::MPT], Get get) {
  typedef K3Cfg<CHI> C;
#pragma unroll
  for (int f = 0; f < 3; ++f)
#pragma unroll
    for (int j = 0; j < C::MPT; ++j) {
      const int i = threadIdx.x + j * C::THREADS;
      if (i >= C::S2) continue;
      const int r = i / CHI, c = i % CHI;
      x[f][j] = FULL || (r < m.q[f] && c < m.q[f]) ? get(f, r, c) : czero();
    }
}

template <int CHI>
__device__ __forceinline__ void k3_store_blocks(cd *sM, const cd (&x)[3][K3Cfg<CHI>::MPT]) {
  typedef K3Cfg<CHI> C;
#pragma unroll
  for (int f = 0; f < 3; ++f)
#pragma unroll
    for (int j = 0; j < C::MPT; ++j) {
      const int i = threadIdx.x + j * C::THREADS;
      if (i < C::S2) sM[f * CHI * C::MS + (i / CHI) * C::MS + i % CHI] = x[f][j];
    }
}

// One warp's share of a CHI x CHI output in fragment order (position p = pos * 32
// + lane): conflict-free to write and to sum; k3_pos gives row and column.
template <int CHI>
__device__ __forceinline__ void k3_put_share(const CTile<CHI / 8, CHI / 8> &o, cd *dst) {
  const int lane = threadIdx.x & 31;
  int pos = 0;
#pragma unroll
  for (int r = 0; r < CHI / 8; ++r)
#pragma unroll
    for (int n = 0; n < CHI / 8; ++n)
#pragma unroll
      for (int i = 0; i < 2; ++i) dst[(pos++) * 32 + lane] = mk(o.re[r][n][i], o.im[r][n][i]);
}
template <int CHI>
__device__ __forceinline__ void k3_pos(int x, int &row, int &col) {
  const int pos = x >> 5, ln = x & 31;
  row = 8 * (pos / (2 * (CHI / 8))) + (ln >> 2);
  col = 8 * ((pos / 2) % (CHI / 8)) + 2 * (ln & 3) + (pos & 1);
}

inline int k3_sm_count() {
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}

}  // namespace dqz
