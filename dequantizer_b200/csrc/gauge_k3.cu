// FP64 tensor-core forms of two gauge operations for degree-3 nodes (slabs,
// padding and fragments: k3.cuh, dmma.cuh):
//  * absorb  -- tensor_ops.py:88-93 (absorb_by_node): T x_f G_f^T on every bond,
//               divided by its norm (three bonds of 8 or 16, physical dimension 2);
//  * density -- mappings/density_matrix.py:16-37: T x_f m_f on every bond, then
//               the d x d matrix of its products with conj(T), over its trace
//               (bonds up to 16).
// Both are three mode products a slab. Bond 0 is contracted slab-wide into a
// second slab (warp w: index w of bond 1); bonds 1 and 2 then stay with the warp
// that owns an index of bond 0, the second product taking the first one's tile
// from the registers, and the result never returns to shared memory: the
// absorbed tensor waits in registers for the node's norm, the density sums its
// products with conj(T) at once.
//
// Bound: the FP64 tensor pipe, 6,144 m8n8k4 a slab pair for absorb at bond 16 (13
// us a node and SM), twice that for density's two slabs of each factor.
// Measured (1,024 nodes, bond 16): absorb 189 us (230 with register-tiled FMAs),
// density 193 us (842 with the generic kernel in global scratch).
#include "k3.cuh"

using namespace dqz;

namespace {

// The table entries of node v into m (message blocks at arena + offset); the
// whole CTA, with a barrier before and after.
template <int CHI, bool FULL>
__device__ __forceinline__ bool gk3_item(const dqz_graph_t &g, const cd *arena, int v, K3Item &m) {
  const int tid = threadIdx.x;
  __syncthreads();
  if (tid < 3) {
    const int k = g.node_degree[v], d = g.node_phys[v];
    int chi = 0;
    long long off = 0;
    if (k == 3) {
      const int h = g.node_half[v] + tid;
      const int e = g.half_edge[h];
      chi = e >= 0 ? g.edge_chi[e] : 0;
      off = g.half_msg_off[h];
    }
    m.q[tid] = chi;
    m.msg[tid] = arena + off;
    const bool fine = k == 3 && (FULL ? d == 2 && chi == CHI : chi >= 1 && chi <= CHI);
    const unsigned all = __ballot_sync(0x7u, fine);
    if (tid == 0) {
      m.ok = all == 0x7u;
      m.d = d;
      m.toff = g.node_off[v];
    }
  }
  __syncthreads();
  return m.ok;
}

// U[a'][b][c] = sum_a M(a', a) T[a][b][c] for the warp's indices b.
template <int CHI, typename M0>
__device__ __forceinline__ void gk3_bond0(const cd *sT, cd *U, M0 m0) {
  typedef K3Cfg<CHI> C;
  constexpr int TN = C::TN, SB = C::SB, SA = C::SA;
  const int w = threadIdx.x >> 5;
#pragma unroll 1
  for (int j = 0; j < CHI / C::WARPS; ++j) {
    const int b = w + j * C::WARPS;
    CTile<TN, TN> t;
    t.clear();
    cgemm<false, false, TN>(t, m0, [&](int k, int c) { return sT[k * SA + b * SB + c]; });
    ctile_each(t, [&](int a, int c, cd v) { U[a * SA + b * SB + c] = v; });
  }
}

// y = M1 U_a M2^T (rows b', columns c') for one index a of bond 0.
template <int CHI, typename M1, typename M2>
__device__ __forceinline__ void gk3_bond12(const cd *U, int a, CTile<CHI / 8, CHI / 8> &y, M1 m1, M2 m2) {
  typedef K3Cfg<CHI> C;
  constexpr int TN = C::TN, SB = C::SB, SA = C::SA;
  CTile<TN, TN> t;
  t.clear();
  cgemm<false, false, TN>(t, m1, [&](int k, int c) { return U[a * SA + k * SB + c]; });
  y.clear();
  cgemm_regs<false, false>(y, t, m2);
}

template <int CHI>
__global__ void __launch_bounds__(K3Cfg<CHI>::THREADS, K3Cfg<CHI>::MIN_BLOCKS)
    absorb_k3_dmma(dqz_graph_t g, const cd *__restrict__ Tin, const cd *__restrict__ orth, cd *Tout,
                   const int32_t *__restrict__ sel, int total, int *error_flag) {
  typedef K3Cfg<CHI> C;
  constexpr int TN = C::TN, MS = C::MS, PER = CHI / C::WARPS;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cd *slab = reinterpret_cast<cd *>(smem_raw);
  cd *U = slab + 2 * C::SLAB, *sG = slab + 3 * C::SLAB;
  __shared__ K3Item meta;
  __shared__ double red[48];
  const int w = threadIdx.x >> 5;
  for (int item = blockIdx.x; item < total; item += gridDim.x) {
    if (!gk3_item<CHI, true>(g, orth, sel ? sel[item] : item, meta)) {
      if (threadIdx.x == 0) atomicExch(error_flag, 1);
      continue;
    }
    const K3Item &m = meta;
    k3_load_slab<CHI, true>(Tin, m, 0, slab);
    k3_load_slab<CHI, true>(Tin, m, 1, slab + C::SLAB);
    {
      cd x[3][C::MPT];
      k3_load_blocks<CHI, true>(m, x, [&](int f, int r, int c) { return m.msg[f][r * CHI + c]; });
      k3_store_blocks<CHI>(sG, x);
    }
    const cd *G0 = sG, *G1 = sG + CHI * MS, *G2 = sG + 2 * CHI * MS;  // G_f[a][a'], row-major
    CTile<TN, TN> y[2][PER];
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      if (s == 0)
        cp_async_wait<1>();
      else
        cp_async_wait<0>();
      __syncthreads();
      gk3_bond0<CHI>(slab + s * C::SLAB, U, [&](int a, int k) { return G0[k * MS + a]; });
      __syncthreads();
#pragma unroll
      for (int j = 0; j < PER; ++j)
        gk3_bond12<CHI>(
            U, w + j * C::WARPS, y[s][j], [&](int b, int k) { return G1[k * MS + b]; },
            [&](int k, int c) { return G2[k * MS + c]; });
    }
    double n2 = 0.0;
#pragma unroll
    for (int s = 0; s < 2; ++s)
#pragma unroll
      for (int j = 0; j < PER; ++j) ctile_each(y[s][j], [&](int, int, cd v) { n2 += cabs2(v); });
    const double inv = 1.0 / sqrt(block_sum(n2, red));
    cd *O = Tout + m.toff;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      const int a = w + j * C::WARPS;
#pragma unroll
      for (int s = 0; s < 2; ++s)
        ctile_each(y[s][j], [&](int b, int c, cd v) { O[((a * CHI + b) * CHI + c) * 2 + s] = cscale(v, inv); });
    }
  }
}

template <int CHI, bool FULL>
__global__ void __launch_bounds__(K3Cfg<CHI>::THREADS, K3Cfg<CHI>::MIN_BLOCKS)
    density_k3_dmma(dqz_graph_t g, const cd *__restrict__ T, const cd *__restrict__ e2n,
                    const int32_t *__restrict__ nodes, int total, cd *rho, int *error_flag) {
  typedef K3Cfg<CHI> C;
  constexpr int TN = C::TN, MS = C::MS, SB = C::SB, SA = C::SA, PER = CHI / C::WARPS;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cd *slab = reinterpret_cast<cd *>(smem_raw);
  cd *U = slab + 2 * C::SLAB, *sM = slab + 3 * C::SLAB;
  __shared__ K3Item meta;
  __shared__ cd part[C::WARPS];
  __shared__ cd rho_sh[DQZ_MAX_PHYS * DQZ_MAX_PHYS];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  for (int item = blockIdx.x; item < total; item += gridDim.x) {
    if (!gk3_item<CHI, FULL>(g, e2n, nodes[item], meta)) {
      if (tid == 0) atomicExch(error_flag, 1);
      continue;
    }
    const K3Item &m = meta;
    const int d = FULL ? 2 : m.d;
    {
      cd x[3][C::MPT];
      k3_load_blocks<CHI, FULL>(m, x, [&](int f, int r, int c) { return m.msg[f][r * (FULL ? CHI : m.q[f]) + c]; });
      k3_store_blocks<CHI>(sM, x);
    }
    const cd *m0 = sM, *m1 = sM + CHI * MS, *m2 = sM + 2 * CHI * MS;
    // rho[s][s2] = sum (T_s x m) conj(T_s2): T_s in the first slab, T_s2 in either
    for (int s = 0; s < d; ++s) {
      __syncthreads();
      k3_load_slab<CHI, FULL>(T, m, s, slab);
      const int first = s == 0 ? 1 : 0;
      if (d > 1) k3_load_slab<CHI, FULL>(T, m, first, slab + C::SLAB);
      if (d > 1)
        cp_async_wait<1>();
      else
        cp_async_wait<0>();
      __syncthreads();
      gk3_bond0<CHI>(slab, U, [&](int a, int k) { return m0[a * MS + k]; });
      cp_async_wait<0>();
      __syncthreads();
      CTile<TN, TN> y[PER];
#pragma unroll
      for (int j = 0; j < PER; ++j)
        gk3_bond12<CHI>(
            U, w + j * C::WARPS, y[j], [&](int b, int k) { return m1[b * MS + k]; },
            [&](int k, int c) { return m2[c * MS + k]; });
      for (int s2 = 0; s2 < d; ++s2) {
        const cd *other = slab;
        if (s2 != s) {
          if (s2 != first) {  // a third slice and on: the second slab again
            __syncthreads();
            k3_load_slab<CHI, FULL>(T, m, s2, slab + C::SLAB);
            cp_async_wait<0>();
            __syncthreads();
          }
          other = slab + C::SLAB;
        }
        cd acc = czero();
#pragma unroll
        for (int j = 0; j < PER; ++j) {
          const cd *Ta = other + (w + j * C::WARPS) * SA;
          ctile_each(y[j], [&](int b, int c, cd v) { cfmac(acc, Ta[b * SB + c], v); });
        }
        acc = warp_csum(acc);
        if (lane == 0) part[w] = acc;
        __syncthreads();
        if (tid == 0) {
          cd sum = part[0];
          for (int i = 1; i < C::WARPS; ++i) sum = cadd(sum, part[i]);
          rho_sh[s * d + s2] = sum;
        }
        __syncthreads();
      }
    }
    cd tr = czero();
    for (int i = 0; i < d; ++i) tr = cadd(tr, rho_sh[i * d + i]);
    cd *out = rho + (long long)item * DQZ_MAX_PHYS * DQZ_MAX_PHYS;
    for (int i = tid; i < d * d; i += C::THREADS) out[i] = cdiv(rho_sh[i], tr);
  }
}

template <int CHI>
int launch_absorb(const dqz_graph_t *g, const void *tin, const void *orth, void *tout, const int32_t *sel, int total,
                  int *error_flag, cudaStream_t stream) {
  typedef K3Cfg<CHI> C;
  DQZ_SMEM_ATTR_ONCE(absorb_k3_dmma<CHI>, C::SMEM);
  const int slots = k3_sm_count() * C::MIN_BLOCKS;
  absorb_k3_dmma<CHI><<<total < slots ? total : slots, C::THREADS, C::SMEM, stream>>>(
      *g, (const cd *)tin, (const cd *)orth, (cd *)tout, sel, total, error_flag);
  DQZ_CHECK_LAUNCH();
  return DQZ_OK;
}

template <int CHI, bool FULL>
int launch_density(const dqz_graph_t *g, const void *T, const void *e2n, const int32_t *nodes, int total, void *rho,
                   int *error_flag, cudaStream_t stream) {
  typedef K3Cfg<CHI> C;
  DQZ_SMEM_ATTR_ONCE((density_k3_dmma<CHI, FULL>), C::SMEM);
  const int slots = k3_sm_count() * C::MIN_BLOCKS;
  density_k3_dmma<CHI, FULL><<<total < slots ? total : slots, C::THREADS, C::SMEM, stream>>>(
      *g, (const cd *)T, (const cd *)e2n, nodes, total, (cd *)rho, error_flag);
  DQZ_CHECK_LAUNCH();
  return DQZ_OK;
}

}  // namespace

extern "C" int dqz_absorb_k3(const dqz_graph_t *g, int32_t chi, const void *tensors_in, const void *orth,
                             void *tensors_out, const int32_t *nodes, int32_t n_sel, int32_t *error_flag,
                             cudaStream_t stream) {
  if (!g || !tensors_in || !orth || !tensors_out || !error_flag) return DQZ_ERR_ARG;
  if (nodes && (n_sel < 0 || n_sel > g->n_nodes)) return DQZ_ERR_ARG;
  const int total = nodes ? n_sel : g->n_nodes;
  if (total == 0) return DQZ_OK;
  if (chi == 16) return launch_absorb<16>(g, tensors_in, orth, tensors_out, nodes, total, error_flag, stream);
  if (chi == 8) return launch_absorb<8>(g, tensors_in, orth, tensors_out, nodes, total, error_flag, stream);
  return DQZ_ERR_UNSUPPORTED;
}

extern "C" int dqz_density_k3(const dqz_graph_t *g, int32_t max_chi, int32_t uniform, const void *tensors,
                              const void *e2n, const int32_t *nodes, int32_t n_nodes, void *rho, int32_t *error_flag,
                              cudaStream_t stream) {
  if (!g || !tensors || !e2n || !nodes || !rho || !error_flag || n_nodes < 0) return DQZ_ERR_ARG;
  if (max_chi <= 0 || max_chi > 16 || (uniform && max_chi != 8 && max_chi != 16)) return DQZ_ERR_UNSUPPORTED;
  if (n_nodes == 0) return DQZ_OK;
  if (uniform)
    return max_chi == 16 ? launch_density<16, true>(g, tensors, e2n, nodes, n_nodes, rho, error_flag, stream)
                         : launch_density<8, true>(g, tensors, e2n, nodes, n_nodes, rho, error_flag, stream);
  return max_chi > 8 ? launch_density<16, false>(g, tensors, e2n, nodes, n_nodes, rho, error_flag, stream)
                     : launch_density<8, false>(g, tensors, e2n, nodes, n_nodes, rho, error_flag, stream);
}
