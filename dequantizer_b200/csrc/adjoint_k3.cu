// Adjoint of the BP node update for degree-3 nodes with bonds up to 16 on the
// FP64 tensor cores: the transposed message sweep of the implicit adjoint (the
// same derivatives as adjoint.cu, which keeps the other shapes).
//
// With M_e the unnormalised outgoing message of bond e, G_e its cotangent and
//   gM_e = G_e / conj(tr M_e) - conj(sum(conj(G_e) M_e) / (tr M_e)^2) I,  P_e = gM_e^T,
// the cotangent of the incoming message of bond f is
//   gm_f[b][a] = sum over e != f, g the third bond, of
//                sum conj((T x_g m_g)[.., a@f, ..]) (T x_e P_e)[.., b@f, ..].
// Per physical slice that is six contractions of pairs of the six mode products
// A_g = T x_g m_g, B_e = T x_e P_e. Three slabs of shared memory hold T and two
// of them at a time; the other factor of a pair is contracted from the
// accumulator registers where its own bond is the contracted index (dmma.cuh),
// and B_0 is formed twice instead of stored: 13 contractions of 16^4. The M_e do
// not depend on the cotangent, so a caller's loop forms them once
// (dqz_bp_sweep_k3, raw) where the general kernel forms them in every call.
//
// Bound: the FP64 tensor pipe, 26,624 m8n8k4 a node at bond 16 = 56 us a node and
// SM. Measured (random 3-regular graph, 128 nodes, bond 16): a forward and backward
// pass of 21 sweeps and 22 transposed sweeps 4.35 ms, 50.6 ms with adjoint.cu's
// kernel (one warp per entry of a Gram matrix, every buffer in global scratch).
#include "k3.cuh"

using namespace dqz;

namespace {

// A node's table entries and P_e (in sP); the whole CTA, ends with a barrier.
template <int CHI, bool FULL>
__device__ __forceinline__ bool vjp_start(const dqz_graph_t &g, const cd *e2n, const cd *n2e_cot, const cd *raw, int v,
                                          const cd *__restrict__ T, K3Item &m, cd *slab0, cd *sP) {
  typedef K3Cfg<CHI> C;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  __syncthreads();  // the previous node's last reads
  if (tid < 3) {
    const int k = g.node_degree[v], d = g.node_phys[v];
    int chi = 0, tw = -1;
    long long off = 0;
    if (k == 3) {
      const int h = g.node_half[v] + tid;
      const int e = g.half_edge[h];
      chi = e >= 0 ? g.edge_chi[e] : 0;
      off = g.half_msg_off[h];
      tw = g.half_twin[h];
    }
    m.q[tid] = chi;
    m.hoff[tid] = off;
    m.twoff[tid] = tw >= 0 ? g.half_msg_off[tw] : -1;
    m.msg[tid] = e2n + off;
    const bool fine = k == 3 && (FULL ? d == 2 && chi == CHI : chi >= 1 && chi <= CHI);
    const unsigned all = __ballot_sync(0x7u, fine);
    if (tid == 0) {
      m.ok = all == 0x7u;
      m.d = d;
      m.toff = g.node_off[v];
    }
  }
  __syncthreads();
  if (!m.ok) return false;
  k3_load_slab<CHI, FULL>(T, m, 0, slab0);
  if (w < 3) {  // one warp per bond
    const int q = FULL ? CHI : m.q[w];
    const cd *G = n2e_cot + m.hoff[w], *M = raw + m.hoff[w];
    cd t = czero(), s = czero();
    for (int i = lane; i < q; i += 32) t = cadd(t, M[i * q + i]);
    for (int i = lane; i < q * q; i += 32) cfmac(s, G[i], M[i]);
    t = warp_csum(t);
    s = warp_csum(s);
    const cd ct = cconj(t), cs = cconj(cdiv(s, cmul(t, t)));
    cd *P = sP + w * CHI * C::MS;
    for (int i = lane; i < C::S2; i += 32) {  // P[a][a'] = gM[a'][a]
      const int a = i / CHI, ap = i % CHI;
      cd x = czero();
      if (a < q && ap < q) {
        x = cdiv(G[ap * q + a], ct);
        if (a == ap) x = csub(x, cs);
      }
      P[a * C::MS + ap] = x;
    }
  }
  return true;
}

// `add`: e2n_cot receives add + (cotangents swapped to the far ends), i.e. the
// next iterate of x = add + J^H x, and `change` the largest |next - x| entry's bits.
template <int CHI, bool FULL>
__global__ void __launch_bounds__(K3Cfg<CHI>::THREADS, K3Cfg<CHI>::MIN_BLOCKS)
    bp_vjp_k3(dqz_graph_t g, const cd *__restrict__ T, const cd *__restrict__ e2n, const cd *__restrict__ n2e_cot,
              const cd *__restrict__ raw, cd *e2n_cot, const cd *__restrict__ add, unsigned long long *change,
              const int32_t *__restrict__ nodes, int n_nodes, int *error_flag) {
  typedef K3Cfg<CHI> C;
  constexpr int TN = C::TN, SB = C::SB, SA = C::SA, MS = C::MS, S2 = C::S2, NT = C::THREADS;
  constexpr int PER = CHI / C::WARPS;
  typedef CTile<TN, TN> Tile;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cd *slab = reinterpret_cast<cd *>(smem_raw);
  cd *sP = slab + 3 * C::SLAB;
  __shared__ K3Item m;
  const int tid = threadIdx.x, w = tid >> 5;
  const cd *P0 = sP, *P1 = sP + CHI * MS, *P2 = sP + 2 * CHI * MS;
  for (int item = blockIdx.x; item < n_nodes; item += gridDim.x) {
    if (!vjp_start<CHI, FULL>(g, e2n, n2e_cot, raw, nodes[item], T, m, slab, sP)) {
      if (tid == 0) atomicExch(error_flag, 1);
      continue;
    }
    // m_f[i][j] (global, L1-resident; zero in the padding)
    const cd *g0 = m.msg[0], *g1 = m.msg[1], *g2 = m.msg[2];
    const int q0 = FULL ? CHI : m.q[0], q1 = FULL ? CHI : m.q[1], q2 = FULL ? CHI : m.q[2];
    auto at = [&](const cd *p, int q, int i, int j) { return FULL || (i < q && j < q) ? p[i * q + j] : czero(); };
    Tile o0, o1, o2;
    o0.clear();
    o1.clear();
    o2.clear();
    const int d = FULL ? 2 : m.d;
    int p = 0;
#pragma unroll 1
    for (int s = 0; s < d; ++s) {
      const cd *sT = slab + p * C::SLAB;
      cd *X = slab + ((p + 1) % 3) * C::SLAB, *Y = slab + ((p + 2) % 3) * C::SLAB;
      cp_async_wait<0>();
      __syncthreads();
#pragma unroll 1
      for (int j = 0; j < PER; ++j) {  // X = A_2
        const int a = w + j * C::WARPS;
        Tile t;
        t.clear();
        cgemm<false, false, TN>(
            t, [&](int b, int k) { return sT[a * SA + b * SB + k]; }, [&](int k, int c) { return at(g2, q2, c, k); });
        ctile_each(t, [&](int b, int c, cd v) { X[a * SA + b * SB + c] = v; });
      }
      __syncthreads();
#pragma unroll 1
      for (int j = 0; j < PER; ++j) {  // Y = B_1; gm_0 += B_1 conj(A_2)
        const int c = w + j * C::WARPS;
        Tile t;
        t.clear();
        cgemm<false, false, TN>(
            t, [&](int a, int k) { return sT[a * SA + k * SB + c]; }, [&](int k, int b) { return P1[b * MS + k]; });
        ctile_each(t, [&](int a, int b, cd v) { Y[a * SA + b * SB + c] = v; });
        cgemm_regs<false, true>(o0, t, [&](int b, int z) { return X[z * SA + b * SB + c]; });
        // gm_1 += B_0 conj(A_2)
        t.clear();
        cgemm<false, false, TN>(
            t, [&](int b, int k) { return sT[k * SA + b * SB + c]; }, [&](int k, int a) { return P0[a * MS + k]; });
        cgemm_regs<false, true>(o1, t, [&](int a, int z) { return X[a * SA + z * SB + c]; });
      }
      __syncthreads();
#pragma unroll 1
      for (int j = 0; j < PER; ++j) {  // X = A_0; gm_2 += B_1 conj(A_0), both from shared memory (one orientation)
        const int b = w + j * C::WARPS;
        Tile t;
        t.clear();
        cgemm<false, false, TN>(
            t, [&](int c, int k) { return sT[k * SA + b * SB + c]; }, [&](int k, int a) { return at(g0, q0, a, k); });
        ctile_each(t, [&](int c, int a, cd v) { X[a * SA + b * SB + c] = v; });
        __syncwarp();
        cgemm<false, true, TN>(
            o2, [&](int r, int a) { return Y[a * SA + b * SB + r]; }, [&](int a, int z) { return X[a * SA + b * SB + z]; });
      }
      __syncthreads();
#pragma unroll 1
      for (int j = 0; j < PER; ++j) {  // Y = B_2; gm_1 += B_2 conj(A_0)
        const int a = w + j * C::WARPS;
        Tile t;
        t.clear();
        cgemm<false, false, TN>(
            t, [&](int b, int k) { return sT[a * SA + b * SB + k]; }, [&](int k, int c) { return P2[c * MS + k]; });
        ctile_each(t, [&](int b, int c, cd v) { Y[a * SA + b * SB + c] = v; });
        cgemm_regs<false, true>(o1, t, [&](int c, int z) { return X[a * SA + z * SB + c]; });
      }
      __syncthreads();
#pragma unroll 1
      for (int j = 0; j < PER; ++j) {  // X = A_1; gm_0 += B_2 conj(A_1)
        const int c = w + j * C::WARPS;
        Tile t;
        t.clear();
        cgemm<false, false, TN>(
            t, [&](int a, int k) { return sT[a * SA + k * SB + c]; }, [&](int k, int b) { return at(g1, q1, b, k); });
        ctile_each(t, [&](int a, int b, cd v) { X[a * SA + b * SB + c] = v; });
        __syncwarp();
        cgemm<false, true, TN>(
            o0, [&](int r, int b) { return Y[r * SA + b * SB + c]; }, [&](int b, int z) { return X[z * SA + b * SB + c]; });
      }
      __syncthreads();
      if (s + 1 < d) k3_load_slab<CHI, FULL>(T, m, s + 1, Y);
#pragma unroll 1
      for (int j = 0; j < PER; ++j) {  // gm_2 += B_0 conj(A_1)
        const int b = w + j * C::WARPS;
        Tile t;
        t.clear();
        cgemm<false, false, TN>(
            t, [&](int c, int k) { return sT[k * SA + b * SB + c]; }, [&](int k, int a) { return P0[a * MS + k]; });
        cgemm_regs<false, true>(o2, t, [&](int a, int z) { return X[a * SA + b * SB + z]; });
      }
      p = (p + 2) % 3;
    }
    __syncthreads();
    k3_put_share<CHI>(o0, slab + w * S2);
    k3_put_share<CHI>(o1, slab + C::SLAB + w * S2);
    k3_put_share<CHI>(o2, slab + 2 * C::SLAB + w * S2);
    static_assert(C::WARPS * S2 <= C::SLAB, "the shares fit");
    __syncthreads();
    double far = 0.0;
    for (int i = tid; i < 3 * S2; i += NT) {
      const int f = i / S2;
      const cd *src = slab + f * C::SLAB + i % S2;
      cd sum = src[0];
#pragma unroll
      for (int k = 1; k < C::WARPS; ++k) sum = cadd(sum, src[k * S2]);
      int r, c;
      k3_pos<CHI>(i % S2, r, c);
      const int q = FULL ? CHI : m.q[f];
      if (!FULL && (r >= q || c >= q)) continue;
      const int x = r * q + c;
      if (!add) {
        e2n_cot[m.hoff[f] + x] = sum;
      } else if (m.twoff[f] >= 0) {
        const long long at_far = m.twoff[f] + x;
        const cd next = cadd(add[at_far], sum);
        const double dist = sqrt(cabs2(csub(next, n2e_cot[at_far])));
        far = dist > far || dist != dist ? dist : far;
        e2n_cot[at_far] = next;
      }
    }
    if (add) {
      unsigned long long bits = (unsigned long long)__double_as_longlong(far);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long y = __shfl_xor_sync(0xffffffffu, bits, o);
        bits = y > bits ? y : bits;
      }
      if ((tid & 31) == 0) atomicMax(change, bits);
    }
  }
}

// Cotangent of the node tensor, added into t_cot:
//   sum_e T x_e conj(gM_e) x_{f != e} m_f  +  sum_e T x_e P_e x_{f != e} m_f^H,
// each sum the derivative of T x_0 N_0 x_1 N_1 x_2 N_2 in the direction of the D_e
// (N = m, D = conj(gM); then N = m^H, D = P), by the product rule: seven mode
// products each. The last two bonds stay in one warp's registers and slice.
template <int CHI, bool FULL>
__global__ void __launch_bounds__(K3Cfg<CHI>::THREADS, K3Cfg<CHI>::MIN_BLOCKS)
    bp_vjp_k3_tensor(dqz_graph_t g, const cd *__restrict__ T, const cd *__restrict__ e2n,
                     const cd *__restrict__ n2e_cot, const cd *__restrict__ raw, cd *t_cot,
                     const int32_t *__restrict__ nodes, int n_nodes) {
  typedef K3Cfg<CHI> C;
  constexpr int TN = C::TN, SB = C::SB, SA = C::SA, MS = C::MS;
  constexpr int PER = CHI / C::WARPS;
  typedef CTile<TN, TN> Tile;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cd *slab = reinterpret_cast<cd *>(smem_raw);
  cd *sP = slab + 3 * C::SLAB;
  __shared__ K3Item m;
  const int w = threadIdx.x >> 5;
  cd *sT = slab, *U = slab + C::SLAB, *V = slab + 2 * C::SLAB;
  for (int item = blockIdx.x; item < n_nodes; item += gridDim.x) {
    if (!vjp_start<CHI, FULL>(g, e2n, n2e_cot, raw, nodes[item], T, m, sT, sP)) continue;
    const int d = FULL ? 2 : m.d;
#pragma unroll 1
    for (int s = 0; s < d; ++s) {
      cp_async_wait<0>();
      __syncthreads();
#pragma unroll 1
      for (int term = 0; term < 2; ++term) {
        auto N = [&](int f, int i, int j) {
          const int q = FULL ? CHI : m.q[f];
          if (!FULL && (i >= q || j >= q)) return czero();
          return term == 0 ? m.msg[f][i * q + j] : cconj(m.msg[f][j * q + i]);
        };
        auto D = [&](int f, int i, int j) {
          const cd *P = sP + f * CHI * MS;
          return term == 0 ? cconj(P[j * MS + i]) : P[i * MS + j];
        };
#pragma unroll 1
        for (int j = 0; j < PER; ++j) {  // U = T x_0 N_0, V = T x_0 D_0
          const int b = w + j * C::WARPS;
          auto lt = [&](int k, int c) { return sT[k * SA + b * SB + c]; };
          Tile t;
          t.clear();
          cgemm<false, false, TN>(t, [&](int a, int k) { return N(0, a, k); }, lt);
          ctile_each(t, [&](int a, int c, cd v) { U[a * SA + b * SB + c] = v; });
          t.clear();
          cgemm<false, false, TN>(t, [&](int a, int k) { return D(0, a, k); }, lt);
          ctile_each(t, [&](int a, int c, cd v) { V[a * SA + b * SB + c] = v; });
        }
        __syncthreads();
#pragma unroll 1
        for (int j = 0; j < PER; ++j) {
          const int a = w + j * C::WARPS;
          auto lu = [&](int k, int c) { return U[a * SA + k * SB + c]; };
          auto lv = [&](int k, int c) { return V[a * SA + k * SB + c]; };
          Tile y, t;
          y.clear();
          t.clear();  // t = V x_1 N_1 + U x_1 D_1, then y += t x_2 N_2
          cgemm<false, false, TN>(t, [&](int b, int k) { return N(1, b, k); }, lv);
          cgemm<false, false, TN>(t, [&](int b, int k) { return D(1, b, k); }, lu);
          cgemm_regs<false, false>(y, t, [&](int k, int c) { return N(2, c, k); });
          t.clear();  // t = U x_1 N_1, then y += t x_2 D_2
          cgemm<false, false, TN>(t, [&](int b, int k) { return N(1, b, k); }, lu);
          cgemm_regs<false, false>(y, t, [&](int k, int c) { return D(2, c, k); });
          const int q0 = FULL ? CHI : m.q[0], q1 = FULL ? CHI : m.q[1], q2 = FULL ? CHI : m.q[2];
          cd *out = t_cot + m.toff + s;
          ctile_each(y, [&](int b, int c, cd v) {
            if (!FULL && (a >= q0 || b >= q1 || c >= q2)) return;
            cd &x = out[((a * q1 + b) * q2 + c) * (long long)d];
            x = cadd(x, v);
          });
        }
        __syncthreads();
      }
      if (s + 1 < d) k3_load_slab<CHI, FULL>(T, m, s + 1, sT);
    }
  }
}

template <int CHI, bool FULL>
int launch_vjp(const dqz_graph_t *g, const void *T, const void *e2n, const void *n2e_cot, const void *raw,
               void *e2n_cot, const void *add, double *change, void *t_cot, const int32_t *nodes, int n,
               int *error_flag, cudaStream_t stream) {
  typedef K3Cfg<CHI> C;
  const int slots = k3_sm_count() * C::MIN_BLOCKS, grid = n < slots ? n : slots;
  if (e2n_cot) {
    DQZ_SMEM_ATTR_ONCE((bp_vjp_k3<CHI, FULL>), C::SMEM);
    bp_vjp_k3<CHI, FULL><<<grid, C::THREADS, C::SMEM, stream>>>(
        *g, (const cd *)T, (const cd *)e2n, (const cd *)n2e_cot, (const cd *)raw, (cd *)e2n_cot, (const cd *)add,
        reinterpret_cast<unsigned long long *>(change), nodes, n, error_flag);
    DQZ_CHECK_LAUNCH();
  }
  if (t_cot) {
    DQZ_SMEM_ATTR_ONCE((bp_vjp_k3_tensor<CHI, FULL>), C::SMEM);
    bp_vjp_k3_tensor<CHI, FULL><<<grid, C::THREADS, C::SMEM, stream>>>(
        *g, (const cd *)T, (const cd *)e2n, (const cd *)n2e_cot, (const cd *)raw, (cd *)t_cot, nodes, n);
    DQZ_CHECK_LAUNCH();
  }
  return DQZ_OK;
}

}  // namespace

extern "C" int dqz_bp_vjp_k3(const dqz_graph_t *g, int32_t max_chi, int32_t uniform, const void *tensors,
                             const void *e2n, const void *n2e_cot, const void *raw, void *e2n_cot, const void *add,
                             double *max_change, void *t_cot, const int32_t *nodes, int32_t n_nodes,
                             int32_t *error_flag, cudaStream_t stream) {
  if (!g || !tensors || !e2n || !n2e_cot || !raw || !nodes || !error_flag || n_nodes < 0) return DQZ_ERR_ARG;
  if ((!e2n_cot && !t_cot) || (add && (!max_change || !e2n_cot))) return DQZ_ERR_ARG;
  if (max_chi <= 0 || max_chi > 16 || (uniform && max_chi != 8 && max_chi != 16)) return DQZ_ERR_UNSUPPORTED;
  if (n_nodes == 0) return DQZ_OK;
  if (uniform)
    return max_chi == 16 ? launch_vjp<16, true>(g, tensors, e2n, n2e_cot, raw, e2n_cot, add, max_change, t_cot, nodes,
                                                n_nodes, error_flag, stream)
                         : launch_vjp<8, true>(g, tensors, e2n, n2e_cot, raw, e2n_cot, add, max_change, t_cot, nodes,
                                               n_nodes, error_flag, stream);
  return max_chi > 8 ? launch_vjp<16, false>(g, tensors, e2n, n2e_cot, raw, e2n_cot, add, max_change, t_cot, nodes,
                                             n_nodes, error_flag, stream)
                     : launch_vjp<8, false>(g, tensors, e2n, n2e_cot, raw, e2n_cot, add, max_change, t_cot, nodes,
                                            n_nodes, error_flag, stream);
}
