// FP64 (complex128) BP node update of degree-3 nodes with bonds of dimension
// CHI (8 or 16) and physical dimension 2 on the FP64 tensor cores: the
// random 3-regular workloads' tensor_ops.py:36-60 (pass_through_node), with the
// edge pass (tensor_ops.py:70-76) in the same launch.
//
// With x_f contracting bond f with a message's second index, T_s the physical
// slice s and a, b, c the bonds,
//   out_0[a'][a] = sum_{b,c} conj(T[a',b,c]) (T x_1 m1 x_2 m2)[a,b,c], and cyclic.
// Moving one message of each pair to the conjugated factor leaves four mode
// products for the three outputs instead of six:
//   E0 = T x_0 m0,  E2 = T x_2 m2,  D1 = T x_1 m1^H,  D2 = T x_2 m2^H,
//   out_2 = sum conj(D1) E0,  out_0 = sum conj(D1) E2,  out_1 = sum conj(D2) E0:
// seven 16^4 contractions per slice and node against nine when every output is
// formed alone. D1, D2 and E2 are consumed by the product that follows from
// the accumulator registers; only T, E0 and D1 live in shared memory, three
// slabs with odd strides (dmma.cuh).
//
// One CTA owns one node at a time (persistent grid). Warps split the slices of
// the batch index (two each at bond 16); a slab's three phases are E0 | D1 and
// out_2, D2 and out_1 | E2 and out_0. The buffers rotate: E0's is free after the
// second phase and takes the next slab (the other physical index, or the next
// node) by cp.async while the third runs; the next node's table entries are
// fetched one dependent load per phase, its messages during its predecessor's
// last phase. Each warp keeps its share of the three outputs in registers over
// both slices; they are summed in warp order at the end.
//
// Bound: the FP64 tensor pipe, 57 k cycles of a node's 14,336 m8n8k4 at bond 16
// (30 us a node and SM). Measured at 1,024 nodes, bond 16: 284 us with the edge
// pass (seven rounds of 40 us: 76% of the pipe inside a node), against 657 us for
// the register-tiled FMA kernel (a CTA per half-edge, nine contractions, 41% of
// the DGEMM peak) and its edge-pass launch; 8,190 nodes 2,194 against 5,048 us.
//
// A list of half-edges (HALVES), or one item per output of a short node list
// (SPLIT: a wave of small launches is shorter when the three outputs of a node
// run on three SMs), runs only the three products of that output, in the same
// order, so every form gives the same bits.
#include "dmma.cuh"

using namespace dqz;

namespace {

enum K3Mode { NODES, HALVES, SPLIT };

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
};

// One item's table entries (a node and its three half-edges).
struct K3Item {
  int ok, mask;         // supported shape; outputs to compute, bit e
  long long toff;       // node tensor
  long long hoff[3];    // messages of the node's half-edges
  const cd *msg[3];     // incoming messages
  long long twoff[3];   // messages of the far ends' half-edges, -1 without one
  int new_edge[3];      // the far end reads this sweep's message (edge pass)
};

template <int CHI, K3Mode MODE>
__global__ void __launch_bounds__(K3Cfg<CHI>::THREADS, K3Cfg<CHI>::MIN_BLOCKS)
    bp_k3_dmma(dqz_graph_t g, const cd *__restrict__ T, const cd *n2e_old, const cd *e2n_old, cd *n2e_new, cd *e2n_new,
               const uint8_t *__restrict__ src_sel, const uint8_t *__restrict__ edge_new,
               const int32_t *__restrict__ items, int n_items, int *error_flag) {
  typedef K3Cfg<CHI> C;
  constexpr int TN = C::TN, SB = C::SB, SA = C::SA, MS = C::MS, S2 = C::S2, S3 = C::S3, NT = C::THREADS;
  constexpr int PER = CHI / C::WARPS;
  typedef CTile<TN, TN> Tile;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cd *slab = reinterpret_cast<cd *>(smem_raw);
  cd *sM = slab + 3 * C::SLAB;
  __shared__ K3Item meta[2];
  __shared__ cd trace_sh[3];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;

  // next item's table entries, thread q < 3 for half-edge q, one dependent level a call
  int c_it = -1, c_e = 0, c_v = 0, c_h0 = 0, c_ok = 0, c_he = 0, c_sel = 0, c_tw = 0, c_new = 0, c_chi = 0;
  long long c_toff = 0, c_hoff = 0, c_twoff = 0;
  auto level0 = [&](int i) {
    c_it = items[MODE == SPLIT ? i / 3 : i];
    c_e = MODE == SPLIT ? i % 3 : 0;
  };
  auto level1 = [&]() { c_v = MODE == HALVES ? g.half_node[c_it] : c_it; };
  auto level2 = [&]() {
    c_h0 = g.node_half[c_v];
    c_ok = g.node_degree[c_v] == 3 && g.node_phys[c_v] == 2;
    c_toff = g.node_off[c_v];
  };
  auto level3 = [&]() {
    if (!c_ok) return;
    const int h = c_h0 + tid;
    c_he = g.half_edge[h];
    c_sel = src_sel[h];
    c_hoff = g.half_msg_off[h];
    c_tw = g.half_twin[h];
  };
  auto level4 = [&]() {
    if (!c_ok) return;
    c_chi = c_he >= 0 ? g.edge_chi[c_he] : 0;
    c_twoff = c_tw >= 0 ? g.half_msg_off[c_tw] : -1;
    c_new = (e2n_new && c_tw >= 0) ? edge_new[c_tw] : 0;
  };
  auto publish = [&](K3Item &m) {
    if (tid == 0) {
      m.toff = c_toff;
      m.mask = MODE == NODES ? 7 : 1 << (MODE == HALVES ? c_it - c_h0 : c_e);
    }
    m.hoff[tid] = c_hoff;
    m.twoff[tid] = c_twoff;
    m.new_edge[tid] = c_new;
    const bool own = c_sel == DQZ_SRC_E2N_OLD;
    m.msg[tid] = (own ? e2n_old : (c_sel == DQZ_SRC_N2E_NEW ? n2e_new : n2e_old)) + (own ? c_hoff : c_twoff);
    const bool fine = c_ok && c_chi == CHI && (own || c_twoff >= 0);
    const unsigned all = __ballot_sync(0x7u, fine);
    if (tid == 0) m.ok = all == 0x7u;
  };
  auto load_slab = [&](const K3Item &m, int s, cd *dst) {
    const cd *src = T + m.toff + s;
#pragma unroll 4
    for (int i = tid; i < S3; i += NT) cp_async16(dst + (i / S2) * SA + ((i / CHI) % CHI) * SB + i % CHI, src + 2 * i);
    cp_async_commit();
  };
  constexpr int MPT = (S2 + NT - 1) / NT;  // message entries per thread
  auto load_msgs = [&](const K3Item &m, cd (&x)[3][MPT]) {
#pragma unroll
    for (int q = 0; q < 3; ++q)
#pragma unroll
      for (int j = 0; j < MPT; ++j) {
        const int i = tid + j * NT;
        if (i < S2) x[q][j] = m.msg[q][i];
      }
  };
  auto store_msgs = [&](const cd (&x)[3][MPT]) {
#pragma unroll
    for (int q = 0; q < 3; ++q)
#pragma unroll
      for (int j = 0; j < MPT; ++j) {
        const int i = tid + j * NT;
        if (i < S2) sM[q * CHI * MS + (i / CHI) * MS + i % CHI] = x[q][j];
      }
  };

  // the first item: everything at once
  auto start_item = [&](int i, int buf, cd *dst) {
    if (tid < 3) {
      level0(i);
      level1();
      level2();
      level3();
      level4();
      publish(meta[buf]);
    }
    __syncthreads();
    if (!meta[buf].ok) return;
    load_slab(meta[buf], 0, dst);
    cd x[3][MPT];
    load_msgs(meta[buf], x);
    store_msgs(x);
  };

  int cur = 0, p = 0;  // p: slab buffer holding T
  if (blockIdx.x < n_items) start_item(blockIdx.x, 0, slab);
  for (int item = blockIdx.x; item < n_items; item += gridDim.x) {
    const int next = item + (int)gridDim.x;
    const bool has_next = next < n_items;
    if (!meta[cur].ok) {  // a shape outside this kernel's: flag it, go on
      __syncthreads();  // the previous item's last reads
      if (tid == 0) atomicExch(error_flag, 1);
      if (has_next) start_item(next, cur ^ 1, slab + p * C::SLAB);
      cur ^= 1;
      continue;
    }
    const int mask = MODE == NODES ? 7 : meta[cur].mask;
    Tile o0, o1, o2;  // out_0 transposed, out_1, out_2: this warp's share
    o0.clear();
    o1.clear();
    o2.clear();
    cd xn[3][MPT];  // the next item's messages
#pragma unroll 1
    for (int s = 0; s < 2; ++s) {
      const cd *sT = slab + p * C::SLAB;
      cd *sE = slab + ((p + 1) % 3) * C::SLAB;
      cd *sD = slab + ((p + 2) % 3) * C::SLAB;
      const cd *m0 = sM, *m1 = sM + CHI * MS, *m2 = sM + 2 * CHI * MS;
      if (tid < 3 && has_next) {
        if (s == 0) level0(next);
        else level3();
      }
      cp_async_wait<0>();
      __syncthreads();
      if (mask & 6) {
#pragma unroll 1
        for (int j = 0; j < PER; ++j) {  // E0[a][l][c] = sum_k m0[a][k] T[k][l][c]
          const int l = w + j * C::WARPS;
          Tile e;
          e.clear();
          cgemm<false, false, TN>(
              e, [&](int a, int k) { return m0[a * MS + k]; }, [&](int k, int c) { return sT[k * SA + l * SB + c]; });
          ctile_each(e, [&](int a, int c, cd v) { sE[a * SA + l * SB + c] = v; });
        }
      }
      if (tid < 3 && has_next) {
        if (s == 0) level1();
        else level4();
      }
      __syncthreads();
#pragma unroll 1
      for (int j = 0; j < PER; ++j) {
        const int a = w + j * C::WARPS;
        const cd *Ta = sT + a * SA, *Ea = sE + a * SA;
        if (mask & 5) {  // D1[a][l][c'] = sum_b T[a][b][c'] conj(m1[b][l]), rows c'
          Tile d;
          d.clear();
          cgemm<false, true, TN>(
              d, [&](int c, int b) { return Ta[b * SB + c]; }, [&](int b, int l) { return m1[b * MS + l]; });
          if (mask & 1) ctile_each(d, [&](int c, int l, cd v) { sD[a * SA + l * SB + c] = v; });
          // out_2[c'][c] += sum_l conj(D1[a][l][c']) E0[a][l][c]
          if (mask & 4) cgemm_regs<true, false>(o2, d, [&](int l, int c) { return Ea[l * SB + c]; });
        }
        if (mask & 2) {  // D2[a][b'][k] = sum_c T[a][b'][c] conj(m2[c][k]), rows b'
          Tile d;
          d.clear();
          cgemm<false, true, TN>(
              d, [&](int b, int c) { return Ta[b * SB + c]; }, [&](int c, int k) { return m2[c * MS + k]; });
          // out_1[b'][b] += sum_k conj(D2[a][b'][k]) E0[a][b][k]
          cgemm_regs<true, false>(o1, d, [&](int k, int b) { return Ea[b * SB + k]; });
        }
      }
      if (tid < 3 && has_next) {
        if (s == 0) level2();
        else publish(meta[cur ^ 1]);
      }
      __syncthreads();
      // E0's buffer takes the next slab
      if (s == 0) {
        load_slab(meta[cur], 1, sE);
      } else if (has_next && meta[cur ^ 1].ok) {
        load_slab(meta[cur ^ 1], 0, sE);
        load_msgs(meta[cur ^ 1], xn);
      }
      if (mask & 1) {
#pragma unroll 1
        for (int j = 0; j < PER; ++j) {
          const int l = w + j * C::WARPS;
          const cd *Tl = sT + l * SB, *Dl = sD + l * SB;
          Tile e;  // E2[a][l][c] = sum_k T[a][l][k] m2[c][k], rows a
          e.clear();
          cgemm<false, false, TN>(
              e, [&](int a, int k) { return Tl[a * SA + k]; }, [&](int k, int c) { return m2[c * MS + k]; });
          // out_0[a'][a] += sum_c E2[a][l][c] conj(D1[a'][l][c]), kept as [a][a']
          cgemm_regs<false, true>(o0, e, [&](int c, int ap) { return Dl[ap * SA + c]; });
        }
      }
      p = (p + 1) % 3;
    }
    // ---- sum the warps' shares: T's and D1's buffers of the last slab are free
    cd *r0 = slab + ((p + 2) % 3) * C::SLAB, *r2 = slab + ((p + 1) % 3) * C::SLAB;
    constexpr int WS = C::WARPS * S2;  // one output's shares
    static_assert(2 * WS <= C::SLAB && WS + 3 * CHI * MS <= C::SLAB, "the shares fit two slabs");
    __syncthreads();
    {
      auto part = [&](const Tile &o, cd *dst) {
        int pos = 0;
#pragma unroll
        for (int r = 0; r < TN; ++r)
#pragma unroll
          for (int n = 0; n < TN; ++n)
#pragma unroll
            for (int i = 0; i < 2; ++i) dst[w * S2 + (pos++) * 32 + lane] = mk(o.re[r][n][i], o.im[r][n][i]);
      };
      if (mask & 1) part(o0, r0);
      if (mask & 2) part(o1, r0 + WS);
      if (mask & 4) part(o2, r2);
    }
    if (has_next && meta[cur ^ 1].ok) store_msgs(xn);
    __syncthreads();
    cd *fin = r2 + WS;  // 3 x CHI x MS: the summed outputs, row-major
    for (int i = tid; i < 3 * S2; i += NT) {
      const int e = i / S2, x = i % S2;
      if (!((mask >> e) & 1)) continue;
      const cd *src = (e == 2 ? r2 : r0 + e * WS) + x;
      cd sum = src[0];
#pragma unroll
      for (int k = 1; k < C::WARPS; ++k) sum = cadd(sum, src[k * S2]);
      const int pos = x >> 5, ln = x & 31;
      const int row = 8 * (pos / (2 * TN)) + (ln >> 2), col = 8 * ((pos / 2) % TN) + 2 * (ln & 3) + (pos & 1);
      fin[e * CHI * MS + (e == 0 ? col * MS + row : row * MS + col)] = sum;
    }
    __syncthreads();
    if (tid < 3 && ((mask >> tid) & 1)) {
      cd tr = czero();
      for (int i = 0; i < CHI; ++i) tr = cadd(tr, fin[tid * CHI * MS + i * MS + i]);
      trace_sh[tid] = tr;
    }
    __syncthreads();
    for (int i = tid; i < 3 * S2; i += NT) {
      const int e = i / S2, x = i % S2;
      if (!((mask >> e) & 1)) continue;
      const cd o = cdiv(fin[e * CHI * MS + (x / CHI) * MS + x % CHI], trace_sh[e]);
      const K3Item &m = meta[cur];
      n2e_new[m.hoff[e] + x] = o;
      // edge pass: the far end's incoming message
      if (e2n_new && m.twoff[e] >= 0) e2n_new[m.twoff[e] + x] = m.new_edge[e] ? o : n2e_old[m.hoff[e] + x];
    }
    cur ^= 1;
  }
}

int sm_count() {
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}

template <int CHI, K3Mode MODE>
int launch(const dqz_graph_t *g, const void *T, const void *n2e_old, const void *e2n_old, void *n2e_new, void *e2n_new,
           const uint8_t *src_sel, const uint8_t *edge_new, const int32_t *items, int n, int *error_flag,
           cudaStream_t stream) {
  typedef K3Cfg<CHI> C;
  DQZ_SMEM_ATTR_ONCE((bp_k3_dmma<CHI, MODE>), C::SMEM);
  const int slots = sm_count() * C::MIN_BLOCKS;
  bp_k3_dmma<CHI, MODE><<<n < slots ? n : slots, C::THREADS, C::SMEM, stream>>>(
      *g, (const cd *)T, (const cd *)n2e_old, (const cd *)e2n_old, (cd *)n2e_new, (cd *)e2n_new, src_sel, edge_new,
      items, n, error_flag);
  DQZ_CHECK_LAUNCH();
  return DQZ_OK;
}

// A wave of whole nodes lasts seven products, a wave of single outputs three:
// SPLIT where its waves are the shorter (at most a third of a wave of nodes, or
// two thirds). Measured at bond 16, us: 49 nodes 24.7 split, 43 whole; 98 nodes
// 44 split, 43 whole; 99 nodes 62 split, 42 whole; 296 nodes 121 split, 80 whole.
template <int CHI>
int sweep(const dqz_graph_t *g, const void *T, const void *n2e_old, const void *e2n_old, void *n2e_new, void *e2n_new,
          const uint8_t *src_sel, const uint8_t *edge_new, const int32_t *nodes, int n, int *error_flag,
          cudaStream_t stream) {
  const long long slots = (long long)sm_count() * K3Cfg<CHI>::MIN_BLOCKS;
  const bool split = 3 * ((3ll * n + slots - 1) / slots) < 7 * ((n + slots - 1) / slots);
  if (split)
    return launch<CHI, SPLIT>(g, T, n2e_old, e2n_old, n2e_new, e2n_new, src_sel, edge_new, nodes, 3 * n, error_flag,
                              stream);
  return launch<CHI, NODES>(g, T, n2e_old, e2n_old, n2e_new, e2n_new, src_sel, edge_new, nodes, n, error_flag, stream);
}

}  // namespace

namespace dqz {

int bp_k3_halves(const dqz_graph_t *g, int chi, const void *T, const void *n2e_old, const void *e2n_old, void *n2e_new,
                 const uint8_t *src_sel, const int32_t *halves, int n, int *error_flag, cudaStream_t stream) {
  if (chi == 16)
    return launch<16, HALVES>(g, T, n2e_old, e2n_old, n2e_new, nullptr, src_sel, nullptr, halves, n, error_flag, stream);
  if (chi == 8)
    return launch<8, HALVES>(g, T, n2e_old, e2n_old, n2e_new, nullptr, src_sel, nullptr, halves, n, error_flag, stream);
  return DQZ_ERR_UNSUPPORTED;
}

}  // namespace dqz

extern "C" int dqz_bp_sweep_k3(const dqz_graph_t *g, int32_t chi, const void *tensors, const void *n2e_old,
                               const void *e2n_old, void *n2e_new, void *e2n_new, const uint8_t *src_sel,
                               const uint8_t *edge_new, const int32_t *nodes, int32_t n_nodes, int32_t *error_flag,
                               cudaStream_t stream) {
  if (!g || !tensors || !n2e_old || !e2n_old || !n2e_new || !src_sel || !nodes || !error_flag || n_nodes < 0)
    return DQZ_ERR_ARG;
  if (e2n_new && !edge_new) return DQZ_ERR_ARG;
  if (n_nodes == 0) return DQZ_OK;
  if (chi == 16)
    return sweep<16>(g, tensors, n2e_old, e2n_old, n2e_new, e2n_new, src_sel, edge_new, nodes, n_nodes, error_flag,
                     stream);
  if (chi == 8)
    return sweep<8>(g, tensors, n2e_old, e2n_old, n2e_new, e2n_new, src_sel, edge_new, nodes, n_nodes, error_flag,
                    stream);
  return DQZ_ERR_UNSUPPORTED;
}
