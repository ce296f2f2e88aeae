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
#include "k3.cuh"

using namespace dqz;

namespace {

enum K3Mode { NODES, HALVES, SPLIT };

// `raw`: the outputs without the division by the trace (then no edge pass).
// `change`: the largest |n2e_new - n2e_old| entry, as its bits (non-negative
// doubles order like integers; a NaN orders above all of them and stays).
template <int CHI, K3Mode MODE, bool FULL>
__global__ void __launch_bounds__(K3Cfg<CHI>::THREADS, K3Cfg<CHI>::MIN_BLOCKS)
    bp_k3_dmma(dqz_graph_t g, const cd *__restrict__ T, const cd *n2e_old, const cd *e2n_old, cd *n2e_new, cd *e2n_new,
               const uint8_t *__restrict__ src_sel, const uint8_t *__restrict__ edge_new,
               const int32_t *__restrict__ items, int n_items, int raw, unsigned long long *change,
               int *error_flag) {
  typedef K3Cfg<CHI> C;
  constexpr int TN = C::TN, SB = C::SB, SA = C::SA, MS = C::MS, S2 = C::S2, NT = C::THREADS;
  constexpr int PER = CHI / C::WARPS;
  typedef CTile<TN, TN> Tile;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cd *slab = reinterpret_cast<cd *>(smem_raw);
  cd *sM = slab + 3 * C::SLAB;
  __shared__ K3Item meta[2];
  __shared__ cd trace_sh[3];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;

  // next item's table entries, thread q < 3 for half-edge q, one dependent level a call
  int c_it = -1, c_e = 0, c_v = 0, c_h0 = 0, c_k = 0, c_d = 0, c_he = -1, c_sel = 0, c_tw = -1, c_new = 0, c_chi = 0;
  long long c_toff = 0, c_hoff = 0, c_twoff = -1;
  auto level0 = [&](int i) {
    c_it = items[MODE == SPLIT ? i / 3 : i];
    c_e = MODE == SPLIT ? i % 3 : 0;
  };
  auto level1 = [&]() { c_v = MODE == HALVES ? g.half_node[c_it] : c_it; };
  auto level2 = [&]() {
    c_h0 = g.node_half[c_v];
    c_k = g.node_degree[c_v];
    c_d = g.node_phys[c_v];
    c_toff = g.node_off[c_v];
  };
  auto level3 = [&]() {
    c_he = c_tw = -1;
    c_sel = DQZ_SRC_E2N_OLD;
    if (c_k != 3) return;
    const int h = c_h0 + tid;
    c_he = g.half_edge[h];
    c_sel = src_sel[h];
    c_hoff = g.half_msg_off[h];
    c_tw = g.half_twin[h];
  };
  auto level4 = [&]() {
    c_chi = c_he >= 0 ? g.edge_chi[c_he] : 0;
    c_twoff = c_tw >= 0 ? g.half_msg_off[c_tw] : -1;
    c_new = (e2n_new && c_tw >= 0) ? edge_new[c_tw] : 0;
  };
  auto publish = [&](K3Item &m) {
    const bool own = c_sel == DQZ_SRC_E2N_OLD;
    m.q[tid] = c_chi;
    m.hoff[tid] = c_hoff;
    m.twoff[tid] = c_twoff;
    m.new_edge[tid] = c_new;
    m.msg[tid] = (own ? e2n_old : (c_sel == DQZ_SRC_N2E_NEW ? n2e_new : n2e_old)) + (own ? c_hoff : c_twoff);
    const bool shape = c_k == 3 && (FULL ? c_d == 2 && c_chi == CHI : c_chi >= 1 && c_chi <= CHI);
    const unsigned all = __ballot_sync(0x7u, shape && (own || c_twoff >= 0));
    if (tid == 0) {
      m.ok = all == 0x7u;
      m.toff = c_toff;
      m.d = c_d;
      m.mask = MODE == NODES ? 7 : 1 << (MODE == HALVES ? c_it - c_h0 : c_e);
    }
  };
  auto load_msgs = [&](const K3Item &m, cd (&x)[3][C::MPT]) {
    k3_load_blocks<CHI, FULL>(m, x, [&](int f, int r, int c) { return m.msg[f][r * (FULL ? CHI : m.q[f]) + c]; });
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
    k3_load_slab<CHI, FULL>(T, meta[buf], 0, dst);
    cd x[3][C::MPT];
    load_msgs(meta[buf], x);
    k3_store_blocks<CHI>(sM, x);
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
    const int d = FULL ? 2 : meta[cur].d;
    Tile o0, o1, o2;  // out_0 transposed, out_1, out_2: this warp's share
    o0.clear();
    o1.clear();
    o2.clear();
    cd xn[3][C::MPT];  // the next item's messages
#pragma unroll 1
    for (int s = 0; s < d; ++s) {
      const bool last = s == d - 1;
      const cd *sT = slab + p * C::SLAB;
      cd *sE = slab + ((p + 1) % 3) * C::SLAB;
      cd *sD = slab + ((p + 2) % 3) * C::SLAB;
      const cd *m0 = sM, *m1 = sM + CHI * MS, *m2 = sM + 2 * CHI * MS;
      if (tid < 3 && has_next) {
        if (FULL && s == 0) level0(next);
        if (FULL && s == 1) level3();
        if (!FULL && last) {
          level0(next);
          level1();
        }
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
        if (FULL && s == 0) level1();
        if (FULL && s == 1) level4();
        if (!FULL && last) {
          level2();
          level3();
        }
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
        if (FULL && s == 0) level2();
        if (!FULL && last) level4();
        if (last) publish(meta[cur ^ 1]);
      }
      __syncthreads();
      // E0's buffer takes the next slab
      if (!last) {
        k3_load_slab<CHI, FULL>(T, meta[cur], s + 1, sE);
      } else if (has_next && meta[cur ^ 1].ok) {
        k3_load_slab<CHI, FULL>(T, meta[cur ^ 1], 0, sE);
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
    if (mask & 1) k3_put_share<CHI>(o0, r0 + w * S2);
    if (mask & 2) k3_put_share<CHI>(o1, r0 + WS + w * S2);
    if (mask & 4) k3_put_share<CHI>(o2, r2 + w * S2);
    if (has_next && meta[cur ^ 1].ok) k3_store_blocks<CHI>(sM, xn);
    __syncthreads();
    const K3Item &m = meta[cur];
    cd *fin = r2 + WS;  // 3 x CHI x MS: the summed outputs, row-major
    for (int i = tid; i < 3 * S2; i += NT) {
      const int e = i / S2, x = i % S2;
      if (!((mask >> e) & 1)) continue;
      const cd *src = (e == 2 ? r2 : r0 + e * WS) + x;
      cd sum = src[0];
#pragma unroll
      for (int k = 1; k < C::WARPS; ++k) sum = cadd(sum, src[k * S2]);
      int row, col;
      k3_pos<CHI>(x, row, col);
      fin[e * CHI * MS + (e == 0 ? col * MS + row : row * MS + col)] = sum;
    }
    __syncthreads();
    if (tid < 3 && ((mask >> tid) & 1)) {
      cd tr = czero();
      for (int i = 0; i < (FULL ? CHI : m.q[tid]); ++i) tr = cadd(tr, fin[tid * CHI * MS + i * MS + i]);
      trace_sh[tid] = tr;
    }
    __syncthreads();
    double far = 0.0;
    for (int i = tid; i < 3 * S2; i += NT) {
      const int e = i / S2, r = (i % S2) / CHI, c = i % CHI;
      if (!((mask >> e) & 1)) continue;
      const int qe = FULL ? CHI : m.q[e];
      if (!FULL && (r >= qe || c >= qe)) continue;
      const int x = r * qe + c;
      const cd y = fin[e * CHI * MS + r * MS + c];
      const cd o = raw ? y : cdiv(y, trace_sh[e]);
      if (change) {
        const double dist = sqrt(cabs2(csub(o, n2e_old[m.hoff[e] + x])));
        far = dist > far || dist != dist ? dist : far;
      }
      n2e_new[m.hoff[e] + x] = o;
      // edge pass: the far end's incoming message
      if (e2n_new && m.twoff[e] >= 0) e2n_new[m.twoff[e] + x] = m.new_edge[e] ? o : n2e_old[m.hoff[e] + x];
    }
    if (change) {
      unsigned long long bits = (unsigned long long)__double_as_longlong(far);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long y = __shfl_xor_sync(0xffffffffu, bits, o);
        bits = y > bits ? y : bits;
      }
      if (lane == 0) atomicMax(change, bits);
    }
    cur ^= 1;
  }
}

struct K3Args {
  const dqz_graph_t *g;
  const void *T, *n2e_old, *e2n_old;
  void *n2e_new, *e2n_new;
  const uint8_t *src_sel, *edge_new;
  int raw;
  unsigned long long *change;
  int *error_flag;
  cudaStream_t stream;
};

template <int CHI, K3Mode MODE, bool FULL>
int launch(const K3Args &a, const int32_t *items, int n) {
  typedef K3Cfg<CHI> C;
  DQZ_SMEM_ATTR_ONCE((bp_k3_dmma<CHI, MODE, FULL>), C::SMEM);
  const int slots = k3_sm_count() * C::MIN_BLOCKS;
  bp_k3_dmma<CHI, MODE, FULL><<<n < slots ? n : slots, C::THREADS, C::SMEM, a.stream>>>(
      *a.g, (const cd *)a.T, (const cd *)a.n2e_old, (const cd *)a.e2n_old, (cd *)a.n2e_new, (cd *)a.e2n_new, a.src_sel,
      a.edge_new, items, n, a.raw, a.change, a.error_flag);
  DQZ_CHECK_LAUNCH();
  return DQZ_OK;
}

// A wave of whole nodes lasts seven products, a wave of single outputs three:
// SPLIT where its waves are the shorter (at most a third of a wave of nodes, or
// two thirds). Measured at bond 16, us: 49 nodes 24.7 split, 43 whole; 98 nodes
// 44 split, 43 whole; 99 nodes 62 split, 42 whole; 296 nodes 121 split, 80 whole.
template <int CHI, bool FULL>
int sweep(const K3Args &a, const int32_t *nodes, int n) {
  const long long slots = (long long)k3_sm_count() * K3Cfg<CHI>::MIN_BLOCKS;
  if (3 * ((3ll * n + slots - 1) / slots) < 7 * ((n + slots - 1) / slots))
    return launch<CHI, SPLIT, FULL>(a, nodes, 3 * n);
  return launch<CHI, NODES, FULL>(a, nodes, n);
}

}  // namespace

namespace dqz {

int bp_k3_halves(const dqz_graph_t *g, int chi, const void *T, const void *n2e_old, const void *e2n_old, void *n2e_new,
                 const uint8_t *src_sel, const int32_t *halves, int n, int *error_flag, cudaStream_t stream) {
  const K3Args a{g, T, n2e_old, e2n_old, n2e_new, nullptr, src_sel, nullptr, 0, nullptr, error_flag, stream};
  if (chi == 16) return launch<16, HALVES, true>(a, halves, n);
  if (chi == 8) return launch<8, HALVES, true>(a, halves, n);
  return DQZ_ERR_UNSUPPORTED;
}

}  // namespace dqz

extern "C" int dqz_bp_sweep_k3(const dqz_graph_t *g, int32_t max_chi, int32_t uniform, const void *tensors,
                               const void *n2e_old, const void *e2n_old, void *n2e_new, void *e2n_new,
                               const uint8_t *src_sel, const uint8_t *edge_new, const int32_t *nodes, int32_t n_nodes,
                               int32_t raw, double *max_change, int32_t *error_flag, cudaStream_t stream) {
  if (!g || !tensors || !n2e_old || !e2n_old || !n2e_new || !src_sel || !nodes || !error_flag || n_nodes < 0)
    return DQZ_ERR_ARG;
  if (e2n_new && (!edge_new || raw)) return DQZ_ERR_ARG;
  if (max_chi <= 0 || max_chi > 16 || (uniform && max_chi != 8 && max_chi != 16)) return DQZ_ERR_UNSUPPORTED;
  if (n_nodes == 0) return DQZ_OK;
  const K3Args a{g, tensors, n2e_old, e2n_old, n2e_new, e2n_new, src_sel, edge_new, raw,
                 reinterpret_cast<unsigned long long *>(max_change), error_flag, stream};
  if (uniform) return max_chi == 16 ? sweep<16, true>(a, nodes, n_nodes) : sweep<8, true>(a, nodes, n_nodes);
  return max_chi > 8 ? sweep<16, false>(a, nodes, n_nodes) : sweep<8, false>(a, nodes, n_nodes);
}
