// FP32 (complex64) BP node update of degree-3 nodes with bonds of dimension CHI (8
// or 16) and physical dimension 2 (tensor_ops.py:36-60), the edge pass
// (tensor_ops.py:70-76) in the same launch: the seven products, phases and buffers
// of bp_k3.cu on FP32 multiply-adds.
//
// A half-warp owns a value of the batch index, all CHI of them at once: its lanes
// form a 4 x 4 grid, each with CHI / 4 rows and columns of the CHI x CHI products in
// registers (rows r0 + 4 r, columns c0 + 4 c). At bond 16 that is 64 multiply-adds
// for eight 8-byte loads a step, where the shared-memory port (128 bytes a cycle
// into registers) and the FP32 pipe take the same time; two by four outputs a lane,
// as before, kept the port busy one and a half times as long as the pipe. D1 is read
// back from its slab, D2 and E2 pass through a block of the half-warp's own.
//
// Sums: 64 products of a half-warp's share in order, the shares as a balanced tree.
// Bound: FP32 pipe and shared-memory port alike (28.7 k cycles of a node's 3.7 M
// multiply-adds and as many of its loads, at bond 16). Measured at 1,024 nodes, bond
// 16: 220 us with the edge pass, against 354 us for a CTA per half-edge, nine
// contractions, with its edge-pass launch. Step loop unrolled by 2: 235, by 8: 226.
#include "k3.cuh"

using namespace dqz;

namespace {

typedef float2 cf;

template <int CHI>
struct F3Cfg {
  static constexpr int THREADS = 16 * CHI, WARPS = CHI / 2;
  static constexpr int RT = CHI / 4;
  static constexpr int S2 = CHI * CHI, S3 = CHI * S2;
  static constexpr int SB = CHI + 1, SA = CHI * SB + 1, SLAB = CHI * SA, MS = CHI + 1;
  static constexpr int OWN = CHI * MS;  // a half-warp's block
  static constexpr size_t SMEM = (3 * (size_t)SLAB + 3 * (size_t)CHI * MS + (size_t)CHI * OWN) * sizeof(cf);
  static constexpr int MIN_BLOCKS = CHI == 16 ? 1 : 4;
};

template <int RT>
struct FTile {
  float re[RT][RT], im[RT][RT];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int r = 0; r < RT; ++r)
#pragma unroll
      for (int c = 0; c < RT; ++c) re[r][c] = im[r][c] = 0.0f;
  }
};

// t += A B over k < CHI; A conjugated when CA, B when CB.
template <int CHI, bool CA, bool CB, typename LA, typename LB>
__device__ __forceinline__ void fgemm(FTile<CHI / 4> &t, LA la, LB lb) {
  constexpr int RT = CHI / 4;
  const int r0 = (threadIdx.x & 15) >> 2, c0 = threadIdx.x & 3;
#pragma unroll 4
  for (int k = 0; k < CHI; ++k) {
    cf a[RT], b[RT];
#pragma unroll
    for (int r = 0; r < RT; ++r) a[r] = la(r0 + 4 * r, k);
#pragma unroll
    for (int c = 0; c < RT; ++c) b[c] = lb(k, c0 + 4 * c);
#pragma unroll
    for (int r = 0; r < RT; ++r) {
      const float ay = CA ? -a[r].y : a[r].y;
#pragma unroll
      for (int c = 0; c < RT; ++c) {
        const float by = CB ? -b[c].y : b[c].y;
        t.re[r][c] = fmaf(a[r].x, b[c].x, t.re[r][c]);
        t.im[r][c] = fmaf(a[r].x, by, t.im[r][c]);
        t.re[r][c] = fmaf(-ay, by, t.re[r][c]);
        t.im[r][c] = fmaf(ay, b[c].x, t.im[r][c]);
      }
    }
  }
}

template <int RT, typename Put>
__device__ __forceinline__ void ftile_each(const FTile<RT> &t, Put put) {
  const int r0 = (threadIdx.x & 15) >> 2, c0 = threadIdx.x & 3;
#pragma unroll
  for (int r = 0; r < RT; ++r)
#pragma unroll
    for (int c = 0; c < RT; ++c) put(r0 + 4 * r, c0 + 4 * c, make_float2(t.re[r][c], t.im[r][c]));
}

// A warp's share (both half-warps): position (r RT + c) 16 + lane.
template <int RT>
__device__ __forceinline__ void f3_put_share(const FTile<RT> &o, cf *dst) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int r = 0; r < RT; ++r)
#pragma unroll
    for (int c = 0; c < RT; ++c) {
      const float x = o.re[r][c] + __shfl_xor_sync(0xffffffffu, o.re[r][c], 16);
      const float y = o.im[r][c] + __shfl_xor_sync(0xffffffffu, o.im[r][c], 16);
      if (lane < 16) dst[(r * RT + c) * 16 + lane] = make_float2(x, y);
    }
}

__device__ __forceinline__ void cp_async8(void *dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}

template <int CHI>
__device__ __forceinline__ void f3_load_slab(const cf *__restrict__ T, long long toff, int s, cf *dst) {
  typedef F3Cfg<CHI> C;
  const cf *src = T + toff + s;
#pragma unroll 4
  for (int i = threadIdx.x; i < C::S3; i += C::THREADS)
    cp_async8(dst + (i / C::S2) * C::SA + ((i / CHI) % CHI) * C::SB + i % CHI, src + 2 * i);
  cp_async_commit();
}

enum F3Mode { NODES, HALVES, SPLIT };

// A node's table entries.
struct F3Item {
  int ok, mask;
  long long toff, hoff[3], twoff[3];
  const cf *msg[3];
  int new_edge[3];
};

template <int CHI, F3Mode MODE>
__global__ void __launch_bounds__(F3Cfg<CHI>::THREADS, F3Cfg<CHI>::MIN_BLOCKS)
    bp_k3_f32(dqz_graph_t g, const cf *__restrict__ T, const cf *n2e_old, const cf *e2n_old, cf *n2e_new, cf *e2n_new,
              const uint8_t *__restrict__ src_sel, const uint8_t *__restrict__ edge_new,
              const int32_t *__restrict__ items, int n_items, int *error_flag) {
  typedef F3Cfg<CHI> C;
  constexpr int RT = C::RT, SB = C::SB, SA = C::SA, MS = C::MS, S2 = C::S2, NT = C::THREADS;
  typedef FTile<RT> Tile;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cf *slab = reinterpret_cast<cf *>(smem_raw);
  cf *sM = slab + 3 * C::SLAB;
  __shared__ F3Item meta[2];
  __shared__ cf trace_sh[3];
  const int tid = threadIdx.x, w = tid >> 5, own = tid >> 4;
  cf *mine = sM + 3 * CHI * MS + own * C::OWN;

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
  auto publish = [&](F3Item &m) {
    const bool old = c_sel == DQZ_SRC_E2N_OLD;
    m.hoff[tid] = c_hoff;
    m.twoff[tid] = c_twoff;
    m.new_edge[tid] = c_new;
    m.msg[tid] = (old ? e2n_old : (c_sel == DQZ_SRC_N2E_NEW ? n2e_new : n2e_old)) + (old ? c_hoff : c_twoff);
    const unsigned all = __ballot_sync(0x7u, c_k == 3 && c_d == 2 && c_chi == CHI && (old || c_twoff >= 0));
    if (tid == 0) {
      m.ok = all == 0x7u;
      m.toff = c_toff;
      m.mask = MODE == NODES ? 7 : 1 << (MODE == HALVES ? c_it - c_h0 : c_e);
    }
  };
  constexpr int MPT = (S2 + NT - 1) / NT;
  auto load_msgs = [&](const F3Item &m, cf (&x)[3][MPT]) {
#pragma unroll
    for (int f = 0; f < 3; ++f)
#pragma unroll
      for (int j = 0; j < MPT; ++j)
        if (tid + j * NT < S2) x[f][j] = m.msg[f][tid + j * NT];
  };
  auto store_msgs = [&](const cf (&x)[3][MPT]) {
#pragma unroll
    for (int f = 0; f < 3; ++f)
#pragma unroll
      for (int j = 0; j < MPT; ++j) {
        const int i = tid + j * NT;
        if (i < S2) sM[f * CHI * MS + (i / CHI) * MS + i % CHI] = x[f][j];
      }
  };
  // the first item: everything at once
  auto start_item = [&](int i, int buf, cf *dst) {
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
    f3_load_slab<CHI>(T, meta[buf].toff, 0, dst);
    cf x[3][MPT];
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
    Tile o0, o1, o2;  // out_0 transposed, out_1, out_2: this half-warp's share
    o0.clear();
    o1.clear();
    o2.clear();
    cf xn[3][MPT];  // the next item's messages
#pragma unroll 1
    for (int s = 0; s < 2; ++s) {
      const cf *sT = slab + p * C::SLAB;
      cf *sE = slab + ((p + 1) % 3) * C::SLAB;
      cf *sD = slab + ((p + 2) % 3) * C::SLAB;
      const cf *m0 = sM, *m1 = sM + CHI * MS, *m2 = sM + 2 * CHI * MS;
      if (tid < 3 && has_next) {
        if (s == 0)
          level0(next);
        else
          level3();
      }
      cp_async_wait<0>();
      __syncthreads();
      if (mask & 6) {  // E0[a][l][c] = sum_k m0[a][k] T[k][l][c]
        const int l = own;
        Tile e;
        e.clear();
        fgemm<CHI, false, false>(
            e, [&](int a, int k) { return m0[a * MS + k]; }, [&](int k, int c) { return sT[k * SA + l * SB + c]; });
        ftile_each(e, [&](int a, int c, cf v) { sE[a * SA + l * SB + c] = v; });
      }
      if (tid < 3 && has_next) {
        if (s == 0)
          level1();
        else
          level4();
      }
      __syncthreads();
      {
        const int a = own;
        const cf *Ta = sT + a * SA, *Ea = sE + a * SA;
        cf *Da = sD + a * SA;
        if (mask & 5) {  // D1[a][l][c'] = sum_b T[a][b][c'] conj(m1[b][l]), rows c'
          Tile d;
          d.clear();
          fgemm<CHI, false, true>(
              d, [&](int c, int b) { return Ta[b * SB + c]; }, [&](int b, int l) { return m1[b * MS + l]; });
          ftile_each(d, [&](int c, int l, cf v) { Da[l * SB + c] = v; });
          __syncwarp();
          // out_2[c'][c] += sum_l conj(D1[a][l][c']) E0[a][l][c]
          if (mask & 4)
            fgemm<CHI, true, false>(
                o2, [&](int c, int l) { return Da[l * SB + c]; }, [&](int l, int c) { return Ea[l * SB + c]; });
        }
        if (mask & 2) {  // D2[a][b'][k] = sum_c T[a][b'][c] conj(m2[c][k]), rows b'
          Tile d;
          d.clear();
          fgemm<CHI, false, true>(
              d, [&](int b, int c) { return Ta[b * SB + c]; }, [&](int c, int k) { return m2[c * MS + k]; });
          ftile_each(d, [&](int b, int k, cf v) { mine[b * MS + k] = v; });
          __syncwarp();
          // out_1[b'][b] += sum_k conj(D2[a][b'][k]) E0[a][b][k]
          fgemm<CHI, true, false>(
              o1, [&](int b, int k) { return mine[b * MS + k]; }, [&](int k, int b) { return Ea[b * SB + k]; });
        }
      }
      if (tid < 3 && has_next) {
        if (s == 0)
          level2();
        else
          publish(meta[cur ^ 1]);
      }
      __syncthreads();
      // E0's buffer takes the next slab
      if (s == 0) {
        f3_load_slab<CHI>(T, meta[cur].toff, 1, sE);
      } else if (has_next && meta[cur ^ 1].ok) {
        f3_load_slab<CHI>(T, meta[cur ^ 1].toff, 0, sE);
        load_msgs(meta[cur ^ 1], xn);
      }
      if (mask & 1) {  // E2[a][l][c] = sum_k T[a][l][k] m2[c][k], rows a
        const int l = own;
        const cf *Tl = sT + l * SB, *Dl = sD + l * SB;
        Tile e;
        e.clear();
        fgemm<CHI, false, false>(
            e, [&](int a, int k) { return Tl[a * SA + k]; }, [&](int k, int c) { return m2[c * MS + k]; });
        ftile_each(e, [&](int a, int c, cf v) { mine[a * MS + c] = v; });
        __syncwarp();
        // out_0[a'][a] += sum_c E2[a][l][c] conj(D1[a'][l][c]), kept as [a][a']
        fgemm<CHI, false, true>(
            o0, [&](int a, int c) { return mine[a * MS + c]; }, [&](int c, int ap) { return Dl[ap * SA + c]; });
        __syncwarp();
      }
      p = (p + 1) % 3;
    }
    // ---- sum the warps' shares: T's and D1's buffers of the last slab are free
    cf *r0 = slab + ((p + 2) % 3) * C::SLAB, *r2 = slab + ((p + 1) % 3) * C::SLAB;
    constexpr int WS = C::WARPS * S2;  // one output's shares
    static_assert(2 * WS <= C::SLAB && WS + 3 * CHI * MS <= C::SLAB, "the shares fit two slabs");
    __syncthreads();
    if (mask & 1) f3_put_share(o0, r0 + w * S2);
    if (mask & 2) f3_put_share(o1, r0 + WS + w * S2);
    if (mask & 4) f3_put_share(o2, r2 + w * S2);
    if (has_next && meta[cur ^ 1].ok) store_msgs(xn);
    __syncthreads();
    const F3Item &m = meta[cur];
    cf *fin = r2 + WS;  // 3 x CHI x MS: the summed outputs, row-major
    for (int i = tid; i < 3 * S2; i += NT) {
      const int e = i / S2, x = i % S2;
      if (!((mask >> e) & 1)) continue;
      const cf *src = (e == 2 ? r2 : r0 + e * WS) + x;
      cf v[C::WARPS];
#pragma unroll
      for (int k = 0; k < C::WARPS; ++k) v[k] = src[k * S2];
#pragma unroll
      for (int h = C::WARPS / 2; h > 0; h >>= 1)
#pragma unroll
        for (int k = 0; k < h; ++k) v[k] = make_float2(v[k].x + v[k + h].x, v[k].y + v[k + h].y);
      const int ln = x & 15, pos = x >> 4, row = (ln >> 2) + 4 * (pos / RT), col = (ln & 3) + 4 * (pos % RT);
      fin[e * CHI * MS + (e == 0 ? col * MS + row : row * MS + col)] = v[0];
    }
    __syncthreads();
    if (tid < 3 && ((mask >> tid) & 1)) {
      cf tr = make_float2(0.0f, 0.0f);
      for (int i = 0; i < CHI; ++i) {
        const cf d = fin[tid * CHI * MS + i * MS + i];
        tr = make_float2(tr.x + d.x, tr.y + d.y);
      }
      trace_sh[tid] = tr;
    }
    __syncthreads();
    for (int i = tid; i < 3 * S2; i += NT) {
      const int e = i / S2, x = i % S2;
      if (!((mask >> e) & 1)) continue;
      const cf y = fin[e * CHI * MS + (x / CHI) * MS + x % CHI], tr = trace_sh[e];
      const float den = tr.x * tr.x + tr.y * tr.y;
      const cf o = make_float2((y.x * tr.x + y.y * tr.y) / den, (y.y * tr.x - y.x * tr.y) / den);
      n2e_new[m.hoff[e] + x] = o;
      // edge pass: the far end's incoming message
      if (e2n_new && m.twoff[e] >= 0) e2n_new[m.twoff[e] + x] = m.new_edge[e] ? o : n2e_old[m.hoff[e] + x];
    }
    cur ^= 1;
  }
}

struct F3Args {
  const dqz_graph_t *g;
  const void *T, *n2e_old, *e2n_old;
  void *n2e_new, *e2n_new;
  const uint8_t *src_sel, *edge_new;
  int *error_flag;
  cudaStream_t stream;
};

template <int CHI, F3Mode MODE>
int launch(const F3Args &a, const int32_t *items, int n) {
  typedef F3Cfg<CHI> C;
  DQZ_SMEM_ATTR_ONCE((bp_k3_f32<CHI, MODE>), C::SMEM);
  const int slots = k3_sm_count() * C::MIN_BLOCKS;
  bp_k3_f32<CHI, MODE><<<n < slots ? n : slots, C::THREADS, C::SMEM, a.stream>>>(
      *a.g, (const cf *)a.T, (const cf *)a.n2e_old, (const cf *)a.e2n_old, (cf *)a.n2e_new, (cf *)a.e2n_new, a.src_sel,
      a.edge_new, items, n, a.error_flag);
  DQZ_CHECK_LAUNCH();
  return DQZ_OK;
}

// Single outputs where their waves (three products of seven) are the shorter, as in bp_k3.cu.
template <int CHI>
int sweep(const F3Args &a, const int32_t *nodes, int n) {
  const long long slots = (long long)k3_sm_count() * F3Cfg<CHI>::MIN_BLOCKS;
  if (3 * ((3ll * n + slots - 1) / slots) < 7 * ((n + slots - 1) / slots)) return launch<CHI, SPLIT>(a, nodes, 3 * n);
  return launch<CHI, NODES>(a, nodes, n);
}

}  // namespace

namespace dqz {

int bp_k3_halves_c64(const dqz_graph_t *g, int chi, const void *T, const void *n2e_old, const void *e2n_old,
                     void *n2e_new, const uint8_t *src_sel, const int32_t *halves, int n, int *error_flag,
                     cudaStream_t stream) {
  const F3Args a{g, T, n2e_old, e2n_old, n2e_new, nullptr, src_sel, nullptr, error_flag, stream};
  if (chi == 16) return launch<16, HALVES>(a, halves, n);
  if (chi == 8) return launch<8, HALVES>(a, halves, n);
  return DQZ_ERR_UNSUPPORTED;
}

}  // namespace dqz

extern "C" int dqz_bp_sweep_k3_c64(const dqz_graph_t *g, int32_t chi, const void *tensors, const void *n2e_old,
                                   const void *e2n_old, void *n2e_new, void *e2n_new, const uint8_t *src_sel,
                                   const uint8_t *edge_new, const int32_t *nodes, int32_t n_nodes, int32_t *error_flag,
                                   cudaStream_t stream) {
  if (!g || !tensors || !n2e_old || !e2n_old || !n2e_new || !src_sel || !nodes || !error_flag || n_nodes < 0)
    return DQZ_ERR_ARG;
  if (e2n_new && !edge_new) return DQZ_ERR_ARG;
  if (chi != 8 && chi != 16) return DQZ_ERR_UNSUPPORTED;
  if (n_nodes == 0) return DQZ_OK;
  const F3Args a{g, tensors, n2e_old, e2n_old, n2e_new, e2n_new, src_sel, edge_new, error_flag, stream};
  return chi == 16 ? sweep<16>(a, nodes, n_nodes) : sweep<8>(a, nodes, n_nodes);
}
