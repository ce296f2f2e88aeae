// Belief-propagation kernels (FP64 / complex128, generic shapes).
//
// Node update, replacing dequantizer/src/tensor_ops.py:36-60
// (pass_through_node) inside the sweep of mappings/belief_propagation.py:24-64.
// One CTA owns one half-edge h = (node v, bond e). It walks the bond-e slices
// T[.., a_e = a, ..] of the node tensor, contracts each slice with the k-1
// incoming messages (mode products in shared memory or CTA scratch), and
// accumulates column a of the outgoing message,
//     m_out[a', a] = sum_x conj(T_slice(a')[x]) Y_a[x],
// then divides by the trace.
//
// The incoming message of every bond is chosen per half-edge (src_sel), which
// reproduces the reference's synchronous sweep (all DQZ_SRC_E2N_OLD), its
// asynchronous sweep in traversal order (a mix, with nodes launched level by
// level) and a flooding schedule (all DQZ_SRC_N2E_OLD).
#include "bp_slices.cuh"

using namespace dqz;

namespace {

constexpr int BP_THREADS = 256;
static_assert(BP_THREADS == SL_THREADS, "the one-launch sweep runs both forms");

__device__ __forceinline__ const cd *incoming_msg(const dqz_graph_t &g, int hf, const cd *n2e_old, const cd *e2n_old,
                                                  const cd *n2e_new, const uint8_t *src_sel) {
  int sel = src_sel[hf];
  if (sel == DQZ_SRC_E2N_OLD) return e2n_old + g.half_msg_off[hf];
  int tw = g.half_twin[hf];
  return (sel == DQZ_SRC_N2E_NEW ? n2e_new : n2e_old) + g.half_msg_off[tw];
}

// Column a of the unnormalised outgoing message of bond e of a node (tensor
// Tv, shape s): out[ap][a] = sum_x conj(T_slice(ap)[x]) Y_a[x], with Y_a the
// bond-e slice a contracted with the k-1 incoming messages; `put(ap, value)`
// stores each entry. bufA / bufB hold two slices. The message at a half-edge h with
// fresh(h) is divided by its trace in `staged`. Whole CTA; ends with a barrier.
struct NeverFresh {
  __device__ __forceinline__ bool operator()(int) const { return false; }
};
template <typename Put, typename Fresh = NeverFresh>
__device__ __forceinline__ void node_slice_column(const dqz_graph_t &g, const cd *__restrict__ Tv, const NodeShape &s,
                                                  int e, const cd *n2e_old, const cd *e2n_old, const cd *n2e_new,
                                                  const uint8_t *__restrict__ src_sel, int a, cd *bufA, cd *bufB,
                                                  Put put, cd *staged = nullptr, Fresh fresh = Fresh()) {
  const int ce = s.dims[e];
  const long long Re = s.stride[e];
  const long long P = s.size / ce;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  // P < 2^31 for every slice held on chip: the division by Re via FastDiv
  const bool small = P * ce < (1ll << 31);
  const FastDiv fRe((unsigned)(small ? Re : 1));
  if (small) {
    for (unsigned x = threadIdx.x; x < (unsigned)P; x += blockDim.x) {
      const unsigned l = fRe.div(x), r = x - l * (unsigned)Re;
      bufA[x] = Tv[(l * (unsigned)ce + (unsigned)a) * (unsigned)Re + r];
    }
  } else {
    for (long long x = threadIdx.x; x < P; x += blockDim.x) {
      long long l = x / Re, r = x - l * Re;
      bufA[x] = Tv[(l * ce + a) * Re + r];
    }
  }
  __syncthreads();
  cd *cur = bufA, *nxt = bufB;
  long long Lj = 1;
  for (int f = 0; f < s.k; ++f) {
    if (f == e) continue;
    const int q = s.dims[f];
    const long long R = P / Lj / q;
    const cd *m = incoming_msg(g, s.half0 + f, n2e_old, e2n_old, n2e_new, src_sel);
    if (fresh(s.half0 + f)) {
      cd tr = czero();
      for (int i = 0; i < q; ++i) tr = cadd(tr, __ldcg(m + i * q + i));
      for (int i = threadIdx.x; i < q * q; i += blockDim.x) staged[i] = cdiv(__ldcg(m + i), tr);
      __syncthreads();
      m = staged;
    }
    mode_product<false>(cur, nxt, Lj, q, q, R, m, q, 1);
    __syncthreads();
    cd *t = cur;
    cur = nxt;
    nxt = t;
    Lj *= q;
  }
  for (int ap = warp; ap < ce; ap += nw) {
    cd acc = czero();
    if (small) {
      for (unsigned x = lane; x < (unsigned)P; x += 32) {
        const unsigned l = fRe.div(x), r = x - l * (unsigned)Re;
        cfmac(acc, Tv[(l * (unsigned)ce + (unsigned)ap) * (unsigned)Re + r], cur[x]);
      }
    } else {
      for (long long x = lane; x < P; x += 32) {
        long long l = x / Re, r = x - l * Re;
        cfmac(acc, Tv[(l * ce + ap) * Re + r], cur[x]);
      }
    }
    acc = warp_csum(acc);
    if (lane == 0) put(ap, acc);
  }
  __syncthreads();
}

// dst (ce x ce) /= its trace, the trace summed by one thread in index order.
// Whole CTA; src may equal dst.
__device__ __forceinline__ void normalise_by_trace(const cd *src, cd *dst, int ce, cd &trace_sh) {
  if (threadIdx.x == 0) {
    cd tr = czero();
    for (int i = 0; i < ce; ++i) tr = cadd(tr, src[i * ce + i]);
    trace_sh = tr;
  }
  __syncthreads();
  const cd tr = trace_sh;
  for (int i = threadIdx.x; i < ce * ce; i += blockDim.x) dst[i] = cdiv(src[i], tr);
  __syncthreads();
}

// n2e_new[h] for one half-edge h by the whole CTA (out: ce x ce, bufA / bufB:
// two slices, trace_sh: one shared complex). Ends with a barrier.
__device__ __forceinline__ void node_update_half(const dqz_graph_t &g, const cd *__restrict__ T, const cd *n2e_old,
                                                 const cd *e2n_old, cd *n2e_new, const uint8_t *__restrict__ src_sel,
                                                 int h, cd *out, cd *bufA, cd *bufB, cd &trace_sh) {
  const int v = g.half_node[h];
  NodeShape s;
  load_shape(g, v, s);
  const int e = h - s.half0;
  const int ce = s.dims[e];
  const cd *Tv = T + g.node_off[v];
  for (int a = 0; a < ce; ++a)
    node_slice_column(g, Tv, s, e, n2e_old, e2n_old, n2e_new, src_sel, a, bufA, bufB,
                      [&](int ap, cd val) { out[ap * ce + a] = val; });
  normalise_by_trace(out, n2e_new + g.half_msg_off[h], ce, trace_sh);
}

__global__ void __launch_bounds__(BP_THREADS) bp_node_generic(dqz_graph_t g, const cd *__restrict__ T,
                                                              const cd *n2e_old, const cd *e2n_old, cd *n2e_new,
                                                              const uint8_t *__restrict__ src_sel,
                                                              const int32_t *__restrict__ halves, int n_halves,
                                                              int max_slice, int max_chi, cd *scratch) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cd *out = reinterpret_cast<cd *>(smem_raw + 48 * sizeof(double));  // max_chi^2
  cd *bufA, *bufB;
  if (scratch) {
    bufA = scratch + (long long)blockIdx.x * 2 * max_slice;
  } else {
    bufA = out + (long long)max_chi * max_chi;
  }
  bufB = bufA + max_slice;
  __shared__ cd trace_sh;
  for (int item = blockIdx.x; item < n_halves; item += gridDim.x)
    node_update_half(g, T, n2e_old, e2n_old, n2e_new, src_sel, halves[item], out, bufA, bufB, trace_sh);
}

// Bonds from SL_MIN_CHI: the node update by blocks of slices on the FP64 tensor
// cores (bp_slices.cuh), block blockIdx.y of half-edge halves[blockIdx.x], columns
// left unnormalised for bp_trace_kernel. Nodes outside that form's shapes share the
// generic update's columns out among the same CTAs (two slices in shared memory):
// 4-regular graph of 200 nodes, bond 8, 378 us (400 by one CTA a half-edge here, 382
// by the generic kernel alone); 26 nodes 73 us (113, 102). Below the bound the one-launch sweeps of small nodes are faster, and must agree with
// this entry bit for bit.
constexpr int SL_MIN_CHI = 8;

__global__ void __launch_bounds__(SL_THREADS, 2) bp_node_slices(dqz_graph_t g, const cd *__restrict__ T,
                                                             const cd *n2e_old, const cd *e2n_old, cd *n2e_new,
                                                             const uint8_t *__restrict__ src_sel,
                                                             const int32_t *__restrict__ halves, int max_slice) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cd *buf = reinterpret_cast<cd *>(smem_raw);
  const int h = halves[blockIdx.x];
  const int v = g.half_node[h];
  NodeShape s;
  load_shape(g, v, s);
  const int e = h - s.half0;
  SliceItem it;
  cd *dst = n2e_new + g.half_msg_off[h];
  const cd *Tv = T + g.node_off[v];
  if (sl_geometry(s, e, it.g)) {
    const int n = sl_count(it.g), ce = it.g.ce;
    it.a0 = blockIdx.y * n;
    if (it.a0 >= ce) return;
    it.n = ce - it.a0 < n ? ce - it.a0 : n;
    it.T = Tv;
    it.Re = (unsigned)s.stride[e];
    sl_load(it, buf);
    const cd *mx =
        it.g.nb > 0 ? incoming_msg(g, s.half0 + it.g.fx, n2e_old, e2n_old, n2e_new, src_sel) : nullptr;
    const cd *my =
        it.g.nb > 1 ? incoming_msg(g, s.half0 + it.g.fy, n2e_old, e2n_old, n2e_new, src_sel) : nullptr;
    sl_columns(it, mx, false, my, false, buf, buf + SL_BUF, [&](int ap, int a, cd val) { dst[ap * ce + a] = val; });
    return;
  }
  const int ce = s.dims[e];
  for (int a = blockIdx.y; a < ce; a += gridDim.y)
    node_slice_column(g, Tv, s, e, n2e_old, e2n_old, n2e_new, src_sel, a, buf, buf + max_slice,
                      [&](int ap, cd val) { dst[ap * ce + a] = val; });
}

// The listed messages divided by their traces, one CTA each.
__global__ void __launch_bounds__(SL_THREADS) bp_trace_kernel(dqz_graph_t g, cd *n2e_new,
                                                              const int32_t *__restrict__ halves) {
  __shared__ cd trace_sh;
  const int h = halves[blockIdx.x];
  const int e = g.half_edge[h];
  if (e < 0) return;
  cd *m = n2e_new + g.half_msg_off[h];
  normalise_by_trace(m, m, g.edge_chi[e], trace_sh);
}

// ---- one warp per half-edge, for small nodes. The same elements in the same
// order as node_update_half (each mode-product output by one lane, the final
// column by the lanes' partial sums and warp_csum, the trace by one lane), so
// the messages are bit-identical; phases are separated by __syncwarp only.
__device__ __forceinline__ void warp_mode_product(const cd *__restrict__ X, cd *__restrict__ Y, unsigned L, int q,
                                                  unsigned R, const cd *__restrict__ m) {
  // plain 32-bit divisions: a lane runs a handful of outputs here (small
  // nodes), fewer than it takes to amortise a FastDiv set-up
  const unsigned total = L * (unsigned)q * R;
  for (unsigned o = threadIdx.x & 31; o < total; o += 32) {
    const unsigned t = o / R;
    const unsigned r = o - t * R;
    const unsigned l = t / (unsigned)q;
    const int i = (int)(t - l * (unsigned)q);
    const cd *x = X + (l * (unsigned)q) * R + r;
    cd acc = czero();
    for (int b = 0; b < q; ++b) cfma(acc, m[(long long)i * q + b], x[(long long)b * R]);
    Y[o] = acc;
  }
}

__device__ __forceinline__ void warp_node_update_half(const dqz_graph_t &g, const cd *__restrict__ T, const cd *n2e_old,
                                                      const cd *e2n_old, cd *n2e_new,
                                                      const uint8_t *__restrict__ src_sel, int h, cd *out, cd *bufA,
                                                      cd *bufB, cd *Ts, cd *Ms) {
  const int lane = threadIdx.x & 31;
  const int v = g.half_node[h];
  NodeShape s;
  load_shape(g, v, s);
  const int e = h - s.half0;
  const int ce = s.dims[e];
  const unsigned Re = (unsigned)s.stride[e];
  const unsigned P = (unsigned)(s.size / ce);
  const FastDiv fRe(Re);
  // the node tensor and the k-1 incoming messages staged once (their global
  // loads all in flight together), then everything runs from shared memory
  {
    const cd *Tv = T + g.node_off[v];
    for (unsigned x = lane; x < (unsigned)s.size; x += 32) Ts[x] = Tv[x];
    int off = 0;
    for (int f = 0; f < s.k; ++f) {
      if (f == e) continue;
      const int q2 = s.dims[f] * s.dims[f];
      const cd *m = incoming_msg(g, s.half0 + f, n2e_old, e2n_old, n2e_new, src_sel);
      for (int x = lane; x < q2; x += 32) Ms[off + x] = m[x];
      off += q2;
    }
    __syncwarp();
  }
  for (int a = 0; a < ce; ++a) {
    for (unsigned x = lane; x < P; x += 32) {
      const unsigned l = fRe.div(x), r = x - l * Re;
      bufA[x] = Ts[(l * (unsigned)ce + (unsigned)a) * Re + r];
    }
    __syncwarp();
    cd *cur = bufA, *nxt = bufB;
    unsigned Lj = 1;
    int off = 0;
    for (int f = 0; f < s.k; ++f) {
      if (f == e) continue;
      const int q = s.dims[f];
      const unsigned R = P / Lj / (unsigned)q;
      warp_mode_product(cur, nxt, Lj, q, R, Ms + off);
      __syncwarp();
      cd *t = cur;
      cur = nxt;
      nxt = t;
      Lj *= (unsigned)q;
      off += q * q;
    }
    for (int ap = 0; ap < ce; ++ap) {
      cd acc = czero();
      for (unsigned x = lane; x < P; x += 32) {
        const unsigned l = fRe.div(x), r = x - l * Re;
        cfmac(acc, Ts[(l * (unsigned)ce + (unsigned)ap) * Re + r], cur[x]);
      }
      acc = warp_csum(acc);
      if (lane == 0) out[ap * ce + a] = acc;
    }
    __syncwarp();
  }
  cd tr = czero();
  if (lane == 0)
    for (int i = 0; i < ce; ++i) tr = cadd(tr, out[i * ce + i]);
  tr.x = __shfl_sync(0xffffffffu, tr.x, 0);
  tr.y = __shfl_sync(0xffffffffu, tr.y, 0);
  cd *dst = n2e_new + g.half_msg_off[h];
  for (int i = lane; i < ce * ce; i += 32) dst[i] = cdiv(out[i], tr);
  __syncwarp();
}

// A whole asynchronous sweep in one CTA, for graphs of small nodes: the
// warps take the half-edges of a level (one each), a __syncthreads closes the
// level, then the edge pass. No grid barrier; bit-identical to the per-level
// launches. Per warp: out (max_chi^2) and two slices in shared memory.
constexpr int ONECTA_THREADS = 1024;
// per warp: out (max_chi^2), two slices, the node tensor (max_slice x max_chi),
// the incoming messages ((DQZ_MAX_DEGREE - 1) x max_chi^2)
__host__ __device__ inline size_t round_up16(size_t x) { return (x + 15) & ~(size_t)15; }
__host__ __device__ inline size_t onecta_warp_elems(int max_slice, int max_chi) {
  return (size_t)max_chi * max_chi + 2 * (size_t)max_slice + (size_t)max_slice * max_chi +
         (size_t)(DQZ_MAX_DEGREE - 1) * max_chi * max_chi;
}

__global__ void __launch_bounds__(ONECTA_THREADS) bp_sweep_onecta_kernel(
    dqz_graph_t g, const cd *__restrict__ T, const cd *n2e_old, const cd *e2n_old, cd *n2e_new, cd *e2n_new,
    const uint8_t *__restrict__ src_sel, const uint8_t *__restrict__ edge_new, const int32_t *__restrict__ halves,
    const int32_t *__restrict__ level_off, int n_levels, int max_slice, int max_chi) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  cd *out = reinterpret_cast<cd *>(smem_raw) + (size_t)warp * onecta_warp_elems(max_slice, max_chi);
  cd *bufA = out + (size_t)max_chi * max_chi;
  cd *bufB = bufA + max_slice;
  cd *Ts = bufB + max_slice;
  cd *Ms = Ts + (size_t)max_slice * max_chi;
  for (int lv = 0; lv < n_levels; ++lv) {
    for (int item = level_off[lv] + warp; item < level_off[lv + 1]; item += nw)
      warp_node_update_half(g, T, n2e_old, e2n_old, n2e_new, src_sel, halves[item], out, bufA, bufB, Ts, Ms);
    __syncthreads();
  }
  for (int h = warp; h < g.n_halves; h += nw) {
    const int e = g.half_edge[h];
    const int tw = g.half_twin[h];
    if (e < 0 || tw < 0) continue;
    const int c = g.edge_chi[e];
    const cd *src = (edge_new[h] ? n2e_new : n2e_old) + g.half_msg_off[tw];
    cd *dst = e2n_new + g.half_msg_off[h];
    warp_copy16(reinterpret_cast<uint4 *>(dst), reinterpret_cast<const uint4 *>(src), c * c);
  }
}

// ---- the one-CTA sweep with a host-built plan: per item (the order of the
// level table) DQZ_PLAN_WORDS words: node offset, degree k, physical
// dimension d, slot e of the outgoing bond, outgoing message offset, the k
// bond dimensions (DQZ_MAX_DEGREE words), then per other bond in bond order
// its incoming message as offset * 4 + source (DQZ_SRC_*). A warp reads its
// item's words in one coalesced load instead of walking node -> half-edges
// -> edges -> twins (six dependent loads), then stages the tensor and the
// messages at once. Same arithmetic as warp_node_update_half.
__device__ __forceinline__ void warp_plan_item(const long long *pw, const cd *__restrict__ T, const cd *n2e_old,
                                               const cd *e2n_old, cd *n2e_new, cd *out, cd *bufA, cd *bufB, cd *Ts,
                                               cd *Ms) {
  const int lane = threadIdx.x & 31;
  const int k = (int)pw[1], d = (int)pw[2], e = (int)pw[3];
  const long long *dims = pw + 5;
  unsigned size = (unsigned)d, Re = (unsigned)d;
  for (int f = k - 1; f >= 0; --f) {
    if (f == e) Re = size;
    size *= (unsigned)dims[f];
  }
  const int ce = (int)dims[e];
  const unsigned P = size / (unsigned)ce;
  {
    const cd *Tv = T + pw[0];
    for (unsigned x = lane; x < size; x += 32) Ts[x] = Tv[x];
    int off = 0, slot = 0;
    for (int f = 0; f < k; ++f) {
      if (f == e) continue;
      const int q2 = (int)(dims[f] * dims[f]);
      const long long code = pw[5 + DQZ_MAX_DEGREE + slot];
      const int src = (int)(code & 3);
      const cd *m = (src == DQZ_SRC_E2N_OLD ? e2n_old : (src == DQZ_SRC_N2E_NEW ? n2e_new : n2e_old)) + (code >> 2);
      for (int x = lane; x < q2; x += 32) Ms[off + x] = m[x];
      off += q2;
      ++slot;
    }
    __syncwarp();
  }
  for (int a = 0; a < ce; ++a) {
    for (unsigned x = lane; x < P; x += 32) {
      const unsigned l = x / Re, r = x - l * Re;
      bufA[x] = Ts[(l * (unsigned)ce + (unsigned)a) * Re + r];
    }
    __syncwarp();
    cd *cur = bufA, *nxt = bufB;
    unsigned Lj = 1;
    int off = 0;
    for (int f = 0; f < k; ++f) {
      if (f == e) continue;
      const int q = (int)dims[f];
      const unsigned R = P / Lj / (unsigned)q;
      warp_mode_product(cur, nxt, Lj, q, R, Ms + off);
      __syncwarp();
      cd *t = cur;
      cur = nxt;
      nxt = t;
      Lj *= (unsigned)q;
      off += q * q;
    }
    for (int ap = 0; ap < ce; ++ap) {
      cd acc = czero();
      for (unsigned x = lane; x < P; x += 32) {
        const unsigned l = x / Re, r = x - l * Re;
        cfmac(acc, Ts[(l * (unsigned)ce + (unsigned)ap) * Re + r], cur[x]);
      }
      acc = warp_csum(acc);
      if (lane == 0) out[ap * ce + a] = acc;
    }
    __syncwarp();
  }
  cd tr = czero();
  if (lane == 0)
    for (int i = 0; i < ce; ++i) tr = cadd(tr, out[i * ce + i]);
  tr.x = __shfl_sync(0xffffffffu, tr.x, 0);
  tr.y = __shfl_sync(0xffffffffu, tr.y, 0);
  cd *dst = n2e_new + pw[4];
  for (int i = lane; i < ce * ce; i += 32) dst[i] = cdiv(out[i], tr);
  __syncwarp();
}

// ---- the same with all slices of an item at once: the mode products run on the
// whole tensor (the outgoing bond is one more batch index), so an item is degree -
// 1 dependent phases instead of that many per slice, and a lane has several outputs
// of a phase in flight. Every entry is the same sum in the same order. What does not
// depend on other items of the sweep happens before the barrier that opens
// its level: the warps take the items of all levels in turn, so that a warp has
// several levels' time to stage its next item (words, strides and reciprocals, the
// addresses of its messages, its tensor by cp.async). A quotient x / y is
// floor((2 x + 1) ceil(2^31 / y) / 2^32): (x + 1/2) / y plus less than (x + 1/2)
// 2^-31, and (x + 1/2) / y lies at least 1 / (2 y) below a whole number, so it is
// exact while x y < 2^30.
// Bound by the levels' chain, and within a level by the SM's shared-memory port (five
// items' operand loads at once). 16 warps: with 32 the registers spill. Measured on the
// 6 x 6 x 6 lattice, bond 2 (206 levels, 5 half-edges each): 572 us, 661 us with an
// output at a time in the products, 1,750 us by slices.
struct PlanWarp {
  long long pw[DQZ_PLAN_WORDS + 1];
  int4 bond[DQZ_MAX_DEGREE];    // stride R, dimension q, small_div's factors of R and q
  int moff[DQZ_MAX_DEGREE];     // the bond's message in Ms
  int size, nm;                 // entries of the tensor and of all messages
};
__device__ __forceinline__ unsigned small_div(unsigned x, unsigned m) { return __umulhi(2 * x + 1, m); }
__device__ __forceinline__ unsigned small_div_factor(unsigned y) { return (0x80000000u + y - 1) / y; }

// The words of the next item, `word` in lane < DQZ_PLAN_WORDS, and what follows from them.
__device__ __forceinline__ void plan_setup(PlanWarp &W, long long word) {
  const int lane = threadIdx.x & 31;
  __syncwarp();
  if (lane < DQZ_PLAN_WORDS) W.pw[lane] = word;
  __syncwarp();
  const int k = (int)W.pw[1], e = (int)W.pw[3];
  const long long *dims = W.pw + 5;
  if (lane < k) {
    int R = (int)W.pw[2], off = 0;
    for (int f = k - 1; f > lane; --f) R *= (int)dims[f];
    for (int f = 0; f < lane; ++f)
      if (f != e) off += (int)(dims[f] * dims[f]);
    const int q = (int)dims[lane];
    W.bond[lane] = make_int4(R, q, (int)small_div_factor((unsigned)R), (int)small_div_factor((unsigned)q));
    W.moff[lane] = off;
    if (lane == 0) W.size = R * q;
    if (lane == k - 1) W.nm = off + (lane != e ? q * q : 0);
  }
  __syncwarp();
}
// Address of entry x of the item's messages, laid one after another.
__device__ __forceinline__ const cd *plan_message(const PlanWarp &W, int x, const cd *n2e_old, const cd *e2n_old,
                                                  const cd *n2e_new) {
  const int k = (int)W.pw[1], e = (int)W.pw[3];
  int slot = 0, at = x;
  for (int f = 0; f < k; ++f) {
    if (f == e) continue;
    if (x >= W.moff[f]) {
      at = x - W.moff[f];
      slot = f < e ? f : f - 1;
    }
  }
  const long long code = W.pw[5 + DQZ_MAX_DEGREE + slot];
  const int src = (int)(code & 3);
  return (src == DQZ_SRC_E2N_OLD ? e2n_old : (src == DQZ_SRC_N2E_NEW ? n2e_new : n2e_old)) + (code >> 2) + at;
}
__device__ __forceinline__ void plan_load_tensor(const PlanWarp &W, const cd *__restrict__ T, cd *Ts) {
  const cd *Tv = T + W.pw[0];
  for (int x = threadIdx.x & 31; x < W.size; x += 32) cp_async16(Ts + x, Tv + x);
  cp_async_commit();
}

// Y = X x_f m over the whole tensor, Q the bond's dimension: a lane takes whole
// fibers (all Q entries along the bond, U fibers at a time), so each entry of X is
// read once, and a row of m once for all of them. For bonds up to 4; above, Q U
// entries a lane spill the registers.
template <int Q, int U>
__device__ __forceinline__ void plan_fibers(const int4 &bond, unsigned size, const cd *X, cd *Y, const cd *m) {
  const unsigned R = (unsigned)bond.x, fR = (unsigned)bond.z, fibers = size / Q;
  for (unsigned o0 = threadIdx.x & 31; o0 < fibers; o0 += 32 * U) {
    cd x[U][Q];
    unsigned at[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const unsigned o = o0 + 32 * u < fibers ? o0 + 32 * u : o0;
      at[u] = o + small_div(o, fR) * (Q - 1) * R;
#pragma unroll
      for (int b = 0; b < Q; ++b) x[u][b] = X[at[u] + b * R];
    }
#pragma unroll
    for (int i = 0; i < Q; ++i) {
      cd row[Q];
#pragma unroll
      for (int b = 0; b < Q; ++b) row[b] = m[i * Q + b];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        cd acc = czero();
#pragma unroll
        for (int b = 0; b < Q; ++b) cfma(acc, row[b], x[u][b]);
        if (o0 + 32 * u < fibers) Y[at[u] + i * R] = acc;
      }
    }
  }
}
// The same for any bond, an output a time.
template <int U>
__device__ __forceinline__ void plan_product(const int4 &bond, unsigned size, const cd *X, cd *Y, const cd *m) {
  const unsigned R = (unsigned)bond.x, q = (unsigned)bond.y, fR = (unsigned)bond.z, fq = (unsigned)bond.w;
  for (unsigned o0 = threadIdx.x & 31; o0 < size; o0 += 32 * U) {
    cd acc[U];
    unsigned x[U], mi[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const unsigned o = o0 + 32 * u < size ? o0 + 32 * u : o0;
      const unsigned t = small_div(o, fR), l = small_div(t, fq), i = t - l * q;
      mi[u] = i * q;
      x[u] = o - i * R;
      acc[u] = czero();
    }
#pragma unroll 2
    for (unsigned b = 0; b < q; ++b)
#pragma unroll
      for (int u = 0; u < U; ++u) cfma(acc[u], m[mi[u] + b], X[x[u] + b * R]);
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (o0 + 32 * u < size) Y[o0 + 32 * u] = acc[u];
  }
}

// warp_csum of four values, each lane exchanging only what it will go on with: value
// u's sum, added in the same pairs, ends in lane 8 u.
__device__ __forceinline__ cd warp_csum4(const cd (&v)[4]) {
  const int lane = threadIdx.x & 31;
  const bool hi = lane & 16, mid = lane & 8;
  const auto get = [](cd x, int o) {
    return mk(__shfl_xor_sync(0xffffffffu, x.x, o), __shfl_xor_sync(0xffffffffu, x.y, o));
  };
  const cd a = cadd(hi ? v[2] : v[0], get(hi ? v[0] : v[2], 16));
  const cd b = cadd(hi ? v[3] : v[1], get(hi ? v[1] : v[3], 16));
  cd s = cadd(mid ? b : a, get(mid ? a : b, 8));
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) s = cadd(s, get(s, o));
  return s;
}

// out[p], p = a' ce + a, for four pairs from p0 (up to ce^2): lane-strided sums over x as node_update_half.
__device__ __forceinline__ void plan_pairs(const int4 &bond, unsigned P, const cd *Ts, const cd *Z, int p0,
                                           cd *out) {
  const int lane = threadIdx.x & 31;
  const unsigned Re = (unsigned)bond.x, ce = (unsigned)bond.y, fR = (unsigned)bond.z;
  cd acc[4];
  unsigned tp[4], zp[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const unsigned p = p0 + u < ce * ce ? p0 + u : p0, ap = small_div(p, (unsigned)bond.w);
    tp[u] = ap * Re;
    zp[u] = (p - ap * ce) * Re;
    acc[u] = czero();
  }
#pragma unroll 2
  for (unsigned x = lane; x < P; x += 32) {
    const unsigned l = small_div(x, fR), base = x + l * (ce - 1) * Re;
#pragma unroll
    for (int u = 0; u < 4; ++u) cfmac(acc[u], Ts[base + tp[u]], Z[base + zp[u]]);
  }
  const cd s = warp_csum4(acc);
  const unsigned p = p0 + (lane >> 3);
  if ((lane & 7) == 0 && p < ce * ce) out[p] = s;
}

__host__ __device__ inline size_t plan_warp_elems(int max_slice, int max_chi) {
  return (size_t)max_chi * max_chi + 3 * (size_t)max_slice * max_chi +
         (size_t)(DQZ_MAX_DEGREE - 1) * max_chi * max_chi;
}
__host__ __device__ inline size_t plan_warp_bytes(int max_slice, int max_chi) {
  return plan_warp_elems(max_slice, max_chi) * sizeof(cd) + round_up16(sizeof(PlanWarp));
}
constexpr int PLAN_LEVELS = 1024;  // level offsets kept in shared memory
constexpr int PLAN_THREADS = 512;

// The edge pass of the one-CTA sweeps, a lane per half-edge: the table look-ups of 32
// of them in flight at once.
__device__ __forceinline__ void plan_edge_pass(const dqz_graph_t &g, const cd *n2e_old, const cd *n2e_new, cd *e2n_new,
                                               const uint8_t *__restrict__ edge_new) {
  for (int h = threadIdx.x; h < g.n_halves; h += blockDim.x) {
    const int e = g.half_edge[h];
    const int tw = g.half_twin[h];
    if (e < 0 || tw < 0) continue;
    const int c = g.edge_chi[e];
    const cd *src = (edge_new[h] ? n2e_new : n2e_old) + g.half_msg_off[tw];
    cd *dst = e2n_new + g.half_msg_off[h];
#pragma unroll 4
    for (int i = 0; i < c * c; ++i) dst[i] = src[i];
  }
}

__global__ void __launch_bounds__(PLAN_THREADS) bp_sweep_whole_kernel(
    dqz_graph_t g, const cd *__restrict__ T, const cd *n2e_old, const cd *e2n_old, cd *n2e_new, cd *e2n_new,
    const uint8_t *__restrict__ edge_new, const long long *__restrict__ plan, const int32_t *__restrict__ level_off,
    int n_levels, int max_slice, int max_chi) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int off_sh[PLAN_LEVELS + 1];
  const int warp = threadIdx.x >> 5, nw = blockDim.x >> 5, lane = threadIdx.x & 31;
  unsigned char *mine = smem_raw + (size_t)warp * plan_warp_bytes(max_slice, max_chi);
  PlanWarp &W = *reinterpret_cast<PlanWarp *>(mine);
  cd *out = reinterpret_cast<cd *>(mine + round_up16(sizeof(PlanWarp)));
  cd *Ts = out + (size_t)max_chi * max_chi, *A = Ts + (size_t)max_slice * max_chi,
     *B = A + (size_t)max_slice * max_chi, *Ms = B + (size_t)max_slice * max_chi;
  for (int i = threadIdx.x; i <= n_levels && i <= PLAN_LEVELS; i += blockDim.x) off_sh[i] = level_off[i];
  __syncthreads();
  auto offset = [&](int lv) { return lv <= PLAN_LEVELS ? off_sh[lv] : level_off[lv]; };
  const int total = offset(n_levels);
  int at = warp;  // the staged item: the warps take the items of all levels in turn
  long long later = 0;
  bool pending = false;
  const cd *mp[2] = {nullptr, nullptr};
  auto stage = [&](long long word) {  // the item's words, message addresses and tensor
    plan_setup(W, word);
#pragma unroll
    for (int j = 0; j < 2; ++j)
      if (lane + 32 * j < W.nm) mp[j] = plan_message(W, lane + 32 * j, n2e_old, e2n_old, n2e_new);
    plan_load_tensor(W, T, Ts);
  };
  auto words = [&](int item) {
    return item < total && lane < DQZ_PLAN_WORDS ? plan[(long long)item * DQZ_PLAN_WORDS + lane] : 0;
  };
  if (at < total) stage(words(at));
  for (int lv = 0; lv < n_levels; ++lv) {
    for (const int end = offset(lv + 1); at < end; at += nw) {
      const long long word = words(at + nw);
      const int k = (int)W.pw[1], e = (int)W.pw[3], nm = W.nm;
      const long long *dims = W.pw + 5;
      const int ce = (int)dims[e];
      const long long dst_off = W.pw[4];
#pragma unroll
      for (int j = 0; j < 2; ++j)
        if (lane + 32 * j < nm) Ms[lane + 32 * j] = *mp[j];
      for (int x = lane + 64; x < nm; x += 32) Ms[x] = *plan_message(W, x, n2e_old, e2n_old, n2e_new);
      cp_async_wait<0>();
      __syncwarp();
      const cd *cur = Ts;
      cd *nxt = A;
      const unsigned size = (unsigned)W.size;
      int4 bond = W.bond[e == 0 ? (k > 1 ? 1 : 0) : 0];
      for (int f = e == 0 ? 1 : 0; f < k;) {
        const int after = f + 1 == e ? f + 2 : f + 1;
        const int4 nb = W.bond[after < k ? after : e];  // on its way during the product; the pairs' at the end
        const cd *m = Ms + W.moff[f];
        switch (bond.y) {
          case 2: plan_fibers<2, 2>(bond, size, cur, nxt, m); break;
          case 3: plan_fibers<3, 2>(bond, size, cur, nxt, m); break;
          case 4: plan_fibers<4, 1>(bond, size, cur, nxt, m); break;
          default: plan_product<4>(bond, size, cur, nxt, m);
        }
        bond = nb;
        f = after;
        __syncwarp();
        cur = nxt;
        nxt = nxt == A ? B : A;
      }
      const unsigned P = size / (unsigned)ce;
      for (int p0 = 0; p0 < ce * ce; p0 += 4) plan_pairs(bond, P, Ts, cur, p0, out);
      __syncwarp();
      cd tr = czero();
      for (int i = 0; i < ce; ++i) tr = cadd(tr, out[i * ce + i]);
      cd *dst = n2e_new + dst_off;
      for (int i = lane; i < ce * ce; i += 32) dst[i] = cdiv(out[i], tr);
      if (at + nw < total) {
        // after the barrier, which the other warps wait at, unless it is for this level
        if (at + nw < end) {
          stage(word);
        } else {
          later = word;
          pending = true;
        }
      }
      __syncwarp();
    }
    __syncthreads();
    if (pending) {
      stage(later);
      pending = false;
    }
  }
  plan_edge_pass(g, n2e_old, n2e_new, e2n_new, edge_new);
}

__global__ void __launch_bounds__(ONECTA_THREADS) bp_sweep_planned_kernel(
    dqz_graph_t g, const cd *__restrict__ T, const cd *n2e_old, const cd *e2n_old, cd *n2e_new, cd *e2n_new,
    const uint8_t *__restrict__ edge_new, const long long *__restrict__ plan, const int32_t *__restrict__ level_off,
    int n_levels, int max_slice, int max_chi) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int warp = threadIdx.x >> 5, nw = blockDim.x >> 5, lane = threadIdx.x & 31;
  long long *pw = reinterpret_cast<long long *>(smem_raw) + (size_t)warp * DQZ_PLAN_WORDS;
  cd *out = reinterpret_cast<cd *>(smem_raw + round_up16((size_t)nw * DQZ_PLAN_WORDS * sizeof(long long))) +
            (size_t)warp * onecta_warp_elems(max_slice, max_chi);
  cd *bufA = out + (size_t)max_chi * max_chi;
  cd *bufB = bufA + max_slice;
  cd *Ts = bufB + max_slice;
  cd *Ms = Ts + (size_t)max_slice * max_chi;
  for (int lv = 0; lv < n_levels; ++lv) {
    for (int item = level_off[lv] + warp; item < level_off[lv + 1]; item += nw) {
      if (lane < DQZ_PLAN_WORDS) pw[lane] = plan[(long long)item * DQZ_PLAN_WORDS + lane];
      __syncwarp();
      warp_plan_item(pw, T, n2e_old, e2n_old, n2e_new, out, bufA, bufB, Ts, Ms);
    }
    __syncthreads();
  }
  plan_edge_pass(g, n2e_old, n2e_new, e2n_new, edge_new);
}

// Grid-wide barrier for a cooperative launch: one arrival counter and one
// generation word (sync[0], sync[1], zero at launch). The last block to arrive
// resets the counter and advances the generation; the others poll it, at
// most `limit` times. Returns false in every thread of a block that gave up
// (it has set *error_flag to 3).
__device__ __forceinline__ bool grid_barrier(unsigned *sync, unsigned &gen, int *error_flag) {
  __shared__ int ok_sh;
  __syncthreads();
  if (threadIdx.x == 0) {
    int ok = 1;
    __threadfence();
    const unsigned target = gen + 1;
    if (atomicAdd(&sync[0], 1u) == gridDim.x - 1) {
      atomicExch(&sync[0], 0u);
      __threadfence();
      atomicExch(&sync[1], target);
    } else {
      ok = 0;
      for (int it = 0; it < (1 << 24); ++it) {
        if (atomicAdd(&sync[1], 0u) == target) {
          ok = 1;
          break;
        }
        __nanosleep(32);
      }
      if (!ok) atomicExch(error_flag, 3);
    }
    __threadfence();
    ok_sh = ok;
  }
  __syncthreads();
  ++gen;
  return ok_sh != 0;
}

// n2e_new[h] by the whole CTA as bp_node_slices and bp_trace_kernel compute it: its
// blocks of slices one after another (nodes outside that form: node_update_half).
// Ends with a barrier.
__device__ __forceinline__ void node_update_half_slices(const dqz_graph_t &g, const cd *__restrict__ T,
                                                        const cd *n2e_old, const cd *e2n_old, cd *n2e_new,
                                                        const uint8_t *__restrict__ src_sel, int h, cd *smem,
                                                        int max_slice, int max_chi, cd &trace_sh) {
  const int v = g.half_node[h];
  NodeShape s;
  load_shape(g, v, s);
  const int e = h - s.half0;
  SliceItem it;
  if (!sl_geometry(s, e, it.g)) {
    cd *bufA = smem + (long long)max_chi * max_chi;
    node_update_half(g, T, n2e_old, e2n_old, n2e_new, src_sel, h, smem, bufA, bufA + max_slice, trace_sh);
    return;
  }
  const int most = sl_count(it.g), ce = it.g.ce;
  cd *dst = n2e_new + g.half_msg_off[h];
  it.T = T + g.node_off[v];
  it.Re = (unsigned)s.stride[e];
  const cd *mx = it.g.nb > 0 ? incoming_msg(g, s.half0 + it.g.fx, n2e_old, e2n_old, n2e_new, src_sel) : nullptr;
  const cd *my = it.g.nb > 1 ? incoming_msg(g, s.half0 + it.g.fy, n2e_old, e2n_old, n2e_new, src_sel) : nullptr;
  for (it.a0 = 0; it.a0 < ce; it.a0 += most) {
    it.n = ce - it.a0 < most ? ce - it.a0 : most;
    sl_load(it, smem);
    sl_columns(it, mx, false, my, false, smem, smem + SL_BUF, [&](int ap, int a, cd val) { dst[ap * ce + a] = val; });
  }
  normalise_by_trace(dst, dst, ce, trace_sh);
}

// A whole sweep in one cooperative launch: node levels in order (the
// asynchronous schedule's dependency levels), a grid barrier after each, then
// the edge pass. Every half-edge is computed exactly as dqz_bp_node_update does:
// by slices (SLICES) from SL_MIN_CHI, as bp_node_generic below.
template <bool SLICES>
__global__ void __launch_bounds__(BP_THREADS) bp_sweep_levels_kernel(
    dqz_graph_t g, const cd *__restrict__ T, const cd *n2e_old, const cd *e2n_old, cd *n2e_new, cd *e2n_new,
    const uint8_t *__restrict__ src_sel, const uint8_t *__restrict__ edge_new, const int32_t *__restrict__ halves,
    const int32_t *__restrict__ level_off, int n_levels, int max_slice, int max_chi, unsigned *sync,
    int *error_flag) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cd *out = reinterpret_cast<cd *>(smem_raw);
  cd *bufA = out + (long long)max_chi * max_chi;
  cd *bufB = bufA + max_slice;
  __shared__ cd trace_sh;
  unsigned gen = 0;
  for (int lv = 0; lv < n_levels; ++lv) {
    for (int item = level_off[lv] + blockIdx.x; item < level_off[lv + 1]; item += gridDim.x) {
      if (SLICES)
        node_update_half_slices(g, T, n2e_old, e2n_old, n2e_new, src_sel, halves[item], out, max_slice, max_chi,
                                trace_sh);
      else
        node_update_half(g, T, n2e_old, e2n_old, n2e_new, src_sel, halves[item], out, bufA, bufB, trace_sh);
    }
    if (!grid_barrier(sync, gen, error_flag)) return;
  }
  // edge pass: e2n_new[h] = (edge_new[h] ? n2e_new : n2e_old)[twin(h)], one warp per half-edge
  const int wpb = blockDim.x >> 5;
  for (int h = blockIdx.x * wpb + (threadIdx.x >> 5); h < g.n_halves; h += gridDim.x * wpb) {
    const int e = g.half_edge[h];
    const int tw = g.half_twin[h];
    if (e < 0 || tw < 0) continue;
    const int c = g.edge_chi[e];
    const cd *src = (edge_new[h] ? n2e_new : n2e_old) + g.half_msg_off[tw];
    cd *dst = e2n_new + g.half_msg_off[h];
    warp_copy16(reinterpret_cast<uint4 *>(dst), reinterpret_cast<const uint4 *>(src), c * c);
  }
}

// One item of the sliced sweep, with its block's range of its level.
constexpr int SL_LEVELS = 128;  // levels looked up ahead
struct SweepItem {
  int item, h, a0, n, ce, begin, end;
  unsigned Re;
  bool fast, fx, fy;
  SliceGeom g;
  const cd *T, *mx, *my;
  cd *dst;
};

// The same sweep with each half-edge's slices spread over the grid (for larger
// bonds, where a level has few half-edges but each carries much work): an item is
// a half-edge and a block of its slices (item_slice: the first one, plus their
// number << 16 when more than one), its unnormalised columns as bp_node_slices
// computes them (nodes outside that form: node_slice_column per slice). A grid
// barrier closes a level. The messages stay unnormalised until the end: readers of
// this sweep's messages divide by the trace as they stage them, so a level needs
// no second barrier; then every listed message is divided in place, a barrier, and
// the edge pass. Messages of half-edges that no level lists are as the caller left
// them, for readers too. Bit-identical to the per-level launches.
// Bound by the levels' chain: an item at bond 32 reads 1 MB of T through L2 (16 k
// cycles an SM) and a level has 16 to 194 of them.
// One CTA per SM: 120 KB with the table, and 217 registers a thread (128, for a
// second one that never fits, spilled).
// Measured at bond 32 on the 127-qubit heavy-hex lattice (72 levels): 1,670 us, 1,838 us
// with the spills; one slice an item and generic arithmetic 3,252 us, without the
// table 2,107 us.
__global__ void __launch_bounds__(SL_THREADS) bp_sweep_sliced_kernel(
    dqz_graph_t g, const cd *__restrict__ T, const cd *n2e_old, const cd *e2n_old, cd *n2e_new, cd *e2n_new,
    const uint8_t *__restrict__ src_sel, const uint8_t *__restrict__ edge_new, const int32_t *__restrict__ halves,
    const int32_t *__restrict__ level_off, const int32_t *__restrict__ item_half,
    const int32_t *__restrict__ item_slice, const int32_t *__restrict__ item_off, int n_levels, int max_slice,
    unsigned *sync, int *error_flag) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cd *buf = reinterpret_cast<cd *>(smem_raw);
  __shared__ cd trace_sh;
  unsigned gen = 0;
  // An item's tables do not depend on other items: the first item of this block in
  // every level is looked up at the start, a thread per level, all the chains of
  // dependent table loads at once (9.7 k cycles a level otherwise), and its block
  // of T is on its way before the barrier that opens the level.
  __shared__ SweepItem table[SL_LEVELS];
  __shared__ SweepItem other;  // further items of a level, and levels beyond the table
  const int n_listed = level_off[n_levels];
  const bool all_listed = n_listed >= g.n_halves;
  auto computed = [&](int hf) {  // the message read at hf is one that this launch computes
    if (src_sel[hf] != DQZ_SRC_N2E_NEW) return false;
    if (all_listed) return true;
    const int tw = g.half_twin[hf];
    for (int i = 0; i < n_listed; ++i)
      if (halves[i] == tw) return true;
    return false;
  };
  auto look_up = [&](int item, SweepItem &d) {
    d.item = item;
    d.h = item_half[item];
    d.a0 = item_slice[item] & 0xffff;
    d.n = item_slice[item] >> 16;
    if (d.n < 1) d.n = 1;
    const int v = g.half_node[d.h];
    NodeShape s;
    load_shape(g, v, s);
    const int e = d.h - s.half0;
    d.ce = s.dims[e];
    d.T = T + g.node_off[v];
    d.dst = n2e_new + g.half_msg_off[d.h];
    d.Re = (unsigned)s.stride[e];
    d.fast = sl_geometry(s, e, d.g);
    const bool x = d.fast && d.g.nb > 0, y = d.fast && d.g.nb > 1;
    const int hx = x ? s.half0 + d.g.fx : d.h, hy = y ? s.half0 + d.g.fy : d.h;
    d.fx = x && computed(hx);
    d.fy = y && computed(hy);
    d.mx = x ? incoming_msg(g, hx, n2e_old, e2n_old, n2e_new, src_sel) : nullptr;
    d.my = y ? incoming_msg(g, hy, n2e_old, e2n_old, n2e_new, src_sel) : nullptr;
  };
  for (int lv = threadIdx.x; lv < n_levels && lv < SL_LEVELS; lv += blockDim.x) {
    table[lv].begin = item_off[lv] + (int)blockIdx.x;
    table[lv].end = item_off[lv + 1];
    if (table[lv].begin < table[lv].end) look_up(table[lv].begin, table[lv]);
  }
  __syncthreads();
  SliceItem it;
  auto load = [&](const SweepItem &d) {
    if (!d.fast) return;
    const int most = sl_count(d.g);
    it.g = d.g;
    it.T = d.T;
    it.Re = d.Re;
    it.a0 = d.a0;
    it.n = d.n < most ? d.n : most;
    sl_load(it, buf);
  };
  int ready = -1;
  for (int lv = 0; lv < n_levels; ++lv) {
    const bool listed = lv < SL_LEVELS;
    const int begin = listed ? table[lv].begin : item_off[lv] + (int)blockIdx.x;
    const int end = listed ? table[lv].end : item_off[lv + 1];
    for (int item = begin; item < end; item += gridDim.x) {
      const bool first = listed && item == begin;
      if (!first) {
        __syncthreads();
        if (threadIdx.x == 0) look_up(item, other);
        __syncthreads();
      }
      const SweepItem &d = first ? table[lv] : other;
      if (item != ready) load(d);
      const int ce = d.ce;
      cd *dst = d.dst;
      if (d.fast) {
        for (int left = d.n;;) {
          sl_columns(it, d.mx, d.fx, d.my, d.fy, buf, buf + SL_BUF,
                     [&](int ap, int a, cd val) { dst[ap * ce + a] = val; });
          left -= it.n;
          if (left <= 0) break;
          it.a0 += it.n;
          if (it.n > left) it.n = left;
          sl_load(it, buf);
        }
      } else {
        // every message of this launch is divided by its trace in a staged copy behind the two slices
        NodeShape s;
        load_shape(g, g.half_node[d.h], s);
        for (int b = 0; b < d.n; ++b)
          node_slice_column(g, d.T, s, d.h - s.half0, n2e_old, e2n_old, n2e_new, src_sel, d.a0 + b, buf,
                            buf + max_slice, [&](int ap, cd val) { dst[ap * ce + d.a0 + b] = val; },
                            buf + 2 * max_slice, computed);
      }
    }
    if (lv + 1 < n_levels && lv + 1 < SL_LEVELS && table[lv + 1].begin < table[lv + 1].end) {
      ready = table[lv + 1].begin;
      load(table[lv + 1]);
    }
    if (!grid_barrier(sync, gen, error_flag)) {
      cp_async_wait<0>();
      return;
    }
  }
  for (int i = blockIdx.x; i < n_listed; i += gridDim.x) {
    const int h = halves[i], e = g.half_edge[h];
    if (e < 0) continue;
    cd *m = n2e_new + g.half_msg_off[h];
    normalise_by_trace(m, m, g.edge_chi[e], trace_sh);
  }
  if (!grid_barrier(sync, gen, error_flag)) return;
  const int wpb = blockDim.x >> 5;
  for (int h = blockIdx.x * wpb + (threadIdx.x >> 5); h < g.n_halves; h += gridDim.x * wpb) {
    const int e = g.half_edge[h];
    const int tw = g.half_twin[h];
    if (e < 0 || tw < 0) continue;
    const int c = g.edge_chi[e];
    const cd *src = (edge_new[h] ? n2e_new : n2e_old) + g.half_msg_off[tw];
    cd *dst = e2n_new + g.half_msg_off[h];
    warp_copy16(reinterpret_cast<uint4 *>(dst), reinterpret_cast<const uint4 *>(src), c * c);
  }
}

__global__ void bp_edge_pass_kernel(dqz_graph_t g, const cd *n2e_old, const cd *n2e_new,
                                    const uint8_t *__restrict__ edge_new, cd *e2n_new) {
  const int nh = g.n_halves;
  // one warp per half-edge
  const int warps_per_block = blockDim.x >> 5;
  for (int h = blockIdx.x * warps_per_block + (threadIdx.x >> 5); h < nh; h += gridDim.x * warps_per_block) {
    const int e = g.half_edge[h];
    const int tw = g.half_twin[h];
    if (e < 0 || tw < 0) continue;
    const int c = g.edge_chi[e];
    const cd *src = (edge_new[h] ? n2e_new : n2e_old) + g.half_msg_off[tw];
    cd *dst = e2n_new + g.half_msg_off[h];
    warp_copy16(reinterpret_cast<uint4 *>(dst), reinterpret_cast<const uint4 *>(src), c * c);
  }
}

// partial[h] = |n2e_a[h] - n2e_b[h]|_F, partial[2E + h] = |e2n_a[h] - e2n_b[h]|_F
__global__ void msg_dist_kernel(dqz_graph_t g, const cd *n2e_a, const cd *n2e_b, const cd *e2n_a, const cd *e2n_b,
                                double *partial) {
  const int nh = g.n_halves;
  const int wpb = blockDim.x >> 5;
  const int lane = threadIdx.x & 31;
  for (int w = blockIdx.x * wpb + (threadIdx.x >> 5); w < 2 * nh; w += gridDim.x * wpb) {
    const int h = w < nh ? w : w - nh;
    const cd *A = (w < nh ? n2e_a : e2n_a) + g.half_msg_off[h];
    const cd *B = (w < nh ? n2e_b : e2n_b) + g.half_msg_off[h];
    const int e = g.half_edge[h];
    if (e < 0) {
      if (lane == 0) partial[w] = 0.0;
      continue;
    }
    const int c = g.edge_chi[e];
    double acc = 0.0;
    for (int i = lane; i < c * c; i += 32) acc += cabs2(csub(A[i], B[i]));
    acc = warp_sum(acc);
    if (lane == 0) partial[w] = sqrt(acc);
  }
}

// partial[h] = |a[h] - b[h]|_F over the node->edge messages of complex64 arenas.
__global__ void msg_dist_c64_kernel(dqz_graph_t g, const float2 *a, const float2 *b, double *partial) {
  const int nh = g.n_halves;
  const int wpb = blockDim.x >> 5;
  const int lane = threadIdx.x & 31;
  for (int h = blockIdx.x * wpb + (threadIdx.x >> 5); h < nh; h += gridDim.x * wpb) {
    const int e = g.half_edge[h];
    if (e < 0) {
      if (lane == 0) partial[h] = 0.0;
      continue;
    }
    const int c = g.edge_chi[e];
    const float2 *A = a + g.half_msg_off[h], *B = b + g.half_msg_off[h];
    double acc = 0.0;
    for (int i = lane; i < c * c; i += 32) {
      const double dx = (double)A[i].x - (double)B[i].x, dy = (double)A[i].y - (double)B[i].y;
      acc += dx * dx + dy * dy;
    }
    acc = warp_sum(acc);
    if (lane == 0) partial[h] = sqrt(acc);
  }
}

// out[0] = sum(partial[0..n)) * scale, deterministic single-CTA reduction.
__global__ void reduce_sum_kernel(const double *partial, int n, double scale, double *out) {
  __shared__ double red[48];
  double acc = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) acc += partial[i];
  acc = block_sum(acc, red);
  if (threadIdx.x == 0) out[0] = acc * scale;
}

size_t bp_smem_bytes(int max_slice, int max_chi, bool use_scratch) {
  size_t b = 48 * sizeof(double) + (size_t)max_chi * max_chi * sizeof(cd);
  if (!use_scratch) b += 2 * (size_t)max_slice * sizeof(cd);
  return b;
}

constexpr size_t BP_SMEM_LIMIT = 200 * 1024;
constexpr int BP_SCRATCH_GRID = 148 * 4;

}  // namespace

extern "C" size_t dqz_bp_node_scratch_bytes(int32_t n_halves, int32_t max_slice, int32_t max_chi) {
  if (bp_smem_bytes(max_slice, max_chi, false) <= BP_SMEM_LIMIT) return 0;
  int grid = n_halves < BP_SCRATCH_GRID ? n_halves : BP_SCRATCH_GRID;
  return (size_t)grid * 2 * (size_t)max_slice * sizeof(cd);
}

extern "C" int dqz_bp_node_update(const dqz_graph_t *g, const void *tensors, const void *n2e_old,
                                  const void *e2n_old, void *n2e_new, const uint8_t *src_sel,
                                  const int32_t *halves, int32_t n_halves, int32_t max_slice, int32_t max_chi,
                                  void *scratch, cudaStream_t stream) {
  if (!g || !tensors || !n2e_new || !src_sel || !halves || n_halves < 0 || max_slice <= 0) return DQZ_ERR_ARG;
  if (max_chi <= 0 || max_chi > DQZ_MAX_CHI) return DQZ_ERR_UNSUPPORTED;
  if (n_halves == 0) return DQZ_OK;
  const bool use_scratch = bp_smem_bytes(max_slice, max_chi, false) > BP_SMEM_LIMIT;
  if (use_scratch && !scratch) return DQZ_ERR_ARG;
  const size_t smem = bp_smem_bytes(max_slice, max_chi, use_scratch);
  if (smem > BP_SMEM_LIMIT) return DQZ_ERR_UNSUPPORTED;
  if (max_chi >= SL_MIN_CHI && !use_scratch) {
    DQZ_SMEM_ATTR_ONCE(bp_node_slices, BP_SMEM_LIMIT);
    // blocks of the largest slice the form takes, less what padding may cost (checked for every
    // shape of up to 32 x 32 x 8: no node has a smaller block); smaller slices need fewer
    const int per = sl_block(max_slice < SL_ELEMS ? max_slice : SL_ELEMS);
    const int fit = per <= 3 ? per : per - 1 - per / 16;
    const int blocks = (max_chi + fit - 1) / fit;
    bp_node_slices<<<dim3(n_halves, blocks), SL_THREADS, smem > SL_SMEM ? smem : SL_SMEM, stream>>>(
        *g, (const cd *)tensors, (const cd *)n2e_old, (const cd *)e2n_old, (cd *)n2e_new, src_sel, halves, max_slice);
    DQZ_CHECK_LAUNCH();
    bp_trace_kernel<<<n_halves, SL_THREADS, 0, stream>>>(*g, (cd *)n2e_new, halves);
    DQZ_CHECK_LAUNCH();
    return DQZ_OK;
  }
  DQZ_SMEM_ATTR_ONCE(bp_node_generic, BP_SMEM_LIMIT);
  int grid = use_scratch ? (n_halves < BP_SCRATCH_GRID ? n_halves : BP_SCRATCH_GRID) : n_halves;
  bp_node_generic<<<grid, BP_THREADS, smem, stream>>>(
      *g, (const cd *)tensors, (const cd *)n2e_old, (const cd *)e2n_old, (cd *)n2e_new, src_sel, halves, n_halves,
      max_slice, max_chi, use_scratch ? (cd *)scratch : nullptr);
  DQZ_CHECK_LAUNCH();
  return DQZ_OK;
}

extern "C" int dqz_bp_edge_pass(const dqz_graph_t *g, const void *n2e_old, const void *n2e_new,
                                const uint8_t *edge_new, void *e2n_new, int32_t max_chi, cudaStream_t stream) {
  if (!g || !n2e_old || !n2e_new || !edge_new || !e2n_new) return DQZ_ERR_ARG;
  if (max_chi <= 0 || max_chi > DQZ_MAX_CHI) return DQZ_ERR_UNSUPPORTED;
  const int nh = g->n_halves;
  if (nh == 0) return DQZ_OK;
  const int wpb = 8;
  int grid = (nh + wpb - 1) / wpb;
  bp_edge_pass_kernel<<<grid, wpb * 32, 0, stream>>>(*g, (const cd *)n2e_old, (const cd *)n2e_new, edge_new,
                                                    (cd *)e2n_new);
  DQZ_CHECK_LAUNCH();
  return DQZ_OK;
}

extern "C" int dqz_messages_distance(const dqz_graph_t *g, const void *n2e_a, const void *n2e_b, const void *e2n_a,
                                     const void *e2n_b, double *partial, double *out, int32_t max_chi,
                                     cudaStream_t stream) {
  if (!g || !n2e_a || !n2e_b || !e2n_a || !e2n_b || !partial || !out) return DQZ_ERR_ARG;
  if (max_chi <= 0 || max_chi > DQZ_MAX_CHI) return DQZ_ERR_UNSUPPORTED;
  const int nh = g->n_halves;
  if (nh == 0) return DQZ_ERR_ARG;
  const int wpb = 8;
  int grid = (2 * nh + wpb - 1) / wpb;
  msg_dist_kernel<<<grid, wpb * 32, 0, stream>>>(*g, (const cd *)n2e_a, (const cd *)n2e_b, (const cd *)e2n_a,
                                                (const cd *)e2n_b, partial);
  DQZ_CHECK_LAUNCH();
  reduce_sum_kernel<<<1, 256, 0, stream>>>(partial, 2 * nh, 1.0 / (2.0 * nh), out);
  DQZ_CHECK_LAUNCH();
  return DQZ_OK;
}

extern "C" int dqz_reduce_sum(const double *partial, int32_t n, double scale, double *out, cudaStream_t stream) {
  if (!partial || !out || n <= 0) return DQZ_ERR_ARG;
  reduce_sum_kernel<<<1, 256, 0, stream>>>(partial, n, scale, out);
  DQZ_CHECK_LAUNCH();
  return DQZ_OK;
}

extern "C" int dqz_bp_sweep_levels(const dqz_graph_t *g, const void *tensors, const void *n2e_old,
                                   const void *e2n_old, void *n2e_new, void *e2n_new, const uint8_t *src_sel,
                                   const uint8_t *edge_new, const int32_t *halves, const int32_t *level_off,
                                   int32_t n_levels, int32_t max_level, int32_t max_slice, int32_t max_chi,
                                   uint32_t *sync, int32_t *error_flag, cudaStream_t stream) {
  if (!g || !tensors || !n2e_old || !e2n_old || !n2e_new || !e2n_new || !src_sel || !edge_new || !halves ||
      !level_off || !sync || !error_flag || n_levels <= 0 || max_level <= 0 || max_slice <= 0)
    return DQZ_ERR_ARG;
  if (max_chi <= 0 || max_chi > DQZ_MAX_CHI) return DQZ_ERR_UNSUPPORTED;
  // Small nodes (bond slices up to 256 elements) and narrow levels (at most
  // two half-edges per warp): the whole sweep in one CTA, a warp per
  // half-edge and __syncthreads between levels (no grid barrier). Knob
  // DQZ_TUNE_SWEEP_ONECTA: 1 = never, 2 = wherever the warps' buffers fit. From
  // SL_MIN_CHI only by the knob: its sums are not those of the node update by slices.
  {
    const int knob = dqz_get_tuning(DQZ_TUNE_SWEEP_ONECTA);
    const size_t per_warp = onecta_warp_elems(max_slice, max_chi) * sizeof(cd);
    int warps = (int)(BP_SMEM_LIMIT / per_warp);
    if (warps > ONECTA_THREADS / 32) warps = ONECTA_THREADS / 32;
    const bool rule = max_chi < SL_MIN_CHI && max_slice <= 256 && warps >= 8 && max_level <= 2 * warps;
    if (knob != 1 && warps >= 1 && (rule || knob == 2)) {
      DQZ_SMEM_ATTR_ONCE(bp_sweep_onecta_kernel, BP_SMEM_LIMIT);
      bp_sweep_onecta_kernel<<<1, 32 * warps, (size_t)warps * per_warp, stream>>>(
          *g, (const cd *)tensors, (const cd *)n2e_old, (const cd *)e2n_old, (cd *)n2e_new, (cd *)e2n_new, src_sel,
          edge_new, halves, level_off, (int)n_levels, (int)max_slice, (int)max_chi);
      DQZ_CHECK_LAUNCH();
      return DQZ_OK;
    }
  }
  size_t smem = bp_smem_bytes(max_slice, max_chi, false);
  if (smem > BP_SMEM_LIMIT) return DQZ_ERR_UNSUPPORTED;  // the per-level launches use global scratch then
  auto *kernel = max_chi >= SL_MIN_CHI ? bp_sweep_levels_kernel<true> : bp_sweep_levels_kernel<false>;
  if (max_chi >= SL_MIN_CHI) {
    if (smem < SL_SMEM) smem = SL_SMEM;
    DQZ_SMEM_ATTR_ONCE(bp_sweep_levels_kernel<true>, BP_SMEM_LIMIT);
  } else {
    DQZ_SMEM_ATTR_ONCE(bp_sweep_levels_kernel<false>, BP_SMEM_LIMIT);
  }
  int dev = 0, sms = 148, per_sm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return DQZ_ERR_CUDA;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, BP_THREADS, smem) !=
          cudaSuccess ||
      per_sm < 1)
    return DQZ_ERR_UNSUPPORTED;
  int grid = max_level;  // one CTA per half-edge of the widest level, all co-resident
  if (grid > sms * per_sm) grid = sms * per_sm;
  if (cudaMemsetAsync(sync, 0, 2 * sizeof(uint32_t), stream) != cudaSuccess) return DQZ_ERR_CUDA;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(BP_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cudaLaunchKernelEx(&cfg, kernel, *g, (const cd *)tensors, (const cd *)n2e_old,
                         (const cd *)e2n_old, (cd *)n2e_new, (cd *)e2n_new, src_sel, edge_new, halves, level_off,
                         (int)n_levels, (int)max_slice, (int)max_chi, (unsigned *)sync, (int *)error_flag) !=
      cudaSuccess)
    return DQZ_ERR_CUDA;
  return DQZ_OK;
}

extern "C" int dqz_bp_sweep_planned(const dqz_graph_t *g, const void *tensors, const void *n2e_old,
                                    const void *e2n_old, void *n2e_new, void *e2n_new, const uint8_t *edge_new,
                                    const int64_t *plan, const int32_t *level_off, int32_t n_levels,
                                    int32_t max_level, int32_t max_slice, int32_t max_chi, cudaStream_t stream) {
  if (!g || !tensors || !n2e_old || !e2n_old || !n2e_new || !e2n_new || !edge_new || !plan || !level_off ||
      n_levels <= 0 || max_level <= 0 || max_slice <= 0)
    return DQZ_ERR_ARG;
  if (max_chi <= 0 || max_chi > DQZ_MAX_CHI) return DQZ_ERR_UNSUPPORTED;
  const size_t per_warp = onecta_warp_elems(max_slice, max_chi) * sizeof(cd);
  int warps = ONECTA_THREADS / 32;
  while (warps > 8 && round_up16((size_t)warps * DQZ_PLAN_WORDS * sizeof(long long)) + warps * per_warp >
                          BP_SMEM_LIMIT)
    --warps;
  size_t smem = round_up16((size_t)warps * DQZ_PLAN_WORDS * sizeof(long long)) + warps * per_warp;
  if (smem > BP_SMEM_LIMIT) return DQZ_ERR_UNSUPPORTED;
  // all slices of an item at once where the tensors' buffers leave as many warps as a
  // level can use, or as the form by slices has
  const size_t per_whole = plan_warp_bytes(max_slice, max_chi);
  int fit = (int)(BP_SMEM_LIMIT / per_whole);
  if (fit > PLAN_THREADS / 32) fit = PLAN_THREADS / 32;
  if (fit >= 1 && (fit >= PLAN_THREADS / 32 || fit >= warps || fit >= max_level)) {
    DQZ_SMEM_ATTR_ONCE(bp_sweep_whole_kernel, BP_SMEM_LIMIT);
    bp_sweep_whole_kernel<<<1, 32 * fit, fit * per_whole, stream>>>(
        *g, (const cd *)tensors, (const cd *)n2e_old, (const cd *)e2n_old, (cd *)n2e_new, (cd *)e2n_new, edge_new,
        (const long long *)plan, level_off, (int)n_levels, (int)max_slice, (int)max_chi);
  } else {
    DQZ_SMEM_ATTR_ONCE(bp_sweep_planned_kernel, BP_SMEM_LIMIT);
    bp_sweep_planned_kernel<<<1, 32 * warps, smem, stream>>>(
        *g, (const cd *)tensors, (const cd *)n2e_old, (const cd *)e2n_old, (cd *)n2e_new, (cd *)e2n_new, edge_new,
        (const long long *)plan, level_off, (int)n_levels, (int)max_slice, (int)max_chi);
  }
  DQZ_CHECK_LAUNCH();
  return DQZ_OK;
}

extern "C" int dqz_message_changes_c64(const dqz_graph_t *g, const void *n2e_a, const void *n2e_b, double *partial,
                                       cudaStream_t stream) {
  if (!g || !n2e_a || !n2e_b || !partial) return DQZ_ERR_ARG;
  const int nh = g->n_halves;
  if (nh == 0) return DQZ_OK;
  const int wpb = 8;
  msg_dist_c64_kernel<<<(nh + wpb - 1) / wpb, wpb * 32, 0, stream>>>(*g, (const float2 *)n2e_a, (const float2 *)n2e_b,
                                                                   partial);
  DQZ_CHECK_LAUNCH();
  return DQZ_OK;
}

extern "C" int dqz_bp_sweep_sliced(const dqz_graph_t *g, const void *tensors, const void *n2e_old,
                                   const void *e2n_old, void *n2e_new, void *e2n_new, const uint8_t *src_sel,
                                   const uint8_t *edge_new, const int32_t *halves, const int32_t *level_off,
                                   const int32_t *item_half, const int32_t *item_slice, const int32_t *item_off,
                                   int32_t n_levels, int32_t max_items, int32_t max_slice, int32_t max_chi,
                                   uint32_t *sync, int32_t *error_flag, cudaStream_t stream) {
  if (!g || !tensors || !n2e_old || !e2n_old || !n2e_new || !e2n_new || !src_sel || !edge_new || !halves ||
      !level_off || !item_half || !item_slice || !item_off || !sync || !error_flag || n_levels <= 0 ||
      max_items <= 0 || max_slice <= 0)
    return DQZ_ERR_ARG;
  if (max_chi <= 0 || max_chi > DQZ_MAX_CHI) return DQZ_ERR_UNSUPPORTED;
  size_t smem = bp_smem_bytes(max_slice, max_chi, false);  // two slices and a staged message
  if (smem > BP_SMEM_LIMIT) return DQZ_ERR_UNSUPPORTED;
  if (smem < SL_SMEM) smem = SL_SMEM;
  DQZ_SMEM_ATTR_ONCE(bp_sweep_sliced_kernel, BP_SMEM_LIMIT);
  int dev = 0, sms = 148, per_sm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return DQZ_ERR_CUDA;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, bp_sweep_sliced_kernel, SL_THREADS, smem) !=
          cudaSuccess ||
      per_sm < 1)
    return DQZ_ERR_UNSUPPORTED;
  int grid = max_items;  // all co-resident
  if (grid > sms * per_sm) grid = sms * per_sm;
  if (cudaMemsetAsync(sync, 0, 2 * sizeof(uint32_t), stream) != cudaSuccess) return DQZ_ERR_CUDA;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(SL_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cudaLaunchKernelEx(&cfg, bp_sweep_sliced_kernel, *g, (const cd *)tensors, (const cd *)n2e_old,
                         (const cd *)e2n_old, (cd *)n2e_new, (cd *)e2n_new, src_sel, edge_new, halves, level_off,
                         item_half, item_slice, item_off, (int)n_levels, (int)max_slice, (unsigned *)sync,
                         (int *)error_flag) != cudaSuccess)
    return DQZ_ERR_CUDA;
  return DQZ_OK;
}
