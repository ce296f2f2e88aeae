// Blocks of bond slices of a BP node update on the FP64 tensor cores, for nodes of
// degree up to 3 with bonds up to 32 (tensor_ops.py:36-60). One CTA takes half-edge
// (v, e) and a block of its slices a: the block T[.., a@e, ..] lies in shared
// memory once, the other bonds' messages are applied in place (8 columns of the
// flattened rest at a time, a warp each: a column's rows are read and rewritten by
// one warp only), and the columns out[:, a] are contracted with conj(T) read
// through L2 once per block.
//
// Every entry is the same chain whatever the block or the grid (mode products:
// m8n8k4 steps in index order; the contraction: lane-strided sums and a warp
// reduction), so the level-by-level launches and the one-launch sweep give the
// same bits.
//
// Bound: per slice of 32 x 32 x 2 the two mode products take 2,048 m8n8k4 (8.2 k
// cycles of an SM) and the contraction 262 k multiply-adds (4.1 k) against 1 MB of
// T; blocks of two slices halve that traffic and let two CTAs of the node update
// share an SM (106 KB each; the one-launch sweep's table of levels adds 14 KB).
// Measured (127-qubit heavy-hex lattice, bond 32, all 144 half-edges in one launch):
// 425 us against 3,128 us of the generic form. Lanes as a' with rows of T read
// whole, for the bonds whose entries lie close together, took 557 us.
#pragma once

#include "dmma.cuh"

namespace dqz {

constexpr int SL_MAX = 32;              // largest bond
constexpr int SL_ELEMS = 4096;          // slice entries of a block (before padding)
constexpr int SL_MS = SL_MAX + 1;       // message row stride
constexpr int SL_THREADS = 256;
// block (strides padded) + two messages + their diagonals
constexpr int SL_BUF = SL_ELEMS + SL_ELEMS / 16 + 64;
constexpr size_t SL_SMEM = (SL_BUF + 2 * (size_t)SL_MAX * SL_MS + 2 * SL_MAX) * sizeof(cd);

// Geometry of a node's slices over bond e: the other bonds x (and y), d.
struct SliceGeom {
  int ce, nb, qx, qy, d;     // nb: other bonds (0, 1, 2)
  int P;                     // entries of a slice
  int sx, slice;             // strides of x and of a slice in the block
  int fx, fy;                // slots of the other bonds
};

__host__ __device__ inline int sl_block(int P) {  // slices of a block
  const int n = SL_ELEMS / P;
  return n < 1 ? 1 : n;
}

__device__ __forceinline__ bool sl_geometry(const NodeShape &s, int e, SliceGeom &g) {
  if (s.k < 1 || s.k > 3) return false;
  g.ce = s.dims[e];
  g.d = s.d;
  g.nb = s.k - 1;
  g.fx = e == 0 ? 1 : 0;
  g.fy = e == 2 ? 1 : 2;
  g.qx = g.nb > 0 ? s.dims[g.fx] : 1;
  g.qy = g.nb > 1 ? s.dims[g.fy] : 1;
  for (int f = 0; f < s.k; ++f)
    if (s.dims[f] > SL_MAX) return false;
  g.P = g.qx * g.qy * g.d;
  if (g.P > SL_ELEMS) return false;
  const int row = g.qy * g.d;
  g.sx = row >= 8 ? row | 1 : row;  // odd where columns run along a row (dmma.cuh)
  g.slice = (g.qx * g.sx) | 1;
  return (long long)sl_block(g.P) * g.slice <= SL_BUF || g.slice <= SL_BUF;
}

// Slices that fit a block of this geometry.
__device__ __forceinline__ int sl_count(const SliceGeom &g) {
  const int block = sl_block(g.P), most = SL_BUF / g.slice, n = block < most ? block : most;
  return n < 1 ? 1 : n;
}

// buf <- m applied to the bond of dimension q and stride ks, in place, for ncol
// columns at base(c). WIDE: eight neighbouring columns are contiguous.
template <typename Base>
__device__ __forceinline__ void sl_mode(cd *buf, const cd *m, int q, int ks, int ncol, bool wide, Base base) {
  const int lane = threadIdx.x & 31, row = lane >> 2, ql = lane & 3, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int mt = (q + 7) >> 3;
  for (int c0 = 8 * w; c0 < ncol; c0 += 8 * nw) {
    double re[4][2], im[4][2];
#pragma unroll
    for (int r = 0; r < 4; ++r) re[r][0] = re[r][1] = im[r][0] = im[r][1] = 0.0;
    const bool in = c0 + row < ncol;
    const cd *src = buf + (in ? base(c0 + row) : 0);
    for (int t = 0; t < mt; ++t)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int k = 8 * t + (wide ? 2 * ql + i : ql + 4 * i);
        const cd b = in && k < q ? src[k * ks] : czero();
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          if (r < mt) {
            const cd a = m[(8 * r + row) * SL_MS + k];
            dmma(re[r], a.x, b.x);
            dmma(im[r], a.x, b.y);
            dmma(re[r], -a.y, b.y);
            dmma(im[r], a.y, b.x);
          }
        }
      }
    __syncwarp();
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int c = c0 + 2 * ql + j;
      if (c >= ncol) continue;
      cd *dst = buf + base(c);
#pragma unroll
      for (int r = 0; r < 4; ++r)
        if (8 * r + row < q) dst[(8 * r + row) * ks] = mk(re[r][j], im[r][j]);
    }
  }
  __syncthreads();
}

// The other bonds' messages (q x q, global) into shared memory, zero-padded to 32
// x 32, divided by their traces where `tx` / `ty` (the sum in index order, as
// normalise_by_trace; the diagonal goes through shared memory, so that every
// global load is in flight at once). `diag`: 64 entries. Whole CTA, no barrier at
// the end.
__device__ __forceinline__ void sl_messages(const SliceGeom &g, const cd *mx, bool tx, const cd *my, bool ty, cd *sM,
                                            cd *diag) {
  constexpr int PT = SL_MAX * SL_MAX / SL_THREADS;
  const int tid = threadIdx.x;
  cd x[2][PT];
#pragma unroll
  for (int f = 0; f < 2; ++f) {
    const int q = f < g.nb ? (f ? g.qy : g.qx) : 0;
    const cd *m = f ? my : mx;
#pragma unroll
    for (int j = 0; j < PT; ++j) {
      const int i = tid + j * SL_THREADS, r = i / SL_MAX, c = i % SL_MAX;
      x[f][j] = r < q && c < q ? __ldcg(m + r * q + c) : czero();
      if (r == c && r < q) diag[f * SL_MAX + r] = x[f][j];
    }
  }
  __syncthreads();
#pragma unroll
  for (int f = 0; f < 2; ++f) {
    if (f >= g.nb) continue;
    const bool by = f ? ty : tx;
    const int q = f ? g.qy : g.qx;
    cd tr = czero();
    if (by)
      for (int i = 0; i < q; ++i) tr = cadd(tr, diag[f * SL_MAX + i]);
#pragma unroll
    for (int j = 0; j < PT; ++j) {
      const int i = tid + j * SL_THREADS, r = i / SL_MAX, c = i % SL_MAX;
      if (by && r < q && c < q) x[f][j] = cdiv(x[f][j], tr);
      sM[f * SL_MAX * SL_MS + r * SL_MS + c] = x[f][j];
    }
  }
}

// One block of slices: T at the node, its stride and the block's columns of dst.
struct SliceItem {
  SliceGeom g;
  const cd *T;
  unsigned Re;
  int a0, n;
};

// The block of T into shared memory. Whole CTA, no barrier.
__device__ __forceinline__ void sl_load(const SliceItem &it, cd *buf) {
  const SliceGeom &g = it.g;
  const unsigned P = (unsigned)g.P, row = (unsigned)(g.qy * g.d), ce = (unsigned)g.ce;
  const FastDiv fP(P), fRe(it.Re), fRow(row);
  for (unsigned i = threadIdx.x; i < (unsigned)it.n * P; i += blockDim.x) {
    const unsigned a = fP.div(i), x = i - a * P, xx = fRow.div(x), l = fRe.div(x);
    cp_async16(buf + a * (unsigned)g.slice + xx * (unsigned)g.sx + (x - xx * row),
               it.T + l * ce * it.Re + (x - l * it.Re) + (unsigned)(it.a0 + a) * it.Re);
  }
  cp_async_commit();
}

// out[a'][a] = sum_x conj(T[x, a']) buf[a][x] for slices b0 .. b0 + JN - 1 of the
// block: a warp takes AP values of a' at a time, U rounds of loads in flight.
template <int JN, int AP, int U, typename Put>
__device__ __forceinline__ void sl_contract(const SliceItem &it, const cd *buf, int b0, Put put) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const SliceGeom &g = it.g;
  const unsigned P = (unsigned)g.P, row = (unsigned)(g.qy * g.d), ce = (unsigned)g.ce, Re = it.Re;
  const FastDiv fRe(Re), fRow(row);
  for (int p0 = AP * w; p0 < g.ce; p0 += AP * nw) {
    cd acc[AP][JN];
#pragma unroll
    for (int i = 0; i < AP; ++i)
#pragma unroll
      for (int j = 0; j < JN; ++j) acc[i][j] = czero();
    for (unsigned x0 = lane; x0 < P; x0 += 32 * U) {
      cd t[U][AP];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const unsigned x = x0 + 32 * u, l = fRe.div(x);
        const cd *src = it.T + l * ce * Re + (x - l * Re);
#pragma unroll
        for (int i = 0; i < AP; ++i) t[u][i] = x < P && p0 + i < g.ce ? src[(unsigned)(p0 + i) * Re] : czero();
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const unsigned x = x0 + 32 * u, xx = fRow.div(x);
        if (x >= P) continue;
        const cd *z = buf + b0 * g.slice + xx * (unsigned)g.sx + (x - xx * row);
#pragma unroll
        for (int j = 0; j < JN; ++j) {
          const cd y = z[j * g.slice];
#pragma unroll
          for (int i = 0; i < AP; ++i) cfmac(acc[i][j], t[u][i], y);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < JN; ++j)
#pragma unroll
      for (int i = 0; i < AP; ++i) {
        const cd v = warp_csum(acc[i][j]);
        if (lane == 0 && p0 + i < g.ce) put(p0 + i, it.a0 + b0 + j, v);
      }
  }
}

// The other bonds' messages applied to the block. Whole CTA; ends with a barrier
// (when there is another bond).
__device__ __forceinline__ void sl_apply(const SliceItem &it, cd *buf, const cd *sM) {
  const SliceGeom &g = it.g;
  const unsigned row = (unsigned)(g.qy * g.d);
  if (g.nb > 0) {
    const FastDiv f(row);
    sl_mode(buf, sM, g.qx, g.sx, it.n * (int)row, row >= 8, [&](int c) {
      const unsigned a = f.div((unsigned)c);
      return (int)(a * (unsigned)g.slice + ((unsigned)c - a * row));
    });
  }
  if (g.nb > 1) {
    const unsigned xd = (unsigned)(g.qx * g.d);
    const FastDiv f(xd), fd((unsigned)g.d);
    sl_mode(buf, sM + SL_MAX * SL_MS, g.qy, g.d, it.n * (int)xd, false, [&](int c) {
      const unsigned a = f.div((unsigned)c), r = (unsigned)c - a * xd, xx = fd.div(r);
      return (int)(a * (unsigned)g.slice + xx * (unsigned)g.sx + (r - xx * (unsigned)g.d));
    });
  }
}

// Columns a0 .. a0 + n - 1 of the unnormalised outgoing message: put(a', a, value).
// sl_load has been issued. mx, my: the other bonds' messages; tx, ty: divide them
// by their traces. Whole CTA; ends with a barrier.
template <typename Put>
__device__ __forceinline__ void sl_columns(const SliceItem &it, const cd *mx, bool tx, const cd *my, bool ty, cd *buf,
                                           cd *sM, Put put) {
  sl_messages(it.g, mx, tx, my, ty, sM, sM + 2 * SL_MAX * SL_MS);
  cp_async_wait<0>();
  __syncthreads();
  sl_apply(it, buf, sM);
  int b0 = 0;
  for (; b0 + 4 <= it.n; b0 += 4) sl_contract<4, 2, 4>(it, buf, b0, put);
  if (b0 + 2 <= it.n) {
    sl_contract<2, 4, 4>(it, buf, b0, put);
    b0 += 2;
  }
  if (b0 < it.n) sl_contract<1, 4, 4>(it, buf, b0, put);
  __syncthreads();
}

}  // namespace dqz
