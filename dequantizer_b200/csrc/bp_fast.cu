// Node updates of uniform degree-3 nodes by half-edge (the kernels are in bp_k3.cu,
// FP64, and bp_k3_f32.cu, FP32) and the edge pass of complex64 arenas.
#include "common.cuh"

using namespace dqz;

namespace dqz {
int bp_k3_halves(const dqz_graph_t *g, int chi, const void *T, const void *n2e_old, const void *e2n_old, void *n2e_new,
                 const uint8_t *src_sel, const int32_t *halves, int n, int *error_flag, cudaStream_t stream);
int bp_k3_halves_c64(const dqz_graph_t *g, int chi, const void *T, const void *n2e_old, const void *e2n_old,
                     void *n2e_new, const uint8_t *src_sel, const int32_t *halves, int n, int *error_flag,
                     cudaStream_t stream);
}  // namespace dqz

namespace {

template <typename W>
__global__ void edge_pass_words(dqz_graph_t g, const W *n2e_old, const W *n2e_new, const uint8_t *edge_new,
                                W *e2n_new) {
  const int wpb = blockDim.x >> 5, lane = threadIdx.x & 31;
  for (int h = blockIdx.x * wpb + (threadIdx.x >> 5); h < g.n_halves; h += gridDim.x * wpb) {
    const int e = g.half_edge[h], tw = g.half_twin[h];
    if (e < 0 || tw < 0) continue;
    const int c = g.edge_chi[e];
    const W *src = (edge_new[h] ? n2e_new : n2e_old) + g.half_msg_off[tw];
    W *dst = e2n_new + g.half_msg_off[h];
    const int bytes = c * c * (int)sizeof(W);
    if (bytes % 16 == 0 && ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15) == 0)
      warp_copy16(reinterpret_cast<uint4 *>(dst), reinterpret_cast<const uint4 *>(src), bytes / 16);
    else
      for (int i = lane; i < c * c; i += 32) dst[i] = src[i];
  }
}

}  // namespace

extern "C" int dqz_bp_node_update_k3(const dqz_graph_t *g, int32_t chi, int32_t precision, const void *tensors,
                                     const void *n2e_old, const void *e2n_old, void *n2e_new, const uint8_t *src_sel,
                                     const int32_t *halves, int32_t n_halves, int32_t *error_flag,
                                     cudaStream_t stream) {
  if (!g || !tensors || !n2e_old || !e2n_old || !n2e_new || !src_sel || !halves || !error_flag || n_halves < 0)
    return DQZ_ERR_ARG;
  if (n_halves == 0) return DQZ_OK;
  if (precision == 64)
    return bp_k3_halves(g, chi, tensors, n2e_old, e2n_old, n2e_new, src_sel, halves, n_halves, error_flag, stream);
  if (precision == 32)
    return bp_k3_halves_c64(g, chi, tensors, n2e_old, e2n_old, n2e_new, src_sel, halves, n_halves, error_flag, stream);
  return DQZ_ERR_UNSUPPORTED;
}

extern "C" int dqz_bp_edge_pass_c64(const dqz_graph_t *g, const void *n2e_old, const void *n2e_new,
                                    const uint8_t *edge_new, void *e2n_new, cudaStream_t stream) {
  if (!g || !n2e_old || !n2e_new || !edge_new || !e2n_new) return DQZ_ERR_ARG;
  if (g->n_halves == 0) return DQZ_OK;
  const int wpb = 8;
  edge_pass_words<float2><<<(g->n_halves + wpb - 1) / wpb, 32 * wpb, 0, stream>>>(
      *g, (const float2 *)n2e_old, (const float2 *)n2e_new, edge_new, (float2 *)e2n_new);
  DQZ_CHECK_LAUNCH();
  return DQZ_OK;
}
