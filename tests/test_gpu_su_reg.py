"""The register form of the simple update (dqz_simple_update, default knob)
against the one-CTA kernel and the oracle (tensor_ops.py:265-389): bonds at the
edges of its limits, ranks 1, 2 and 4, other physical dimensions, null singular
values, and batches above one workspace chunk.

Tolerances as elsewhere: lambdas, errors, entropies and the two-site tensor
around the updated bond 1e-10 (SVD of matrices of norm 1 in FP64, both sides
backward stable to about 1e-14, divided by lambdas down to 1e-3)."""

import numpy as np
import pytest
import torch

from dequantizer_b200 import _lib, autotune
from dequantizer_b200 import graph as G
from dequantizer_b200 import maps as M
from dequantizer_b200.gates import decompose_gates
from dequantizer_b200.layout import GraphLayout
from dequantizer_b200.tensor_graph_ops import simple_update_shapes
from oracle import maps as OM
from tests.helpers import random_tensors, rel_err, two_site

pytestmark = pytest.mark.gpu
TOL = 1e-10


def gate_of_rank(rank, d, rng):
    """Diagonal phases (rank 2 at most), a product gate (1) or a random unitary (d^2)."""
    if rank == 1:
        a, b = (np.linalg.qr(rng.standard_normal((d, d)) + 1j * rng.standard_normal((d, d)))[0] for _ in range(2))
        return np.einsum("ac,bd->abcd", a, b)
    if rank == 2:
        phase = np.where(np.arange(d)[:, None] == np.arange(d)[None, :], 0.3, -0.4)
        z = np.exp(1j * phase) if d == 2 else np.exp(1j * 0.5 * np.outer(np.arange(d) == 0, np.arange(d) == 0))
        return np.einsum("ab,ac,bd->abcd", z, np.eye(d), np.eye(d))
    z = rng.standard_normal((d * d, d * d)) + 1j * rng.standard_normal((d * d, d * d))
    return np.linalg.qr(z)[0].reshape(d, d, d, d)


# (bonds cycled over the edges, physical dimension, gate rank, cap)
@pytest.mark.parametrize("dims,d,rank,cap", [
    ((16,), 2, 2, 16), ((16,), 2, 1, None), ((15, 16, 1), 2, 2, None), ((8,), 2, 4, 8), ((8,), 2, 4, None),
    ((4, 7), 2, 2, 5), ((1,), 2, 4, 4), ((2,), 2, 1, 2), ((5, 3), 3, 2, 6), ((17, 3), 2, 2, 17), ((4,), 4, 2, None),
])
def test_register_form_matches_oracle(dims, d, rank, cap):
    rng = np.random.default_rng(sum(dims) + d + rank)

    def graph():
        g = G.get_random_regular_graph(6, 3, d, 1, 2)
        for i, e in enumerate(g.edges.values()):
            e.dimension = dims[i % len(dims)]
        g.refresh_bond_shapes()
        return g

    g_ref, g_gpu = graph(), graph()
    tensors = random_tensors(g_ref, 3)
    lambdas = {}
    for eid, e in g_ref.edges.items():
        lam = np.sort(10.0 ** rng.uniform(-3, 0, e.dimension))[::-1]
        lambdas[eid] = lam / np.linalg.norm(lam)
    for a, b in list(g_ref.edges)[:3]:
        gate = gate_of_rank(rank, d, rng)
        g_ref, g_gpu = graph(), graph()
        r_t, r_l = dict(tensors), {k: v.copy() for k, v in lambdas.items()}
        g_t = {k: torch.from_numpy(v).cuda() for k, v in tensors.items()}
        g_l = {k: torch.from_numpy(v.copy()).cuda() for k, v in lambdas.items()}
        _, _, er, en = OM.apply2_to_vidal_canonical(g_ref, a, b, r_t, r_l, gate, 1e-10, None, cap)
        _, _, eg, ng = g_gpu.apply2_to_vidal_canonical(a, b, g_t, g_l, gate, 1e-10, None, cap)
        edge = g_ref.find_edge(a, b)
        assert g_gpu.find_edge(a, b).dimension == edge.dimension
        assert rel_err(g_l[edge.id], r_l[edge.id]) < TOL
        assert abs(float(eg) - er) < TOL and abs(float(ng) - en) < TOL
        i1, i2 = g_ref.get_node(a).indices[edge.id], g_ref.get_node(b).indices[edge.id]
        assert rel_err(two_site(g_t[a], g_t[b], i1, i2, g_l[edge.id]),
                       two_site(r_t[a], r_t[b], i1, i2, r_l[edge.id])) < TOL


@pytest.mark.parametrize("chi,n", [(2, 2000), (8, 300)])
def test_batches_match_the_one_cta_kernel(chi, n):
    """A matching of a random 3-regular graph in one call (2000 nodes: more jobs than one workspace chunk)."""
    g = G.get_random_regular_graph(n, 3, 2, chi, 4)
    topo = M.Topology(list(g.get_traversal_iterator()), True)
    rng = np.random.default_rng(8)
    results = []
    for knob in (0, 1):
        L = GraphLayout(topo.nodes, topo.edges, [chi] * len(topo.edges))
        gen = torch.Generator(device="cuda").manual_seed(5)
        T = torch.randn(L.tensor_elems, dtype=torch.complex128, device="cuda", generator=gen)
        lam = torch.rand(L.lam_elems, dtype=torch.float64, device="cuda", generator=gen) + 0.1
        used, jobs = set(), []
        for e in range(L.n_edges):
            a, b = (int(L.half_node[L.edge_half[2 * e + i]]) for i in (0, 1))
            if not {a, b} & used:
                used |= {a, b}
                jobs.append(e)
        m = len(jobs)
        assert n < 2000 or m > 592
        flat, ranks, _ = decompose_gates(gate_of_rank(2, 2, rng)[None], 1e-10)
        m1, m2, k, _, _ = simple_update_shapes([chi] * 3, 2, 0, [chi] * 3, 2, 0, int(ranks[0]), chi)
        halves = torch.from_numpy(np.repeat(flat.reshape(1, -1), m, 0)).cuda()
        rk = torch.full((m,), int(ranks[0]), dtype=torch.int32, device="cuda")
        edges = torch.tensor(jobs, dtype=torch.int32, device="cuda")
        first = torch.ones(m, dtype=torch.uint8, device="cuda")
        err, ent = (torch.empty(m, dtype=torch.float64, device="cuda") for _ in range(2))
        scratch = torch.empty(_lib.lib().dqz_simple_update_scratch_bytes(m, max(m1, m2), k), dtype=torch.uint8,
                              device="cuda")
        try:
            autotune.set_knobs({"su_onchip": knob})
            _lib.call("dqz_simple_update", L.gptr, T.data_ptr(), lam.data_ptr(), edges.data_ptr(), first.data_ptr(),
                      halves.data_ptr(), rk.data_ptr(), m, 1e-10, chi, max(m1, m2), k, err.data_ptr(),
                      ent.data_ptr(), scratch.data_ptr(), _lib.stream_handle())
            torch.cuda.synchronize()
        finally:
            autotune.set_knobs({"su_onchip": 0})
        theta = []
        for e in jobs[:: max(1, m // 50)] + jobs[-3:]:
            h0, h1 = int(L.edge_half[2 * e]), int(L.edge_half[2 * e + 1])
            ts = L.unpack_tensors(T)
            a, b = int(L.half_node[h0]), int(L.half_node[h1])
            theta.append(two_site(ts[a], ts[b], h0 - int(L.node_half[a]), h1 - int(L.node_half[b]),
                                  L.lambda_view(lam, e)))
        results.append((lam, err, ent, theta))
    for x, y in zip(results[0][:3], results[1][:3]):
        assert float((x - y).abs().max()) < TOL
    for x, y in zip(results[0][3], results[1][3]):
        assert rel_err(x, y) < TOL
