"""The one-warp Vidal-gauge kernels and the degree-3 tensor-core absorb and
density kernels against the one-CTA / generic forms and plain FP64 torch
(tensor_ops.py:88-175, density_matrix.py:16-37), at every bond up to 16."""

import numpy as np
import pytest
import torch

from dequantizer_b200 import _lib, autotune
from dequantizer_b200 import graph as G
from dequantizer_b200 import maps as M
from dequantizer_b200.layout import GraphLayout

pytestmark = pytest.mark.gpu
EPS = 1e-10


def layout_of(g):
    topo = M.Topology(list(g.get_traversal_iterator()), True)
    return GraphLayout(topo.nodes, topo.edges, [e.dimension for e in topo.edges])


def rr3(n, dims, phys=2):
    g = G.get_random_regular_graph(n, 3, phys, 1, 5)
    for i, e in enumerate(g.edges.values()):
        e.dimension = dims[i % len(dims)]
    g.refresh_bond_shapes()
    return g


def messages(L, rng, decades, deficient):
    """Positive matrices with eigenvalues log-uniform over ``decades`` (trace 1), a
    third of them set to 1e-12 when ``deficient``."""
    arena = np.zeros(L.msg_elems, dtype=np.complex128)
    for h in range(L.n_halves):
        c = int(L.edge_chi[L.half_edge[h]])
        z = rng.standard_normal((c, c)) + 1j * rng.standard_normal((c, c))
        q, _ = np.linalg.qr(z)
        w = 10.0 ** -rng.uniform(0, decades, c)
        w[0], w[-1] = 1.0, 10.0 ** -decades if c > 1 else 1.0
        if deficient:
            w[: c // 3] = 1e-12
        m = (q * (w / w.sum())) @ q.conj().T
        arena[L.half_msg_off[h]: L.half_msg_off[h] + c * c] = m.ravel()
    return torch.from_numpy(arena).cuda()


def edges_by(L, n2e, path):
    orth, lam = torch.zeros_like(n2e), L.new_lam_arena()
    nb = _lib.lib().dqz_vidal_edges_scratch_bytes(L.n_edges, L.max_chi())
    scratch = torch.empty(max(nb, 1), dtype=torch.uint8, device="cuda")
    try:
        autotune.set_knobs({"gauge_path": path})
        _lib.call("dqz_vidal_edges", L.gptr, n2e.data_ptr(), EPS, orth.data_ptr(), lam.data_ptr(), L.max_chi(), None, 0,
                  scratch.data_ptr(), _lib.stream_handle())
        torch.cuda.synchronize()
    finally:
        autotune.set_knobs({"gauge_path": 0})
    return orth, lam


# the factored form (well above the threshold), eigenvalues down to 1e-8, and messages with dropped
# eigenvalues (left to the eigendecompositions)
@pytest.mark.parametrize("decades,deficient", [(2, False), (7, False), (2, True)])
@pytest.mark.parametrize("dims", [(1,), (2,), (3, 8, 16), (7, 15), (16,)])
def test_edge_orthogonalisers(dims, decades, deficient):
    """lambda equals the one-CTA kernel's, G_f diag(lambda) G_b^T (free of the
    singular vectors' phases) too, and without dropped eigenvalues it is a
    multiple of 1 and G_f^H m_f G_f = 1 / rank. Rounding, kappa the condition of
    the messages: their entries carry eps, a relative eps kappa of the smallest
    eigenvalue, so the Gram product and the reference form's G_f lambda G_b^T
    differ from 1 by up to c eps kappa (4 c eps kappa allowed); the factored
    form's product is L^-H U' U'^H L^H, where U' U'^H - 1 of c eps a row grows
    with the condition of L only (4 c^2 eps kappa^(1/2))."""
    L = layout_of(rr3(10, dims))
    n2e = messages(L, np.random.default_rng(3), decades, deficient)
    orth, lam = edges_by(L, n2e, 0)
    ref_orth, ref_lam = edges_by(L, n2e, 2)
    assert bool(torch.isfinite(lam).all())
    assert float((lam - ref_lam).abs().max()) < 1e-13
    for e in range(L.n_edges):
        h0, h1 = int(L.edge_half[2 * e]), int(L.edge_half[2 * e + 1])
        c = int(L.edge_chi[e])
        one = torch.eye(c, device="cuda")
        le = L.lambda_view(lam, e).to(torch.complex128)
        bound = 4 * c * 2.2e-16 * 10.0 ** (12 if deficient else decades)
        p = (L.message_view(orth, h0) * le) @ L.message_view(orth, h1).mT
        r = (L.message_view(ref_orth, h0) * le) @ L.message_view(ref_orth, h1).mT
        assert float((p - r).norm() / r.norm()) < bound
        if not deficient:
            assert float((c * p / p.diagonal().sum() - one).norm()) < 4 * c * c * 2.2e-16 * 10.0 ** (0.5 * decades)
            for h in (h0, h1):
                o, m = L.message_view(orth, h), L.message_view(n2e, h)
                assert float((c * (o.mH @ m @ o) - one).norm()) < bound


@pytest.mark.parametrize("graph", ["rr3", "lattice", "hex", "rr4"])
def test_distance_terms_at_every_bond(graph):
    """Each half-edge's trace norm against the oracle's, mixed bonds up to 16 and
    physical dimension 3: the reduced matrix sums at most 3 * 16^2 products and
    the eigenvalues carry n eps of the norm, so 1e-13 of the terms' scale (below 2)."""
    g = {"rr3": lambda: rr3(12, (1, 2, 9, 16, 5), 3), "lattice": lambda: G.get_nd_lattice([3, 4], 3, 1, True),
         "hex": G.get_heavy_hex_ibm_eagle_lattice_infinite,
         "rr4": lambda: G.get_random_regular_graph(9, 4, 2, 1, 2)}[graph]()
    dims = {"lattice": (4, 7, 2), "hex": (3, 16, 10), "rr4": (3, 5, 8)}.get(graph)
    if dims:
        for i, e in enumerate(g.edges.values()):
            e.dimension = dims[i % len(dims)]
        g.refresh_bond_shapes()
    L = layout_of(g)
    rng = np.random.default_rng(4)
    T = torch.from_numpy(rng.standard_normal(L.tensor_elems) + 1j * rng.standard_normal(L.tensor_elems)).cuda()
    lam_h = np.concatenate([np.sort(10.0 ** -rng.uniform(0, 4, int(c)))[::-1] for c in L.edge_chi])
    lam = torch.from_numpy(lam_h).cuda()
    part = M.vidal_distance_partial(L, T, lam, EPS).cpu().numpy()
    lams = [L.lambda_view(lam, i).cpu().numpy() for i in range(L.n_edges)]
    for v, t in enumerate(L.unpack_tensors(T)):
        h0, k = int(L.node_half[v]), int(L.degree[v])
        ls = [lams[int(L.half_edge[h0 + f])] for f in range(k)]
        t = t.cpu().numpy()
        for f in range(k):
            y = t
            for f2 in range(k):
                if f2 != f:
                    shape = [1] * t.ndim
                    shape[f2] = -1
                    y = y * ls[f2].reshape(shape)
            y = np.moveaxis(y, f, 0).reshape(t.shape[f], -1)
            r = y.conj() @ y.T
            r = r / np.trace(r)
            on = r.diagonal().real > EPS
            ref = np.abs(np.linalg.eigvalsh(r - np.diag(on / on.sum()))).sum()
            assert abs(part[h0 + f] - ref) < 1e-13


def test_distance_of_non_finite_tensors_is_not_finite():
    L = layout_of(rr3(10, (4,)))
    T = torch.ones(L.tensor_elems, dtype=torch.complex128, device="cuda")
    T[5] = complex("nan")
    T[int(L.node_off[3]) + 1] = complex("inf")
    lam = torch.ones(L.lam_elems, dtype=torch.float64, device="cuda")
    part = M.vidal_distance_partial(L, T, lam, EPS).cpu().numpy()
    for v in (0, 3):
        h0 = int(L.node_half[v])
        assert not np.isfinite(part[h0:h0 + 3]).any()
    assert not np.isfinite(float(M.vidal_distance_packed(L, T, lam, EPS)))


@pytest.mark.parametrize("n,dims,phys", [(10, (16,), 2), (302, (16,), 2), (760, (8,), 2), (12, (5, 16, 3), 2),
                                         (12, (2, 8), 3), (10, (9, 4), 1), (160, (12,), 4)])
def test_degree3_density_and_absorb(n, dims, phys):
    """Density: rho has at most 4 * 16^3 terms in a chain of three products, its
    trace positive terms (positive messages): 1e-13. Absorb (uniform shapes): a
    chain of three 16-term products, 1e-13 of the unit norm."""
    L = layout_of(rr3(n, dims, phys))
    rng = np.random.default_rng(6)
    T = torch.from_numpy(rng.standard_normal(L.tensor_elems) + 1j * rng.standard_normal(L.tensor_elems)).cuda()
    e2n = messages(L, rng, 2, False)
    nodes = list(range(0, n, 3)) + [1]
    assert L.k3_shape()
    rho = M.density_packed(L, T, e2n, nodes)
    ts = L.unpack_tensors(T)
    orth = torch.from_numpy(rng.standard_normal(L.msg_elems) + 1j * rng.standard_normal(L.msg_elems)).cuda()
    chi = L.uniform_k3_chi()
    if chi:
        out = torch.full_like(T, 7.0)
        _lib.call("dqz_absorb_k3", L.gptr, chi, T.data_ptr(), orth.data_ptr(), out.data_ptr(), None, 0,
                  M.error_flag(L.device).data_ptr(), _lib.stream_handle())
        outs = L.unpack_tensors(out)
    for j, v in enumerate(nodes):
        h0 = int(L.node_half[v])
        y, x = ts[v], ts[v]
        for f in range(3):
            y = torch.movedim(torch.tensordot(L.message_view(e2n, h0 + f), y, dims=([1], [f])), 0, f)
            x = torch.movedim(torch.tensordot(L.message_view(orth, h0 + f), x, dims=([0], [f])), 0, f)
        r = torch.einsum("abci,abcj->ij", y, ts[v].conj())
        r = r / r.diagonal().sum()
        assert float((rho[j] - r).abs().max()) < 1e-13
        if chi:
            assert float((outs[v] - x / x.norm()).norm()) < 1e-13
    assert int(M.error_flag(L.device)) == 0
