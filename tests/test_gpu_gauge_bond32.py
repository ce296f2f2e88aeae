"""Vidal gauge kernels of bonds from 17 to 32 (tensor_ops.py:88-175)."""

import numpy as np
import pytest
import torch

from dequantizer_b200 import graph as G
from dequantizer_b200 import maps as M
from tests.test_gpu_gauge_kernels import edges_by, layout_of, messages, rr3

pytestmark = pytest.mark.gpu
EPS64 = 2.2e-16


# mixed with small bonds (one CTA takes any up to 32), odd, and the largest; a third of the eigenvalues dropped
@pytest.mark.parametrize("decades,deficient", [(2, False), (7, False), (2, True)])
@pytest.mark.parametrize("dims", [(17,), (1, 32, 2), (20, 31, 5), (32,)])
def test_edge_orthogonalisers(dims, decades, deficient):
    """Against the one-CTA form with two-sided rotations. Eigenvalues carry c eps
    of the message (trace 1), so its square root c eps sqrt(kappa) and lambda
    that over |sigma| >= c^(-1/2): 4 c^(3/2) eps sqrt(kappa) allowed. G_f lambda
    G_b^T and the Gram product as for bonds up to 16: 4 c eps kappa, kappa 1e12
    with dropped eigenvalues."""
    L = layout_of(rr3(10, dims))
    n2e = messages(L, np.random.default_rng(3), decades, deficient)
    orth, lam = edges_by(L, n2e, 0)
    ref_orth, ref_lam = edges_by(L, n2e, 2)
    assert bool(torch.isfinite(lam).all())
    for e in range(L.n_edges):
        h0, h1 = int(L.edge_half[2 * e]), int(L.edge_half[2 * e + 1])
        c = int(L.edge_chi[e])
        d = (L.lambda_view(lam, e) - L.lambda_view(ref_lam, e)).abs().max()
        assert float(d) < 4 * c ** 1.5 * EPS64 * 10.0 ** (0.5 * decades)
        le = L.lambda_view(lam, e).to(torch.complex128)
        bound = 4 * c * EPS64 * 10.0 ** (12 if deficient else decades)
        p = (L.message_view(orth, h0) * le) @ L.message_view(orth, h1).mT
        r = (L.message_view(ref_orth, h0) * le) @ L.message_view(ref_orth, h1).mT
        assert float((p - r).norm() / r.norm()) < bound
        if not deficient:
            for h in (h0, h1):
                o, m = L.message_view(orth, h), L.message_view(n2e, h)
                assert float((c * (o.mH @ m @ o) - torch.eye(c, device="cuda")).norm()) < bound


def test_indefinite_and_non_finite_messages_take_the_two_sided_form():
    """Eigenvalues of both signs and one size, a zero message and a NaN: the same bits as the form they are left to."""
    L = layout_of(rr3(10, (24,)))
    n2e = messages(L, np.random.default_rng(5), 2, False)
    rng = np.random.default_rng(6)
    for e in range(L.n_edges):
        q, _ = np.linalg.qr(rng.standard_normal((24, 24)) + 1j * rng.standard_normal((24, 24)))
        w = np.where(np.arange(24) % 2, -1.0, 1.0) * (1 + np.arange(24) // 2)
        L.message_view(n2e, int(L.edge_half[2 * e + e % 2])).copy_(torch.from_numpy((q * w) @ q.conj().T).cuda())
    L.message_view(n2e, int(L.edge_half[0])).zero_()
    L.message_view(n2e, int(L.edge_half[3]))[4, 4] = complex("nan")
    for a, b in zip(edges_by(L, n2e, 0), edges_by(L, n2e, 2)):
        assert torch.equal(torch.nan_to_num(torch.view_as_real(a) if a.is_complex() else a, nan=3e33),
                           torch.nan_to_num(torch.view_as_real(b) if b.is_complex() else b, nan=3e33))


# blocks of one, two and many slices, leaves, over 592 nodes; slices above a block and degree 4 (whole-node form)
@pytest.mark.parametrize("graph,n,dims,phys", [("rr3", 10, (32, 17, 31), 2), ("rr3", 8, (32,), 4), ("rr3", 8, (31, 32, 7), 3),
                                               ("rr3", 600, (17, 3, 22), 8), ("tree", 9, (32, 29), 8), ("rr3", 6, (24,), 1),
                                               ("rr3", 6, (17, 31, 20), 8), ("rr4", 6, (9, 10), 2)])
def test_density(graph, n, dims, phys):
    """A chain of three 32-term products and lane-strided sums of at most 32^3 / 32
    terms, 1,100 eps = 2.4e-13 of sum |T| |m T| <= |T| |m T|, which is below 3 per
    bond (eigenvalues over two decades) times the trace: 1e-11."""
    g = {"rr3": lambda: G.get_random_regular_graph(n, 3, phys, 1, 5), "rr4": lambda: G.get_random_regular_graph(n, 4, phys, 1, 5),
         "tree": lambda: G.get_random_tree_tensor_graph(n, phys, [1], 5)}[graph]()
    for i, e in enumerate(g.edges.values()):
        e.dimension = dims[i % len(dims)]
    g.refresh_bond_shapes()
    L = layout_of(g)
    rng = np.random.default_rng(6)
    T = torch.from_numpy(rng.standard_normal(L.tensor_elems) + 1j * rng.standard_normal(L.tensor_elems)).cuda()
    e2n = messages(L, rng, 2, False)
    nodes = list(range(L.n_nodes)) + [1]
    assert not L.k3_shape()
    rho = M.density_packed(L, T, e2n, nodes)
    ts = L.unpack_tensors(T)
    for j, v in enumerate(nodes):
        h0, y = int(L.node_half[v]), ts[v]
        for f in range(int(L.degree[v])):
            y = torch.movedim(torch.tensordot(L.message_view(e2n, h0 + f), y, dims=([1], [f])), 0, f)
        r = torch.einsum("bi,bj->ij", y.reshape(-1, phys), ts[v].conj().reshape(-1, phys))
        assert float((rho[j] - r / r.diagonal().sum()).abs().max()) < 1e-11
