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


@pytest.mark.parametrize("dims,phys", [((17,), 2), ((32, 1, 30), 3), ((32,), 2), ((31, 2, 33), 2)])
def test_distance_terms(dims, phys):
    """Each half-edge's trace norm (33: the form above bond 32). R sums at most 3 *
    32^2 products a split, 768 eps = 1.7e-13 of a trace of 1, its trace norm moves
    by at most 32^(1/2) times the Frobenius norm of that: 1e-12."""
    L = layout_of(rr3(8, dims, phys))
    rng = np.random.default_rng(4)
    T = torch.from_numpy(rng.standard_normal(L.tensor_elems) + 1j * rng.standard_normal(L.tensor_elems)).cuda()
    lam_h = np.concatenate([np.sort(10.0 ** -rng.uniform(0, 4, int(c)))[::-1] for c in L.edge_chi])
    lam = torch.from_numpy(lam_h).cuda()
    part = M.vidal_distance_partial(L, T, lam, 1e-10).cpu().numpy()
    for v, t in enumerate(L.unpack_tensors(T)):
        h0 = int(L.node_half[v])
        ls = [L.lambda_view(lam, int(L.half_edge[h0 + f])) for f in range(3)]
        for f in range(3):
            y = t
            for f2 in range(3):
                if f2 != f:
                    y = y * ls[f2].reshape([-1 if i == f2 else 1 for i in range(4)])
            y = torch.movedim(y, f, 0).reshape(t.shape[f], -1).cpu().numpy()
            r = y.conj() @ y.T
            r = r / np.trace(r)
            on = r.diagonal().real > 1e-10
            ref = np.abs(np.linalg.eigvalsh(r - np.diag(on / on.sum()))).sum()
            assert abs(part[h0 + f] - ref) < 1e-12


def test_distance_of_diagonal_zero_and_non_finite_tensors():
    """Graded and diagonal reduced matrices (no reflector, tiny off-diagonals), a zero and a NaN tensor."""
    L = layout_of(rr3(8, (32,)))
    T = torch.zeros(L.tensor_elems, dtype=torch.complex128, device="cuda")
    for v, t in enumerate(L.unpack_tensors(T)):
        base = int(L.node_off[v])
        i = torch.arange(32, device="cuda")
        idx = ((i * 32 + i) * 32 + i) * 2
        T[base + idx] = (10.0 ** (-0.5 * i)).to(torch.complex128)
    T[int(L.node_off[5]):int(L.node_off[5]) + 65536] = 0.0
    T[int(L.node_off[6]) + 7] = complex("nan")
    lam = torch.ones(L.lam_elems, dtype=torch.float64, device="cuda")
    part = M.vidal_distance_partial(L, T, lam, 1e-10).cpu().numpy()
    w = ((10.0 ** (-0.5 * i)).to(torch.complex128).abs() ** 2).cpu().numpy()  # of the entries as stored
    w /= w.sum()
    on = w > 1e-10
    ref = np.abs(w - on / on.sum()).sum()
    for v in range(8):
        h0 = int(L.node_half[v])
        if v in (5, 6):
            assert not np.isfinite(part[h0:h0 + 3]).any()
        else:
            assert np.abs(part[h0:h0 + 3] - ref).max() < 1e-13


@pytest.mark.parametrize("dims,phys", [((32,), 2), ((1, 31, 8), 3), ((2, 5), 1)])
def test_symmetric_gauge(dims, phys):
    """T times the square roots of the kept lambdas over its norm: a product of
    three roots and one division, the norm's sum 65,536 / 512 terms a lane in
    chains: 128 eps = 3e-14 of an entry, 1e-13."""
    from dequantizer_b200 import _lib
    L = layout_of(rr3(8, dims, phys))
    rng = np.random.default_rng(4)
    T = torch.from_numpy(rng.standard_normal(L.tensor_elems) + 1j * rng.standard_normal(L.tensor_elems)).cuda()
    lam = torch.from_numpy(10.0 ** -rng.uniform(0, 12, L.lam_elems)).cuda()
    out = torch.zeros_like(T)
    _lib.call("dqz_symmetric_gauge", L.gptr, T.data_ptr(), lam.data_ptr(), 1e-10, out.data_ptr(), _lib.stream_handle())
    for v, (t, o) in enumerate(zip(L.unpack_tensors(T), L.unpack_tensors(out))):
        h0 = int(L.node_half[v])
        for f in range(3):
            le = L.lambda_view(lam, int(L.half_edge[h0 + f]))
            t = t * torch.where(le > 1e-10, le, 0.0).sqrt().reshape([-1 if i == f else 1 for i in range(4)])
        t = t / t.norm()
        assert float(((o - t).abs() - 1e-13 * t.abs()).max()) <= 0.0
