"""Vidal edges of messages far from unit scale (tensor_ops.py:108-130): lambdas
are normalised, so a common factor of the messages only scales the
orthogonalisers."""

import numpy as np
import pytest
import torch

from dequantizer_b200 import _lib
from dequantizer_b200 import graph as G
from dequantizer_b200 import maps as M
from dequantizer_b200.layout import GraphLayout

pytestmark = pytest.mark.gpu


# the factored form (up to 16) and the one-CTA Jacobi (17 to 32); at 1e73 the scalar products of two columns of C are
# 1e146 and their squares, 1e292, still finite
@pytest.mark.parametrize("chi", [2, 5, 16, 17, 32])
@pytest.mark.parametrize("scale", [1e40, 1e73])
def test_edges_of_scaled_messages(chi, scale):
    """Against scale 1, conditions up to 1e2: lambdas to 1e-13, G_f diag(lambda)
    G_b^T (free of the singular vectors' phases) to 4 chi^2 eps 1e2 < 1e-10 of its norm."""
    g = G.get_random_regular_graph(8, 3, 2, chi, 5)
    topo = M.Topology(list(g.get_traversal_iterator()), True)
    L = GraphLayout(topo.nodes, topo.edges, [chi] * len(topo.edges))
    rng = np.random.default_rng(chi)
    mats = []
    for _ in range(L.n_halves):
        q, _ = np.linalg.qr(rng.standard_normal((chi, chi)) + 1j * rng.standard_normal((chi, chi)))
        mats.append((q * 10.0 ** -rng.uniform(0, 2, chi)) @ q.conj().T)
    out = []
    for s in (1.0, scale):
        n2e = torch.from_numpy(s * np.concatenate([m.ravel() for m in mats])).cuda()
        orth, lam = torch.zeros_like(n2e), L.new_lam_arena()
        nb = _lib.lib().dqz_vidal_edges_scratch_bytes(L.n_edges, chi)
        scratch = torch.empty(max(nb, 1), dtype=torch.uint8, device="cuda")
        _lib.call("dqz_vidal_edges", L.gptr, n2e.data_ptr(), 1e-10, orth.data_ptr(), lam.data_ptr(), chi, None, 0,
                  scratch.data_ptr(), _lib.stream_handle())
        out.append((lam, [s * (L.message_view(orth, int(L.edge_half[2 * e])) * L.lambda_view(lam, e))
                          @ L.message_view(orth, int(L.edge_half[2 * e + 1])).mT for e in range(L.n_edges)]))
    assert float((out[0][0] - out[1][0]).abs().max()) < 1e-13
    for p, r in zip(out[1][1], out[0][1]):
        assert float((p - r).norm() / r.norm()) < 1e-10
