"""Vidal edges that the factored form leaves (rank-deficient, indefinite and
non-finite messages among positive ones), by a CTA or a warp each
(tensor_ops.py:108-130)."""

import numpy as np
import pytest
import torch

from dequantizer_b200 import graph as G
from tests.test_gpu_gauge_kernels import edges_by, layout_of, messages

pytestmark = pytest.mark.gpu


# 294 edges: a CTA per marked edge from bond 3; 303: a warp, from bond 15 a CTA
@pytest.mark.parametrize("n,chi", [(196, 3), (196, 16), (202, 3), (202, 14), (202, 15), (196, 2), (202, 2)])
def test_marked_edges_among_others(n, chi):
    """Against the one-CTA form with two-sided rotations, conditions up to 1e2 with
    some eigenvalues zero: lambdas to 1e-13, G_f lambda G_b^T to 4 c eps 1e2 / the
    smallest kept weight, below 1e-11 of its norm; a non-finite message stays with its edge."""
    L = layout_of(G.get_random_regular_graph(n, 3, 2, chi, 3))
    rng = np.random.default_rng(n + chi)
    n2e = messages(L, rng, 2, False)
    few = [0, 7, L.n_edges // 2, L.n_edges - 1]
    for i, e in enumerate(few):  # rank 1 and about half, on either side
        z = rng.standard_normal((chi, 1 if i % 2 else (chi + 1) // 2)) + 1j * rng.standard_normal(
            (chi, 1 if i % 2 else (chi + 1) // 2))
        m = z @ z.conj().T
        L.message_view(n2e, int(L.edge_half[2 * e + (i // 2) % 2])).copy_(torch.from_numpy(m / np.trace(m)).cuda())
    q, _ = np.linalg.qr(rng.standard_normal((chi, chi)) + 1j * rng.standard_normal((chi, chi)))
    w = np.where(np.arange(chi) % 2, -1.0, 1.0) * (1 + np.arange(chi) // 2)
    L.message_view(n2e, int(L.edge_half[2 * 11])).copy_(torch.from_numpy((q * w) @ q.conj().T).cuda())
    L.message_view(n2e, int(L.edge_half[2 * 23]))[0, 0] = complex("nan")
    orth, lam = edges_by(L, n2e, 0)
    ref_orth, ref_lam = edges_by(L, n2e, 2)
    for e in range(L.n_edges):
        le, lr = L.lambda_view(lam, e), L.lambda_view(ref_lam, e)
        if e == 23:
            continue
        assert float((le - lr).abs().max()) < 1e-13
        h0, h1 = int(L.edge_half[2 * e]), int(L.edge_half[2 * e + 1])
        p = (L.message_view(orth, h0) * le) @ L.message_view(orth, h1).mT
        r = (L.message_view(ref_orth, h0) * lr) @ L.message_view(ref_orth, h1).mT
        assert float((p - r).norm() / r.norm()) < 1e-11
