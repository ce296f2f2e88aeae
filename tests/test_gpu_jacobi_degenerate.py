"""One-sided Jacobi of matrices with nearly equal singular values: the Vidal
edges of bonds from 17 on, whose eigendecompositions and SVD are such iterations
(tensor_ops.py:108-130), on messages next to the identity."""

import numpy as np
import pytest
import torch

from dequantizer_b200 import graph as G
from tests.test_gpu_gauge_kernels import edges_by, layout_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chi", [17, 24, 32])
@pytest.mark.parametrize("size", [3e-10, 1e-11, 1e-13])
def test_messages_next_to_the_identity(chi, size):
    """m = (1 + size H) / c with H of norm about 1: condition 1, so G_f^H m_f G_f,
    G_b^H m_b G_b and G_f lambda G_b^T are multiples of 1 to a few c^(3/2) eps in
    Frobenius norm (sums of c products of orthonormal columns): 8 c^(3/2) eps."""
    L = layout_of(G.get_random_regular_graph(8, 3, 2, chi, 5))
    rng = np.random.default_rng(chi)
    n2e = np.zeros(L.msg_elems, dtype=complex)
    for h in range(L.n_halves):
        z = rng.standard_normal((chi, chi)) + 1j * rng.standard_normal((chi, chi))
        m = (np.eye(chi) + size * (z + z.conj().T) / np.linalg.norm(z, 2)) / chi
        n2e[L.half_msg_off[h]: L.half_msg_off[h] + chi * chi] = m.ravel()
    n2e = torch.from_numpy(n2e).cuda()
    orth, lam = edges_by(L, n2e, 0)
    one, bound = torch.eye(chi, device="cuda"), 8 * chi ** 1.5 * 2.2e-16
    for e in range(L.n_edges):
        h0, h1 = int(L.edge_half[2 * e]), int(L.edge_half[2 * e + 1])
        for h in (h0, h1):
            o, m = L.message_view(orth, h), L.message_view(n2e, h)
            assert float((chi * (o.mH @ m @ o) - one).norm()) < bound
        p = (L.message_view(orth, h0) * L.lambda_view(lam, e)) @ L.message_view(orth, h1).mT
        assert float((chi * p / p.diagonal().sum() - one).norm()) < bound
