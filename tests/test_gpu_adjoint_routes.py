"""The implicit adjoint of the BP fixed point by the degree-3 tensor-core form and by
the generic one (the derivatives of tensor_ops.py:36-76), on both sides of the rule
between them."""

import pytest
import torch

from dequantizer_b200 import graph as G
from dequantizer_b200.adjoint import FixedPointProblem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chi,phys,tensor_core", [(2, 8, False), (3, 6, False), (3, 4, True), (4, 8, True)])
def test_both_forms_agree(chi, phys, tensor_core):
    """Ten transposed sweeps of up to 3 x 8 x 4^3 products an entry and the tensor
    cotangent: 1e-11 of the largest entry (rounding 1e-13 a sweep at most)."""
    g = G.get_random_regular_graph(12, 3, phys, chi, 5)
    P = FixedPointProblem(g)
    assert bool(P._k3_vjp) == tensor_core
    L = P.layout
    gen = torch.Generator(device="cuda").manual_seed(3)
    T = torch.randn(L.tensor_elems, dtype=torch.complex128, device="cuda", generator=gen)
    a = torch.randn(L.n_halves, chi, chi, dtype=torch.complex128, device="cuda", generator=gen)
    m = a @ a.mH
    n2e, e2n, _ = P.converge(T, (m / m.diagonal(dim1=1, dim2=2).sum(1)[:, None, None]).reshape(-1).contiguous(), 1e-13, 60)
    cot = torch.randn(n2e.numel(), dtype=torch.complex128, device="cuda", generator=gen)
    out = []
    for form in (L.k3_shape(), None):
        P._k3_vjp = form
        t_cot = torch.zeros_like(T)
        out.append((P.solve_adjoint(T, e2n, cot, 0.0, 10, t_cot), t_cot))
    for got, want in zip(*out):
        assert float((got - want).abs().max()) < 1e-11 * float(want.abs().max())
