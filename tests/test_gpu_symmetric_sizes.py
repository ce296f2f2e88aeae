"""The symmetric gauge of graphs of up to two nodes per SM and above
(tensor_ops.py:189-199)."""

import numpy as np
import pytest
import torch

from dequantizer_b200 import _lib
from tests.test_gpu_gauge_kernels import layout_of, rr3

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [296, 298])
@pytest.mark.parametrize("dims,phys", [((1, 2), 1), ((2, 5, 16), 2)])
def test_symmetric_gauge(n, dims, phys):
    """Products of three square roots and a norm of at most 2 x 16^3 terms: 1e-13 of the unit norm."""
    L = layout_of(rr3(n, dims, phys))
    rng = np.random.default_rng(n)
    T = torch.from_numpy(rng.standard_normal(L.tensor_elems) + 1j * rng.standard_normal(L.tensor_elems)).cuda()
    lam = torch.from_numpy(10.0 ** -rng.uniform(0, 3, L.lam_elems)).cuda()
    out = torch.empty_like(T)
    _lib.call("dqz_symmetric_gauge", L.gptr, T.data_ptr(), lam.data_ptr(), 1e-10, out.data_ptr(), _lib.stream_handle())
    for v, (t, got) in enumerate(zip(L.unpack_tensors(T), L.unpack_tensors(out))):
        h0 = int(L.node_half[v])
        for f in range(3):
            shape = [1] * 4
            shape[f] = -1
            t = t * L.lambda_view(lam, int(L.half_edge[h0 + f])).sqrt().reshape(shape)
        assert float((got - t / t.norm()).norm()) < 1e-13
