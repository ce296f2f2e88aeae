"""One-site densities of degree-3 nodes by the tensor-core form and by the generic one
(density_matrix.py:16-37), over shapes on both sides of the rule between them."""

import numpy as np
import pytest
import torch

from dequantizer_b200 import _lib
from dequantizer_b200 import maps as M
from tests.test_gpu_gauge_kernels import layout_of, messages, rr3

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,dims,phys,tensor_core", [
    (60, (5, 2, 1), 2, True), (60, (9,), 2, False), (60, (11, 12), 2, False), (60, (12,), 2, True), (60, (16, 3, 2), 2, False),
    (60, (4,), 3, False), (60, (6,), 3, True), (36, (12,), 4, False), (40, (12,), 4, True), (40, (8,), 8, True),
    (36, (16,), 8, False)])
def test_both_forms_agree(n, dims, phys, tensor_core):
    """At most 8 * 16^3 terms in a chain of three products, a trace of positive terms: 1e-13 each."""
    L = layout_of(rr3(n, dims, phys))
    assert L.k3_density(n) == tensor_core
    rng = np.random.default_rng(6)
    T = torch.from_numpy(rng.standard_normal(L.tensor_elems) + 1j * rng.standard_normal(L.tensor_elems)).cuda()
    e2n = messages(L, rng, 2, False)
    idx = torch.arange(n, dtype=torch.int32, device="cuda")
    out = []
    for k3 in (True, False):
        rho = torch.zeros((n, 64), dtype=torch.complex128, device="cuda")
        if k3:
            _lib.call("dqz_density_k3", L.gptr, *L.k3_shape(), T.data_ptr(), e2n.data_ptr(), idx.data_ptr(), n,
                      rho.data_ptr(), M.error_flag(L.device).data_ptr(), _lib.stream_handle())
        else:
            nb = _lib.lib().dqz_density_scratch_bytes(n, L.max_size())
            scratch = torch.empty(max(nb, 1), dtype=torch.uint8, device="cuda")
            _lib.call("dqz_density_matrices", L.gptr, T.data_ptr(), e2n.data_ptr(), idx.data_ptr(), n, rho.data_ptr(),
                      L.max_size(), scratch.data_ptr(), _lib.stream_handle())
        out.append(rho[:, : phys * phys].reshape(n, phys, phys))
    assert float((out[0] - out[1]).abs().max()) < 2e-13
    got = M.density_packed(L, T, e2n, list(range(n)))
    assert torch.equal(got, out[0] if tensor_core else out[1])
    assert int(M.error_flag(L.device)) == 0
