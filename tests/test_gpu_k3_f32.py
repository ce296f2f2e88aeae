"""The FP32 sweep of degree-3 nodes (dqz_bp_sweep_k3_c64 and the half-edge form of
dqz_bp_node_update_k3) against the FP64 sweep on the same values
(tensor_ops.py:36-76).

Tolerance: as in test_gpu_k3.py with eps = 6e-8: sqrt(8192) eps = 5.4e-6 of |M|,
2.7e-5 allowed, and |dm| <= that times |m| (1 + |m|) after the division by the
trace.
"""

import pytest
import torch

from dequantizer_b200 import _lib
from dequantizer_b200 import graph as G
from dequantizer_b200.engine import BPEngine

pytestmark = pytest.mark.gpu


# 4 nodes: one item per output; 110, 302: whole nodes, below and above one wave of SMs; 1000 at bond 8 above a wave
@pytest.mark.parametrize("chi,n,schedule", [(16, 4, "sync"), (16, 110, "flooding"), (16, 302, "sync"), (16, 30, "async"),
                                            (8, 4, "flooding"), (8, 600, "sync"), (8, 1000, "flooding"), (8, 60, "async")])
def test_fp32_sweep_matches_fp64(chi, n, schedule):
    g = G.get_random_regular_graph(n, 3, 2, chi, 3)
    eng, ref = BPEngine(g, schedule=schedule, precision="fp32"), BPEngine(g, schedule=schedule)
    gen = torch.Generator(device="cuda").manual_seed(7)
    for a, b in ((eng.T, ref.T), (eng.n2e, ref.n2e), (eng.e2n, ref.e2n)):
        a.copy_(torch.randn(a.numel(), dtype=torch.complex64, device="cuda", generator=gen))
        b.copy_(a)
    n2e, e2n = eng.n2e.clone(), eng.e2n.clone()
    eng.sweep()
    ref.sweep()
    eng.check()
    levels = 1 if schedule != "async" else len(eng.topo.levels)
    for got, want in ((eng.n2e, ref.n2e), (eng.e2n, ref.e2n)):
        m = want.view(-1, chi * chi).norm(dim=1)
        d = (got - want).view(-1, chi * chi).norm(dim=1) / (m * (1 + m))
        # later levels of a schedule read messages that carry such errors themselves: the first level's only
        sel = torch.as_tensor(eng.topo.levels[0], device="cuda").long() if levels > 1 else slice(None)
        if levels == 1 or got is eng.n2e:
            assert float(d[sel].max()) < 2.7e-5
    # the half-edge form: the same bits
    L, topo = eng.layout, eng.topo
    src_sel, _, lv = topo.device_tables(L.device)
    out = torch.zeros_like(n2e)
    flag = torch.zeros(1, dtype=torch.int32, device=L.device)
    for halves in lv:
        _lib.call("dqz_bp_node_update_k3", L.gptr, chi, 32, eng.T.data_ptr(), n2e.data_ptr(), e2n.data_ptr(),
                  out.data_ptr(), src_sel.data_ptr(), halves.data_ptr(), halves.numel(), flag.data_ptr(),
                  _lib.stream_handle())
    assert torch.equal(out, eng.n2e) and int(flag) == 0
