"""dqz_bp_sweep_levels from bond 8 on equals one dqz_bp_node_update launch per level
and dqz_bp_edge_pass bit for bit (tensor_ops.py:36-76)."""

import pytest
import torch

from dequantizer_b200 import _lib
from dequantizer_b200 import graph as G
from dequantizer_b200 import maps as M
from dequantizer_b200.engine import BPEngine

pytestmark = pytest.mark.gpu


# blocks of several slices and of one, small nodes that one CTA could take whole, degree 4 and bonds above 32 (generic)
@pytest.mark.parametrize("make,dims", [
    (lambda: G.get_random_regular_graph(24, 3, 2, 1, 3), (8, 16, 11)), (lambda: G.get_heavy_hex_ibm_eagle_lattice_infinite(), (8,)),
    (lambda: G.get_random_regular_graph(6, 3, 2, 1, 3), (32, 31)), (lambda: G.get_nd_lattice([4, 4], 2, 1), (8, 3, 9)),
    (lambda: G.get_nd_lattice([12], 2, 1), (40, 33, 8))])
def test_one_launch_equals_level_launches(make, dims):
    g = make()
    for i, e in enumerate(g.edges.values()):
        e.dimension = dims[i % len(dims)]
    g.refresh_bond_shapes()
    eng = BPEngine(g, schedule="async")
    L, topo = eng.layout, eng.topo
    gen = torch.Generator(device="cuda").manual_seed(7)
    for arena in (eng.T, eng.n2e, eng.e2n):
        arena.copy_(torch.randn(arena.numel(), dtype=torch.complex128, device="cuda", generator=gen))
    src_sel, edge_new, levels = topo.device_tables(L.device)
    flat, off, widest, sync = topo.device_level_tables(L.device)
    stream = _lib.stream_handle()
    n2e, e2n = torch.zeros_like(eng.n2e), torch.zeros_like(eng.e2n)
    _lib.call("dqz_bp_sweep_levels", L.gptr, eng.T.data_ptr(), eng.n2e.data_ptr(), eng.e2n.data_ptr(), n2e.data_ptr(),
              e2n.data_ptr(), src_sel.data_ptr(), edge_new.data_ptr(), flat.data_ptr(), off.data_ptr(),
              len(topo.levels), widest, L.max_slice(), L.max_chi(), sync.data_ptr(),
              M.error_flag(L.device).data_ptr(), stream)
    ref_n, ref_e = torch.zeros_like(eng.n2e), torch.zeros_like(eng.e2n)
    for halves in levels:
        _lib.call("dqz_bp_node_update", L.gptr, eng.T.data_ptr(), eng.n2e.data_ptr(), eng.e2n.data_ptr(),
                  ref_n.data_ptr(), src_sel.data_ptr(), halves.data_ptr(), halves.numel(), L.max_slice(), L.max_chi(),
                  None, stream)
    _lib.call("dqz_bp_edge_pass", L.gptr, eng.n2e.data_ptr(), ref_n.data_ptr(), edge_new.data_ptr(), ref_e.data_ptr(),
              L.max_chi(), stream)
    assert len(topo.levels) > 2
    assert torch.equal(n2e, ref_n) and torch.equal(e2n, ref_e)
    assert int(M.error_flag(L.device).item()) == 0
