"""The one-CTA asynchronous sweep (dqz_bp_sweep_planned) equals one
dqz_bp_node_update launch per level and dqz_bp_edge_pass bit for bit: every
entry is the same sum in the same order."""

import pytest
import torch

from dequantizer_b200 import _lib
from dequantizer_b200 import graph as G
from dequantizer_b200.engine import BPEngine

pytestmark = pytest.mark.gpu


# bonds 1 .. 7, physical 1 .. 3, degrees 1 .. 6; levels above the warps (several items a warp); tensors of more than 128
# entries a phase, and too large for all slices at once (bond 7)
@pytest.mark.parametrize("make,dims,phys", [
    (lambda p: G.get_nd_lattice([3, 3, 3], p, 1, False), (2,), 2), (lambda p: G.get_nd_lattice([3, 4, 2], p, 1, True), (2, 1, 3), 3),
    (lambda p: G.get_nd_lattice([9, 4], p, 1, True), (5, 4, 2), 1), (lambda p: G.get_random_regular_graph(60, 3, p, 1, 3), (6, 7, 4), 2),
    (lambda p: G.get_random_regular_graph(60, 3, p, 1, 3), (7,), 2), (lambda p: G.get_random_regular_graph(400, 3, p, 1, 3), (2, 3), 2),
    (lambda p: G.get_random_tree_tensor_graph(60, p, [1], 5), (2, 1), 2), (lambda p: G.get_random_regular_graph(9, 4, p, 1, 3), (3, 4), 2)])
def test_planned_sweep_equals_level_launches(make, dims, phys):
    g = make(phys)
    for i, e in enumerate(g.edges.values()):
        e.dimension = dims[i % len(dims)]
    g.refresh_bond_shapes()
    eng = BPEngine(g, schedule="async")
    L, topo = eng.layout, eng.topo
    gen = torch.Generator(device="cuda").manual_seed(7)
    for arena in (eng.T, eng.n2e, eng.e2n):
        arena.copy_(torch.randn(arena.numel(), dtype=torch.complex128, device="cuda", generator=gen))
    src_sel, edge_new, levels = topo.device_tables(L.device)
    _, off, widest, _ = topo.device_level_tables(L.device)
    stream = _lib.stream_handle()
    n2e, e2n = torch.zeros_like(eng.n2e), torch.zeros_like(eng.e2n)
    status = _lib.lib().dqz_bp_sweep_planned(
        L.gptr, eng.T.data_ptr(), eng.n2e.data_ptr(), eng.e2n.data_ptr(), n2e.data_ptr(), e2n.data_ptr(),
        edge_new.data_ptr(), topo.device_plan(L, L.device).data_ptr(), off.data_ptr(), len(topo.levels), widest,
        L.max_slice(), L.max_chi(), stream)
    assert status == _lib.DQZ_OK
    ref_n, ref_e = torch.zeros_like(eng.n2e), torch.zeros_like(eng.e2n)
    for halves in levels:
        _lib.call("dqz_bp_node_update", L.gptr, eng.T.data_ptr(), eng.n2e.data_ptr(), eng.e2n.data_ptr(),
                  ref_n.data_ptr(), src_sel.data_ptr(), halves.data_ptr(), halves.numel(), L.max_slice(), L.max_chi(),
                  None, stream)
    _lib.call("dqz_bp_edge_pass", L.gptr, eng.n2e.data_ptr(), ref_n.data_ptr(), edge_new.data_ptr(), ref_e.data_ptr(),
              L.max_chi(), stream)
    assert torch.equal(n2e, ref_n) and torch.equal(e2n, ref_e)
