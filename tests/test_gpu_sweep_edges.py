"""Sweeps at the ends of their tables (tensor_ops.py:36-76): more levels than the
sliced sweep looks up ahead, and the measured change of non-finite messages."""

import math

import pytest
import torch

from dequantizer_b200 import _lib
from dequantizer_b200 import graph as G
from dequantizer_b200 import maps as M
from dequantizer_b200.engine import BPEngine

pytestmark = pytest.mark.gpu


def random_engine(g, schedule):
    eng = BPEngine(g, schedule=schedule)
    gen = torch.Generator(device="cuda").manual_seed(7)
    for arena in (eng.T, eng.n2e, eng.e2n):
        arena.copy_(torch.randn(arena.numel(), dtype=torch.complex128, device="cuda", generator=gen))
    return eng


# degree 3 (by slices) and degree 4 (generic), the table ending in the middle of the schedule
@pytest.mark.parametrize("degree,chi", [(3, 9), (4, 8)])
def test_more_levels_than_the_table(degree, chi):
    """Bit for bit the launches level by level."""
    eng = random_engine(G.get_random_regular_graph(200, degree, 2, chi, 1), "async")
    L, topo = eng.layout, eng.topo
    assert len(topo.levels) > 128
    src_sel, edge_new, levels = topo.device_tables(L.device)
    n2e, e2n, T = eng.n2e.clone(), eng.e2n.clone(), eng.T
    eng.sweep()
    ref_n, ref_e = torch.zeros_like(n2e), torch.zeros_like(e2n)
    for halves in levels:
        _lib.call("dqz_bp_node_update", L.gptr, T.data_ptr(), n2e.data_ptr(), e2n.data_ptr(), ref_n.data_ptr(),
                  src_sel.data_ptr(), halves.data_ptr(), halves.numel(), L.max_slice(), L.max_chi(), None,
                  _lib.stream_handle())
    _lib.call("dqz_bp_edge_pass", L.gptr, n2e.data_ptr(), ref_n.data_ptr(), edge_new.data_ptr(), ref_e.data_ptr(),
              L.max_chi(), _lib.stream_handle())
    assert torch.equal(eng.n2e, ref_n) and torch.equal(eng.e2n, ref_e)
    assert int(M.error_flag(L.device).item()) == 0


@pytest.mark.parametrize("chi,n", [(16, 60), (16, 400), (5, 60)])
def test_change_of_non_finite_messages(chi, n):
    """max_change is the largest |new - old| entry, and NaN when one is NaN."""
    eng = random_engine(G.get_random_regular_graph(n, 3, 2, chi, 1), "flooding")
    L = eng.layout
    src_sel, edge_new, _ = eng.topo.device_tables(L.device)
    nodes = torch.arange(L.n_nodes, dtype=torch.int32, device="cuda")
    for bad in (False, True):
        if bad:
            eng.T[int(L.node_off[n // 2]) + 3] = complex("nan")
        n2e, e2n = torch.empty_like(eng.n2e), torch.empty_like(eng.e2n)
        change = torch.zeros(1, dtype=torch.float64, device="cuda")
        _lib.call("dqz_bp_sweep_k3", L.gptr, *L.k3_shape(), eng.T.data_ptr(), eng.n2e.data_ptr(), eng.e2n.data_ptr(),
                  n2e.data_ptr(), e2n.data_ptr(), src_sel.data_ptr(), edge_new.data_ptr(), nodes.data_ptr(), n, 0,
                  change.data_ptr(), M.error_flag(L.device).data_ptr(), _lib.stream_handle())
        if bad:
            assert math.isnan(float(change))
        else:
            want = float((n2e - eng.n2e).abs().max())
            assert abs(float(change) - want) <= 4 * 2.2e-16 * want
