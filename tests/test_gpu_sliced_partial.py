"""dqz_bp_sweep_sliced on part of a schedule (tensor_ops.py:36-76): half-edges that
no level lists keep their messages, and their readers see them as they are."""

import numpy as np
import pytest
import torch

from dequantizer_b200 import _lib
from dequantizer_b200 import graph as G
from dequantizer_b200 import maps as M
from dequantizer_b200.layout import GraphLayout

pytestmark = pytest.mark.gpu

CASES = {
    "regular": (lambda: G.get_random_regular_graph(20, 3, 2, 2, 11), [8, 16, 9]),
    "degree4": (lambda: G.get_nd_lattice([4, 4], 2, 2), [8, 3, 9]),
}


@pytest.mark.parametrize("per_item", [1, 3])
@pytest.mark.parametrize("case", list(CASES))
def test_unlisted_messages_are_left_alone(case, per_item):
    """Bit for bit dqz_bp_node_update on the same lists, n2e_new filled with
    messages of trace 3 before, then dqz_bp_edge_pass."""
    make, dims = CASES[case]
    g = make()
    for i, e in enumerate(g.edges.values()):
        e.dimension = dims[i % len(dims)]
    g.refresh_bond_shapes()
    topo = M.Topology(list(g.get_traversal_iterator(ordering="dfs")), False)
    L = GraphLayout(topo.nodes, topo.edges, [e.dimension for e in topo.edges])
    rng = np.random.default_rng(9)

    def messages(trace):
        out = np.zeros(L.msg_elems, dtype=complex)
        for h, c in enumerate(L.half_chi()):
            a = rng.standard_normal((c, c)) + 1j * rng.standard_normal((c, c))
            m = a @ a.conj().T
            out[L.half_msg_off[h]: L.half_msg_off[h] + c * c] = (trace * m / np.trace(m).real).ravel()
        return torch.from_numpy(out).cuda()

    z = rng.standard_normal((L.tensor_elems, 2))
    T = torch.from_numpy(z[:, 0] + 1j * z[:, 1]).cuda()
    n2e, e2n, filled = messages(1.0), messages(1.0), messages(3.0)
    src_sel, edge_new, _ = topo.device_tables(T.device)
    levels = [lv[rng.random(len(lv)) < 0.6] for lv in topo.levels]
    levels = [lv for lv in levels if len(lv)]
    listed = np.concatenate(levels)
    twin_listed = np.isin(L.half_twin, listed)
    new = topo.src_sel == _lib.SRC_N2E_NEW
    assert (new & twin_listed).any() and (new & ~twin_listed).any() and len(listed) < L.n_halves

    ih, isl, ioff = [], [], [0]
    for lv in levels:
        for h in lv:
            c = int(L.half_chi()[h])
            for a in range(0, c, per_item):
                ih.append(h)
                isl.append(a + (min(per_item, c - a) << 16 if per_item > 1 else 0))
        ioff.append(len(ih))
    i32 = [torch.tensor(np.asarray(x, dtype=np.int32)).cuda()
           for x in (listed, np.cumsum([0] + [len(lv) for lv in levels]), ih, isl, ioff)]
    got, got_e = filled.clone(), torch.zeros_like(e2n)
    sync = torch.zeros(2, dtype=torch.int32, device="cuda")
    _lib.call("dqz_bp_sweep_sliced", L.gptr, T.data_ptr(), n2e.data_ptr(), e2n.data_ptr(), got.data_ptr(),
              got_e.data_ptr(), src_sel.data_ptr(), edge_new.data_ptr(), *(x.data_ptr() for x in i32), len(levels),
              int(np.diff(ioff).max()), L.max_slice(), L.max_chi(), sync.data_ptr(),
              M.error_flag(T.device).data_ptr(), _lib.stream_handle())
    want, want_e = filled.clone(), torch.zeros_like(e2n)
    for lv in levels:
        halves = torch.from_numpy(lv).cuda()
        _lib.call("dqz_bp_node_update", L.gptr, T.data_ptr(), n2e.data_ptr(), e2n.data_ptr(), want.data_ptr(),
                  src_sel.data_ptr(), halves.data_ptr(), halves.numel(), L.max_slice(), L.max_chi(), None,
                  _lib.stream_handle())
    _lib.call("dqz_bp_edge_pass", L.gptr, n2e.data_ptr(), want.data_ptr(), edge_new.data_ptr(), want_e.data_ptr(),
              L.max_chi(), _lib.stream_handle())
    assert torch.equal(got, want) and torch.equal(got_e, want_e)
    assert int(M.error_flag(T.device).item()) == 0
