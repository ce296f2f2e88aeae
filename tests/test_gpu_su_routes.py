"""Which form takes a simple-update job above the register form's limits
(tensor_ops.py:265-389): the cluster forms, whatever the physical dimension and
the gate rank; no job of 256 rows or more is left to the one-CTA kernel."""

import numpy as np
import pytest
import torch

from dequantizer_b200 import _lib, autotune
from dequantizer_b200 import graph as G
from dequantizer_b200.gates import decompose_gates
from dequantizer_b200.layout import GraphLayout
from tests.helpers import rel_err, two_site
from tests.test_gpu_su_reg import gate_of_rank

pytestmark = pytest.mark.gpu


# each just outside one limit: S of 90 rows; S of 128; 289 rows of other bonds; B of 34 columns (a product gate)
@pytest.mark.parametrize("d,bond,others,rank", [(3, 10, 10, 2), (4, 8, 8, 2), (1, 16, 17, 1), (2, 17, 12, 1)])
@pytest.mark.parametrize("n_nodes", [40, 420])
def test_jobs_above_the_register_form(n_nodes, d, bond, others, rank):
    """Marks (the first bytes of the scratch) of every job, and the values of the
    one-CTA kernel: lambdas, errors, entropies 1e-12, two-site tensors 1e-10."""
    g = G.get_random_regular_graph(n_nodes, 3, d, 1, 7)
    edges = list(g.edges.values())
    taken, jobs = set(), []
    for i, e in enumerate(edges):
        if not {n.id for n in e.neighbors} & taken:
            taken |= {n.id for n in e.neighbors}
            jobs.append(i)
    chis = np.full(len(edges), others)
    chis[jobs] = bond
    for e, c in zip(edges, chis):
        e.dimension = int(c)
    g.refresh_bond_shapes()
    L = GraphLayout(list(g.nodes.values()), edges, [int(c) for c in chis])
    rng = np.random.default_rng(d + bond)
    n = len(jobs)
    assert (n <= 148) == (n_nodes == 40)
    z = rng.standard_normal((L.tensor_elems, 2))
    T0 = torch.from_numpy(z[:, 0] + 1j * z[:, 1]).cuda()
    lam0 = torch.from_numpy(np.concatenate([np.sort(10 ** rng.uniform(-3, 0, int(c)))[::-1] for c in chis])).cuda()
    flat, ranks, _ = decompose_gates(gate_of_rank(rank, d, rng)[None], 1e-10)
    assert int(ranks[0]) == rank
    rows, cols = d * others * others, bond * rank
    assert rows >= 256
    ed = torch.tensor(jobs, dtype=torch.int32, device="cuda")
    first = torch.ones(n, dtype=torch.uint8, device="cuda")
    halves = torch.from_numpy(np.repeat(flat.reshape(1, -1), n, 0)).cuda()
    rk = torch.full((n,), rank, dtype=torch.int32, device="cuda")
    out = {}
    try:
        for knob in (1, 0):
            autotune.set_knobs({"su_onchip": knob})
            L.edge_chi[:] = chis
            L.push_edge_chi()
            T, lam = T0.clone(), lam0.clone()
            err, ent = (torch.empty(n, dtype=torch.float64, device="cuda") for _ in range(2))
            nb = _lib.lib().dqz_simple_update_workspace_bytes(n, rows, cols)
            scratch = torch.full((nb,), 0xA5, dtype=torch.uint8, device="cuda")
            _lib.call("dqz_simple_update_ws", L.gptr, T.data_ptr(), lam.data_ptr(), ed.data_ptr(), first.data_ptr(),
                      halves.data_ptr(), rk.data_ptr(), n, 1e-10, bond, rows, cols, err.data_ptr(), ent.data_ptr(),
                      scratch.data_ptr(), nb, _lib.stream_handle())
            torch.cuda.synchronize()
            if knob == 0:
                assert bool((scratch[:n] == 1).all())
            ts, sites = L.unpack_tensors(T), []
            for e in jobs[:5]:
                ha, hb = int(L.edge_half[2 * e]), int(L.edge_half[2 * e + 1])
                a, b = int(L.half_node[ha]), int(L.half_node[hb])
                sites.append(two_site(ts[a], ts[b], ha - int(L.node_half[a]), hb - int(L.node_half[b]),
                                      L.lambda_view(lam, e)))
            out[knob] = (torch.cat([L.lambda_view(lam, e) for e in jobs]), err, ent, sites)
    finally:
        autotune.set_knobs({"su_onchip": 0})
    for got, want in zip(out[0][:3], out[1][:3]):
        assert float((got - want).abs().max()) < 1e-12
    for got, want in zip(out[0][3], out[1][3]):
        assert rel_err(got, want) < 1e-10


# both sides of the rule between the register form and the one-CTA kernel, and more jobs than one workspace chunk
@pytest.mark.parametrize("bond,rank,n_nodes,register", [
    (3, 2, 30, False), (4, 2, 120, True), (4, 2, 160, False), (7, 2, 300, True), (7, 2, 480, False), (8, 2, 500, True),
    (9, 2, 480, False), (8, 1, 120, True), (8, 1, 160, False), (11, 2, 1500, True)])
def test_rule_of_the_register_form(bond, rank, n_nodes, register):
    """The marks show whether the register form ran (untouched bytes: it did not);
    values as above against the one-CTA kernel."""
    g = G.get_random_regular_graph(n_nodes, 3, 2, bond, 7)
    edges = list(g.edges.values())
    taken, jobs = set(), []
    for i, e in enumerate(edges):
        if not {n.id for n in e.neighbors} & taken:
            taken |= {n.id for n in e.neighbors}
            jobs.append(i)
    n = len(jobs)
    assert bond != 11 or n > 592
    L = GraphLayout(list(g.nodes.values()), edges, [bond] * len(edges))
    rng = np.random.default_rng(bond + n)
    z = rng.standard_normal((L.tensor_elems, 2))
    T0 = torch.from_numpy(z[:, 0] + 1j * z[:, 1]).cuda()
    lam0 = torch.from_numpy(np.sort(10 ** rng.uniform(-3, 0, (len(edges), bond)))[:, ::-1].ravel().copy()).cuda()
    flat, ranks, _ = decompose_gates(gate_of_rank(rank, 2, rng)[None], 1e-10)
    assert int(ranks[0]) == rank
    rows, cols = 2 * bond * bond, bond * rank
    ed = torch.tensor(jobs, dtype=torch.int32, device="cuda")
    first = torch.ones(n, dtype=torch.uint8, device="cuda")
    halves = torch.from_numpy(np.repeat(flat.reshape(1, -1), n, 0)).cuda()
    rk = torch.full((n,), rank, dtype=torch.int32, device="cuda")
    out = {}
    try:
        for knob in (1, 0):
            autotune.set_knobs({"su_onchip": knob})
            T, lam = T0.clone(), lam0.clone()
            err, ent = (torch.empty(n, dtype=torch.float64, device="cuda") for _ in range(2))
            nb = _lib.lib().dqz_simple_update_workspace_bytes(n, rows, cols)
            scratch = torch.full((nb,), 0xA5, dtype=torch.uint8, device="cuda")
            _lib.call("dqz_simple_update_ws", L.gptr, T.data_ptr(), lam.data_ptr(), ed.data_ptr(), first.data_ptr(),
                      halves.data_ptr(), rk.data_ptr(), n, 1e-10, bond, rows, cols, err.data_ptr(), ent.data_ptr(),
                      scratch.data_ptr(), nb, _lib.stream_handle())
            torch.cuda.synchronize()
            if knob == 0:
                assert bool((scratch[:n] == (1 if register else 0xA5)).all())
            ts, sites = L.unpack_tensors(T), []
            for e in jobs[:3] + jobs[-2:]:
                ha, hb = int(L.edge_half[2 * e]), int(L.edge_half[2 * e + 1])
                a, b = int(L.half_node[ha]), int(L.half_node[hb])
                sites.append(two_site(ts[a], ts[b], ha - int(L.node_half[a]), hb - int(L.node_half[b]),
                                      L.lambda_view(lam, e)))
            out[knob] = (lam, err, ent, sites)
    finally:
        autotune.set_knobs({"su_onchip": 0})
    for got, want in zip(out[0][:3], out[1][:3]):
        assert float((got - want).abs().max()) < 1e-12
    for got, want in zip(out[0][3], out[1][3]):
        assert rel_err(got, want) < 1e-10
