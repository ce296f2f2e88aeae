"""The forms of the simple update chained in one dqz_simple_update call
(tensor_ops.py:265-389): a node-disjoint batch whose jobs the register form,
the shared-memory cluster form and the global-workspace cluster form divide
among themselves, against the one-CTA kernel. Every launch of such a call reads
which jobs the launches before it did."""

import numpy as np
import pytest
import torch

from dequantizer_b200 import _lib, autotune
from dequantizer_b200 import graph as G
from dequantizer_b200.gates import decompose_gates
from dequantizer_b200.layout import GraphLayout
from tests.helpers import rel_err, two_site

pytestmark = pytest.mark.gpu
CAP = 8  # kept rank of every job: no bond grows above its storage
SMEM_ENTRIES = 220 * 1024 // 16


def form_of(bond, others, d=2, r=2):
    """Which form takes a side of a job (su_reg.cu's and gates.cu's limits)."""
    mb, kb, ks = int(np.prod(others)), bond * d, bond * r
    mub = min(mb, kb)
    ms = mub * d
    if mb <= 256 and kb <= 32 and ks <= 32 and ms <= 64:
        return 0
    need = ms * ks + mb * kb + max(2 * ks * ks, mub * max(mub, d * CAP)) + max(ms * CAP, ks * ks) + min(ms, ks) + mub
    return 1 if need + 8 <= SMEM_ENTRIES else 2


# up to one job per SM (shared-memory form, then the workspace form), and more (workspace form only)
@pytest.mark.parametrize("n_nodes", [96, 420])
def test_mixed_batch_matches_the_one_cta_kernel(n_nodes):
    """Lambdas, errors and entropies agree to 1e-12 and the two-site tensors
    around the updated bonds to 1e-10 relative, as for the uniform batches: SVDs
    of matrices of norm 1 in FP64, divided by lambdas down to 1e-3."""
    g = G.get_random_regular_graph(n_nodes, 3, 2, 1, 7)
    edges = list(g.edges.values())
    taken, jobs = set(), []
    for i, e in enumerate(edges):
        if not {n.id for n in e.neighbors} & taken:
            taken |= {n.id for n in e.neighbors}
            jobs.append(i)
    rng = np.random.default_rng(n_nodes)
    chis = rng.choice([16, 32], size=len(edges), p=[0.7, 0.3])
    chis[jobs] = np.array([16, 8, 32])[np.arange(len(jobs)) % 3]
    for e, c in zip(edges, chis):
        e.dimension = int(c)
    g.refresh_bond_shapes()
    L = GraphLayout(list(g.nodes.values()), edges, [int(c) for c in chis])
    forms = []
    for e in jobs:
        sides = []
        for i in (0, 1):
            h = int(L.edge_half[2 * e + i])
            v = int(L.half_node[h])
            dims = L.node_dims(v)
            slot = h - int(L.node_half[v])
            sides.append(form_of(dims[slot], dims[:slot] + dims[slot + 1:]))
        forms.append(max(sides))
    assert all(forms.count(f) > 2 for f in (0, 1, 2))
    n = len(jobs)
    assert (n <= 148) == (n_nodes == 96)

    z = rng.standard_normal((L.tensor_elems, 2))
    T0 = torch.from_numpy(z[:, 0] + 1j * z[:, 1]).cuda()
    lam0 = torch.from_numpy(np.concatenate([np.sort(10 ** rng.uniform(-3, 0, int(c)))[::-1] for c in chis])).cuda()
    gates = np.zeros((n, 4, 4), complex)
    gates[:, range(4), range(4)] = np.exp(1j * rng.uniform(-3, 3, (n, 4)))
    flat, ranks, _ = decompose_gates(gates.reshape(n, 2, 2, 2, 2), 1e-10)
    assert (ranks == 2).all()
    rows, cols = 2 * 32 * 32, 64
    ed = torch.tensor(jobs, dtype=torch.int32, device="cuda")
    first = torch.from_numpy((np.arange(n) % 2).astype(np.uint8)).cuda()
    halves, rk = torch.from_numpy(flat.reshape(n, -1)).cuda(), torch.from_numpy(ranks).cuda()
    out = {}
    try:
        for knob in (1, 0):
            autotune.set_knobs({"su_onchip": knob})
            L.edge_chi[:] = chis
            L.push_edge_chi()
            T, lam = T0.clone(), lam0.clone()
            err, ent = (torch.empty(n, dtype=torch.float64, device="cuda") for _ in range(2))
            nb = _lib.lib().dqz_simple_update_workspace_bytes(n, rows, cols)
            scratch = torch.full((nb,), 0xA5, dtype=torch.uint8, device="cuda")  # no mark of an earlier call
            _lib.call("dqz_simple_update_ws", L.gptr, T.data_ptr(), lam.data_ptr(), ed.data_ptr(), first.data_ptr(),
                      halves.data_ptr(), rk.data_ptr(), n, 1e-10, CAP, rows, cols, err.data_ptr(), ent.data_ptr(),
                      scratch.data_ptr(), nb, _lib.stream_handle())
            torch.cuda.synchronize()
            L.edge_chi[jobs] = CAP
            sites = []
            ts = L.unpack_tensors(T)
            for e in jobs:
                ha, hb = int(L.edge_half[2 * e]), int(L.edge_half[2 * e + 1])
                a, b = int(L.half_node[ha]), int(L.half_node[hb])
                sites.append(two_site(ts[a], ts[b], ha - int(L.node_half[a]), hb - int(L.node_half[b]),
                                      L.lambda_view(lam, e)) if len(sites) < 9 else None)
            out[knob] = (torch.cat([L.lambda_view(lam, e) for e in jobs]), err, ent, sites)
    finally:
        autotune.set_knobs({"su_onchip": 0})
    for got, want in zip(out[0][:3], out[1][:3]):
        assert float((got - want).abs().max()) < 1e-12
    for got, want in zip(out[0][3], out[1][3]):
        assert got is None or rel_err(got, want) < 1e-10
