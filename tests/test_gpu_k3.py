"""The FP64 tensor-core node update of degree-3 nodes (dqz_bp_sweep_k3 and the
half-edge form of dqz_bp_node_update_k3) against the generic node update and
the edge pass (tensor_ops.py:36-76).

Tolerance: an entry of M is a chain of three contractions, at most 2 * 16^3
terms in all, so two orders of summation differ by about sqrt(8192) eps = 2e-14
of |M|; 1e-13 is allowed. The message is m = M / tr M, and tr M carries the same
absolute error: |dm| <= 1e-13 |M / tr M| (1 + |M / tr M|) = 1e-13 |m| (1 + |m|)
(the random messages here are not positive, so |m| is not near 1).
"""

import numpy as np
import pytest
import torch

from dequantizer_b200 import _lib
from dequantizer_b200 import graph as G
from dequantizer_b200.engine import BPEngine

pytestmark = pytest.mark.gpu
TOL = 1e-13


def engine(g, schedule="sync"):
    eng = BPEngine(g, schedule=schedule)
    gen = torch.Generator(device="cuda").manual_seed(7)
    L = eng.layout
    eng.T.copy_(torch.randn(L.tensor_elems, dtype=torch.complex128, device="cuda", generator=gen))
    for arena in (eng.n2e, eng.e2n):
        arena.copy_(torch.randn(L.msg_elems, dtype=torch.complex128, device="cuda", generator=gen))
    return eng


def generic_sweep(eng):
    """Level by level with the generic kernel, then the edge pass."""
    L, topo = eng.layout, eng.topo
    src_sel, edge_new, levels = topo.device_tables(L.device)
    n2e_new, e2n_new = torch.zeros_like(eng.n2e), torch.zeros_like(eng.e2n)
    stream = _lib.stream_handle()
    for halves in levels:
        _lib.call("dqz_bp_node_update", L.gptr, eng.T.data_ptr(), eng.n2e.data_ptr(), eng.e2n.data_ptr(),
                  n2e_new.data_ptr(), src_sel.data_ptr(), halves.data_ptr(), halves.numel(), L.max_slice(),
                  L.max_chi(), None, stream)
    _lib.call("dqz_bp_edge_pass", L.gptr, eng.n2e.data_ptr(), n2e_new.data_ptr(), edge_new.data_ptr(),
              e2n_new.data_ptr(), L.max_chi(), stream)
    return n2e_new, e2n_new


# 4 nodes: one item per output; 110 and 302: whole nodes, below and above one wave of SMs; 1000 at bond 8
# crosses its wave of five CTAs per SM
@pytest.mark.parametrize("chi,n,schedule", [(16, 4, "sync"), (16, 110, "flooding"), (16, 302, "sync"),
                                            (16, 30, "async"), (8, 4, "flooding"), (8, 600, "sync"),
                                            (8, 1000, "flooding"), (8, 60, "async")])
def test_sweep_matches_generic_and_half_edge_form(chi, n, schedule):
    eng = engine(G.get_random_regular_graph(n, 3, 2, chi, 3), schedule)
    ref_n, ref_e = generic_sweep(eng)
    L, topo = eng.layout, eng.topo
    src_sel, _, levels = topo.device_tables(L.device)
    n2e, e2n = eng.n2e, eng.e2n
    eng.sweep()
    eng.check()
    for got, ref in ((eng.n2e, ref_n), (eng.e2n, ref_e)):
        m = ref.view(-1, chi * chi).norm(dim=1)
        d = (got - ref).view(-1, chi * chi).norm(dim=1)
        assert float((d / (m * (1 + m))).max()) < TOL
    halves_new = torch.zeros_like(n2e)
    flag = torch.zeros(1, dtype=torch.int32, device=L.device)
    for halves in levels:
        _lib.call("dqz_bp_node_update_k3", L.gptr, chi, 64, eng.T.data_ptr(), n2e.data_ptr(), e2n.data_ptr(),
                  halves_new.data_ptr(), src_sel.data_ptr(), halves.data_ptr(), halves.numel(), flag.data_ptr(),
                  _lib.stream_handle())
    assert torch.equal(halves_new, eng.n2e) and int(flag) == 0


@pytest.mark.parametrize("chi", [8, 16])
@pytest.mark.parametrize("repeat", [1, 60])
def test_other_shapes_are_flagged_and_skipped(chi, repeat):
    """The heavy-hex cell: degree-2 nodes between the degree-3 ones, listed together (repeated past one wave)."""
    g = G.get_heavy_hex_ibm_eagle_lattice_infinite()
    for e in g.edges.values():
        e.dimension = chi
    g.refresh_bond_shapes()
    eng = engine(g)
    ref_n, _ = generic_sweep(eng)
    L = eng.layout
    src_sel, _, _ = eng.topo.device_tables(L.device)
    out = torch.full_like(eng.n2e, 7.0)
    flag = torch.zeros(1, dtype=torch.int32, device=L.device)
    nodes = torch.arange(L.n_nodes, dtype=torch.int32, device=L.device).repeat(repeat)
    _lib.call("dqz_bp_sweep_k3", L.gptr, chi, 1, eng.T.data_ptr(), eng.n2e.data_ptr(), eng.e2n.data_ptr(),
              out.data_ptr(), None, src_sel.data_ptr(), None, nodes.data_ptr(), nodes.numel(), 0, None,
              flag.data_ptr(), _lib.stream_handle())
    assert int(flag) == 1
    for v in range(L.n_nodes):
        for h in range(L.node_half[v], L.node_half[v] + L.degree[v]):
            got, ref = L.message_view(out, h), L.message_view(ref_n, h)
            if L.degree[v] == 3:
                assert float((got - ref).norm() / (ref.norm() * (1 + ref.norm()))) < TOL
            else:
                assert bool((got == 7.0).all())


def uneven_graph(n, dims, phys):
    """Random 3-regular graph whose bond dimensions cycle through ``dims``."""
    g = G.get_random_regular_graph(n, 3, phys, 1, 5)
    for i, e in enumerate(g.edges.values()):
        e.dimension = dims[i % len(dims)]
    g.refresh_bond_shapes()
    return g


def positive_messages(eng, gen):
    L = eng.layout
    arena = torch.zeros_like(eng.n2e)
    for h in range(L.n_halves):
        c = int(L.edge_chi[L.half_edge[h]])
        a = torch.randn((c, c), dtype=torch.complex128, device="cuda", generator=gen)
        m = a @ a.mH
        L.message_view(arena, h).copy_(m / m.diagonal().sum().real)
    return arena


SHAPES = [(10, (16,), 2), (302, (16,), 2), (10, (8,), 2), (1000, (8,), 2),  # uniform: compile-time strides
          (10, (5,), 2), (160, (12,), 2), (12, (1, 3, 8), 3), (12, (2, 9, 16, 7), 1), (160, (15, 1, 4), 3)]


@pytest.mark.parametrize("n,dims,phys", SHAPES)
def test_padded_sweep_raw_and_change(n, dims, phys):
    """Messages, unnormalised messages and the largest change, against the generic kernel."""
    g = uneven_graph(n, dims, phys)
    eng = engine(g, "flooding")
    gen = torch.Generator(device="cuda").manual_seed(11)
    eng.n2e = positive_messages(eng, gen)
    eng.e2n = positive_messages(eng, gen)
    ref_n, ref_e = generic_sweep(eng)
    L = eng.layout
    shape = L.k3_shape()
    assert shape == (max(dims), int(dims in ((8,), (16,)) and phys == 2))
    src_sel, edge_new, _ = eng.topo.device_tables(L.device)
    nodes = torch.arange(L.n_nodes, dtype=torch.int32, device=L.device)
    out_n, out_e, raw = (torch.zeros_like(eng.n2e) for _ in range(3))
    change = torch.zeros(1, dtype=torch.float64, device=L.device)
    flag = torch.zeros(1, dtype=torch.int32, device=L.device)
    for n_new, e_new, is_raw, ch in ((out_n, out_e, 0, change), (raw, None, 1, None)):
        _lib.call("dqz_bp_sweep_k3", L.gptr, *shape, eng.T.data_ptr(), eng.n2e.data_ptr(), eng.e2n.data_ptr(),
                  n_new.data_ptr(), _lib.ptr(e_new), src_sel.data_ptr(), edge_new.data_ptr(), nodes.data_ptr(),
                  L.n_nodes, is_raw, _lib.ptr(ch), flag.data_ptr(), _lib.stream_handle())
    assert int(flag) == 0
    assert float(change) == pytest.approx(float((out_n - eng.n2e).abs().max()), rel=1e-14)
    for h in range(L.n_halves):
        for got, ref in ((out_n, ref_n), (out_e, ref_e)):
            x, y = L.message_view(got, h), L.message_view(ref, h)
            assert float((x - y).norm()) < TOL * float(y.norm() * (1 + y.norm()))
        r = L.message_view(raw, h)
        assert float((r / r.diagonal().sum() - L.message_view(out_n, h)).norm()) < TOL


@pytest.mark.parametrize("n,dims,phys", SHAPES)
def test_transposed_sweep_matches_generic_adjoint(n, dims, phys):
    """dqz_bp_vjp_k3 against dqz_bp_node_vjp, both outputs and the fused iterate. A cotangent entry is a few
    chains of three contractions of at most 2 * 16^3 terms (error about 2e-14 of the norm each, positive
    messages: no cancellation in the trace): 1e-12 of the arena's norm."""
    g = uneven_graph(n, dims, phys)
    eng = engine(g, "flooding")
    gen = torch.Generator(device="cuda").manual_seed(13)
    e2n = positive_messages(eng, gen)
    L = eng.layout
    cot, add = (torch.randn(L.msg_elems, dtype=torch.complex128, device="cuda", generator=gen) for _ in range(2))
    nodes = torch.arange(L.n_nodes, dtype=torch.int32, device=L.device)
    stream = _lib.stream_handle()
    ref, ref_t = torch.zeros_like(cot), torch.ones_like(eng.T)
    scratch = torch.empty(_lib.lib().dqz_bp_node_vjp_scratch_bytes(L.n_nodes, L.max_size()), dtype=torch.uint8,
                          device=L.device)
    _lib.call("dqz_bp_node_vjp", L.gptr, eng.T.data_ptr(), e2n.data_ptr(), cot.data_ptr(), ref.data_ptr(),
              ref_t.data_ptr(), nodes.data_ptr(), L.n_nodes, L.max_size(), L.max_chi(), scratch.data_ptr(), stream)
    shape = L.k3_shape()
    flag = torch.zeros(1, dtype=torch.int32, device=L.device)
    own = torch.zeros(L.n_halves, dtype=torch.uint8, device=L.device)
    raw, got, nxt = (torch.zeros_like(cot) for _ in range(3))
    got_t = torch.ones_like(eng.T)
    change = torch.zeros(1, dtype=torch.float64, device=L.device)
    _lib.call("dqz_bp_sweep_k3", L.gptr, *shape, eng.T.data_ptr(), e2n.data_ptr(), e2n.data_ptr(), raw.data_ptr(),
              None, own.data_ptr(), None, nodes.data_ptr(), L.n_nodes, 1, None, flag.data_ptr(), stream)
    for out, ad, ch, tc in ((got, None, None, got_t), (nxt, add, change, None)):
        _lib.call("dqz_bp_vjp_k3", L.gptr, *shape, eng.T.data_ptr(), e2n.data_ptr(), cot.data_ptr(), raw.data_ptr(),
                  out.data_ptr(), _lib.ptr(ad), _lib.ptr(ch), _lib.ptr(tc), nodes.data_ptr(), L.n_nodes,
                  flag.data_ptr(), stream)
    assert int(flag) == 0
    assert float((got - ref).norm() / ref.norm()) < 1e-12
    assert float((got_t - ref_t).norm() / ref_t.norm()) < 1e-12
    want = add.clone()
    for h in range(L.n_halves):
        L.message_view(want, int(L.half_twin[h])).add_(L.message_view(got, h))
    assert float((nxt - want).norm() / want.norm()) < 1e-14
    assert float(change) == pytest.approx(float((nxt - cot).abs().max()), rel=1e-14)
