"""BPEngine.launches_per_sweep against the kernels that one sweep launches."""

import pytest
import torch

from dequantizer_b200 import graph as G
from dequantizer_b200.engine import BPEngine

pytestmark = pytest.mark.gpu


def hex_graph(chi):
    g = G.get_heavy_hex_ibm_eagle_lattice_infinite()
    for e in g.edges.values():
        e.dimension = chi
    g.refresh_bond_shapes()
    return g


@pytest.mark.parametrize("make,schedule,precision,expected", [
    (lambda: G.get_nd_lattice([3, 4], 2, 4, True), "sync", "fp64", 2), (lambda: hex_graph(9), "sync", "fp64", 3),
    (lambda: hex_graph(9), "async", "fp64", 1), (lambda: hex_graph(4), "async", "fp64", 1),
    (lambda: G.get_random_regular_graph(20, 3, 2, 16, 1), "sync", "fp64", 1),
    (lambda: G.get_random_regular_graph(20, 3, 2, 16, 1), "flooding", "fp32", 1),
    (lambda: G.get_random_regular_graph(20, 3, 2, 16, 1), "sync", "bf16", 2),
    (lambda: G.get_nd_lattice([3, 3], 2, 16, True), "sync", "fp64", 2)])
def test_launches_per_sweep(make, schedule, precision, expected):
    """The last shape is above shared memory: the generic kernel in global scratch and the edge pass."""
    eng = BPEngine(make(), schedule=schedule, precision=precision)
    for arena in (eng.T, eng.n2e, eng.e2n):
        arena.copy_(torch.ones_like(arena))
    eng.sweep()
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        eng.sweep()
        torch.cuda.synchronize()
    names = [e.name for e in prof.events() if e.device_type == torch.autograd.DeviceType.CUDA
             and "(dqz_graph_t" in e.name]
    assert eng.launches_per_sweep() == expected
    if not names:
        pytest.skip("no kernel trace on this machine")
    assert len(names) == expected, names
