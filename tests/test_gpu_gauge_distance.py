"""The Vidal distance of the gauge that the factored edge kernel gives (bonds up
to 16) on ill-conditioned messages, against the one of the kernel with
eigendecompositions (tensor_ops.py:108-175)."""

import numpy as np
import pytest
import torch

from dequantizer_b200 import autotune
from dequantizer_b200 import graph as G
from dequantizer_b200.engine import BPEngine

pytestmark = pytest.mark.gpu
EPS = 1e-10


def loaded_engine(graph, seed):
    """Tensors whose bond indices fall over two decades, random positive messages, one sweep."""
    eng = BPEngine(graph)
    L, rng = eng.layout, np.random.default_rng(seed)
    tensors = []
    for v in range(L.n_nodes):
        shape = L.node_shape(v)
        t = rng.standard_normal(shape) + 1j * rng.standard_normal(shape)
        for f, c in enumerate(shape[:-1]):
            w = 10.0 ** (-2.0 * np.arange(c) / max(c - 1, 1))
            t = t * w.reshape([-1 if i == f else 1 for i in range(len(shape))])
        tensors.append(t)
    eng.load_tensors(tensors)
    sets = []
    for _ in range(2):
        mats = []
        for c in L.half_chi():
            a = rng.standard_normal((c, c)) + 1j * rng.standard_normal((c, c))
            m = a @ a.conj().T
            mats.append(m / np.trace(m).real)
        sets.append(mats)
    eng.load_messages(*sets)
    eng.sweep()
    return eng


@pytest.mark.parametrize("make", [
    lambda: G.get_nd_lattice([6, 6, 6], 2, 2, True), lambda: G.get_nd_lattice([4, 4, 4], 2, 2, True),
    lambda: G.get_random_regular_graph(26, 4, 2, 2, 3), lambda: G.get_random_regular_graph(40, 3, 2, 8, 3),
    lambda: G.get_nd_lattice([5, 5], 3, 9, True)], ids=["lattice-2", "cube-2", "rr4-2", "rr3-8", "lattice-9-phys3"])
@pytest.mark.parametrize("seed", [1, 2, 3])
def test_distance_of_the_factored_gauge(make, seed):
    """The distance is a mean of trace norms below 2, unchanged by rotations
    within a bond, so it takes the rounding of a unitary basis (a few c eps,
    c <= 9) and of products of up to 2 x 8^2 terms: 1e-14 = 45 eps. A gauge
    whose columns carry eps over their own singular value (down to 1e-6 of the
    largest here) is 1e-13 to 1e-12 off."""
    eng = loaded_engine(make(), seed)
    dist = []
    try:
        for path in (0, 2):
            autotune.set_knobs({"gauge_path": path})
            gamma, lam = eng.vidal_gauge(EPS)
            autotune.set_knobs({"gauge_path": 0})
            dist.append(float(eng.vidal_distance(gamma, lam, EPS)))
            assert float(lam.min()) > 0.0  # nothing dropped
    finally:
        autotune.set_knobs({"gauge_path": 0})
    assert abs(dist[0] - dist[1]) < 1e-14
