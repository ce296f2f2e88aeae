"""Node updates by blocks of bond slices (bonds from 8: dqz_bp_node_update and
dqz_bp_sweep_sliced) against the FP64 oracle (tensor_ops.py:36-60).

Tolerance: an entry is a chain of at most 32 + 32 + 8192 products; the worst
growth 8256 eps = 1.8e-12 of the absolute sum, positive messages and the trace
division adding small factors: 1e-11 of the message.
"""

import pytest
import torch

from dequantizer_b200 import graph as G
from dequantizer_b200 import maps as M
from oracle import maps as OM
from tests.helpers import random_messages, random_tensors, rel_err

pytestmark = pytest.mark.gpu
TOL = 1e-11

# chains, trees and 3-regular graphs over slice and block remainders (bond 31, 32: a block of two slices at d = 2, of
# one at d = 4; physical 1 and 8; bond 1); slices above a block (17 x 31 x 8) and degree 4 take the generic form
CASES = {
    "chain_32_phys8": (lambda: G.get_nd_lattice([5], 8, 2), [32, 9]),
    "tree_uneven_phys1": (lambda: G.get_random_tree_tensor_graph(9, 1, [1], 5), [32, 1, 17, 8]),
    "regular_uneven_phys3": (lambda: G.get_random_regular_graph(6, 3, 3, 2, 11), [8, 11, 16, 13]),
    "regular_31_phys2": (lambda: G.get_random_regular_graph(4, 3, 2, 2, 3), [31, 32, 7]),
    "regular_32_phys4": (lambda: G.get_random_regular_graph(4, 3, 4, 2, 3), [32]),
    "regular_large_slices": (lambda: G.get_random_regular_graph(4, 3, 8, 2, 3), [17, 31, 20]),
    "lattice_degree4": (lambda: G.get_nd_lattice([3, 3], 2, 2), [8, 3, 9, 2]),
}


@pytest.mark.parametrize("sync", [True, False])
@pytest.mark.parametrize("case", list(CASES))
def test_sweep_by_slices_matches_oracle(case, sync):
    make, dims = CASES[case]
    g = make()
    for i, e in enumerate(g.edges.values()):
        e.dimension = dims[i % len(dims)]
    g.refresh_bond_shapes()
    trav = list(g.get_traversal_iterator(ordering="dfs"))
    tensors, messages = random_tensors(g, 3), random_messages(g, 4)
    want = OM.get_belief_propagation_map(trav, sync)(tensors, messages)
    got = M.get_belief_propagation_map(trav, sync)(tensors, messages)
    for k in want:
        assert rel_err(got[k], want[k]) < TOL, k
    assert int(M.error_flag(torch.device("cuda", 0)).item()) == 0
