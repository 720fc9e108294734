"""GPU suite: sets of different shared-memory plans side by side; the plan of the one made last must not limit the launches
on the others."""

import numpy as np
import pytest

from graphtsetlinmachine_b200.tm import MultiClassGraphTsetlinMachine
from util import random_graphs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("depth,nodes,small", [(2, 100, 5), (3, 300, 140), (1, 9, 1), (2, 1100, 1030)])
def test_a_smaller_set_does_not_limit_a_larger_one(engine_lib, depth, nodes, small):
    rng = np.random.default_rng(nodes)
    np.random.seed(nodes)
    models = []
    for hv, n in ((120, nodes), (8, small)):                   # the larger plan first
        graphs = random_graphs(6, rng, hv_size=hv, max_nodes=n, fixed_nodes=n, max_degree=1)
        tm = MultiClassGraphTsetlinMachine(300, 100, 2.0, depth=depth, message_size=256 if n == nodes else 32)
        tm.fit(graphs, np.arange(6, dtype=np.uint32) % 2, epochs=1)
        models.append((tm, graphs, tm.score(graphs)))
    for tm, graphs, want in models:
        assert np.array_equal(tm.score(graphs), want)
        assert np.array_equal(tm.transform(graphs)[1], want)
