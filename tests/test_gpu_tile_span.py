"""GPU suite, tile scoring kernel beyond one quad: graphs of 129..1,024 nodes (a tile each, planes of eight node words),
17..32 classes (two passes of the votes), clause outputs.  Whole numbers: everything equals the CPU checker's."""

import numpy as np
import pytest

from graphtsetlinmachine_b200 import _lib

from oracle.oracle import OracleTM
from util import EngineTM, encode_labels, random_graphs

pytestmark = pytest.mark.gpu


def compare(n, seed, *, clauses, classes, hv, depth, ms, mb=2, max_nodes, node_types=2, edge_types=3, fixed=None):
    rng = np.random.default_rng(seed)
    np.random.seed(seed)
    graphs = random_graphs(n, rng, hv_size=hv, hv_bits=2, max_nodes=max_nodes, node_types=node_types, edge_types=edge_types,
                           fixed_nodes=fixed)
    encY = encode_labels(rng.integers(0, classes, size=n), classes, 15)
    hvs = np.stack([rng.choice(ms, size=mb, replace=False) for _ in range(clauses)]).astype(np.uint32)
    kw = dict(clauses=clauses, classes=classes, literals=2 * hv, threshold=15, s=2.0, depth=depth, message_size=ms,
              message_bits=mb, max_nodes=max_nodes, hypervectors=hvs, seed=seed)
    cpu, gpu = OracleTM(**kw), EngineTM(**kw)
    for tm in (cpu, gpu):
        tm.set_graphs(graphs)
        tm.prepare()
    assert np.array_equal(gpu.score(), cpu.score())              # every clause empty: true on all nodes of its type
    cpu.fit(encY)
    gpu.load_from(cpu)
    want = cpu.score()
    assert np.array_equal(gpu.score(), want)
    words = [(int(k) + 31) // 32 for k in graphs.number_of_graph_nodes]          # the checker leaves words past a graph's nodes alone
    nodes = [cpu.evaluate_graph(e)["cno"][-1][:, :words[e]] for e in range(n)]
    fired = np.stack([np.any(x != 0, axis=1) for x in nodes]).astype(np.int32)
    for first, count in [(0, n), (1, n - 2), (n - 1, 1)]:
        out, sums = gpu.transform(first, count)
        assert np.array_equal(out, fired[first:first + count])
        assert np.array_equal(sums, want[first:first + count])
        assert np.array_equal(gpu.score(first, count), want[first:first + count])
    gpu.close()


@pytest.mark.parametrize("nodes", [129, 256, 257, 383, 512, 513, 900, 1024])
def test_graphs_that_span_quads(engine_lib, nodes):
    compare(5, nodes, clauses=70, classes=3, hv=40, depth=3, ms=50, max_nodes=nodes, fixed=nodes)


@pytest.mark.parametrize("max_nodes,depth,ms", [(140, 2, 64), (300, 4, 33), (1000, 1, 32)])
def test_ragged_sets_with_graphs_that_span_quads(engine_lib, max_nodes, depth, ms):
    compare(9, max_nodes, clauses=333, classes=2, hv=31, depth=depth, ms=ms, max_nodes=max_nodes, node_types=3)


@pytest.mark.parametrize("classes", [16, 17, 20, 31, 32])
@pytest.mark.parametrize("max_nodes", [30, 200])
def test_class_counts(engine_lib, classes, max_nodes):
    compare(12, classes, clauses=90, classes=classes, hv=20, depth=2, ms=40, max_nodes=max_nodes)


@pytest.mark.parametrize("fixed", [1, 4, None])
@pytest.mark.parametrize("classes", [2, 19])
def test_transform_of_models_without_message_layers(engine_lib, fixed, classes):
    compare(150, 7 + classes, clauses=101, classes=classes, hv=33, depth=1, ms=32, max_nodes=fixed or 9, node_types=1, fixed=fixed)


def test_tiles_of_a_transform_do_not_serve_the_forced_kernel(engine_lib):
    """A set of a model without message layers that came without tiles gets them on its first transform; forcing the tile kernel
    afterwards stays an error, as it is without the transform."""
    rng = np.random.default_rng(8)
    np.random.seed(8)
    graphs = random_graphs(30, rng, hv_size=20, max_nodes=4)
    gpu = EngineTM(clauses=40, classes=3, literals=40, threshold=50, s=3.0, max_nodes=4)
    gpu.set_graphs(graphs)
    gpu.prepare()
    want = gpu.score()
    for transformed in (False, True):
        if transformed:
            assert np.array_equal(gpu.transform()[1], want)
        _lib.check(engine_lib.gtm_set_option(gpu.model, b"score_kernel", 3))
        with pytest.raises(_lib.GtmError):
            gpu.score()
        _lib.check(engine_lib.gtm_set_option(gpu.model, b"score_kernel", 0))
        assert np.array_equal(gpu.score(), want)
    gpu.close()
