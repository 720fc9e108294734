"""GPU suite, learning kernel for one GPU (gtm_fit_chain): automata, weights, draws and scores equal the CPU checker's bit for
bit at the edges of its dispatch - node-word sizes of the transposed rows, row-wise graphs, classes per decision pass, layers
of more than 32 words, layers of different probabilities, one CTA or many, planes in global memory, and what it leaves to
the other learning kernels (large edge types, more classes, wider automata)."""

import numpy as np
import pytest

from cases import state_of
from graphtsetlinmachine_b200 import _lib
from oracle.oracle import OracleTM
from util import EngineTM, encode_labels, random_graphs

pytestmark = pytest.mark.gpu


def agree(kw, graphs, classes, seed, epochs=2, options=None):
    rng = np.random.default_rng(seed)
    encY = encode_labels(rng.integers(0, classes, size=graphs.number_of_graphs), classes, kw["threshold"])
    cpu, gpu = OracleTM(**kw), EngineTM(**kw, options=options)
    for tm in (cpu, gpu):
        tm.set_graphs(graphs)
        tm.prepare()
    for _ in range(epochs):
        for tm in (cpu, gpu):
            tm.fit(encY)
        a, b = state_of(cpu, kw["depth"]), state_of(gpu, kw["depth"])
        assert np.array_equal(a["ta_state"], b["ta_state"])
        for x, y in zip(a["message_ta_state"], b["message_ta_state"]):
            assert np.array_equal(x, y)
        assert np.array_equal(a["clause_weights"], b["clause_weights"])
        assert np.array_equal(a["draws"], b["draws"])
    assert np.array_equal(cpu.score(), gpu.score())
    ran = gpu.last_fit_kernel()
    gpu.close()
    return ran


def model(rng, *, clauses, classes, hv, depth, ms, s=2.5, **more):
    hvs = np.stack([rng.choice(ms, size=2, replace=False) for _ in range(clauses)]).astype(np.uint32)
    return dict(clauses=clauses, classes=classes, literals=2 * hv, threshold=20, s=s, depth=depth, message_size=ms, message_bits=2,
                hypervectors=hvs, **more)


@pytest.mark.parametrize("nodes,depth,clauses,classes,hv,ms,n", [
    (1, 1, 4, 2, 3, 8, 40), (1, 1, 5, 2, 3, 8, 40),                                             # row-wise, a few literals: one CTA / five
    (3, 2, 16, 15, 16, 33, 25), (3, 2, 40, 15, 16, 33, 25),                                     # with messages; a full decision pass
    (4, 3, 33, 16, 40, 32, 25),             # just past row-wise; the second decision pass has one class
    (32, 2, 300, 31, 33, 100, 8), (33, 2, 300, 32, 32, 64, 8),                                  # one node word / more
    (128, 3, 90, 3, 64, 37, 6), (129, 2, 90, 3, 65, 40, 6),
    (512, 2, 150, 2, 20, 70, 3), (513, 2, 150, 2, 20, 70, 3), (1024, 2, 150, 2, 20, 64, 2), (1025, 2, 70, 2, 20, 64, 2),
    (20, 3, 200, 4, 600, 700, 6),           # layers of more than 32 words: updates as work items
])
def test_sizes(engine_lib, nodes, depth, clauses, classes, hv, ms, n):
    rng = np.random.default_rng(nodes + clauses)
    np.random.seed(nodes)
    graphs = random_graphs(n, rng, hv_size=hv, max_nodes=nodes, node_types=2, edge_types=3, max_degree=2)
    graphs2 = random_graphs(2, rng, init_with=graphs, fixed_nodes=nodes, node_types=2, edge_types=3, max_degree=2)
    for g in (graphs, graphs2):             # mixed sizes, then the largest alone
        kw = model(rng, clauses=clauses, classes=classes, hv=hv, depth=depth, ms=ms, max_nodes=nodes, seed=nodes)
        ran = agree(kw, g, classes, 3)
        most = int(g.max_number_of_graph_nodes)
        words = 1 if most <= 32 else 4 if most <= 128 else 16 if most <= 512 else 32
        if most > 1024: assert ran["kernel"] != 2
        else: assert (ran["kernel"], ran["node_words"], ran["hybrid"], ran["narrow"]) == (2, words, 0, hv < 600)


@pytest.mark.parametrize("more", [dict(s=(2.0, 3.0, 4.0)), dict(s=1.0), dict(boost=0), dict(max_included=3), dict(state_bits=1), dict(state_bits=9),
                                  dict(q=0.3)])
@pytest.mark.parametrize("hv,ms", [(20, 50), (560, 50)])
def test_options(engine_lib, more, hv, ms):
    rng = np.random.default_rng(7)
    np.random.seed(7)
    graphs = random_graphs(15, rng, hv_size=hv, max_nodes=9, node_types=1, edge_types=2)
    kw = model(rng, clauses=70, classes=5, hv=hv, depth=3, ms=ms, max_nodes=9, seed=5, **more)
    agree(kw, graphs, 5, 4)


@pytest.mark.parametrize("largest", [24, 25, 300])
def test_edge_types(engine_lib, largest):
    """The window of pulled messages covers edge types up to 24; beyond, another kernel learns."""
    rng = np.random.default_rng(largest)
    np.random.seed(9)
    graphs = random_graphs(12, rng, hv_size=24, max_nodes=20, edge_types=2, max_degree=3)
    graphs.edge[:, 1] = rng.integers(0, largest + 1, size=len(graphs.edge))
    graphs.edge[0, 1] = largest
    kw = model(rng, clauses=150, classes=3, hv=24, depth=3, ms=45, max_nodes=20, seed=6)
    assert (agree(kw, graphs, 3, 5)["kernel"] == 2) == (largest <= 24)
    # one CTA reads the edges themselves, of any type
    kw = model(rng, clauses=14, classes=3, hv=24, depth=3, ms=45, max_nodes=20, seed=6)
    ran = agree(kw, graphs, 3, 5)
    assert (ran["kernel"], ran["one_cta"]) == (2, 1)


@pytest.mark.parametrize("clauses,depth,hv,ms,nodes,s,words,hybrid,narrow", [
    (7000, 2, 512, 512, 6, 2.5, 1, 0, 1), (16000, 1, 700, 8, 40, 2.5, 4, 0, 0),          # many clauses per CTA, all planes still fit
    (16000, 2, 512, 512, 6, 2.5, 1, 1, 1), (40000, 1, 256, 8, 3, 2.5, 1, 1, 1),
    (12000, 2, 700, 700, 6, 2.5, 1, 1, 0), (30000, 1, 700, 8, 40, 2.5, 4, 1, 0),
    (22000, 2, 256, 256, 100, 2.5, 4, 1, 1), (16000, 1, 700, 8, 200, 2.5, 16, 1, 0),
    (24000, 2, 256, 256, 300, 2.5, 16, 1, 1), (30000, 1, 200, 8, 600, 2.5, 32, 1, 1),
    (37000, 2, 128, 128, 600, (2.0, 3.0), 32, 1, 0),
])
def test_planes_in_global_memory(engine_lib, clauses, depth, hv, ms, nodes, s, words, hybrid, narrow):
    """Models whose automata exceed shared memory keep only the include planes there."""
    rng = np.random.default_rng(clauses)
    np.random.seed(2)
    graphs = random_graphs(4 if nodes < 100 else 2, rng, hv_size=hv, max_nodes=nodes, fixed_nodes=nodes if nodes > 6 else None, edge_types=2)
    kw = model(rng, clauses=clauses, classes=4, hv=hv, depth=depth, ms=ms, s=s, max_nodes=nodes, seed=8)
    ran = agree(kw, graphs, 4, 6)
    assert [ran[k] for k in ("kernel", "node_words", "hybrid", "narrow")] == [2, words, hybrid, narrow]


@pytest.mark.parametrize("clauses,nodes", [(14, 90), (90, 90), (90, 300)])
def test_graphs_of_many_edges(engine_lib, clauses, nodes):
    """Graphs of more than 512 edges are read from global memory: by one CTA, and by many."""
    rng = np.random.default_rng(clauses + nodes)
    np.random.seed(4)
    graphs = random_graphs(5, rng, hv_size=20, max_nodes=nodes, fixed_nodes=nodes, edge_types=3, max_degree=15)
    assert int(np.diff(graphs.edge_index[graphs.node_index]).min()) > 512
    kw = model(rng, clauses=clauses, classes=3, hv=20, depth=3, ms=50, max_nodes=nodes, seed=3)
    ran = agree(kw, graphs, 3, 9)
    assert (ran["kernel"], ran["one_cta"]) == (2, clauses < 20)


@pytest.mark.parametrize("clauses,depth,hv,ms,s", [(400, 2, 40, 40, 2.5), (16000, 2, 512, 512, 2.5), (40000, 1, 256, 8, 2.5), (12000, 2, 700, 700, 2.5)])
def test_wait_that_runs_out(engine_lib, clauses, depth, hv, ms, s):
    """An arrival that never comes ends the launch with GTM_ERR_TIMEOUT; with the state restored the model learns on.  With planes
    in global memory (all but the first) the failed call leaves the model in between, as the header says."""
    rng = np.random.default_rng(clauses)
    np.random.seed(5)
    graphs = random_graphs(3, rng, hv_size=hv, max_nodes=3, edge_types=2)
    kw = model(rng, clauses=clauses, classes=3, hv=hv, depth=depth, ms=ms, s=s, max_nodes=3, seed=8)
    encY = encode_labels(np.arange(3) % 3, 3, kw["threshold"])
    cpu, gpu = OracleTM(**kw), EngineTM(**kw)
    for tm in (cpu, gpu):
        tm.set_graphs(graphs)
        tm.prepare()
        tm.fit(encY)
    assert gpu.last_fit_kernel()["kernel"] == 2 and gpu.last_fit_kernel()["hybrid"] == (clauses > 400)
    for name, value in ((b"fit_wait_ms", 30), (b"fit_missing_cta", 1)):
        _lib.check(engine_lib.gtm_set_option(gpu.model, name, value))
    with pytest.raises(_lib.GtmError) as err:
        gpu.fit(encY)
    assert err.value.status == 4
    for name, value in ((b"fit_wait_ms", 2000), (b"fit_missing_cta", 0)):
        _lib.check(engine_lib.gtm_set_option(gpu.model, name, value))
    if clauses == 400:
        assert np.array_equal(gpu.ta_state, cpu.ta_state) and np.array_equal(gpu.draws_consumed(), cpu.draws_consumed())
    gpu.load_from(cpu)
    for tm in (cpu, gpu):
        tm.fit(encY)
    a, b = state_of(cpu, depth), state_of(gpu, depth)
    assert np.array_equal(a["ta_state"], b["ta_state"]) and np.array_equal(a["clause_weights"], b["clause_weights"])
    assert all(np.array_equal(x, y) for x, y in zip(a["message_ta_state"], b["message_ta_state"]))
    gpu.close()


@pytest.mark.parametrize("per_cta", [1, 7, 60])
def test_clause_ranges(engine_lib, per_cta):
    rng = np.random.default_rng(1)
    np.random.seed(3)
    graphs = random_graphs(20, rng, hv_size=30, max_nodes=12, edge_types=2)
    kw = model(rng, clauses=60, classes=3, hv=30, depth=2, ms=64, max_nodes=12, seed=4)
    agree(kw, graphs, 3, 8, options={"fit_block_clauses": per_cta})


@pytest.mark.parametrize("clauses,depth,nodes,s", [
    (4, 1, 3, 2.5), (5, 1, 3, 2.5),                             # no messages
    (16, 2, 30, 2.5), (17, 2, 30, 2.5), (16, 3, 256, 2.5), (16, 2, 257, 2.5),
    (32, 2, 3, 1.0), (33, 2, 3, 1.0), (32, 2, 4, 1.0),          # few nodes and no masks to draw
])
def test_one_cta_or_many(engine_lib, clauses, depth, nodes, s):
    """Both sides of the lines of the rule that has one CTA learn a model alone."""
    rng = np.random.default_rng(nodes)
    np.random.seed(clauses)
    graphs = random_graphs(6, rng, hv_size=20, fixed_nodes=nodes, max_nodes=nodes, edge_types=2, max_degree=2)
    kw = model(rng, clauses=clauses, classes=3, hv=20, depth=depth, ms=70, s=s, max_nodes=nodes, seed=9)
    ran = agree(kw, graphs, 3, 7)
    one = clauses <= (4 if depth == 1 else 32 if s == 1.0 and nodes <= 3 else 16) and nodes <= 256
    assert (ran["kernel"], ran["one_cta"]) == (2, one)


def test_two_models_in_two_threads(engine_lib):
    """Models of one kernel variant and different shared-memory plans, learned in two threads: as each learns alone."""
    import threading

    rng = np.random.default_rng(12)
    np.random.seed(12)
    jobs = []
    for clauses in (150, 900):
        graphs = random_graphs(12, rng, hv_size=60, max_nodes=3, max_degree=2)
        kw = model(rng, clauses=clauses, classes=3, hv=60, depth=2, ms=60, max_nodes=3, seed=clauses)
        encY = encode_labels(rng.integers(0, 3, size=12), 3, kw["threshold"])
        tms = [EngineTM(**kw) for _ in range(2)]
        for tm in tms:
            tm.set_graphs(graphs)
            tm.prepare()
        for _ in range(60):
            tms[0].fit(encY)
        jobs.append((tms, encY))
    errors = []

    def learn(tm, encY):
        try:
            for _ in range(60):
                tm.fit(encY)
        except Exception as e:
            errors.append(e)

    threads = [threading.Thread(target=learn, args=(tms[1], encY)) for tms, encY in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for (alone, beside), _ in jobs:
        a, b = state_of(alone, 2), state_of(beside, 2)
        assert np.array_equal(a["ta_state"], b["ta_state"]) and np.array_equal(a["message_ta_state"][0], b["message_ta_state"][0])
        assert np.array_equal(a["clause_weights"], b["clause_weights"]) and np.array_equal(a["draws"], b["draws"])
        alone.close()
        beside.close()
