"""Performance cases of the engine: what its users call, over the sizes that they call it with.

A user encodes graphs on the host (``Graphs``), learns from them one epoch at a time (``fit(..., incremental=True)``),
and scores graph sets with the trained model: sets that are new to it (uploaded and scored in one call), or the
evaluation set that stays with it from epoch to epoch.  All of it goes in and out as numpy arrays.

A case is (what is called, which graphs, which model):

``op``     "score_new"    class sums of two graph sets, each new to the model when its turn comes
           "score_again"  class sums of a set that the model has scored before
           "fit"          one more epoch, then the whole model state comes back (``save``), as for a checkpoint
           "epoch"        the training loop of the demos: one more epoch, predictions for the test set and for the
                          training set, layer-0 automata and weights (``get_state``)
           "transform"    clause outputs and class sums of a set
``kind``   "xor"          2-node graphs (Noisy XOR)
           "images"       one node per image, a symbol per pixel that is on
           "patches"      one node per 10x10 (or smaller) patch of an image
           "sequences"    directed paths, one symbol per node
           "multigraphs"  random directed multigraphs of ragged sizes, several node and edge types
``graphs`` graphs per set (the evaluation set of "epoch" has as many as ``test`` says), ``warm`` epochs over
``train`` graphs learned beforehand.  The other fields are arguments of the model and of the encoding.
"""

import math

import numpy as np

from graphtsetlinmachine_b200 import datasets
from graphtsetlinmachine_b200.graphs import Graphs
from graphtsetlinmachine_b200.tm import MultiClassGraphTsetlinMachine

# The five benchmark configurations: model and encoding.
XOR = dict(kind="xor", clauses=10, T=100, s=1.0, depth=2, message=256, hv=32, max_included=4, classes=2)
IMAGES = dict(kind="images", clauses=2500, T=3125, s=10.0, depth=1, message=256, hv=128, classes=10, side=28)
PATCHES = dict(kind="patches", clauses=2500, T=3125, s=10.0, depth=1, message=256, hv=128, classes=10, side=28, patch=10)
SEQUENCES = dict(kind="sequences", clauses=2000, T=2000, s=5.0, depth=3, message=512, hv=256, classes=2, length=1000)
MULTIGRAPHS = dict(kind="multigraphs", clauses=20000, T=10000, s=10.0, depth=3, message=1024, hv=1024, classes=10,
                   min_nodes=8, max_nodes=32, node_types=1, edge_types=4, symbols=256)
# Sizes that fit no word and no tile: 3..90 nodes, 200 literals, 2 x 50 message literals, 20 classes, three node types.
RAGGED = dict(kind="multigraphs", clauses=333, T=400, s=4.0, depth=3, message=50, hv=100, classes=20,
              min_nodes=3, max_nodes=90, node_types=3, edge_types=3, symbols=61)


def listed():
    return [
        # online inference: a request is one image
        dict(IMAGES, name="serve_image", op="score_new", graphs=1, train=1000, warm=1),
        # batch inference over images that arrive in large sets
        dict(IMAGES, name="score_images", op="score_new", graphs=120000, train=1000, warm=1),
        # evaluation of a small model on a large set of tiny graphs
        dict(XOR, name="score_xor", op="score_again", graphs=250000, train=2000, warm=1),
        # evaluation on long sequences, depth 3
        dict(SEQUENCES, name="score_sequences", op="score_again", graphs=400, train=100, warm=1),
        # batch inference with the largest model, depth 3
        dict(MULTIGRAPHS, name="score_multigraphs", op="score_new", graphs=6000, train=300, warm=1),
        # clause outputs as features for another learner
        dict(MULTIGRAPHS, name="transform_multigraphs", op="transform", graphs=500, clauses=5000, T=2500, train=300, warm=1),
        # learning, from the smallest model to the largest
        dict(XOR, name="fit_xor", op="fit", graphs=10000, train=10000, warm=1),
        dict(IMAGES, name="fit_images", op="fit", graphs=4000, train=4000, warm=1),
        dict(SEQUENCES, name="fit_sequences", op="fit", graphs=200, train=200, warm=1),
        dict(MULTIGRAPHS, name="fit_multigraphs", op="fit", graphs=300, train=300, warm=1),
        # the demos' loop on convolution-shaped images, and on ragged graphs
        dict(PATCHES, name="epoch_patches", op="epoch", graphs=400, train=400, test=800, warm=1),
        dict(RAGGED, name="epoch_ragged", op="epoch", graphs=700, train=700, test=700, warm=1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["xor", "images", "patches", "sequences", "multigraphs", "multigraphs"])
    op = rng.choice(["score_new", "score_again", "fit", "epoch", "transform"])
    if kind == "xor":
        case = dict(XOR, clauses=_log(rng, 4, 64), message=_log(rng, 33, 512), hv=rng.randint(20, 64), s=rng.choice([1.0, 1.7, 3.0]))
        nodes = 2
    elif kind == "images":
        case = dict(IMAGES, clauses=_log(rng, 90, 5000), hv=rng.randint(60, 256), classes=rng.randint(2, 20))
        nodes = 1
    elif kind == "patches":
        case = dict(PATCHES, clauses=_log(rng, 90, 2500), side=rng.randint(12, 28), patch=rng.randint(3, 10), classes=rng.randint(2, 12))
        nodes = (case["side"] - case["patch"] + 1) ** 2
    elif kind == "sequences":
        case = dict(SEQUENCES, clauses=_log(rng, 90, 2000), length=_log(rng, 20, 1000), depth=rng.randint(2, 4),
                    message=_log(rng, 60, 512), hv=rng.randint(40, 256))
        nodes = case["length"]
    else:
        top = rng.randint(8, 100)
        case = dict(MULTIGRAPHS, clauses=_log(rng, 90, 20000), depth=rng.randint(1, 4), message=_log(rng, 33, 1024),
                    hv=_log(rng, 33, 1024), classes=rng.randint(2, 20), min_nodes=rng.randint(1, 8), max_nodes=top,
                    node_types=rng.randint(1, 3), edge_types=rng.randint(1, 5), symbols=rng.randint(20, 256),
                    s=rng.choice([2.0, 5.0, 10.0]))
        nodes = (case["min_nodes"] + top) // 2
    case["T"] = max(10, case["clauses"] * rng.choice([1, 2]) // 2) if kind != "xor" else 100
    # set sizes by use, within what one pass of the largest listed case costs
    dense = nodes * case["clauses"] * (case["hv"] + (case["depth"] - 1) * case["message"]) / 16      # word tests of one graph
    most = {"fit": 1e10, "epoch": 1e10, "transform": 2e10}.get(op, 2e11) / dense
    most = min(most, 300000 / nodes, {"fit": 4000, "epoch": 2000, "transform": min(4000, 3e6 / case["clauses"])}.get(op, 100000))
    case.update(op=op, warm=1)
    case["graphs"] = _log(rng, 1 if op == "score_new" else 50, max(60, most))
    case["train"] = case["graphs"] if op in ("fit", "epoch") else max(30, min(500, int(1e10 / dense)))
    if op == "epoch":
        case["test"] = _log(rng, 50, max(60, 2 * case["graphs"]))
    return case


# ------------------------------------------------------------------------------------------------ graph sets
def _multigraphs(case, n_graphs, seed, init_with=None):
    """Random directed multigraphs: node count, node type, Poisson(3) out-degree, targets, edge types and one to five
    symbols per node; the label follows from a linear score over the symbol counts."""
    rng = np.random.default_rng(seed)
    n_sym, n_types = case["symbols"], case["node_types"]
    g = Graphs(n_graphs, init_with=init_with) if init_with is not None else \
        Graphs(n_graphs, symbols=list(range(n_sym)), hypervector_size=case["hv"], hypervector_bits=2)
    n = rng.integers(case["min_nodes"], case["max_nodes"] + 1, size=n_graphs)
    g.set_number_of_graph_nodes_bulk(n)
    g.prepare_node_configuration()
    total = int(n.sum())
    degree = rng.poisson(3.0, size=total).astype(np.uint32)
    g.set_nodes_bulk(degree, rng.integers(0, n_types, size=total), ["type %d" % t for t in range(n_types)])
    g.prepare_edge_configuration()
    node_graph = np.repeat(np.arange(n_graphs), n)
    room = n[np.repeat(node_graph, degree)]
    g.set_edges_bulk((rng.random(len(room)) * room).astype(np.uint32), rng.integers(0, case["edge_types"], size=len(room)),
                     ["edge %d" % t for t in range(case["edge_types"])])
    rows = np.repeat(np.arange(total), rng.integers(1, 6, size=total))
    symbols = rng.integers(0, n_sym, size=len(rows))
    g.add_graph_node_properties_bulk(rows, symbols)
    counts = np.zeros((n_graphs, n_sym), dtype=np.float32)
    np.add.at(counts, (node_graph[rows], symbols), 1.0)
    scores = counts @ np.random.default_rng(12345).normal(size=(n_sym, case["classes"])).astype(np.float32)
    g.encode()
    return g, np.argmax(scores, axis=1).astype(np.uint32)


def _graph_set(case, n_graphs, seed, init_with=None):
    kind, hv = case["kind"], case["hv"]
    # large sets repeat a few thousand distinct graphs
    distinct = min(n_graphs, 6000 if kind == "images" else 60000)
    if kind == "xor":
        g, y = datasets.noisy_xor(distinct, seed, hv_size=hv, init_with=init_with)
    elif kind in ("images", "patches"):
        protos = datasets.image_prototypes(1, classes=case["classes"], side=case["side"])
        if kind == "images":
            g, y = datasets.vanilla_images(distinct, seed, protos, hv_size=hv, init_with=init_with)
        else:
            g, y = datasets.convolution_images(distinct, seed, protos, patch=case["patch"], hv_size=hv, init_with=init_with)
    elif kind == "sequences":
        g, y = datasets.sequences(distinct, seed, length=case["length"], hv_size=hv, init_with=init_with)
    else:
        g, y = _multigraphs(case, distinct, seed, init_with)
    if distinct < n_graphs:
        g, y = g[np.arange(n_graphs) % distinct], np.resize(y, n_graphs)
    return g, y


def prepare(case, seed):
    """The encoded graph sets on the host and a model that has learned for a while."""
    np.random.seed(seed % (1 << 32))                      # symbol and clause hypervectors
    train, y = _graph_set(case, case["train"], 5 * seed)
    y[: case["classes"]] = np.arange(case["classes"])[: len(y)]      # every class occurs
    tm = MultiClassGraphTsetlinMachine(case["clauses"], case["T"], case["s"], depth=case["depth"], message_size=case["message"],
                                       max_included_literals=case.get("max_included"), seed=seed)
    tm.fit(train, y, epochs=case["warm"])
    op, state = case["op"], dict(op=case["op"], tm=tm)
    if op in ("fit", "epoch"):
        state.update(train=train, y=y)
    if op == "epoch":
        state["test"] = _graph_set(case, case["test"], 5 * seed + 1, init_with=train)[0]
    if op not in ("fit", "epoch"):
        sets = 2 if op == "score_new" else 1
        state["sets"] = [_graph_set(case, case["graphs"], 5 * seed + 1 + k, init_with=train)[0] for k in range(sets)]
    return state


def run(state):
    op, tm = state["op"], state["tm"]
    if op in ("score_new", "score_again"):
        return [tm.score(g) for g in state["sets"]]
    if op == "transform":
        return tm.transform(state["sets"][0])
    tm.fit(state["train"], state["y"], epochs=1, incremental=True)
    if op == "fit":
        saved = tm.save()
        return [saved["ta_state"], list(saved["message_ta_state"]), saved["clause_weights"]]
    return [tm.predict(state["test"]), tm.predict(state["train"]), list(tm.get_state()[:2])]


# ----------------------------------------------------------------------------------------------------- work
def _mean_nodes_edges(case):
    kind = case["kind"]
    if kind == "xor":
        return 2.0, 2.0
    if kind == "images":
        return 1.0, 0.0
    if kind == "patches":
        return float((case["side"] - case["patch"] + 1) ** 2), 0.0
    if kind == "sequences":
        return float(case["length"]), 2.0 * (case["length"] - 1)
    nodes = (case["min_nodes"] + case["max_nodes"]) / 2
    return nodes, 3.0 * nodes


def work(case):
    """Bytes: graph arrays (literals, node type, degree, edge index; edges; node index and count) read once, include
    bits of the model read once, results written once; a fit reads targets and reads and writes every automaton once.
    Operations: one word operation per 32 nodes for every clause and layer, which is the least that evaluates them."""
    nodes, edges = _mean_nodes_edges(case)
    words0, words_m = -(-2 * case["hv"] // 32), -(-2 * case["message"] // 32)
    words = words0 + (case["depth"] - 1) * words_m                       # words of one automaton plane, all layers
    graph = 4 * nodes * words0 + 12 * nodes + 8 * edges + 8
    C, K, op = case["clauses"], case["classes"], case["op"]
    state = 4 * C * (8 * words + K)
    evaluate = C * case["depth"] * nodes / 32
    if op == "fit":
        n_eval, size = case["graphs"], case["graphs"] * (graph + 4 * K) + 2 * state
    elif op == "epoch":
        n_eval = 2 * case["graphs"] + case["test"]
        size = n_eval * (graph + 4 * K) + 2 * state + 4 * case["graphs"] * K
    else:
        n_eval = case["graphs"] * (2 if op == "score_new" else 1)
        size = n_eval * (graph + 4 * K + (4 * C if op == "transform" else 0)) + 4 * C * (words + K)
    return dict(bytes=float(size), flops=float(n_eval * evaluate))


def tolerance(case):
    return "exact"                                       # bits, integers and automata: every result is a whole number
