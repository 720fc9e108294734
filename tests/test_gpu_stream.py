"""GPU suite, node-stream scoring (depth 1) and the host path around scoring: class sums equal the CPU checker's bit for bit
where the dispatch can go wrong - tile edges, clause-block remainders, class counts at the edges of the vote fragments,
weights of one to four signed bytes, clause shares, sets on both sides of the small-set and chunk limits."""

import ctypes as C

import numpy as np
import pytest

from graphtsetlinmachine_b200 import _lib, hostmem
from oracle.oracle import OracleTM
from util import EngineTM, random_graphs

pytestmark = pytest.mark.gpu


def sparse_model(cpu, rng, include, most_weight):
    """Random include masks with about `include` literals per clause and weights up to the given size."""
    cpu.ta_state[...] = 0xffffffff
    plane = np.zeros((cpu.C, cpu.la_chunks), dtype=np.uint32)
    for c in range(cpu.C):
        for lit in rng.choice(cpu.literals, size=min(cpu.literals, int(rng.integers(0, 2 * include + 1))), replace=False):
            plane[c, lit // 32] |= np.uint32(1 << (lit % 32))
    cpu.ta_state[:, :, cpu.SB - 1] = plane
    cpu.clause_weights[...] = rng.integers(-most_weight, most_weight + 1, size=cpu.clause_weights.shape)
    cpu.clause_weights[0, 0], cpu.clause_weights[-1, -1] = most_weight, -most_weight


def scored_create(tm, graphs):
    """gtm_dataset_create_scored, the upload-and-score call behind the model classes' `score`."""
    u32 = lambda a: np.ascontiguousarray(a, dtype=np.uint32)
    arrays = [u32(graphs.X), u32(graphs.node_type), u32(graphs.number_of_graph_node_edges), u32(graphs.edge_index),
              u32(graphs.edge) if graphs.edge.size else None, u32(graphs.node_index), u32(graphs.number_of_graph_nodes)]
    v = _lib.GraphsView()
    (v.X, v.node_type, v.number_of_graph_node_edges, v.edge_index, v.edge, v.node_index, v.number_of_graph_nodes) = [
        None if a is None else a.ctypes.data for a in arrays]
    v.number_of_graphs, v.total_nodes = int(graphs.number_of_graphs), int(arrays[0].shape[0])
    v.total_edges = int(graphs.edge.shape[0]) if graphs.edge.size else 0
    v.max_number_of_graph_nodes = int(graphs.max_number_of_graph_nodes)
    out = hostmem.empty((graphs.number_of_graphs, tm.K), np.int32)
    ds = C.c_void_p()
    _lib.check(tm.lib.gtm_dataset_create_scored(tm.model, C.byref(v), graphs.number_of_node_types(), out.ctypes.data, C.byref(ds)))
    tm.lib.gtm_dataset_destroy(ds)
    return out


@pytest.mark.parametrize("n,max_nodes,clauses,classes,hv,types,most_weight", [
    (1, 1, 1, 1, 3, 1, 1),                  # the smallest of everything
    (33, 1, 255, 2, 20, 2, 127),            # one byte, one clause short of a block
    (128, 1, 257, 16, 40, 1, 128),          # just over one byte; the last class of the first row block
    (1025, 1, 600, 17, 50, 3, 32640),       # over one tile; the first class of the second row block; three bytes
    (600, 1, 300, 32, 16, 1, 2 ** 31 - 1),  # most classes, four bytes: sums wrap as the reference's additions do
    (300, 9, 130, 5, 30, 2, 40),            # small multi-node graphs
    (40, 90, 513, 3, 33, 1, 200),           # large graphs: voted from the node words
    (4, 700, 70, 10, 64, 2, 30),            # more node words than a quad
])
def test_class_sums(engine_lib, n, max_nodes, clauses, classes, hv, types, most_weight):
    rng = np.random.default_rng(n + clauses)
    np.random.seed(n)
    graphs = random_graphs(n, rng, hv_size=hv, hv_bits=2, max_nodes=max_nodes, node_types=types, max_degree=1, fixed_nodes=1 if max_nodes == 1 else None)
    kw = dict(clauses=clauses, classes=classes, literals=2 * hv, threshold=50, s=3.0, max_nodes=max_nodes, seed=n)
    cpu, gpu = OracleTM(**kw), EngineTM(**kw, options={"score_kernel": 2})
    sparse_model(cpu, rng, 2, most_weight)
    for tm in (cpu, gpu):
        tm.set_graphs(graphs)
    gpu.load_from(cpu)
    want = cpu.score()
    assert np.array_equal(gpu.score(), want)
    assert np.array_equal(scored_create(gpu, graphs), want)
    for first, count in [(n // 2, n - n // 2), (n - 1, 1)]:
        assert np.array_equal(gpu.score(first, count), want[first:first + count])
    gpu.close()


@pytest.mark.parametrize("n,nodes,depth", [(30000, 1, 1), (30000, None, 1), (9000, 3, 2), (9000, None, 2)])
def test_pipelined_chunks(engine_lib, n, nodes, depth):
    """Sets that go up and come back in several chunks, with constant and with varying arrays: equal to scoring the resident
    set in pieces, and to the checker on a few graphs."""
    rng = np.random.default_rng(n)
    np.random.seed(5)
    base = random_graphs(300, rng, hv_size=128, max_nodes=4, node_types=1 if nodes else 3, max_degree=0 if nodes else 2, fixed_nodes=nodes)
    graphs = base[np.arange(n) % 300]
    kw = dict(clauses=200, classes=9, literals=256, threshold=50, s=3.0, depth=depth, message_size=64, max_nodes=4, seed=2,
              hypervectors=np.stack([rng.choice(64, size=2, replace=False) for _ in range(200)]).astype(np.uint32))
    cpu, gpu = OracleTM(**kw), EngineTM(**kw)
    cpu.set_graphs(base)
    cpu.prepare()
    cpu.fit(np.where(rng.integers(0, 9, size=300)[:, None] == np.arange(9)[None, :], 50, -50).astype(np.int32))
    gpu.set_graphs(graphs)
    gpu.load_from(cpu)
    want = np.resize(cpu.score(), (n, 9))
    for _ in range(2):
        assert np.array_equal(gpu.score(), want)
        assert np.array_equal(scored_create(gpu, graphs), want)
    assert np.array_equal(gpu.score(299, n - 300), want[299:n - 1])
    gpu.close()


@pytest.mark.parametrize("depth", [1, 2])
@pytest.mark.parametrize("first", [3, 8000])
def test_shifted_ranges_are_refused_chunk_by_chunk(engine_lib, depth, first):
    """A set that goes up in chunks is checked chunk by chunk, each before it is copied; the model scores on."""
    rng = np.random.default_rng(first)
    np.random.seed(6)
    base = random_graphs(300, rng, hv_size=128, max_nodes=4, max_degree=2)
    base.edge[:, 0] = 0
    kw = dict(clauses=200, classes=9, literals=256, threshold=50, s=3.0, depth=depth, message_size=64, max_nodes=4, seed=2,
              hypervectors=np.stack([rng.choice(64, size=2, replace=False) for _ in range(200)]).astype(np.uint32))
    gpu = EngineTM(**kw)
    gpu.set_graphs(base)
    gpu.prepare()
    want = np.resize(gpu.score(), (16000, 9))
    for name, shift in [("node_index", 2 ** 30), ("edge_index", 2 ** 30)]:
        graphs = base[np.arange(16000) % 300]
        at = first if name == "node_index" else int(graphs.node_index[first])
        array = np.array(getattr(graphs, name))
        array[at:] += np.uint32(shift)
        setattr(graphs, name, array)
        with pytest.raises(Exception, match=name):
            scored_create(gpu, graphs)
    assert np.array_equal(scored_create(gpu, base[np.arange(16000) % 300]), want)
    gpu.close()


def test_results_outlive_the_pool(engine_lib):
    """An array in recycled page-locked memory keeps its memory while it, or a view of it, is alive."""
    for _ in range(4 * hostmem.PER_BLOCK):                       # a size's first arrays are ordinary memory
        hostmem.empty((1000, 100), np.int32)
    a = hostmem.empty((1000, 100), np.int32)
    a[...] = 7
    view = a[10:20]
    address = a.ctypes.data
    del a
    b = hostmem.empty((1000, 100), np.int32)
    b[...] = 8
    assert b.ctypes.data != address and (view == 7).all()
    del view
    assert hostmem.empty((1000, 100), np.int32).ctypes.data == address


def test_memory_that_cannot_be_locked(engine_lib):
    """A failed page-lock is an error of its own call; the calls behind it, whose launches succeed, are not blamed for it."""
    rng = np.random.default_rng(3)
    np.random.seed(3)
    graphs = random_graphs(40, rng, hv_size=20, max_nodes=3)
    gpu = EngineTM(clauses=30, classes=3, literals=40, threshold=50, s=3.0, max_nodes=3)
    gpu.set_graphs(graphs)
    gpu.prepare()
    want = gpu.score()
    p = C.c_void_p()
    assert engine_lib.gtm_host_alloc(1 << 50, C.byref(p)) in (2, 3) and not p.value
    gpu.prepare()                                                 # a launch with a check behind it
    assert engine_lib.gtm_host_alloc(1 << 50, C.byref(p)) in (2, 3)
    assert np.array_equal(scored_create(gpu, graphs), gpu.score()) and gpu.score().shape == want.shape
    gpu.close()


def test_locked_memory_goes_with_the_last_model(engine_lib):
    """Free blocks are given back when the last model is closed; a block in use stays until its array goes."""
    import gc

    from graphtsetlinmachine_b200.tm import MultiClassGraphTsetlinMachine
    gc.collect()
    np.random.seed(4)
    graphs = random_graphs(8, np.random.default_rng(4), hv_size=16, max_nodes=3)
    models = [MultiClassGraphTsetlinMachine(20, 50, 2.0, depth=1) for _ in range(2)]
    for tm in models:
        tm.fit(graphs, np.arange(8, dtype=np.uint32) % 2, epochs=1)
    others = len(hostmem._models) - 2
    shape = (1 << 17, 3)
    kept = [hostmem.empty(shape, np.int32) for _ in range(3 * hostmem.PER_BLOCK)]
    locked = hostmem._locked
    assert locked >= 3 * kept[0].nbytes
    held = next(a for a in kept if not a.flags.owndata)
    held[...] = 5
    del kept
    models[0]._release()
    assert hostmem._locked == locked
    models[1]._release()
    models[1]._release()                                         # once is enough
    if others == 0:
        assert held.nbytes <= hostmem._locked < 2 * held.nbytes and (held == 5).all()
        del held
        assert hostmem._locked == 0 and not any(hostmem._free.values())
    a = hostmem.empty(shape, np.int32)                           # and the module serves on
    a[...] = 1


@pytest.mark.parametrize("n", [40, 30000])                        # packed in one copy / in chunks
def test_device_memory_is_refused_where_host_memory_is_meant(engine_lib, n):
    import torch

    rng = np.random.default_rng(n)
    np.random.seed(1)
    graphs = random_graphs(40, rng, hv_size=20, max_nodes=3)[np.arange(n) % 40]
    gpu = EngineTM(clauses=30, classes=3, literals=40, threshold=50, s=3.0, max_nodes=3)
    gpu.set_graphs(graphs)
    gpu.prepare()
    want = gpu.score()
    dev = torch.zeros(max(n * 30, 30 * 2 * 8), dtype=torch.int32, device="cuda")
    p = C.c_void_p(dev.data_ptr())
    refused = lambda status: status == 1 and b"device memory" in engine_lib.gtm_last_error()
    assert refused(engine_lib.gtm_score(gpu.model, gpu.ds, 1, 0, n, p))
    assert refused(engine_lib.gtm_transform(gpu.model, gpu.ds, 1, 0, n, p, None))
    assert refused(engine_lib.gtm_get_ta_state(gpu.model, 0, p))
    arrays = [np.ascontiguousarray(a, dtype=np.uint32) for a in (graphs.X, graphs.node_type, graphs.number_of_graph_node_edges, graphs.edge_index,
                                                                 graphs.edge, graphs.node_index, graphs.number_of_graph_nodes)]
    copies = [torch.from_numpy(a.view(np.int32)).cuda() for a in arrays]
    names = ("X", "node_type", "number_of_graph_node_edges", "edge_index", "edge", "node_index", "number_of_graph_nodes")
    out, ds = np.zeros((n, 3), dtype=np.int32), C.c_void_p()
    for name, copy in zip(names, copies):
        v = _lib.GraphsView()
        for field, a in zip(names, arrays):
            setattr(v, field, a.ctypes.data)
        setattr(v, name, copy.data_ptr())
        v.number_of_graphs, v.total_nodes, v.total_edges, v.max_number_of_graph_nodes = n, len(arrays[0]), len(arrays[4]), 3
        assert refused(engine_lib.gtm_dataset_create(gpu.model, C.byref(v), C.byref(ds))) and not ds.value
        assert refused(engine_lib.gtm_dataset_create_scored(gpu.model, C.byref(v), 1, out.ctypes.data, C.byref(ds))) and not ds.value
    assert np.array_equal(gpu.score(), want)
    gpu.close()
