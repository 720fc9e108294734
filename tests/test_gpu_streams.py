"""GPU suite: one model, several streams.  `gtm_score_device` returns with its kernels in flight; what follows on another stream
must neither disturb them nor be disturbed by them, and no call may leave anything behind that changes a later one."""

import ctypes as C

import numpy as np
import pytest
import torch

from graphtsetlinmachine_b200 import _lib
from util import EngineTM, encode_labels, random_graphs

pytestmark = pytest.mark.gpu


def learned(depth, clauses=600, classes=7, nodes=None, max_nodes=9):
    """A model that has learned a little, and a base set of 200 graphs."""
    rng = np.random.default_rng(depth)
    np.random.seed(depth)
    base = random_graphs(200, rng, hv_size=40, max_nodes=max_nodes, fixed_nodes=nodes, max_degree=2 if depth > 1 else 0)
    hvs = np.stack([rng.choice(64, size=2, replace=False) for _ in range(clauses)]).astype(np.uint32)
    tm = EngineTM(clauses=clauses, classes=classes, literals=80, threshold=50, s=3.0, depth=depth, message_size=64, max_nodes=max_nodes,
                  hypervectors=hvs, seed=3)
    tm.set_graphs(base)
    tm.prepare()
    tm.fit(encode_labels(rng.integers(0, classes, size=200), classes, 50))
    return tm, base


def resident(tm, graphs):
    """A set of the model's beside the one it has: (handle, expected sums)."""
    tm.ds, keep = C.c_void_p(), (tm.ds, tm.graphs, tm.number_of_graphs)
    tm.set_graphs(graphs)
    want = tm.score()
    ds = tm.ds
    tm.ds, tm.graphs, tm.number_of_graphs = keep
    return ds, want


def queue(tm, ds, stream, out):
    _lib.check(tm.lib.gtm_set_stream(tm.model, C.c_void_p(stream.cuda_stream)))
    _lib.check(tm.lib.gtm_score_device(tm.model, ds, tm.n_types, 0, out.shape[0], C.c_void_p(out.data_ptr())))


def sums(n, tm):
    return torch.full((n, tm.K), -77, dtype=torch.int32, device="cuda")


@pytest.mark.parametrize("depth,nodes", [(1, 1), (1, None), (2, 4), (3, None)])
def test_two_sets_on_two_streams(engine_lib, depth, nodes):
    """Launches in flight on two streams at the same time, more tiles than thread blocks in both; then one call after."""
    tm, base = learned(depth, nodes=nodes)
    sets = [resident(tm, base[(np.arange(n) * 7 + n) % 200]) for n in (60000, 45000)]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    outs = [sums(len(want), tm) for _, want in sets]
    torch.cuda.synchronize()
    for _ in range(3):
        for (ds, _), stream, out in zip(sets, streams, outs):
            queue(tm, ds, stream, out)
        torch.cuda.synchronize()
        for (_, want), out in zip(sets, outs):
            assert np.array_equal(out.cpu().numpy(), want)
            out.fill_(-77)
        torch.cuda.synchronize()
    small, want = resident(tm, base[:50])
    out = sums(50, tm)
    torch.cuda.synchronize()
    queue(tm, small, streams[0], out)
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy(), want)
    for ds in (small, sets[0][0], sets[1][0]):
        tm.lib.gtm_dataset_destroy(ds)
    tm.close()


@pytest.mark.parametrize("depth", [1, 2])
def test_captured_launch(engine_lib, depth):
    """A launch recorded into a CUDA graph replays correctly between and after launches on larger sets."""
    tm, base = learned(depth)
    ds, want = resident(tm, base[np.arange(3000) % 200])
    out, stream = sums(3000, tm), torch.cuda.Stream()
    torch.cuda.synchronize()
    queue(tm, ds, stream, out)                                     # lists and kernels are there before the capture
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        queue(tm, ds, stream, out)
    other, other_want = resident(tm, base[np.arange(20000) % 200])
    other_out = sums(20000, tm)
    for _ in range(2):
        out.fill_(-77)
        torch.cuda.synchronize()
        graph.replay()
        queue(tm, other, stream, other_out)
        torch.cuda.synchronize()
        assert np.array_equal(out.cpu().numpy(), want) and np.array_equal(other_out.cpu().numpy(), other_want)
    tm.lib.gtm_dataset_destroy(other)
    out.fill_(-77)
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy(), want)
    del graph
    tm.lib.gtm_dataset_destroy(ds)
    tm.close()


@pytest.mark.parametrize("depth", [1, 2])
def test_lists_of_one_stream_on_the_next(engine_lib, depth):
    """The first launch after new automata makes the literal lists; a launch on another stream right behind it waits for them.
    Later automata on a third stream leave launches in flight alone."""
    tm, base = learned(depth, clauses=4000)
    large, _ = resident(tm, base[np.arange(40000) % 200])
    small, old_want = resident(tm, base[:100])
    planes = [tm.get_ta(d) for d in range(depth)]
    streams = [torch.cuda.Stream() for _ in range(3)]
    out_large, out_small, out_last = sums(40000, tm), sums(100, tm), sums(100, tm)
    for turn in range(4):
        changed = turn % 2 == 0                            # include planes shifted by a clause, then as they were
        for d, p in enumerate(planes):
            tm.set_ta(d, np.roll(p, 1, axis=0) if changed else p)
        queue(tm, large, streams[0], out_large)
        queue(tm, small, streams[1], out_small)
        queue(tm, small, streams[2], out_last)
        torch.cuda.synchronize()
        got = out_small.cpu().numpy()
        tm.ds, keep = small, tm.ds
        want = tm.score(0, 100)
        tm.ds = keep
        assert np.array_equal(got, want) and np.array_equal(out_last.cpu().numpy(), want)
        assert np.array_equal(out_large.cpu().numpy()[:100], want)
        assert changed or np.array_equal(want, old_want)
    for ds in (large, small):
        tm.lib.gtm_dataset_destroy(ds)
    tm.close()


@pytest.mark.parametrize("depth,max_nodes", [(1, 9), (2, 9)])
def test_set_destroyed_behind_its_launch(engine_lib, depth, max_nodes):
    """A set of ragged graphs, made on one stream, scored on another and destroyed at once: its tile tables outlive the launch,
    although the next set is made on the first stream in the memory that became free."""
    tm, base = learned(depth, clauses=3000, max_nodes=max_nodes)
    first, second = torch.cuda.Stream(), torch.cuda.Stream()
    order = [(np.arange(30000) * 13 + k) % 200 for k in range(2)]
    want = resident(tm, base)[1]
    outs = [sums(30000, tm) for _ in order]
    torch.cuda.synchronize()
    for _ in range(3):
        for k, out in zip(order, outs):
            _lib.check(tm.lib.gtm_set_stream(tm.model, C.c_void_p(first.cuda_stream)))
            tm.ds, keep = C.c_void_p(), (tm.ds, tm.graphs, tm.number_of_graphs)
            tm.set_graphs(base[k])
            ds = tm.ds
            tm.ds, tm.graphs, tm.number_of_graphs = keep
            queue(tm, ds, second, out)
            tm.lib.gtm_dataset_destroy(ds)
        torch.cuda.synchronize()
        for k, out in zip(order, outs):
            assert np.array_equal(out.cpu().numpy(), want[k])
            out.fill_(-77)
        torch.cuda.synchronize()
    tm.close()
