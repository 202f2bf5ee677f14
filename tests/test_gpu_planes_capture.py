"""A launch that the caller captured into a graph of its own answers whatever is
staged later: weighted queries after unweighted ones, queries of more items
than the planes take, and batches staged after the table's planes were built
although the capture is older."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N, D = 30_000, 40


def _queries(genie, rng, values, m, weighted):
    q = 8
    dim = np.concatenate([rng.choice(D, m, replace=m > D) for _ in range(q)]).astype(np.int32)
    centre = values[np.repeat(rng.integers(0, N, q), m), dim]
    r = rng.integers(0, 3, q * m)
    w = rng.uniform(0.5, 2.0, q * m).astype(np.float32) if weighted else None
    return genie.QueryBatch(np.arange(q + 1) * m, dim, (centre - r).astype(np.int32), (centre + r).astype(np.int32), 10, w,
                            np.ones(q, np.uint8) if weighted else None)


def _build_planes(genie, table):
    wide = genie.QueryBatch(np.arange(61) * D, np.tile(np.arange(D), 60), np.zeros(60 * D, np.int32),
                            np.full(60 * D, 49, np.int32), 1)
    genie.search(table, wide)


@pytest.mark.parametrize("planes_first", [False, True])
def test_captured_launch(genie, oracle, planes_first):
    import torch
    rng = np.random.default_rng(4)
    values = rng.integers(0, 50, size=(N, D)).astype(np.int32)
    values[0], values[1] = 0, 49
    table = genie.Table.from_values(values)
    ox = oracle.Index(values)
    if planes_first:
        _build_planes(genie, table)
    batches = [_queries(genie, rng, values, m, w) for m, w in ((20, False), (20, True), (300, False), (20, False))]
    b = genie.Batch(table, 8, 8 * 300, 10, use_graph=False, max_units=16 * 8 * 300)
    stream = torch.cuda.Stream()
    b.stage(batches[0])
    b.launch(stream.cuda_stream)              # directories and bitmaps are there before the capture
    stream.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
        b.launch(torch.cuda.current_stream().cuda_stream)
    if not planes_first:
        _build_planes(genie, table)
    ids, counts = np.zeros(80, np.uint32), np.zeros(80, np.uint32)
    for qb in batches:
        b.stage(qb)
        graph.replay()
        torch.cuda.synchronize()
        assert genie.lib().genie_batch_fetch(b._h, ids.ctypes.data, counts.ctypes.data, ctypes.c_void_p()) == 0
        expect = ox.search(qb.as_oracle_batch())
        assert np.array_equal(counts, expect[1]) and np.array_equal(ids, expect[0])
