"""Which kernels a search launches: the planes of a byte-valued table, built and
used when and only when they should be.  A table of one tile shows it by the
launches of an unweighted batch: the plan and one planes kernel, against the
plan and the three list kernels."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PLANES, LISTS = 2, 4


def _table(genie, n=5_000, d=24, width=60, seed=1):
    values = np.random.default_rng(seed).integers(0, width, size=(n, d)).astype(np.int32)
    values[0], values[1] = 0, width - 1
    return genie.Table.from_values(values), values


def _exact(genie, values, q, m, k=10, seed=2, weighted=False):
    rng = np.random.default_rng(seed)
    n, d = values.shape
    dim = np.concatenate([rng.choice(d, m, replace=m > d) for _ in range(q)]).astype(np.int32)
    low = values[np.repeat(rng.integers(0, n, q), m), dim]
    w = rng.uniform(0.5, 2.0, q * m).astype(np.float32) if weighted else None
    return genie.QueryBatch(np.arange(q + 1) * m, dim, low, low, k, w, np.ones(q, np.uint8) if weighted else None)


def _wide(genie, table, times=1):
    """Searches that touch `times` as many posting ids as the planes have bytes."""
    lay = table.layout()
    d, n = len(lay["dim_min"]), table.info().n_objects
    tiles = -(-n // 16384)
    row = 2048 if tiles > 1 else 16 * -(-n // 128)
    q = 1 + int(times * tiles * row * (len(lay["key_offsets"]) + 1) / (n * d))
    lo, up = int(lay["dim_min"].min()), int(lay["dim_max"].max())
    return genie.QueryBatch(np.arange(q + 1) * d, np.tile(np.arange(d), q), np.full(q * d, lo), np.full(q * d, up), 1)


def test_searches_off_the_planes_do_not_build_them(genie):
    table, values = _table(genie)
    wide, few = _wide(genie, table, 3), _exact(genie, values, 1, 2)
    off = genie.Batch(table, wide.n_queries, len(wide.dim), 1, max_units=len(wide.dim) * 61)
    off.set_tuning(dense_bitmaps=-1)
    off.run(wide)
    on = genie.Batch(table, 1, 2, 10)
    on.run(few)
    assert on.last_stats()[0] == LISTS
    genie.search(table, wide)
    on.run(few)
    assert on.last_stats()[0] == PLANES
    off.run(wide)
    assert off.last_stats()[0] == LISTS


@pytest.mark.parametrize("weighted", [False, True])
def test_autotuning_keeps_the_planes(genie, weighted):
    """Tuned before the planes exist, a batch uses them when they do."""
    table, values = _table(genie)
    sample = _exact(genie, values, 4, 3, weighted=weighted)
    b = genie.Batch(table, 4, 12, 10)
    assert b.autotune(sample)["dense_bitmaps"] > 0
    genie.search(table, _wide(genie, table))
    b.run(sample)
    assert b.last_stats()[0] == PLANES


def test_planes_are_given_back_to_a_failing_allocation(genie, oracle):
    """An allocation that finds the device full takes the planes back, the
    searches go on from the lists and earn them again; the planes that a launch
    captured by its caller reads stay."""
    import torch
    table, values = _table(genie)
    wide, few = _wide(genie, table), _exact(genie, values, 3, 12)
    expect = oracle.Index(values).search(few.as_oracle_batch())
    before = genie.Table.info(table).device_bytes
    b = genie.Batch(table, 3, 36, 10, use_graph=False)

    def run():
        ids, counts = b.run(few)
        assert np.array_equal(counts, expect[1]) and np.array_equal(ids, expect[0])
        return b.last_stats()[0]

    def too_much():      # part results of half a terabyte
        with pytest.raises(genie.gpu_bad_alloc):
            genie.Batch(table, 1 << 19, 16, 2048)

    def held():
        table._info = None
        return table.info().device_bytes - before

    assert run() == LISTS and held() == 0
    genie.search(table, wide)
    assert run() == PLANES and held() > 0
    too_much()
    assert held() == 0 and run() == LISTS
    genie.search(table, wide)
    assert run() == PLANES and held() > 0
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
        b.launch(torch.cuda.current_stream().cuda_stream)
    too_much()
    assert held() > 0 and run() == PLANES
