"""Tables of several tiles: which way a batch is counted (planes, lists, or each
query its own way), by its launches.  Results are whole numbers and fixed-point
sums, compared exactly."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PLANES, LISTS, BOTH = 3, 4, 6        # plan, tiles, merge; plan and three list kernels; all of them


def _ready(genie, values):
    """A table with its planes built."""
    t = genie.Table.from_values(values)
    n, d = values.shape
    lo, up = int(values.min()), int(values.max())
    q = 2 + -(-n // 16384) * 2048 * (len(t.layout()["key_offsets"]) + 1) // (n * d)
    genie.search(t, genie.QueryBatch(np.arange(q + 1) * d, np.tile(np.arange(d), q), np.full(q * d, lo), np.full(q * d, up), 1))
    return t


def _run(genie, oracle, table, values, qb, direct=False):
    expect = oracle.Index(values).search(qb.as_oracle_batch())
    b = genie.Batch(table, qb.n_queries, len(qb.dim), int(qb.k_array.max()), use_graph=not direct,
                    max_units=64 * len(qb.dim))
    for got in (b.run(qb, scores=True), genie.search(table, qb, scores=True)):
        for x, y in zip(got, expect):
            assert np.array_equal(x, y)
    return b.last_stats()[0]


def _table(rng, n, d, rare):
    """Values below `rare` are common, the others are listed a few times each."""
    values = rng.integers(0, rare, size=(n, d)).astype(np.int32)
    for j in range(d):
        values[rng.choice(n, 200, replace=False), j] = rare + rng.integers(0, 8, 200)
    return values


def _batch(genie, rng, q, m, d, low, up, k, weighted):
    w = rng.uniform(0.5, 2.0, q * m).astype(np.float32) if weighted else None
    dim = np.concatenate([rng.permutation(d)[:m] for _ in range(q)])
    return genie.QueryBatch(np.arange(q + 1) * m, dim, low, up, k, w, np.ones(q, np.uint8) if weighted else None)


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("n", [16385, 100_001])
def test_batches_go_the_cheaper_way(genie, oracle, n, weighted):
    rng = np.random.default_rng(n)
    values = _table(rng, n, 12, 12)
    table = _ready(genie, values)
    q, m = 40, 12
    low = rng.integers(12, 20, q * m)
    few = _batch(genie, rng, q, m, 12, low, low, 10, weighted)
    assert _run(genie, oracle, table, values, few) == LISTS
    low = rng.integers(0, 8, q * m)
    many = _batch(genie, rng, q, m, 12, low, low + 3, 10, weighted)
    assert _run(genie, oracle, table, values, many) == PLANES


def test_many_results_of_few_queries(genie, oracle):
    """512 results of two weighted queries of eight items: on planes every tile
    would sum its candidates before any bound is known."""
    rng = np.random.default_rng(7)
    values = rng.integers(0, 30, size=(200_000, 16)).astype(np.int32)
    table = _ready(genie, values)
    low = rng.integers(0, 26, 16)
    assert _run(genie, oracle, table, values, _batch(genie, rng, 2, 8, 16, low, low + 3, 512, True)) == LISTS
    assert _run(genie, oracle, table, values, _batch(genie, rng, 2, 8, 16, low, low + 3, 10, True)) == PLANES


@pytest.mark.parametrize("weighted", [False, True])
def test_unlike_queries_each_their_own_way(genie, oracle, weighted):
    """Half of a large batch touches a few ids a query, half a third of the
    table an item: 1,500 queries of rare values would take 25 tiles each."""
    rng = np.random.default_rng(11)
    n, d, q, m = 400_000, 6, 3000, 6
    values = _table(rng, n, d, 10)
    table = _ready(genie, values)
    low = rng.integers(10, 18, (q, m))
    low[::2] = rng.integers(0, 3, (q, m))[::2]
    up = low.copy()
    up[::2] += 2
    assert _run(genie, oracle, table, values, _batch(genie, rng, q, m, d, low.ravel(), up.ravel(), 5, weighted)) == BOTH


@pytest.mark.parametrize("n", [16385, 50_001, 98_304])
@pytest.mark.parametrize("weights", ["", "half", "all"])
def test_counts_of_several_tiles_on_planes(genie, oracle, n, weights):
    """Items of up to half the values, and ones that match nothing or all."""
    from test_gpu_planes import _queries
    rng = np.random.default_rng(n)
    values = rng.integers(0, 40, size=(n, 24)).astype(np.int32)
    values[0], values[1] = 0, 39
    table = _ready(genie, values)
    ms, ks = [1, 7, 8, 9, 16, 17, 24, 80], [1, 10, 64, 33]
    qb = _queries(genie, rng, n, 24, 64, lambda i: ms[i % 8], lambda i: ks[(i * 3) % 4], values, weights, 20)
    assert _run(genie, oracle, table, values, qb) == (PLANES + 1 if weights == "half" else PLANES)


def _one_tile(genie, rng, n, d, span):
    values = rng.integers(0, span, size=(n, d)).astype(np.int32)
    values[0], values[1] = 0, span - 1
    return values, _ready(genie, values)


@pytest.mark.parametrize("items,span,k,weighted,launches", [
    (255, 256, 10, False, 2), (256, 256, 10, False, LISTS), (255, 257, 10, False, LISTS), (20, 256, 2048, False, 2),
    (255, 256, 128, True, 2), (256, 256, 128, True, LISTS), (20, 60, 129, True, LISTS)])
def test_limits_on_one_tile(genie, oracle, items, span, k, weighted, launches):
    """255 items, 256 values a dim and 128 weighted results (of few objects) are
    the most that the planes take."""
    rng = np.random.default_rng(items + span + k)
    values, table = _one_tile(genie, rng, 6_000, 20, span)
    low = rng.integers(0, span, 3 * items)
    w = rng.uniform(0.5, 2.0, 3 * items).astype(np.float32) if weighted else None
    qb = genie.QueryBatch(np.arange(4) * items, np.tile(np.arange(20), 3 * items)[:3 * items], low, low + 4, k, w,
                          np.ones(3, np.uint8) if weighted else None)
    assert _run(genie, oracle, table, values, qb) == launches


def test_few_queries_beside_ones_of_the_lists(genie, oracle):
    """Every other of 48 weighted queries wants more results than the planes of
    a small table give: all go by the lists, whose kernels run anyway."""
    rng = np.random.default_rng(3)
    values, table = _one_tile(genie, rng, 5_000, 24, 50)
    low = rng.integers(0, 40, 48 * 20)
    k = np.where(np.arange(48) % 2, 500, 10).astype(np.uint32)
    assert _run(genie, oracle, table, values, _batch(genie, rng, 48, 20, 24, low, low + 6, k, True)) == LISTS


@pytest.mark.parametrize("k,launches", [(512, PLANES), (513, LISTS)])
def test_most_weighted_results(genie, oracle, k, launches):
    """Of many objects 512 weighted results, for queries that touch most of them."""
    rng = np.random.default_rng(k)
    n, d, q, m = 140_000, 20, 600, 20
    values = rng.integers(0, 30, size=(n, d)).astype(np.int32)
    table = _ready(genie, values)
    low = rng.integers(0, 3, q * m)
    assert _run(genie, oracle, table, values, _batch(genie, rng, q, m, d, low, low + 24, k, True)) == launches
