"""Tables of several tiles: the merge of many tiles' keys.  Every result is a
whole number and compared exactly."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PLANES = 3        # launches: plan, tiles, merge


def _ready(genie, values):
    """A table with its planes built."""
    t = genie.Table.from_values(values)
    n, d = values.shape
    lo, up = int(values.min()), int(values.max())
    q = 2 + -(-n // 16384) * 2048 * (len(t.layout()["key_offsets"]) + 1) // (n * d)
    genie.search(t, genie.QueryBatch(np.arange(q + 1) * d, np.tile(np.arange(d), q), np.full(q * d, lo), np.full(q * d, up), 1))
    return t


def _batch(genie, rng, q, m, d, low, up, k, weighted):
    w = rng.uniform(0.5, 2.0, q * m).astype(np.float32) if weighted else None
    dim = np.concatenate([rng.permutation(d)[:m] for _ in range(q)])
    return genie.QueryBatch(np.arange(q + 1) * m, dim, low, up, k, w, np.ones(q, np.uint8) if weighted else None)


@pytest.mark.parametrize("k", [500, 1024, 1025, 2048])
@pytest.mark.parametrize("n", [400_000, 700_001])
def test_merge_of_many_keys(genie, oracle, n, k):
    """A query alone: all its tiles write k keys each, most of them tied, far
    more than the merge's buffer holds at once (beyond k = 1,024 it selects)."""
    rng = np.random.default_rng(n + k)
    values = rng.integers(0, 9, size=(n, 8)).astype(np.int32)
    table = _ready(genie, values)
    low = rng.integers(0, 7, 8)
    qb = _batch(genie, rng, 1, 8, 8, low, low + 2, k, False)
    expect = oracle.Index(values).search(qb.as_oracle_batch())
    got = genie.search(table, qb)
    assert np.array_equal(got[1], expect[1]) and np.array_equal(got[0], expect[0])


def test_more_keys_than_the_largest_regions(genie, oracle):
    """Ties in every tile of a batch whose keys do not all fit: the queries are
    counted again, tile by tile."""
    rng = np.random.default_rng(5)
    n, q, k = 2_000_000, 2600, 400
    values = rng.integers(0, 50, size=(n, 2)).astype(np.int32)
    table = _ready(genie, values)
    qb = genie.QueryBatch(np.arange(q + 1), np.zeros(q, np.int32), np.arange(q) % 40, np.arange(q) % 40, k)
    expect = oracle.Index(values).search(genie.QueryBatch(np.arange(41), np.zeros(40, np.int32), np.arange(40),
                                                          np.arange(40), k).as_oracle_batch())
    b = genie.Batch(table, q, q, k)
    ids, counts = b.run(qb)
    assert b.last_stats()[0] == PLANES
    at = np.arange(q) % 40
    assert np.array_equal(ids.reshape(q, k), expect[0].reshape(40, k)[at])
    assert np.array_equal(counts.reshape(q, k), expect[1].reshape(40, k)[at])


@pytest.mark.parametrize("weighted", [False, True])
def test_ties_below_k_in_every_tile(genie, oracle, weighted):
    """420 objects of one value a tile, 512 wanted: no tile alone bounds the
    query, and all 123 write more keys than its region holds."""
    rng = np.random.default_rng(6)
    n, q, k, v = 2_000_000, 2100, 512, 39
    values = rng.integers(0, v, size=(n, 2)).astype(np.int32)
    table = _ready(genie, values)
    at = np.arange(q) % v
    w = np.full(q, 1.5, np.float32) if weighted else None
    wf = np.ones(q, np.uint8) if weighted else None
    few = slice(0, v)
    qb = genie.QueryBatch(np.arange(q + 1), np.zeros(q, np.int32), at, at, k, w, wf)
    one = genie.QueryBatch(np.arange(v + 1), np.zeros(v, np.int32), at[few], at[few], k, None if w is None else w[few],
                           None if wf is None else wf[few])
    expect = oracle.Index(values).search(one.as_oracle_batch())
    b = genie.Batch(table, q, q, k)
    got = b.run(qb, scores=True)
    assert b.last_stats()[0] == PLANES
    for x, y in zip(got, expect):
        assert np.array_equal(x.reshape(q, k), y.reshape(v, k)[at])
