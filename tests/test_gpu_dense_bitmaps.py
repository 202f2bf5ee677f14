"""Dense lists counted from bitmaps: bag rows that list an object several times
(one bitmap row a listing, up to the 16 a list may have and past them), more
rows than a chunk holds, object counts around a vector and a tile, and whole queries
a part, against the oracle.  Whole numbers and fixed-point sums."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _bag(rng, n, terms, repeat):
    length = rng.integers(3, 9, n)
    off = np.concatenate([[0], np.cumsum(length)]).astype(np.int64)
    values = rng.integers(0, terms, off[-1]).astype(np.int32)
    heavy = rng.integers(0, n, 200)          # rows of one term, listed up to `repeat` times
    extra = [np.full(int(rng.integers(2, repeat + 1)), int(rng.integers(0, terms)), np.int32) for _ in heavy]
    rows = [values[off[i]:off[i + 1]] for i in range(n)]
    for r, x in zip(heavy, extra):
        rows[r] = x
    off = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int64)
    return np.concatenate(rows), off


@pytest.mark.parametrize("n", [65_536, 65_569, 150_001])
@pytest.mark.parametrize("repeat", [5, 16, 20])
def test_bag(genie, oracle, n, repeat):
    rng = np.random.default_rng(n + repeat)
    values, off = _bag(rng, n, 40, repeat)
    t = genie.Table.from_bag_arrays(values, off)
    ox = oracle.Index(bag=(values, off))
    q, ms = 12, [1, 5, 12, 40, 300, 700]
    m = np.array([ms[i % 6] for i in range(q)])
    o = np.concatenate([[0], np.cumsum(m)]).astype(np.int64)
    low = rng.integers(0, 40, o[-1]).astype(np.int32)
    qb = genie.QueryBatch(o, np.zeros(o[-1], np.int32), low, low, np.array([10, 100, 33] * 4, np.uint32))
    expect = ox.search(qb.as_oracle_batch())
    # 4-byte counters when the items may add up to more than 255, also from bitmaps with 2 and 3
    for tuning in (dict(dense_bitmaps=1), dict(dense_bitmaps=3), dict(dense_bitmaps=-1), dict(dense_bitmaps=3, dense_tile=40192)):
        b = genie.Batch(t, q, int(o[-1]), 100, max_units=int(4 * o[-1]))
        b.set_tuning(sparse_max_total=1, bitmap_bits=-1, **tuning)
        ids, cnt = b.run(qb)
        assert np.array_equal(cnt, expect[1]) and np.array_equal(ids, expect[0]), tuning


@pytest.mark.parametrize("n", [131_072, 147_457, 300_011])
@pytest.mark.parametrize("codec", [0, 13])
def test_wide_valued_tables(genie, oracle, n, codec):
    """Dims of more than 256 values (no planes): common values from bitmaps, the
    others from ids or segments; few and many queries (parts of one tile, and
    whole queries)."""
    from genie_gb300 import workloads
    rng = np.random.default_rng(n)
    values = workloads.zipf_ranks(rng, (n, 12), n_terms=3000)
    t = genie.Table.compressed(values, codec, 128) if codec else genie.Table.from_values(values)
    ox = oracle.Index(values)
    for q in (3, 700):
        low = workloads.zipf_ranks(rng, (q, 12), n_terms=3000).ravel()
        qb = genie.QueryBatch(np.arange(q + 1) * 12, np.tile(np.arange(12), q), low, low + (np.arange(q * 12) % 7 == 0), 20)
        expect = ox.search(qb.as_oracle_batch())
        b = genie.Batch(t, q, q * 12, 20)
        b.set_tuning(sparse_max_total=1, bitmap_bits=-1)
        ids, cnt = b.run(qb)
        assert np.array_equal(cnt, expect[1]) and np.array_equal(ids, expect[0])
