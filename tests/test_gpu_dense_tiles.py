"""The largest counter tiles that a batch accepts (they leave no room for the
starts of the lists) and the first that it refuses."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile", [173_568, 173_824, 177_664])
@pytest.mark.parametrize("weighted", [False, True])
def test_largest_tiles(genie, oracle, tile, weighted):
    rng = np.random.default_rng(tile)
    n, d, q = 400_000, 6, 5
    values = rng.integers(0, 900, size=(n, d)).astype(np.int32)       # more values than planes hold
    table = genie.Table.from_values(values)
    low = rng.integers(0, 900, q * d).astype(np.int32)
    w = rng.uniform(0.5, 2, q * d).astype(np.float32) if weighted else None
    qb = genie.QueryBatch(np.arange(q + 1) * d, np.tile(np.arange(d), q), low, low + 40, 50, w,
                          np.ones(q, np.uint8) if weighted else None)
    expect = oracle.Index(values).search(qb.as_oracle_batch())
    b = genie.Batch(table, q, q * d, 50, max_units=q * d * 42)
    b.set_tuning(dense_tile=tile, sparse_max_total=1, bitmap_bits=-1, dense_part_work=2 * tile)
    ids, counts = b.run(qb)
    assert np.array_equal(counts, expect[1]) and np.array_equal(ids, expect[0])


def test_a_larger_tile_is_refused(genie):
    table = genie.Table.from_values(np.arange(4096, dtype=np.int32).reshape(-1, 2))
    b = genie.Batch(table, 1, 2, 1)
    with pytest.raises(Exception):
        b.set_tuning(dense_tile=177_920)
    assert b.tuning()["dense_tile"] == 147_456


@pytest.mark.parametrize("tile", [40_192, 40_448])
def test_four_byte_tiles_of_an_odd_number_of_words(genie, oracle, tile):
    """4-byte tiles (10,048 and 10,112 objects) that are no multiple of 128
    objects, or are, count dense lists from their bitmaps alike."""
    rng = np.random.default_rng(tile)
    n, d, q = 90_001, 5, 6
    values = rng.integers(0, 300, size=(n, d)).astype(np.int32)       # more values than planes hold
    values[rng.random((n, d)) < 0.3] = 7                               # and a list that has a bitmap in every dim
    table = genie.Table.from_values(values)
    low = np.where(np.arange(q * d) % 2, 7, rng.integers(0, 300, q * d)).astype(np.int32)
    qb = genie.QueryBatch(np.arange(q + 1) * d, np.tile(np.arange(d), q), low, low + 5, 100,
                          rng.uniform(0.5, 2, q * d).astype(np.float32), np.ones(q, np.uint8))
    expect = oracle.Index(values).search(qb.as_oracle_batch())
    b = genie.Batch(table, q, q * d, 100, max_units=q * d * 8)
    b.set_tuning(dense_tile=tile, sparse_max_total=1, bitmap_bits=-1, dense_bitmaps=3)
    ids, counts, scores = b.run(qb, scores=True)
    assert np.array_equal(ids, expect[0]) and np.array_equal(counts, expect[1]) and np.array_equal(scores, expect[2])
