"""Byte-valued tables counted from their cumulative planes, against the
oracle: object counts around a vector and a tile, item counts around the
eight-item groups and the 255-item limit, every k class, ties, weights, and a
query whose keys outgrow its region.  Whole numbers and fixed-point sums, so
every comparison is exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _queries(genie, rng, n, d, q, m_of, k_of, values, weights, spread):
    off = np.zeros(q + 1, np.int64)
    m = np.array([m_of(i) for i in range(q)])
    off[1:] = np.cumsum(m)
    dim = np.concatenate([rng.choice(d, x, replace=x > d) for x in m]).astype(np.int32)
    row = np.repeat(rng.integers(0, n, q), m)
    centre = values[row, dim]
    r = np.repeat(rng.integers(0, spread + 1, q), m)
    low, up = centre - r, centre + r
    low[::17] = values.max() + 1          # matches nothing
    up[5::23] = 1 << 20                   # open above, and every object when low <= min
    low[9::29] = -5
    dim[11::31] = d + 3                   # no such dim
    w = wf = None
    if weights:
        w = rng.uniform(0.01, 3.0, off[-1]).astype(np.float32)
        w[3::7] = w[0]
        wf = np.ones(q, np.uint8) if weights == "all" else (np.arange(q) % 2).astype(np.uint8)
    return genie.QueryBatch(off, dim, low.astype(np.int32), up.astype(np.int32),
                            np.array([k_of(i) for i in range(q)], np.uint32), w, wf)


def _check(genie, oracle, values, qb, batch=False):
    """Every pass of enough to have the planes built (they are, once the
    searches have touched four times their bytes) and used."""
    from genie_gb300 import workloads
    t = genie.Table.from_values(values)
    lay = t.layout()
    n = len(values)
    row = 2048 * -(-n // 16384) if n > 16384 else 16 * -(-n // 128)
    touched = workloads.algorithmic_bytes(lay["key_offsets"], lay["key_base"], lay["dim_min"], lay["dim_max"],
                                          qb.as_oracle_batch())
    passes = 3 + int(4 * row * (len(lay["key_offsets"]) + 1) / max(1, touched))
    assert passes < 2000
    oid, ocnt, osc, _ = oracle.Index(values).search(qb.as_oracle_batch())
    b = genie.Batch(t, qb.n_queries, len(qb.dim), int(qb.k_array.max())) if batch else None
    for _ in range(passes):
        ids, cnt, sc = b.run(qb, scores=True) if batch else genie.search(t, qb, scores=True)
        assert np.array_equal(cnt, ocnt) and np.array_equal(ids, oid) and np.array_equal(sc, osc)


@pytest.mark.parametrize("n", [1, 31, 127, 129, 1000, 16383, 16384, 16385, 50_001])
@pytest.mark.parametrize("weights", ["", "all"])
def test_sizes(genie, oracle, n, weights):
    rng = np.random.default_rng(n)
    values = rng.integers(0, 40, size=(n, 24)).astype(np.int32)
    values[n // 2] = 39
    values[0, 1:] = 0
    ms = [1, 7, 8, 9, 16, 17, 24, 3]
    ks = [1, 10, 100, 300, 512, 16, 64, 5]
    qb = _queries(genie, rng, n, 24, 16, lambda i: ms[i % 8], lambda i: ks[(i * 3) % 8], values, weights, 4)
    _check(genie, oracle, values, qb, batch=bool(n % 2))


@pytest.mark.parametrize("m", [254, 255, 256])
@pytest.mark.parametrize("span", [2, 256, 257])
def test_item_and_value_limits(genie, oracle, m, span):
    """255 items are the most of the planes (256 take the counter tiles), and
    256 values a dim (257 keep the table on its lists)."""
    rng = np.random.default_rng(m + span)
    values = rng.integers(0, span, size=(20_000, 40)).astype(np.int32) - 7
    values[0], values[1] = -7, span - 8
    qb = _queries(genie, rng, 20_000, 40, 6, lambda i: m, lambda i: [2048, 10, 50][i % 3], values, "half", span // 3)
    _check(genie, oracle, values, qb)


def test_uneven_weights(genie, oracle):
    """Weights over many orders of magnitude, equal ones, and k at its limits."""
    rng = np.random.default_rng(3)
    values = rng.integers(0, 30, size=(70_000, 60)).astype(np.int32)
    qb = _queries(genie, rng, 70_000, 60, 12, lambda i: [5, 60, 33][i % 3], lambda i: [512, 513, 1, 200][i % 4], values,
                  "all", 3)
    w = qb.weight
    w[: len(w) // 2] = (10.0 ** rng.uniform(-9, 3, len(w) // 2)).astype(np.float32)
    w[len(w) // 2: len(w) // 2 + 100] = 1.0
    _check(genie, oracle, values, qb)


def test_more_ties_than_a_region_holds(genie, oracle):
    """Each tile holds fewer than k objects of one count, all tiles together
    far more than the query's region: redone with compaction, smallest ids."""
    rng = np.random.default_rng(5)
    n, q, k = 2_000_000, 256, 100
    values = rng.integers(0, 200, size=(n, 2)).astype(np.int32)
    off = np.arange(q + 1, dtype=np.int64)
    low = rng.integers(0, 200, q).astype(np.int32)
    w = np.full(q, 1.5, np.float32)
    for wf in (None, np.ones(q, np.uint8)):
        qb = genie.QueryBatch(off, np.zeros(q, np.int32), low, low, np.full(q, k, np.uint32), w, wf)
        _check(genie, oracle, values, qb, batch=True)


@pytest.mark.parametrize("n,k", [(20_000, 128), (20_000, 129), (131_072, 512), (131_071, 512), (131_072, 513)])
@pytest.mark.parametrize("m", [12, 48, 49, 90])
def test_weighted_k_and_many_candidates(genie, oracle, n, k, m):
    """The k up to which weighted queries take the planes, and tiles whose many
    candidates are summed a thread each (up to 48 items) or a warp four."""
    rng = np.random.default_rng(n + k + m)
    values = rng.integers(0, 25, size=(n, 90)).astype(np.int32)
    qb = _queries(genie, rng, n, 90, 10, lambda i: m, lambda i: k, values, "half", 3)
    _check(genie, oracle, values, qb)


@pytest.mark.parametrize("n", [1, 128, 129, 300, 4096, 8192, 8193])
def test_small_tables_split_their_items(genie, oracle, n):
    """Rows shorter than a block: runs of its threads count a part of the items
    each (1 to 128 runs, some without items)."""
    rng = np.random.default_rng(n)
    values = rng.integers(0, 20, size=(n, 60)).astype(np.int32)
    values[-1] = 19
    ms = [1, 8, 9, 60, 128, 129, 254, 255]
    qb = _queries(genie, rng, n, 60, 16, lambda i: ms[i % 8], lambda i: [1, 10, 100, 2048][i % 4], values, "", 4)
    _check(genie, oracle, values, qb, batch=bool(n % 2))
