"""One batch handle, and several threads, across the building of a table's
planes: unweighted, weighted and long queries in turn, exact at every step."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N, D, WIDTH = 40_000, 32, 50


@pytest.fixture(scope="module")
def world(genie, oracle):
    rng = np.random.default_rng(21)
    values = rng.integers(0, WIDTH, size=(N, D)).astype(np.int32)
    values[0], values[1] = 0, WIDTH - 1
    ox = oracle.Index(values)
    batches = []
    for m, weighted, spread in ((20, False, 12), (20, True, 12), (300, False, 3), (2, False, 0), (20, False, 12), (9, True, 20)):
        q = 24
        dim = rng.integers(0, D, q * m).astype(np.int32)
        centre = rng.integers(0, WIDTH, q * m).astype(np.int32)
        w = rng.uniform(0.5, 2.0, q * m).astype(np.float32) if weighted else None
        qb = genie.QueryBatch(np.arange(q + 1) * m, dim, centre - spread, centre + spread, 10, w,
                              np.ones(q, np.uint8) if weighted else None)
        batches.append((qb, ox.search(qb.as_oracle_batch())))
    wide = genie.QueryBatch(np.arange(61) * D, np.tile(np.arange(D), 60), np.zeros(60 * D, np.int32),
                            np.full(60 * D, WIDTH, np.int32), 1)
    return values, batches, wide


def _same(got, expect):
    return all(np.array_equal(x, y) for x, y in zip(got, expect))


@pytest.mark.parametrize("graph", [False, True])
def test_one_handle(genie, world, graph):
    values, batches, wide = world
    table = genie.Table.from_values(values)
    b = genie.Batch(table, 24, 24 * 300, 10, use_graph=graph, max_units=24 * 300 * 16)
    for step in range(4):
        for qb, expect in batches:
            assert _same(b.run(qb, scores=True), expect)
            assert _same(genie.search(table, qb, scores=True), expect)
        if step == 1:
            genie.search(table, wide)      # the planes are there from now on


def test_threads(genie, world):
    values, batches, wide = world
    table = genie.Table.from_values(values)
    before = table.info().device_bytes
    wrong = []

    def work(i):
        try:
            b = genie.Batch(table, 24, 24 * 300, 10, max_units=24 * 300 * 16)
            for r in range(30):
                qb, expect = batches[(i + r) % len(batches)]
                got = b.run(qb, scores=True) if (i + r) % 2 else genie.search(table, qb, scores=True)
                if not _same(got, expect):
                    wrong.append((i, r))
                if i == 0 and r in (5, 6, 7):
                    genie.search(table, wide)
        except BaseException as e:      # noqa: BLE001
            wrong.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong
    table._info = None
    assert table.info().device_bytes > before
