"""Index files that describe valid lists no builder makes: an object that a dim
does not list, lists twice or repeats in one list, and a list past its dim's
largest value.  Searches of such a table count its lists, however often it is
searched and whatever is derived from it meanwhile."""
import struct

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _write(path, n, dims, bag=0):
    """dims: (least value, largest value, lists) of each dim."""
    lists = [np.asarray(x, np.uint32) for d in dims for x in d[2]]
    key_off = np.concatenate([[0], np.cumsum([len(x) for x in lists])]).astype(np.int64)
    key_base = np.concatenate([[0], np.cumsum([len(d[2]) for d in dims])]).astype(np.int64)
    ids = np.concatenate(lists)
    data = struct.pack("<8sIIqiiiiqqqq", b"GENIEGB3", 1, bag, n, len(dims), 1, 0, 0, len(lists), len(ids), 0, 0)
    data += np.array([d[0] for d in dims], np.int32).tobytes() + np.array([d[1] for d in dims], np.int32).tobytes()
    data += key_base.tobytes() + key_off.tobytes() + ids.tobytes()
    h = 1469598103934665603
    for b in data:
        h = (h ^ b) * 1099511628211 & 0xFFFFFFFFFFFFFFFF
    path.write_bytes(data + struct.pack("<Q", h))


def _lists(column, width):
    return [np.flatnonzero(column == v) for v in range(width)]


def _expect(n, dims, dim, low, up, off, k):
    ids, counts = [], []
    for q in range(len(off) - 1):
        c = np.zeros(n, np.int64)
        for i in range(off[q], off[q + 1]):
            mn, mx, lists = dims[dim[i]]
            for v in range(max(low[i], mn), min(up[i], mx) + 1):
                np.add.at(c, lists[v - mn], 1)
        at = np.lexsort((np.arange(n), -c))[:k]
        at = at[c[at] > 0]
        ids.append(np.pad(at, (0, k - len(at))))
        counts.append(np.pad(c[at], (0, k - len(at))))
    return np.concatenate(ids), np.concatenate(counts)


def _spoil(kind, dims):
    mn, mx, lists = dims[1]
    lists = [x.copy() for x in lists]
    if kind == "missing":
        lists[2] = lists[2][1:]
    elif kind == "twice":                  # as many ids as objects, one of them in two lists
        lists[3] = np.sort(np.append(lists[3], lists[2][0]))
        lists[4] = lists[4][1:]
    elif kind == "repeated":
        lists[2] = np.sort(np.append(lists[2], lists[2][5]))
    elif kind == "outside":
        mx -= 1
    return dims[:1] + [(mn, mx, lists)] + dims[2:]


@pytest.mark.parametrize("n,width,d", [(300, 8, 6), (20_000, 5, 3), (70_000, 30, 2)])
@pytest.mark.parametrize("kind", ["none", "missing", "twice", "repeated", "outside"])
def test_counts_of_the_lists(genie, tmp_path, n, width, d, kind):
    rng = np.random.default_rng(n)
    values = rng.integers(0, width, size=(n, d))
    dims = _spoil(kind, [(0, width - 1, _lists(values[:, j], width)) for j in range(d)])
    _write(tmp_path / "t.bin", n, dims)
    table = genie.LoadTableFromBinary(str(tmp_path / "t.bin"))
    q, m, k = 8, 2 * d, 20
    off = np.arange(q + 1) * m
    dim = np.tile(np.arange(d), 2 * q)
    low = rng.integers(0, width, q * m)
    up = low + rng.integers(0, 3, q * m)
    low[::5], up[::5] = 0, width - 1       # every value of the dim
    expect = _expect(n, dims, dim, low, up, off, k)
    qb = genie.QueryBatch(off, dim.astype(np.int32), low.astype(np.int32), up.astype(np.int32), k)
    bt = genie.Batch(table, q, q * m, k)
    lists = genie.Batch(table, q, q * m, k)
    lists.set_tuning(sparse_max_total=1, bitmap_bits=-1)
    for _ in range(6):                     # a sound table of these sizes has its planes by then
        for ids, counts in (genie.search(table, qb), bt.run(qb), lists.run(qb)):
            assert np.array_equal(counts, expect[1]) and np.array_equal(ids, expect[0])
