"""The device builder at the edges of its chunks, warps and value classes: the
layout equals a stable sort of every column."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 33, 1023, 1025, 8191, 8192, 8193, 32769, 100_003])
@pytest.mark.parametrize("d", [1, 33])
def test_columns_are_stably_sorted(genie, n, d):
    rng = np.random.default_rng(1000 * d + n)
    bins = np.array([1, 2, 255, 256, 1024, 1025, 16384, 31])[(np.arange(d) + n) % 8]
    values = (rng.integers(0, 1 << 30, size=(n, d)) % bins - 17).astype(np.int32)
    if n > 1:
        values[0], values[-1] = -17, bins - 18
    skew = rng.random(n) < 0.5
    values[skew, d // 2] = values[0, d // 2]          # one long list
    t = genie.Table.from_values(values, builder="device")
    lay = t.layout()
    assert np.array_equal(lay["dim_min"], values.min(0)) and np.array_equal(lay["dim_max"], values.max(0))
    ids = t.ids()
    for j in range(d):
        assert np.array_equal(ids[j * n:(j + 1) * n], np.argsort(values[:, j], kind="stable")), j
        k0, k1 = lay["key_base"][j], lay["key_base"][j + 1]
        count = np.bincount(values[:, j] - values[:, j].min(), minlength=k1 - k0)
        assert np.array_equal(lay["key_offsets"][k0:k1 + 1], j * n + np.concatenate([[0], np.cumsum(count)])), j
