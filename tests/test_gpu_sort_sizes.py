"""The key sort at the edges of its two forms (one block up to 8,192 keys, digit passes above) against numpy's
stable sort: sizes, key widths that end inside a digit, and keys that are all equal."""
import numpy as np
import pytest

from novaphy_gb300 import capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 33, 1023, 1025, 8191, 8192, 8193, 16385])
@pytest.mark.parametrize("bits", [1, 5, 8, 9, 17, 32])
def test_stable(n, bits):
    rng = np.random.default_rng(n * 64 + bits)
    for keys in (rng.integers(0, 1 << bits, n, dtype=np.uint64), np.full(n, (1 << bits) - 1, np.uint64)):
        keys = keys.astype(np.uint32)
        ko, vo = capi.sort_pairs(keys, bits)
        order = np.argsort(keys, kind="stable")
        assert np.array_equal(vo, order) and np.array_equal(ko, keys[order])
