"""Radix sort at the edges of its tiles of 1,024 keys and at the count where it
changes to tiles of 3,072, against numpy's stable order."""
import numpy as np
import pytest
from test_sort_gpu import _keys, _sort

pytestmark = pytest.mark.gpu
FEW_MAX = 148 * 2 * 1024   # keys up to which a tile holds 1,024


@pytest.mark.parametrize("n", [1_023, 1_024, 1_025, 32 * 1_024 + 1, FEW_MAX - 1, FEW_MAX, FEW_MAX + 1])
@pytest.mark.parametrize("dtype,bits", [(np.uint64, 39), (np.uint64, 56), (np.uint32, 30)])
@pytest.mark.parametrize("kind", ["uniform", "few"])
def test_sort_tiles(rtd, cuda, n, dtype, bits, kind):
    keys = _keys(np.random.default_rng(n + bits), n, bits, kind, dtype)
    sk, sv = _sort(rtd.load(), keys, bits)
    order = np.argsort(keys, kind="stable")
    np.testing.assert_array_equal(sk, keys[order])
    np.testing.assert_array_equal(sv, order)
