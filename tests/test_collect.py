"""The library's record collector and its decoding: records across the ends of
the decoded pieces, empty sides, and a buffer that grows."""
import ctypes

import numpy as np
import pytest

from gmkbe_b200 import api


@pytest.mark.parametrize("slab", [1, 2, 7, 64, 1 << 20])
@pytest.mark.parametrize("n", [0, 1, 5000])
def test_collected_records_come_back_as_they_went_in(n, slab):
    rng = np.random.default_rng(n)
    want = [tuple(tuple(int(v) for v in rng.integers(0, 2**32, rng.integers(0, 12))) for _ in range(2))
            for _ in range(n)]
    store = api._Collector()
    cb, user = api.Graph._sink(True, None, store)
    try:
        for x, y in want:
            assert cb(user, (ctypes.c_uint32 * len(x))(*x), len(x), (ctypes.c_uint32 * len(y))(*y), len(y)) == 0
        assert api.Graph._records(store, slab) == want
    finally:
        api.load_library().gmk_collect_free(ctypes.byref(store))
    assert store.data is None and store.len == 0
