"""The encoder's placing of chunks on its own (sleek_selftest_chunk_scan): places from the
scanner's ring and, for groups that the ring has lost, from the group sums; and the
alignment hint, which is the same in every lane of a warp however the lanes arrive."""
import ctypes as C

import numpy as np
import pytest

from sleek_b200 import _capi

pytestmark = pytest.mark.gpu

GROUP, RING = 64, 128


@pytest.mark.parametrize("chunks", [1, 64, 65, 100 * GROUP, 400 * GROUP + 17])
def test_places_in_and_behind_the_ring(cuda, chunks):
    rng = np.random.default_rng(chunks)
    sizes = rng.integers(1, 16385, chunks, dtype=np.uint32)
    last = (chunks + GROUP - 1) // GROUP - 1  # groups known when the scanner is through
    groups = {0, 1, 2, 10, last - RING, last - RING + 32, last - RING + 33, last - 1, last}
    index = np.array(sorted({c for g in groups for c in (g * GROUP, g * GROUP + 1, g * GROUP + 63) if 0 <= c < chunks}),
                     dtype=np.int64)
    want = np.concatenate([[0], np.cumsum(sizes.astype(np.int64))])[index]
    got = np.full(index.size, -7, dtype=np.int64)
    uneven = C.c_uint(77)
    _capi.check(_capi.lib().sleek_selftest_chunk_scan(sizes.ctypes.data, chunks, index.ctypes.data, index.size,
                                                      got.ctypes.data, C.byref(uneven)))
    assert np.array_equal(got, want)
    assert uneven.value == 0
