"""Radix sort around the sizes where the digit pass changes its tile: the
smallest device passes, the end of the short tiles, the start of the long
ones, and sizes one off a whole number of tiles."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def own(gbc):
    # a context of its own: no other test's tuning entries choose the shape
    c = gbc.Context()
    yield c
    c.close()


@pytest.mark.parametrize("dtype", [np.uint32, np.int32, np.float32, np.uint64])
@pytest.mark.parametrize("with_values", [False, True])
@pytest.mark.parametrize("n", [8193, 5 * 2048 - 1, 5 * 2048 + 1, (1 << 18) - 1, 1 << 18, (1 << 18) + 1,
                               (1 << 21) - 1, 1 << 21, 257 * 8192 + 1])
def test_sizes_where_the_tile_changes(own, gbc, orc, dtype, with_values, n):
    rng = np.random.default_rng(n)
    bits = rng.integers(0, 2**64, size=n, dtype=np.uint64).astype(np.uint64 if dtype == np.uint64 else np.uint32)
    bits[::5] &= bits[:: 5][::-1]  # some digits far more common than others
    bits[1::7] = bits[1]
    keys = bits.view(dtype)
    vals = np.arange(n, dtype=np.uint32) if with_values else None
    for descending in (False, True):
        ek, ev = orc.ref_radix_sort(keys, vals, descending)
        kb = gbc.DeviceBuffer.from_host(own, keys)
        vb = gbc.DeviceBuffer.from_host(own, vals) if with_values else None
        vp = vb.device_pointer if with_values else 0
        gbc.sort_raw(own, kb.device_pointer, kb.device_pointer, dtype, n, vp, vp, descending)
        assert np.array_equal(kb.to_host().view(bits.dtype), ek.view(bits.dtype))
        if with_values:
            assert np.array_equal(vb.to_host(), ev)
