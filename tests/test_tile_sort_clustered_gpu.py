"""One-CTA sorts of keys whose set bits are few, so that the leading digits that a
sample would settle for leave long runs: alone and as segments, stable, against the
std:: oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def clustered(n, words, rng):
    u = rng.integers(0, 2**64, size=n, dtype=np.uint64)
    for _ in range(words - 1):
        u &= rng.integers(0, 2**64, size=n, dtype=np.uint64)
    return u


@pytest.mark.parametrize("words", [2, 3, 4, 6])
@pytest.mark.parametrize("n", [40, 300, 1000, 4097, 8192])
def test_small_arrays(ctx, gbc, orc, n, words):
    keys = clustered(n, words, np.random.default_rng(n + words))
    vals = np.arange(n, dtype=np.uint32)
    ek, ev = orc.std_segmented_sort(keys, np.array([0, n], np.uint32), vals)
    kb, vb = gbc.DeviceBuffer.from_host(ctx, keys), gbc.DeviceBuffer.from_host(ctx, vals)
    gbc.sort_raw(ctx, kb.device_pointer, kb.device_pointer, np.uint64, n, vb.device_pointer, vb.device_pointer)
    assert np.array_equal(kb.to_host(), ek)
    assert np.array_equal(vb.to_host(), ev)


@pytest.mark.parametrize("words", [2, 4])
def test_segments(ctx, gbc, orc, words):
    rng = np.random.default_rng(words)
    off = np.concatenate([[0], np.cumsum(rng.integers(1, 9000, size=200))]).astype(np.uint32)
    keys = clustered(int(off[-1]), words, rng)
    vals = np.arange(keys.size, dtype=np.uint32)
    ek, ev = orc.std_segmented_sort(keys, off, vals)
    kb, vb = gbc.DeviceBuffer.from_host(ctx, keys), gbc.DeviceBuffer.from_host(ctx, vals)
    gbc.segmented_sort(ctx, kb, gbc.DeviceBuffer.from_host(ctx, off), vb)
    assert np.array_equal(kb.to_host(), ek)
    assert np.array_equal(vb.to_host(), ev)
