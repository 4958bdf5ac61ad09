"""Histograms of many bytes (counted in pairs from 2^28 of them): uniform,
skewed and constant inputs, one whose counters wrap after the first batch,
signed bytes, bins of every width, sizes off the vectors, against numpy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 1 << 28


def count(x):
    counts = np.zeros(256, dtype=np.int64)
    for i in range(0, x.size, 1 << 24):
        counts += np.bincount(x[i:i + (1 << 24)].view(np.uint8), minlength=256)
    return counts


def expected(counts, dtype, bins, lower, upper):
    """The float bin rule applied to each value's count."""
    values = np.arange(256, dtype=np.uint8).view(dtype).astype(np.float32)
    scale = np.float32(bins) / (np.float32(upper) - np.float32(lower))
    out = np.zeros(bins, dtype=np.uint64)
    for v, c in zip(values, counts):
        if np.float32(lower) <= v < np.float32(upper):
            out[min(int((v - np.float32(lower)) * scale), bins - 1)] += c
    return out.astype(np.uint32)


def make(kind, n, rng):
    if kind == "constant":
        return np.full(n, 200, dtype=np.uint8)
    x = np.frombuffer(rng.bytes(n), dtype=np.uint8).copy()
    if kind == "skewed":  # one value in most places
        x[x < 160] = 7
    if kind != "late":
        return x
    # uniform at first, then one pair only
    share = n // 16 // 128 * 16
    for start in range(0, n, share):
        x[start + (1 << 17):start + share:2] = 129
        x[start + (1 << 17) + 1:start + share:2] = 255
    return x


@pytest.mark.parametrize("kind,n", [("uniform", N), ("uniform", N + 15), ("skewed", N + 1), ("constant", N + 7),
                                    ("late", N + 33)])
def test_byte_pairs(ctx, gbc, kind, n):
    x = make(kind, n, np.random.default_rng(n))
    counts = count(x)
    xb = gbc.DeviceBuffer.from_host(ctx, x)
    for bins, lower, upper in ((256, 0, 256), (64, 0, 256), (100, 10.5, 201), (1, 0, 300), (5000, -3, 256)):
        hb = gbc.DeviceBuffer(ctx, bins, np.uint32)
        gbc.histogram_even(ctx, xb, hb, lower, upper)
        assert np.array_equal(hb.to_host(), expected(counts, x.dtype, bins, lower, upper)), (bins, lower, upper)


def test_signed_bytes(ctx, gbc):
    x = np.frombuffer(np.random.default_rng(5).bytes(N + 7), dtype=np.int8)
    xb, hb = gbc.DeviceBuffer.from_host(ctx, x), gbc.DeviceBuffer(ctx, 50, np.uint32)
    gbc.histogram_even(ctx, xb, hb, -100, 28)
    assert np.array_equal(hb.to_host(), expected(count(x), x.dtype, 50, -100, 28))
