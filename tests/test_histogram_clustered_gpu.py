"""Histograms of many bytes whose neighbours are alike: runs of equal bytes, few
values, and inputs that change their kind within each CTA's share, which are
counted in pairs and by bytes in turn, against numpy."""
import numpy as np
import pytest
from test_histogram_pairs_gpu import N, count, expected

pytestmark = pytest.mark.gpu


def make(kind, n, rng):
    if kind == "runs":
        return (np.arange(n, dtype=np.uint32) >> 8).astype(np.uint8)
    x = np.frombuffer(rng.bytes(n), dtype=np.uint8).copy()
    if kind == "narrow":
        return x & 15
    # uniform, runs and one value by turns, each some batches long
    part = (np.arange(n, dtype=np.uint32) >> 20) % (3 if kind == "by turns" else 7)
    runs = (np.arange(n, dtype=np.uint32) >> 8).astype(np.uint8)
    x = np.where(part == 1, runs, x)
    x[part == 2] = 77
    return x


@pytest.mark.parametrize("kind,n", [("runs", N), ("narrow", N + 31), ("by turns", N + 1), ("late turns", N + 16 * 1000 + 5)])
def test_clustered_bytes(ctx, gbc, kind, n):
    x = make(kind, n, np.random.default_rng(n))
    counts = count(x)
    xb = gbc.DeviceBuffer.from_host(ctx, x)
    for bins, lower, upper in ((256, 0, 256), (100, 10.5, 201)):
        hb = gbc.DeviceBuffer(ctx, bins, np.uint32)
        gbc.histogram_even(ctx, xb, hb, lower, upper)
        assert np.array_equal(hb.to_host(), expected(counts, x.dtype, bins, lower, upper)), (bins, lower, upper)
