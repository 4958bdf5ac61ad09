"""Large floating-point scans combine in sequence order, op(earlier, later): the
zero that a running minimum or maximum keeps is the first one, and sums that
stay finite in that order do. Compared bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TILE_BYTES = 40960
N_MIN = 1 << 25  # bytes; smaller inputs take another kernel


def run(ctx, gbc, x, op):
    xb, yb = gbc.DeviceBuffer.from_host(ctx, x), gbc.DeviceBuffer(ctx, x.size, x.dtype)
    gbc.inclusive_scan(ctx, xb, yb, op)
    return yb.to_host()


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("opname,rest,first", [("minimum", 5.0, -0.0), ("minimum", 5.0, 0.0), ("maximum", -5.0, 0.0),
                                               ("maximum", -5.0, -0.0)])
@pytest.mark.parametrize("apart", ["rows", "blocks", "32 tiles"])
def test_first_zero_stays(ctx, gbc, dtype, opname, rest, first, apart):
    """A zero, and the zero of the other sign further on."""
    dtype = np.dtype(dtype)
    vec, tile = 16 // dtype.itemsize, TILE_BYTES // dtype.itemsize
    n = N_MIN // dtype.itemsize + 1
    a, b = {"rows": (vec, 32 * vec), "blocks": (vec, 512 * vec),
            "32 tiles": (33 * tile + 5, 64 * tile)}[apart]  # the second zero's row or tile falls to an earlier lane
    x = np.full(n, rest, dtype)
    x[a], x[b] = first, -first
    expected = np.full(n, rest, dtype)
    expected[a:] = first
    got = run(ctx, gbc, x, getattr(gbc.ops, opname)(dtype))
    assert np.array_equal(got.view(np.uint8), expected.view(np.uint8))


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("apart", ["rows", "32 tiles"])
def test_sums_that_cancel_in_order_stay_finite(ctx, gbc, dtype, apart):
    """Near the largest value, each taken away again before the next is added."""
    dtype = np.dtype(dtype)
    vec, tile = 16 // dtype.itemsize, TILE_BYTES // dtype.itemsize
    n = N_MIN // dtype.itemsize + 1
    step, gap = (32 * vec, vec) if apart == "rows" else (32 * tile, tile)
    big = np.finfo(dtype).max * dtype.type(0.75)
    x = np.zeros(n, dtype)
    x[::step] = big
    x[gap::step] = -big
    expected = np.zeros(n, dtype)
    at = np.arange(n) % step < gap
    expected[at] = big
    assert np.array_equal(run(ctx, gbc, x, gbc.ops.plus()), expected)
