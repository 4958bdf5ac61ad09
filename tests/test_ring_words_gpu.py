"""The words that tiles publish for one another live in one ring per context,
and a word is taken for a tile's aggregate by its flag and tag alone. So no call
may leave bare values there: maxima of doubles in [2, 4) that have the bits of
a flag and a tag of tiles to come are followed by calls that read those tiles."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TILE8 = 4096         # elements per tile of the 8-byte scans
TILES8 = 500         # under 16 MiB
TILE4 = 40960 // 4   # elements per tile of the pipelined scan and copy_if
TILES4 = 1600        # their tiles 4 j - 500, j < 500, meet the words of tile j


def crafted():
    j = np.arange(TILES8, dtype=np.uint64)
    bits = ((np.uint64(0x40000000) | (np.uint64(4) * j)) << np.uint64(32)) | (j + np.uint64(1))
    return np.repeat(bits, TILE8).view(np.float64)


@pytest.mark.parametrize("writer", ["scan", "segmented_scan"])
@pytest.mark.parametrize("reader", ["scan", "copy_if"])
def test_values_are_not_taken_for_tiles(gbc, writer, reader):
    ctx = gbc.Context()  # its sequence numbers start at 0
    x = crafted()
    xb, yb = gbc.DeviceBuffer.from_host(ctx, x), gbc.DeviceBuffer(ctx, x.size, x.dtype)
    zeros = gbc.DeviceBuffer.from_host(ctx, np.zeros(TILES4 * TILE4, np.int32))
    out = gbc.DeviceBuffer(ctx, TILES4 * TILE4, np.int32)
    if writer == "scan":
        gbc.inclusive_scan(ctx, xb, yb, gbc.ops.maximum(np.float64))
    else:
        offsets = gbc.DeviceBuffer.from_host(ctx, np.array([0, x.size], np.uint32))
        gbc.segmented_scan(ctx, xb, yb, offsets, gbc.ops.maximum(np.float64))
    if reader == "scan":
        gbc.inclusive_scan(ctx, zeros, out)
        assert not out.to_host().any()
    else:
        assert gbc.copy_if(ctx, zeros, out, "x > 0") == 0
    assert np.array_equal(yb.to_host(), x)
    ctx.close()
