"""The pipelined scan (16-byte aligned inputs from 16 MiB): sizes around its
tiles and rounds, every operator family, in place, with the total. Values are
small integers, so floating-point results are exact too."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TILE_BYTES = 40960
MIN_BYTES = 1 << 24


def reference(x, opname, ident, exclusive):
    wide = x.astype(np.float64) if x.dtype.kind == "f" else x.astype(np.int64)
    if opname == "plus":
        inc = np.cumsum(wide)
    elif opname == "maximum":
        inc = np.maximum.accumulate(wide)
    elif opname == "xor":
        inc = np.bitwise_xor.accumulate(wide)
    else:  # the right projection reproduces the input
        inc = wide
    if exclusive:
        inc = np.concatenate([[ident], inc[:-1]])
    return inc.astype(x.dtype)


@pytest.mark.parametrize("dtype", [np.int32, np.uint32, np.int64, np.float32, np.float64])
@pytest.mark.parametrize("opname", ["plus", "maximum", "xor", "right"])
@pytest.mark.parametrize("tail", ["none", "one", "tile-1", "rounds+3"])
def test_pipelined_scan(ctx, gbc, dtype, opname, tail):
    if opname == "xor" and np.dtype(dtype).kind == "f":
        return
    item = np.dtype(dtype).itemsize
    tile = TILE_BYTES // item
    n = MIN_BYTES // item + {"none": 0, "one": 1, "tile-1": tile - 1, "rounds+3": 700 * tile + 3}[tail]
    rng = np.random.default_rng(n)
    x = rng.integers(0 if dtype == np.uint32 else -3, 4, size=n).astype(dtype)
    op, ident = {"plus": (gbc.ops.plus(), 0),
                 "maximum": (gbc.ops.maximum(dtype), -np.inf if np.dtype(dtype).kind == "f" else np.iinfo(dtype).min),
                 "xor": (gbc.ops.bit_xor(), 0), "right": (gbc.binary_op("b", "0"), 0)}[opname]
    xb, yb = gbc.DeviceBuffer.from_host(ctx, x), gbc.DeviceBuffer(ctx, n, dtype)
    for exclusive in (False, True):
        scan = gbc.exclusive_scan if exclusive else gbc.inclusive_scan
        total = scan(ctx, xb, yb, op, total=True)
        assert np.array_equal(yb.to_host(), reference(x, opname, ident, exclusive))
        assert total == reference(x, opname, ident, False)[-1]
    # in place, without a total, twice on the same buffer size (another tile counter, other sequence numbers)
    gbc.inclusive_scan(ctx, xb, xb, op)
    assert np.array_equal(xb.to_host(), reference(x, opname, ident, False))


def test_unaligned_input_keeps_its_results(ctx, gbc):
    n = (MIN_BYTES // 4) + 5
    x = np.random.default_rng(1).integers(-1000, 1001, size=n + 1).astype(np.int32)
    xb, yb = gbc.DeviceBuffer.from_host(ctx, x), gbc.DeviceBuffer(ctx, n, np.int32)
    gbc.scan_raw(ctx, xb.device_pointer + 4, yb.device_pointer, n, np.int32)
    assert np.array_equal(yb.to_host(), np.cumsum(x[1:].astype(np.int64)).astype(np.int32))
