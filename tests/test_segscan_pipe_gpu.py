"""Segmented scan of large inputs (the pipelined form): head patterns from none
to every element, empty segments, starts on the edges of rows, blocks and tiles,
partial last tiles, and arrays whose address takes the other form."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N0 = 1 << 25
TILE = 10240


def starts(kind, n, rng):
    if kind == "one":
        s = [0]
    elif kind == "every":
        s = np.arange(n)
    elif kind == "edges":  # rows of 128, blocks of 512, tiles; one before and one after
        e = np.concatenate([np.arange(0, n, TILE), np.arange(0, n, 3 * 512), np.arange(0, n, 5 * 128)])
        s = np.concatenate([[0], e, e + 1, e[1:] - 1])
    elif kind == "empty":  # most segments hold nothing
        s = np.repeat(rng.integers(0, n, size=3000), rng.integers(1, 9, size=3000))
    else:
        s = rng.integers(0, n, size=n // kind)
    s = np.sort(np.asarray(s, dtype=np.int64))
    s = s[s < n]
    if s[0] != 0:
        s = np.concatenate([[0], s])
    return np.concatenate([s, [n]]).astype(np.uint32)


@pytest.mark.parametrize("kind", ["one", "every", "edges", "empty", 3, 100, 20000])
@pytest.mark.parametrize("n", [N0, 3300 * TILE, 3300 * TILE - 1])
@pytest.mark.parametrize("exclusive", [False, True])
def test_heads(ctx, gbc, orc, kind, n, exclusive):
    rng = np.random.default_rng(n + exclusive)
    off = starts(kind, n, rng)
    x = rng.integers(-2**31, 2**31, size=n, dtype=np.int64).astype(np.int32)
    xb, yb, ob = gbc.DeviceBuffer.from_host(ctx, x), gbc.DeviceBuffer(ctx, n, np.int32), gbc.DeviceBuffer.from_host(ctx, off)
    gbc.segmented_scan(ctx, xb, yb, ob, gbc.ops.plus(), exclusive)
    assert np.array_equal(yb.to_host(), orc.std_segmented_scan(x, off, orc.OP_PLUS, 0, exclusive))


@pytest.mark.parametrize("dtype", [np.int32, np.uint32, np.float32])
@pytest.mark.parametrize("opname", ["plus", "maximum", "right"])
@pytest.mark.parametrize("shift", [0, 1])  # 1: not 16-byte aligned, the other form
def test_operators(ctx, gbc, orc, dtype, opname, shift):
    n = N0 + 12345
    rng = np.random.default_rng(5)
    off = starts(700, n, rng)
    x = rng.integers(0, 1000, size=n).astype(dtype)  # float sums stay whole numbers below 2^24 over a segment
    assert np.diff(off).max() * 1000 < 1 << 24
    if opname == "plus":
        op, code, ident = gbc.ops.plus(), orc.OP_PLUS, 0
    elif opname == "maximum":
        op, code = gbc.ops.maximum(dtype), orc.OP_MAX
        ident = np.finfo(dtype).min if dtype == np.float32 else np.iinfo(dtype).min
    else:
        op, code, ident = gbc.binary_op("b", "0"), orc.OP_RIGHT, 0
    xb = gbc.DeviceBuffer.from_host(ctx, np.concatenate([x[:shift], x]))
    yb = gbc.DeviceBuffer(ctx, n + shift, dtype)
    ob = gbc.DeviceBuffer.from_host(ctx, off)
    gbc.segmented_scan_raw(ctx, xb.device_pointer + 4 * shift, yb.device_pointer + 4 * shift, n, dtype, ob.device_pointer,
                           off.size - 1, op, exclusive=False)
    assert np.array_equal(yb.to_host()[shift:], orc.std_segmented_scan(x, off, code, ident, False))


def test_captured_without_a_warm_pool(gbc, orc):
    # no head bits in the pool: the call takes the other form and is captured all the same
    c = gbc.Context()
    n = N0 + 7
    rng = np.random.default_rng(9)
    off = starts(50, n, rng)
    x = rng.integers(-1000, 1000, size=n).astype(np.int32)
    xb, yb, ob = gbc.DeviceBuffer.from_host(c, x), gbc.DeviceBuffer(c, n, np.int32), gbc.DeviceBuffer.from_host(c, off)
    call = lambda: gbc.segmented_scan_raw(c, xb.device_pointer, yb.device_pointer, n, np.int32, ob.device_pointer,
                                          off.size - 1, exclusive=True)
    expect = orc.std_segmented_scan(x, off, orc.OP_PLUS, 0, True)
    for _ in range(2):  # the second time with the pool warm
        g = gbc.capture(c, call)
        for _ in range(2):
            gbc.fill(c, yb, 0)
            g.launch()
            assert np.array_equal(yb.to_host(), expect)
        g.release()
        call()
        c.finish()
    c.close()
