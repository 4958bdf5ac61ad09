"""copy_if in one pass (4-byte elements compared with a literal, aligned
input): sizes around its tiles, every comparison, everything and nothing
kept, NaN, against numpy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TILE = 10240
N = 1 << 22


@pytest.mark.parametrize("dtype", [np.int32, np.uint32, np.float32])
@pytest.mark.parametrize("n", [1, 33, 512, TILE - 1, TILE, TILE + 1, 300 * TILE + 511, N + 513])
def test_one_pass_copy_if(ctx, gbc, dtype, n):
    rng = np.random.default_rng(n)
    x = rng.integers(0, 1000, size=n).astype(dtype)
    if dtype == np.int32:
        x -= 500
    if dtype == np.float32:
        x[::97] = np.nan
        x[::89] = -0.0
    xb, yb = gbc.DeviceBuffer.from_host(ctx, x), gbc.DeviceBuffer(ctx, n, dtype)
    suffix = {np.int32: "", np.uint32: "u", np.float32: ".0f"}[dtype]
    for op, keep in ((">", np.greater), ("<=", np.less_equal), ("==", np.equal), ("!=", np.not_equal),
                     (">=", np.greater_equal), ("<", np.less)):
        for literal in (300, 0, 5000):  # some, few or most, all or none
            with np.errstate(invalid="ignore"):
                want = x[keep(x, dtype(literal))]
            count = gbc.copy_if(ctx, xb, yb, f"x {op} {literal}{suffix}")
            assert count == want.size
            assert np.array_equal(yb.to_host(count).view(np.uint32), want.view(np.uint32)), (op, literal)
