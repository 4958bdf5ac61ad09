"""64-bit sorts that order the leading digits first, in the forms that their own
test leaves out: from 2^27 keys with all digits, with more digits than the first
plan takes and with keys that the sample misjudges; and captured in a graph whose
replays sort other keys."""
import numpy as np
import pytest
from test_sort_partial_gpu import N_LEAST, N_SEGMENTED, expected, make_keys

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["misjudged", "groups", "seven_digits"])
def test_all_digits_after_all(ctx, gbc, kind):
    keys = make_keys(kind, N_SEGMENTED, np.random.default_rng(21))
    ek, ev = expected(keys)
    kb, vb = gbc.DeviceBuffer.from_host(ctx, keys), gbc.DeviceBuffer.from_host(ctx, np.arange(keys.size, dtype=np.uint32))
    gbc.sort_ex(ctx, kb, vb)
    assert np.array_equal(kb.to_host(), ek)
    assert np.array_equal(vb.to_host(), ev)


@pytest.mark.parametrize("n", [N_LEAST + 5, N_SEGMENTED])
def test_captured(gbc, n):
    ctx = gbc.Context()
    rng = np.random.default_rng(n)
    kin, vin = gbc.DeviceBuffer(ctx, n, np.uint64), gbc.DeviceBuffer.from_host(ctx, np.arange(n, dtype=np.uint32))
    kout, vout = gbc.DeviceBuffer(ctx, n, np.uint64), gbc.DeviceBuffer(ctx, n, np.uint32)

    def sort():
        gbc.sort_raw(ctx, kin.device_pointer, kout.device_pointer, np.uint64, n, vin.device_pointer, vout.device_pointer)

    kin.write(make_keys("uniform", n, rng))
    sort()  # the pool is warm from here on
    ctx.finish()
    graph = gbc.capture(ctx, sort)
    for kind in ("long_runs", "low_digits", "uniform", "misjudged"):
        keys = make_keys(kind, n, rng)
        kin.write(keys)
        graph.launch()
        ctx.finish()
        ek, ev = expected(keys)
        assert np.array_equal(kout.to_host(), ek), kind
        assert np.array_equal(vout.to_host(), ev), kind
    graph.release()
    ctx.close()
