"""A pass of the batched sort that computes places outside its segment writes
nothing there, and the call reports it instead of returning incomplete results."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_places_outside_a_segment_are_reported(gbc, ctx):
    assert gbc.lib.clc_selftest_misplaced(ctx.handle) == gbc.ERROR_OPENCL
    assert b"outside" in gbc.lib.clc_last_error()
    # the error was consumed, and the context sorts
    ctx.finish()
    keys = np.random.default_rng(1).integers(0, 2**32, size=50000, dtype=np.uint32)
    kb = gbc.DeviceBuffer.from_host(ctx, keys)
    gbc.segmented_sort(ctx, kb, gbc.DeviceBuffer.from_host(ctx, np.array([0, 20000, 50000], np.uint32)))
    ctx.finish()
    assert np.array_equal(kb.to_host(), np.concatenate([np.sort(keys[:20000]), np.sort(keys[20000:])]))
