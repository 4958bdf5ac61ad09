"""64-bit sorts that order the leading digits first: runs of every short length
that agree in those digits, equal keys among them, inside the tiles that check
them and across their edges."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = (1 << 23) + 77


def sort_pairs(ctx, gbc, keys):
    kb, vb = gbc.DeviceBuffer.from_host(ctx, keys), gbc.DeviceBuffer.from_host(ctx, np.arange(keys.size, dtype=np.uint32))
    ko, vo = gbc.DeviceBuffer(ctx, keys.size, keys.dtype), gbc.DeviceBuffer(ctx, keys.size, np.uint32)
    gbc.sort_raw(ctx, kb.device_pointer, ko.device_pointer, keys.dtype, keys.size, vb.device_pointer, vo.device_pointer)
    return ko.to_host(), vo.to_host()


@pytest.mark.parametrize("distinct", [2, 1 << 32])  # values of the low halves in a run
def test_runs_of_every_short_length(ctx, gbc, distinct):
    rng = np.random.default_rng(distinct)
    lengths = np.repeat(np.arange(2, 53), 60)
    low = np.uint64(0xFFFFFFFF)
    # uniform keys with the runs' keys among them, at random places
    keys = rng.integers(0, 2**64, size=N, dtype=np.uint64)
    at = rng.choice(N, size=int(lengths.sum()), replace=False)
    prefix = rng.integers(0, 2**32, size=lengths.size, dtype=np.uint64) << np.uint64(32)
    keys[at] = np.repeat(prefix, lengths) | (rng.integers(0, distinct, size=at.size, dtype=np.uint64) & low)
    got, order = sort_pairs(ctx, gbc, keys)
    expected = np.argsort(keys, kind="stable").astype(np.uint32)
    assert np.array_equal(order, expected)
    assert np.array_equal(got, keys[expected])


def test_runs_across_every_tile_edge(ctx, gbc):
    """Runs of 3 to 40 keys centred on the edges of the 4,096-key tiles."""
    rng = np.random.default_rng(3)
    top = np.arange(N, dtype=np.uint64)  # rank, made a prefix below: distinct and spread
    for edge in range(4096, N - 64, 4096):
        length = 3 + (edge // 4096) % 38
        b = edge - int(rng.integers(1, min(length, 22)))
        top[b:b + length] = top[b]
    keys = (top * np.uint64(2**32 // N) << np.uint64(32)) | rng.integers(0, 2**32, size=N, dtype=np.uint64)
    keys = rng.permutation(keys)
    got, order = sort_pairs(ctx, gbc, keys)
    expected = np.argsort(keys, kind="stable").astype(np.uint32)
    assert np.array_equal(order, expected)
    assert np.array_equal(got, keys[expected])
