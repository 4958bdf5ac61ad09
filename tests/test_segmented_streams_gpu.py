"""Batches whose two paths run one after the other (most keys in large segments)
or beside each other, with segments that one digit does not split well (a bin with
more than half of the keys), against the std:: oracle; and the one-stream form in
a graph."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def batch(count, mean, dtype, rng):
    bits = np.dtype(dtype).itemsize * 8
    lens = rng.integers(mean // 2, mean * 3 // 2 + 1, size=count)
    off = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint32)
    u = rng.integers(0, 2**64, size=int(off[-1]), dtype=np.uint64) >> np.uint64(64 - bits)
    for i in range(0, count, 2):  # three keys of five share the top digit
        part = u[off[i]:off[i + 1]]
        part[rng.random(part.size) < 0.6] &= np.uint64((1 << (bits - 8)) - 1)
    return off, u.astype(dtype)


@pytest.mark.parametrize("dtype", [np.uint32, np.uint64])
@pytest.mark.parametrize("with_values", [True, False])
@pytest.mark.parametrize("count,mean", [(40, 300), (30, 9500), (30, 13000), (9, 40000), (900, 12000), (300, 60000)])
def test_paths(ctx, gbc, orc, dtype, with_values, count, mean):
    off, keys = batch(count, mean, dtype, np.random.default_rng(mean))
    vals = np.arange(keys.size, dtype=np.uint32) if with_values else None
    ek, ev = orc.std_segmented_sort(keys, off, vals)
    kb, ob = gbc.DeviceBuffer.from_host(ctx, keys), gbc.DeviceBuffer.from_host(ctx, off)
    vb = gbc.DeviceBuffer.from_host(ctx, vals) if with_values else None
    gbc.segmented_sort(ctx, kb, ob, vb)
    assert np.array_equal(kb.to_host(), ek)
    if with_values:
        assert np.array_equal(vb.to_host(), ev)


def test_one_stream_in_a_graph(gbc, orc):
    ctx = gbc.Context()
    rng = np.random.default_rng(8)
    off, keys = batch(20, 30000, np.uint64, rng)
    ob, kb = gbc.DeviceBuffer.from_host(ctx, off), gbc.DeviceBuffer.from_host(ctx, keys)
    gbc.segmented_sort(ctx, kb, ob)  # the pool is warm from here on
    ctx.finish()
    graph = gbc.capture(ctx, lambda: gbc.segmented_sort(ctx, kb, ob))
    for _ in range(2):
        keys = rng.permutation(keys)
        kb.write(keys)
        graph.launch()
        assert np.array_equal(kb.to_host(), orc.std_segmented_sort(keys, off, None)[0])
    graph.release()
    ctx.close()
