"""Bitpack compression where chunks are packed in parts by several warps: many long
chunks and few, a last chunk that ends within its first part, against the oracle
word for word."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,chunk", [((1 << 25) + 77, 65536), ((1 << 25) + 4096, 4096), (65536 + 1, 65536), (5 * 4096 + 1025, 4096)])
@pytest.mark.parametrize("delta", [False, True])
def test_parts_of_chunks(gbc, ctx, orc, n, chunk, delta):
    rng = np.random.default_rng(n + delta)
    x = np.cumsum(rng.integers(0, 3000, size=n)).astype(np.uint32) if delta else rng.integers(0, 1 << 11, size=n, dtype=np.uint32)
    x[chunk // 2] = 0xFFFFFFFF  # one chunk of full width
    comp = gbc.compress_bitpack(ctx, gbc.DeviceBuffer.from_host(ctx, x), delta=delta, chunk_size=chunk)
    assert np.array_equal(comp.data.to_host(), orc.bitpack_compress(x, chunk, delta))
    out = gbc.DeviceBuffer(ctx, n, np.uint32)
    gbc.decompress_bitpack(ctx, comp, out)
    assert np.array_equal(out.to_host(), x)
