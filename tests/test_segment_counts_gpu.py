"""Large segments of a batch above 2^24 keys: one digit is counted first, the
others only where that does not decide the route. Kinds of segments for every
answer, mixed in one batch, against the std:: oracle bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def make(kind, n, bits, rng):
    u = rng.integers(0, 2**64, size=n, dtype=np.uint64) >> np.uint64(64 - bits)
    if kind == 1:  # the top digit is constant
        u = (u & np.uint64((1 << (bits - 8)) - 1)) | np.uint64(0x3A << (bits - 8))
    elif kind == 2:  # ... but for one key, which a sample misses
        u &= np.uint64((1 << (bits - 8)) - 1)
        u[n // 3] |= np.uint64(1 << (bits - 1))
    elif kind == 3:  # half of the keys in one bin of the top digit
        u[rng.random(n) < 0.5] &= np.uint64((1 << (bits - 8)) - 1)
    elif kind == 4:  # one value
        u[:] = u[0]
    elif kind == 5:  # one value but for the last key
        u[:-1] = u[0]
    elif kind == 6:  # few bits, the lowest digit only
        u &= np.uint64(0x3F)
    elif kind == 7:  # in order, so that neighbours are alike
        u = np.sort(u)
    return u


@pytest.mark.parametrize("dtype", [np.uint32, np.float32, np.uint64])
@pytest.mark.parametrize("with_values", [True, False])
@pytest.mark.parametrize("short", [False, True])
def test_mixed_large_segments(ctx, gbc, orc, dtype, with_values, short):
    bits = np.dtype(dtype).itemsize * 8
    rng = np.random.default_rng(bits + short)
    # short: just above one CTA's capacity; otherwise to beyond what 256 bins of it hold
    lens = [16385, 17000, 25000, 40001] if short else [16385, 130000, 600000, 2100000]
    parts = []
    for n in lens:
        for kind in range(8):
            if n < 1 << 20 or kind in (0, 2, 3):
                parts.append(make(kind, n, bits, rng))
    while sum(p.size for p in parts) <= 1 << 24:  # a batch of few keys counts all digits at once
        parts.append(make(len(parts) % 8, lens[len(parts) % 3], bits, rng))
    parts = [parts[i] for i in rng.permutation(len(parts))]
    off = np.concatenate([[0], np.cumsum([p.size for p in parts])]).astype(np.uint32)
    words = np.concatenate(parts)
    keys = (words.astype(np.uint32) if bits == 32 else words).view(dtype)
    if np.dtype(dtype).kind == "f":
        keys = np.where(np.isnan(keys), dtype(1.5), keys)
    vals = np.arange(keys.size, dtype=np.uint32)
    ek, ev = orc.std_segmented_sort(keys, off, vals if with_values else None)
    ob = gbc.DeviceBuffer.from_host(ctx, off)
    kb = gbc.DeviceBuffer.from_host(ctx, keys)
    vb = gbc.DeviceBuffer.from_host(ctx, vals) if with_values else None

    def size_class(v):
        return f"2^{max(0, int(v) - 1).bit_length()}"

    # the MSD route for every type at this size
    key = (f"segsort:u{bits}{'kv' if with_values else 'k'}:{size_class(keys.size)}:"
           f"avg{size_class(keys.size // len(parts))}:msd")
    try:
        ctx.tuning_set(key, 16384)
        gbc.segmented_sort(ctx, kb, ob, vb)
        assert ctx.tuning_get(key) == 16384
    finally:
        ctx.tuning_set(key, 0)
    assert np.array_equal(kb.to_host().view(np.uint8), ek.view(np.uint8))
    if with_values:
        assert np.array_equal(vb.to_host(), ev)
