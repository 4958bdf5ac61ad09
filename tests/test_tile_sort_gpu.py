"""The one-CTA sort that orders the leading bits and repairs the rest: whole
arrays of up to 8,192 keys and segments of every one-CTA class, and the MSD
route's ranges of neighbouring buckets, against the std:: oracle bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BITS = {np.uint32: 32, np.int32: 32, np.float32: 32, np.uint64: 64, np.int64: 64, np.float64: 64}


def make_keys(kind, n, dtype, seed):
    """Keys whose leading bits decide everything, little, or nothing."""
    rng = np.random.default_rng(seed)
    bits = BITS[dtype]
    u = rng.integers(0, 2**64, size=n, dtype=np.uint64) >> np.uint64(64 - bits)
    low = np.uint64((1 << (bits // 2)) - 1)
    if kind == "uniform":  # a few neighbours share their leading bits: short repairs
        k = u
    elif kind == "short_runs":  # about ten keys per leading value
        groups = rng.integers(0, 2**16, size=max(1, n // 10), dtype=np.uint64) << np.uint64(bits - 16)
        k = groups[rng.integers(0, groups.size, size=n)] | (u & low)
    elif kind == "long_runs":  # four leading values: every digit is needed
        k = (rng.integers(0, 4, size=n, dtype=np.uint64) << np.uint64(bits - 2)) | (u & low)
    elif kind == "duplicates":  # equal keys in long runs, a few strangers among them
        k = (rng.integers(0, 7, size=n, dtype=np.uint64) << np.uint64(bits - 4))
        k[::37] |= u[::37] & np.uint64(0xFF)
    elif kind == "low_bits":  # 13 differing bits
        k = np.uint64(5 << 20) | (u & np.uint64(0x1FFF))
    elif kind == "sorted":
        k = np.sort(u)
    elif kind == "reversed":
        k = np.sort(u)[::-1].copy()
    else:  # one value
        k = np.full(n, u[0])
    words = k.astype(np.uint32) if bits == 32 else k
    keys = words.view(dtype)
    if np.dtype(dtype).kind == "f":
        keys = np.where(np.isnan(keys), dtype(1.5), keys)
    return keys


KINDS = ["uniform", "short_runs", "long_runs", "duplicates", "low_bits", "sorted", "reversed", "constant"]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("dtype", list(BITS))
@pytest.mark.parametrize("n", [2, 15, 33, 257, 1024, 4097, 8191, 8192, 8193])
def test_small_arrays(ctx, gbc, orc, kind, dtype, n):
    keys = make_keys(kind, n, dtype, n)
    off = np.array([0, n], dtype=np.uint32)
    vals = np.arange(n, dtype=np.uint32)
    for descending in (False, True):
        ek, ev = orc.std_segmented_sort(keys, off, vals, descending=descending)
        kb, vb = gbc.DeviceBuffer.from_host(ctx, keys), gbc.DeviceBuffer.from_host(ctx, vals)
        gbc.sort_ex(ctx, kb, vb, descending=descending)
        assert np.array_equal(kb.to_host().view(np.uint8), ek.view(np.uint8))
        assert np.array_equal(vb.to_host(), ev)
        # keys only, out of place from an address one key past a 16-byte boundary
        src = gbc.DeviceBuffer.from_host(ctx, np.concatenate([keys[:1], keys]))
        out = gbc.DeviceBuffer(ctx, n, dtype)
        gbc.sort_raw(ctx, src.device_pointer + keys.itemsize, out.device_pointer, dtype, n, descending=descending)
        assert np.array_equal(out.to_host().view(np.uint8), ek.view(np.uint8))


LENGTHS = [256, 257, 600, 4095, 4096, 4097, 8191, 8192, 8193, 10239, 10240, 10241, 16383, 16384, 16385, 40000, 300000, 1]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("dtype", [np.uint32, np.float32, np.uint64, np.int64])
@pytest.mark.parametrize("with_values", [True, False])
@pytest.mark.parametrize("threads,msd", [(256, True), (256, False), (512, True)])
def test_segments_of_every_class(ctx, gbc, orc, kind, dtype, with_values, threads, msd):
    off = np.concatenate([[0], np.cumsum(LENGTHS)]).astype(np.uint32)
    keys = np.concatenate([make_keys(kind, n, dtype, n) for n in LENGTHS])
    vals = np.arange(keys.size, dtype=np.uint32)
    ek, ev = orc.std_segmented_sort(keys, off, vals if with_values else None)
    ob = gbc.DeviceBuffer.from_host(ctx, off)
    kb = gbc.DeviceBuffer.from_host(ctx, keys)
    vb = gbc.DeviceBuffer.from_host(ctx, vals) if with_values else None

    def size_class(v):
        return f"2^{max(0, int(v) - 1).bit_length()}"

    # the MSD route's capacity, set for this workload's class: 16,384 (cut to the type's largest) or off
    key = (f"segsort:u{keys.itemsize * 8}{'kv' if with_values else 'k'}:{size_class(keys.size)}:"
           f"avg{size_class(keys.size // len(LENGTHS))}:msd")
    try:
        ctx.tuning_set("segsort:cta_threads", threads)
        ctx.tuning_set(key, 16384 if msd else 0)
        gbc.segmented_sort(ctx, kb, ob, vb)
        assert ctx.tuning_get(key) == (16384 if msd else 0)
    finally:
        ctx.tuning_set("segsort:cta_threads", 0)
        ctx.tuning_set(key, 0)
    assert np.array_equal(kb.to_host().view(np.uint8), ek.view(np.uint8))
    if with_values:
        assert np.array_equal(vb.to_host(), ev)
