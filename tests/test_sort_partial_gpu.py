"""64-bit sorts that order the leading digits and repair the rest (from 2^23
keys; from 2^27 long runs go to the segmented sort): distributions that need no
repair, short and long repairs, all digits, and one that the sample misjudges,
against torch's stable sort bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N_LEAST = 1 << 23
N = (1 << 26) + 4321
N_SEGMENTED = (1 << 27) + 4321


def sampled_positions(n):
    sample = 1 << 15
    while sample < 1 << 17 and sample * sample < 32 * n:
        sample *= 2
    i = np.arange(sample, dtype=np.uint64)
    step = n // sample
    return i * np.uint64(step) + (((i * np.uint64(0x9E3779B1)) & np.uint64(0xFFFFFFFF)) >> np.uint64(8)) % np.uint64(step)


def make_keys(kind, n, rng):
    u = rng.integers(0, 2**64, size=n, dtype=np.uint64)
    low = np.uint64(0xFFFFFFFF)
    if kind == "uniform":
        return u
    if kind == "few_values":  # equal keys in long runs, some of them beside strangers
        values = u[:40000].copy()
        values[1::50] = (values[::50] & ~np.uint64(0xFFFF)) | (values[1::50] & np.uint64(0xFFFF))
        return values[(rng.random(n) ** 4 * values.size).astype(np.int64)]
    if kind == "long_runs":  # a few runs of 25 to 50,000 keys that agree in 32 bits
        for length in (25, 26, 49, 100, 5000, 9000, 50000):
            at = rng.integers(0, n, size=length)
            u[at] = (u[length] & ~low) | (u[at] & low)
        return u
    if kind == "groups":  # a hash of 2^14 groups above a sequence number: all digits are needed
        hashed = u[: 1 << 14] & ~low
        return hashed[rng.integers(0, hashed.size, size=n)] | np.arange(n, dtype=np.uint64)[::-1]
    if kind == "low_digits":  # three varying digits, not next to each other
        return (u & np.uint64(0x00FF0000FF00FF00)) | np.uint64(0x1200000000000034)
    if kind == "seven_digits":  # more digits than are sorted at first, all needed
        return (u >> np.uint64(8)) & np.uint64(0x0003000300FFFFFF)
    # every sampled key is uniform, the others share 1,000 leading patterns
    k = (u[:1000] & ~low)[rng.integers(0, 1000, size=n)] | (u & low)
    at = sampled_positions(n).astype(np.int64)
    k[at] = u[at]
    return k


def expected(keys, descending=False):
    """The stably sorted keys' words and their positions."""
    torch = pytest.importorskip("torch")
    u = keys.view(np.uint64)
    sign = np.uint64(1 << 63)
    if keys.dtype.kind == "u":
        u = u ^ sign  # the signed order of these words is the unsigned one of the keys
    elif keys.dtype.kind == "f":
        u = np.where(u & sign, ~u, u | sign) ^ sign
    words = torch.from_numpy((~u if descending else u).view(np.int64)).cuda()
    order = torch.sort(words, stable=True).indices
    torch.cuda.synchronize()
    order = order.cpu().numpy()
    return keys.view(np.uint64)[order], order.astype(np.uint32)


CASES = [(n, k) for n in (N_LEAST, N) for k in ("uniform", "few_values", "long_runs", "groups", "low_digits",
                                                "seven_digits", "misjudged")] + \
        [(N_SEGMENTED, "long_runs")]


@pytest.mark.parametrize("n,kind", CASES)
def test_partial_sort(ctx, gbc, n, kind):
    rng = np.random.default_rng(11)
    keys = make_keys(kind, n, rng)
    vals = np.arange(n, dtype=np.uint32)
    ek, ev = expected(keys)
    # out of place, pairs
    kin, vin = gbc.DeviceBuffer.from_host(ctx, keys), gbc.DeviceBuffer.from_host(ctx, vals)
    kout, vout = gbc.DeviceBuffer(ctx, n, np.uint64), gbc.DeviceBuffer(ctx, n, np.uint32)
    gbc.sort_raw(ctx, kin.device_pointer, kout.device_pointer, np.uint64, n, vin.device_pointer, vout.device_pointer)
    assert np.array_equal(kout.to_host(), ek)
    assert np.array_equal(vout.to_host(), ev)
    assert np.array_equal(kin.to_host(), keys) and np.array_equal(vin.to_host(), vals)
    # in place, keys only
    gbc.sort_ex(ctx, kin)
    assert np.array_equal(kin.to_host(), ek)


@pytest.mark.parametrize("dtype,kind", [(np.int64, "long_runs"), (np.float64, "few_values")])
def test_partial_sort_signed_and_descending(ctx, gbc, dtype, kind):
    rng = np.random.default_rng(12)
    keys = make_keys(kind, N, rng).view(dtype)
    if dtype == np.float64:
        keys = np.where(np.isnan(keys), 0.25, keys)
        keys[::1001] = -0.0
    vals = np.arange(N, dtype=np.uint32)
    ek, ev = expected(keys, descending=True)
    kb, vb = gbc.DeviceBuffer.from_host(ctx, keys), gbc.DeviceBuffer.from_host(ctx, vals)
    gbc.sort_ex(ctx, kb, vb, descending=True)
    assert np.array_equal(kb.to_host().view(np.uint64), ek)
    assert np.array_equal(vb.to_host(), ev)
