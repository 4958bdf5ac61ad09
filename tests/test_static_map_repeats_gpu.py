"""Inserts of many keys into a large table: by regions where a sample shows enough
distinct keys, directly where few values are repeated, and regions with more
pairs than one CTA should take inserted directly by all."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CAP = 1 << 25


def insert(gbc, ctx, keys, vals):
    """The map, the number of new keys and the kernel families that ran."""
    m = gbc.StaticMap(ctx, CAP)
    kb, vb = gbc.DeviceBuffer.from_host(ctx, keys), gbc.DeviceBuffer.from_host(ctx, vals)
    ctx.profile_reset()
    ctx.profile_enable(True)
    added = m.insert(kb, vb)
    ran = {name for name, (launches, _) in ctx.profile().items() if launches}
    ctx.profile_enable(False)
    return m, added, ran


@pytest.mark.parametrize("n", [CAP // 8, CAP // 2 + 3])
@pytest.mark.parametrize("values,by_regions", [(1, False), (1000, False), (CAP // 64, False), (CAP // 4, True)])
def test_route_follows_the_distinct_keys(gbc, ctx, n, values, by_regions):
    rng = np.random.default_rng(n)
    keys = (rng.integers(0, values, size=n).astype(np.uint32) * np.uint32(2654435761)) ^ np.uint32(7)
    vals = np.arange(n, dtype=np.uint32)
    m, added, ran = insert(gbc, ctx, keys, vals)
    assert ("static_map.regions" in ran) == by_regions
    distinct = np.unique(keys)
    assert added == m.size() == distinct.size
    found = gbc.DeviceBuffer(ctx, distinct.size, np.uint32)
    m.find(gbc.DeviceBuffer.from_host(ctx, distinct), found)
    assert np.array_equal(keys[found.to_host()], distinct)  # each with the value of one of its pairs


@pytest.mark.parametrize("extra", ["key", "empty marker"])
def test_a_region_with_many_pairs(gbc, ctx, orc, extra):
    """More than 32,768 pairs for one region, too few of the whole for the sample to see."""
    n = 2 * CAP
    keys = (np.arange(n, dtype=np.uint32) % np.uint32(CAP // 2)) * np.uint32(2654435761)
    keys[500000:536000] = np.uint32(12345 if extra == "key" else 0xFFFFFFFF)
    vals = np.arange(n, dtype=np.uint32)
    m, added, ran = insert(gbc, ctx, keys, vals)
    assert "static_map.regions" in ran
    distinct = np.unique(keys)
    distinct = distinct[distinct != 0xFFFFFFFF]
    assert added == m.size() == distinct.size
    found = gbc.DeviceBuffer(ctx, distinct.size, np.uint32)
    m.find(gbc.DeviceBuffer.from_host(ctx, distinct), found)
    assert np.array_equal(keys[found.to_host()], distinct)
    assert orc.linear_probe_table_ok(m.slots()[0], 0xFFFFFFFF)
