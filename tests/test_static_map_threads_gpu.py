"""Threads with contexts of their own that insert into one map at the same time:
no key may be lost, also where inserts rewrite whole regions of the table."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1 << 14, 1 << 22])  # directly; by regions
def test_inserts_from_several_threads(gbc, ctx, n):
    threads, rounds, cap = 3, 2, 1 << 25
    m = gbc.StaticMap(ctx, cap)
    ctx.finish()
    total = threads * rounds * n
    keys = np.arange(total, dtype=np.uint32) * np.uint32(2654435761)
    start = threading.Barrier(threads)
    added, errors = [0] * threads, []

    def work(t):
        try:
            own = gbc.Context()
            parts = [slice((t * rounds + r) * n, (t * rounds + r + 1) * n) for r in range(rounds)]
            bufs = [(gbc.DeviceBuffer.from_host(own, keys[p]), gbc.DeviceBuffer.from_host(own, ~keys[p])) for p in parts]
            own.finish()
            mine = gbc.StaticMap.__new__(gbc.StaticMap)  # the map, through this thread's context
            start.wait()
            mine.ctx, mine.handle = own, m.handle
            try:
                added[t] = sum(mine.insert(k, v) for k, v in bufs)
            finally:
                mine.handle = None  # the map is the main thread's
        except Exception as e:  # noqa: BLE001  (reported by the main thread)
            errors.append(e)
            start.abort()

    workers = [threading.Thread(target=work, args=(t,)) for t in range(threads)]
    for w in workers:
        w.start()
    for w in workers:
        w.join()
    assert not errors
    assert added == [rounds * n] * threads
    assert m.size() == total
    found = gbc.DeviceBuffer(ctx, total, np.uint32)
    m.find(gbc.DeviceBuffer.from_host(ctx, keys), found)
    assert np.array_equal(found.to_host(), ~keys)
