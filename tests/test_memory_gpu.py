"""The library's per-device memory pool (l3d_memory_trim, l3d_memory_reserved): trimming hands
the memory of destroyed handles back to the driver and leaves the memory of live handles, which
stay usable."""
import numpy as np
import pytest

from luvas3d import memory_reserved, trim_memory
from luvas3d.cloud import PointAccumulator

pytestmark = pytest.mark.gpu


def samples(n, seed):
    rng = np.random.default_rng(seed)
    s = np.zeros((n, 9))
    s[:, :3] = rng.uniform(-1.0, 1.0, (n, 3))
    s[:, 5] = 1.0
    s[:, 6:] = 0.5
    return s


def test_trim_releases_destroyed_handles_memory_and_keeps_live_handles():
    live = PointAccumulator(0.01)
    live.add_points(samples(1000, 1))
    first = live.cloud()
    big = PointAccumulator(0.0005)
    big.add_points(samples(2_000_000, 2))      # about 2 M cells: a table of 4 M slots, 350 MB
    assert big.size > 1_900_000
    r_big, u_big = memory_reserved()
    assert r_big >= u_big >= 300 << 20

    trim_memory(1 << 40)                        # more than the pool holds: nothing to release
    assert memory_reserved()[0] == r_big

    big.destroy()
    trim_memory(0)
    r, u = memory_reserved()
    assert u <= u_big - (300 << 20)             # the big table and its upload buffer are gone
    assert r <= r_big - (300 << 20)             # and their memory went back to the driver
    assert r >= u > 0                           # the live accumulator's table stays

    again = live.cloud()                        # the live handle still works after the trim
    np.testing.assert_array_equal(again.positions, first.positions)
    live.add_points(samples(1000, 3))
    assert live.size > first.positions.shape[0]
    live.destroy()


def test_reads_of_every_size_survive_trimming_and_threads():
    """Read-backs go through two kept pinned buffers of 1 MB: clouds smaller than one, around one and
    two, and of several, read from several threads at once, before and after the buffers are given
    back, equal the samples that went in."""
    import threading

    def check(n, seed):
        rng = np.random.default_rng(seed)
        cell = 0.01
        ids = rng.choice(200 ** 3, n, replace=False)
        at = np.stack([ids % 200, ids // 200 % 200, ids // 40000], 1)
        s = samples(n, seed)
        s[:, :3] = (at + 0.5) * cell
        s[:, 6:] = at % 251
        acc = PointAccumulator(cell)
        acc.add_points(s)
        c = acc.cloud()
        acc.destroy()
        order = np.lexsort((at[:, 0], at[:, 1], at[:, 2]))
        np.testing.assert_array_equal(c.cells, at[order])
        np.testing.assert_array_equal(c.positions, s[order, :3].astype(np.float32))
        np.testing.assert_array_equal(c.colors, (at[order] % 251).astype(np.uint8))
        assert (c.support == 1).all()

    failed = []

    def work(n, seed):
        try:
            check(n, seed)
        except BaseException as e:  # noqa: BLE001
            failed.append((n, e))

    for _ in range(2):
        for n in (1, 25575, 25576, 51150, 51151, 300000):  # 41 bytes a point
            check(n, n)
        threads = [threading.Thread(target=work, args=(30000 + 9000 * i, i)) for i in range(7)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not failed, failed
        trim_memory(0)
