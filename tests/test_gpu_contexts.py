"""Several contexts on one device at once, a thread each.

A context cannot see the others: clusters of slabs (L = 32), launches set up
ahead of the one before (one step a launch), cooperative launches (L = 128) and
the rebuild's launches share the SMs in any order.  Each gives what it gives
alone.
"""
import threading

import numpy as np
import pytest

import elp

pytestmark = pytest.mark.gpu

SPECS = ([dict(L=32, N=100, steps_per_launch=50)] * 6 + [dict(L=28, N=60, steps_per_launch=25)] * 2 +
         [dict(L=64, N=300, steps_per_launch=1)] * 3 + [dict(L=128, N=1000, steps_per_launch=50),
         dict(L=128, N=1000, steps_per_launch=1), dict(L=16, N=50, steps_per_launch=1), dict(L=72, N=300, steps_per_launch=50)])


def intervals(m, out):
    for _ in range(3):
        m.run(50)
        out.append(m.fetch_checked())
    out.append(m.observe(16))


def test_contexts_at_once_give_what_each_gives_alone():
    melts = [elp.Melt(seed=40 + i, **kw) for i, kw in enumerate(SPECS)]
    alone, together = [], []
    for m in melts:
        m.init_melt()
        alone.append([])
        intervals(m, alone[-1])
    for m in melts:
        m.init_melt()
        together.append([])
    threads = [threading.Thread(target=intervals, args=(m, o)) for m, o in zip(melts, together)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for a, b in zip(alone, together):
        assert len(a) == len(b) == 4
        for x, y in zip(a[:3], b[:3]):
            assert x[2] == y[2] == 0 and np.array_equal(x[0], y[0]) and np.array_equal(x[1], y[1])
        assert all(np.array_equal(a[3][k], b[3][k]) for k in a[3])
