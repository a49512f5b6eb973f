"""Fetches into pageable buffers across the change to staged copies.

After 64 copies of a handle, chains of up to 512 KB come to pageable buffers
through pinned memory that is set up once.  Members of a batch of every size,
below and above that bound, smallest first, give the same bytes before, at and
after the change.
"""
import numpy as np
import pytest

import elp

pytestmark = pytest.mark.gpu


def test_a_batch_of_growing_members_fetches_the_same_bytes():
    specs = [dict(L=L, N=N, seed=L) for L, N in ((16, 50), (20, 60), (24, 100), (32, 100), (48, 200), (64, 300), (80, 100))]
    b = elp.Batch(specs)
    b.init_melts()
    b.run(100)
    want = []
    for j, kw in enumerate(specs):
        m = elp.Melt(**kw)
        m.init_melt()
        m.run(100)
        want.append(m.fetch())
    for _ in range(63):
        b.fetch(0)
    for _ in range(2):
        for j, w in enumerate(want):
            got = b.fetch(j)
            assert all(np.array_equal(x, y) for x, y in zip(got, w)), j


@pytest.mark.parametrize("L,N", [(16, 50), (64, 300)])
def test_one_melt_fetches_the_same_bytes(L, N):
    m = elp.Melt(L=L, N=N, seed=9)
    m.init_melt()
    m.run(50)
    want = m.fetch()
    for _ in range(70):
        start, bonds, code = m.fetch_checked()
        assert code == 0 and np.array_equal(start, want[0]) and np.array_equal(bonds, want[1])
