"""Fetches, checks and observables on a device without room for the ranking.

The rebuild by list ranking (csrc/elp_rank.cu) needs 6 to 8 bytes a site, which
a device that is nearly full may not have.  The calls then follow each ring
from its label (csrc/elp_walk.cu, observe_kernel), as they do above L = 512,
and give the same bytes.  elp_debug_scratch bounds a context's scratch to what
the walk needs, so the two are compared on every kind of melt: the walk is
also the oracle of the ranking at sizes that a walk on the host does not reach.
"""
import numpy as np
import pytest

import elp

pytestmark = pytest.mark.gpu


def sizes(m, L, N):
    """Bytes of scratch: observables' sums, rebuilt chains, statuses, visit counters, ranking."""
    S, P = L**3, m.P
    q = 4 if S <= 1 << 22 else 8
    nodes = -(-L // q) * L * L + P
    return dict(obs=8 * (6 * P + 64), out=64 + -(-P * N // 16) * 16 + 12 * P, status=4 * P, visit=4 * S,
                rank=16 * nodes + 4 * S + 4 * P)


def results(m):
    return (*m.fetch(), *m.fetch_checked(), m.check(), m.observe(32))


def assert_same(a, b):
    for x, y in zip(a, b):
        if isinstance(x, dict):
            assert all(np.array_equal(x[k], y[k]) for k in x)
        else:
            assert np.array_equal(x, y)


@pytest.mark.parametrize("L,N,linear,steps", [
    (16, 50, 0, 500), (16, 50, 1, 500), (16, 2000, 0, 400), (20, 40, 0, 300), (32, 100, 1, 1000), (64, 14, 0, 500),
    (64, 200, 1, 500), (64, 65536, 0, 20), (128, 1000, 0, 500), (180, 300, 0, 100), (256, 5000, 0, 300),
])
def test_walks_and_ranking_give_the_same(L, N, linear, steps):
    m = elp.Melt(L=L, N=N, seed=77, linear=linear, steps_per_launch=20)
    m.init_melt()
    z = sizes(m, L, N)
    for k in (0, steps):
        m.run(k)
        m.debug_scratch(0)
        ranked = results(m)
        assert ranked[4] == ranked[5] == 0
        m.debug_scratch(z["obs"] + z["out"] + z["status"] + z["visit"])
        assert_same(results(m), ranked)
        m.debug_scratch(z["obs"])            # the observables alone need no scratch but their sums
        assert_same([m.observe(32)], ranked[6:])


def test_the_ranking_gives_its_scratch_up_to_the_walk():
    """A melt found amiss needs the walk's counters beside the ranking."""
    L, N = 64, 200
    m = elp.Melt(L=L, N=N, seed=78)
    m.init_melt()
    m.run(200)
    z = sizes(m, L, N)
    m.debug_scratch(z["out"] + z["status"] + z["rank"])
    w, r = m.state()
    assert m.check() == 0
    bad = w.copy()
    k = int(np.flatnonzero((w != 0) & ((w & 16) == 0))[7])
    bad[k] = (bad[k] & ~np.uint32(15)) | np.uint32(3)
    m.set_state(bad, r, m.step)
    assert m.check() != 0
    assert m.fetch_checked()[2] != 0
    with pytest.raises(elp.ElpError) as e:
        m.observe(16)
    assert e.value.status == elp.ERR_INTEGRITY
    m.set_state(w, r, m.step)
    assert m.check() == 0 and m.fetch_checked()[2] == 0


def test_no_room_at_all_is_reported_and_the_context_stays_usable():
    m = elp.Melt(L=32, N=100, seed=79)
    m.init_melt()
    m.run(50)
    want = results(m)
    m.debug_scratch(1000)
    for call in (m.fetch, m.fetch_checked, m.check, lambda: m.observe(16)):
        with pytest.raises(elp.ElpError) as e:
            call()
        assert e.value.status == elp.ERR_NOMEM
    m.debug_scratch(0)
    assert_same(results(m), want)
