"""Observables of a melt with runs off its chains (elp_observe).

A plain run on an empty site whose bond leads into a ring is on no ring's path
from monomer 0.  The rebuild by list ranking starts from runs of a sublattice
and so meets it; elp_observe must still return the rings' own observables, as
a walk along each ring gives them, elp_check code 4, and a fetch an error.
"""
import numpy as np
import pytest

import elp

pytestmark = pytest.mark.gpu
VALID = [b for b in range(16) if b not in (0, 3, 12, 15)]


def step(s, b, L):
    t, u, v = s % L, s // L % L, s // (L * L)
    d = b >> 3
    return (t + (b & 1) - d) % L + L * ((u + (b >> 1 & 1) - d) % L + L * ((v + (b >> 2 & 1) - d) % L))


def stray_runs(w, L, q, node, n, rng):
    """Words with n plain runs added on empty sites (of the ranking's
    sublattice, one site in q, or off it) whose bonds lead to plain runs."""
    w, left = w.copy(), n
    for s in rng.permutation(np.flatnonzero(w == 0)):
        s = int(s)
        t, u, v = s % L, s // L % L, s // (L * L)
        if ((t + 2 * u + 3 * v) % q == 0) != node:
            continue
        into = [b for b in VALID if w[step(s, b, L)] and not w[step(s, b, L)] & 16]
        if into:
            w[s] = np.uint32(1 << 16 | into[int(rng.integers(len(into)))])
            left -= 1
            if not left:
                return w
    raise AssertionError("too few empty sites beside the chains")


@pytest.mark.parametrize("L,N,linear,q", [(16, 50, 0, 4), (32, 100, 0, 4), (32, 100, 1, 4), (64, 2000, 0, 4),
                                          (180, 500, 0, 8)])
@pytest.mark.parametrize("node", [True, False])
def test_runs_off_the_chains_leave_the_observables_alone(L, N, linear, q, node):
    m = elp.Melt(L=L, N=N, seed=61, linear=linear, steps_per_launch=20)
    m.init_melt()
    m.run(200)
    w, r = m.state()
    want = m.observe(24)
    m.set_state(stray_runs(w, L, q, node, 40, np.random.default_rng(L)), r, m.step)
    for _ in range(2):
        got = m.observe(24)
        for k in want:
            assert np.array_equal(got[k], want[k]), k
    assert m.check() == 4
    assert m.fetch_checked()[2] == 4
    with pytest.raises(elp.ElpError) as e:
        m.fetch()
    assert e.value.status == elp.ERR_INTEGRITY
    m.set_state(w, r, m.step)            # the context stays usable
    assert m.check() == 0
    got = m.observe(24)
    assert all(np.array_equal(got[k], want[k]) for k in want)
