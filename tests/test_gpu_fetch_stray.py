"""A fetch of melts with words that belong to no chain but lead into one.

A run of no monomers, a second run with a chain's label, a label of no chain:
no monomer is out of place, but such a word reaches a chain's last run, and
elp_fetch_chains refuses the melt (a run leading into another chain).
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


def with_stray(w, L, P, kind, node):
    """One such word on an empty site beside a plain run."""
    w = w.copy()
    for s in np.flatnonzero(w == 0):
        s = int(s)
        t, u, v = s % L, s // L % L, s // (L * L)
        into = [b for b in VALID if w[step(s, b, L)] and not w[step(s, b, L)] & 16]
        if into and ((t + 2 * u + 3 * v) % 4 == 0) == node:
            label = {"empty run": 0, "second label": 5 << 5 | 16, "label of no chain": (P + 3) << 5 | 16}[kind]
            w[s] = np.uint32(label | into[0])
            return w
    raise AssertionError("no empty site beside a chain")


@pytest.mark.parametrize("kind", ["empty run", "second label", "label of no chain"])
@pytest.mark.parametrize("node", [True, False])
@pytest.mark.parametrize("L,linear", [(16, 0), (64, 0), (64, 1)])
def test_words_that_lead_into_a_chain_are_refused(kind, node, L, linear):
    m = elp.Melt(L=L, N=60, seed=83, linear=linear)
    m.init_melt()
    m.run(300)
    w, r = m.state()
    sound = m.fetch()
    m.set_state(with_stray(w, L, m.P, kind, node), r, m.step)
    with pytest.raises(elp.ElpError) as e:
        m.fetch()
    assert e.value.status == elp.ERR_INTEGRITY
    assert m.check() != 0
    m.set_state(w, r, m.step)
    assert all(np.array_equal(a, b) for a, b in zip(m.fetch(), sound))
