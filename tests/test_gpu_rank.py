"""Chains by list ranking (csrc/elp_rank.cu) against a walk on the host.

The rebuild cuts the chains at a sublattice of nodes (one site in four, one in
eight in large boxes; boxes whose edge the four does not divide; one kernel up
to 64^3, launches above), so it is compared, byte for byte, with a walk along
the site words in Python, and its observables with those of the fetched bonds.
"""
import numpy as np
import pytest

import elp
import observables as obs

pytestmark = pytest.mark.gpu
STEP = [((b & 1) - (b >> 3), (b >> 1 & 1) - (b >> 3), (b >> 2 & 1) - (b >> 3)) for b in range(16)]


def host_walk(words, rec, L, N, P):
    start, bonds = np.zeros((P, 3), np.int32), np.zeros((P, N), np.uint8)
    words = words.tolist()
    for p in range(P):
        site, cnt, off = (int(x) for x in rec[p, :3])
        x = [site % L, site // L % L, site // (L * L)]
        start[p] = x
        at, here = 0, cnt - off
        while True:
            b = words[x[0] + L * (x[1] + L * x[2])] & 15
            at += here
            bonds[p, at - 1] = b
            if b == 15:
                break
            x = [(x[k] + STEP[b][k]) % L for k in range(3)]
            s = x[0] + L * (x[1] + L * x[2])
            if s == site:
                break
            here = words[s] >> 16
        assert at + off == N
    return start, bonds


@pytest.mark.parametrize("L,N,linear", [
    (16, 3, 0), (16, 50, 0), (16, 4000, 0), (18, 40, 0), (22, 200, 0), (32, 100, 1), (40, 65, 0), (64, 300, 0),
    (64, 200, 1), (72, 100, 0), (80, 700, 1), (112, 500, 0),
])
def test_ranked_chains_equal_a_host_walk(L, N, linear):
    m = elp.Melt(L=L, N=N, P=0 if N > 3 else 300, seed=91, linear=linear, steps_per_launch=20)
    m.init_melt()
    for steps in (0, 300):
        m.run(steps)
        want = host_walk(*m.state(), L, N, m.P)
        pinned = m.fetch()
        start, bonds, code = m.fetch_checked()
        assert code == 0 and m.check() == 0
        for got in (pinned, (start, bonds)):
            assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
        o = m.observe(24)
        assert np.array_equal(o["run_hist"].astype(np.int64), obs.run_length_hist(bonds, 24))
        assert np.array_equal(o["sl"], (bonds == 0).sum(1) / (N - 1.0 if linear else float(N)))


def test_ranking_node_density_of_the_large_box():
    """One site in eight above 4 Mi sites: the fetched chains, loaded again,
    give back every site word and record."""
    m = elp.Melt(L=192, N=900, seed=92, steps_per_launch=20)
    m.init_melt()
    m.run(200)
    w, r = m.state()
    start, bonds, code = m.fetch_checked()
    assert code == 0
    m.load_chains(start, bonds, 200)
    w2, r2 = m.state()
    assert np.array_equal(w, w2) and np.array_equal(r, r2)
