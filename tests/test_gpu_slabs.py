"""Whole boxes of rings in slabs (csrc/elp_sweep2.cu, sweep_slabs) against the
generic kernel, bit for bit.

One slab (boxes up to 24^3) and the slabs of a cluster (28^3 to 32^3): rings so
short that every substep moves monomers 0 across slab edges, rings longer than
a plane, launches of one step and of several, and the numbers of replicas at
which a batch changes from clusters to one CTA a box.
"""
import numpy as np
import pytest

import elp

pytestmark = pytest.mark.gpu


def relaxed(L, N, P, seed):
    m = elp.Melt(L=L, N=N, P=P, seed=seed, steps_per_launch=50)
    m.init_melt()
    m.run(300)
    assert m.check() == 0
    return m.fetch()


def run(L, N, P, seed, rings, steps, **kw):
    m = elp.Melt(L=L, N=N, P=P, seed=seed, **kw)
    m.load_chains(*rings, 300)
    m.run(steps)
    assert m.check() == 0
    return (*m.state(), m.accepted())


def equal(a, b):
    return np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1]) and a[2] == b[2]


@pytest.mark.parametrize("L,N,P", [
    (16, 3, 600), (16, 1000, 0), (18, 5, 500), (24, 8, 1400), (28, 6, 2048), (28, 3000, 0), (30, 9, 2000),
    (30, 2000, 0), (32, 14, 2048), (32, 16, 2000), (32, 5000, 0),
])
def test_slabs_equal_the_generic_kernel(L, N, P):
    rings = relaxed(L, N, P, 40 + L)
    want = run(L, N, P, 40 + L, rings, 45, kernel=1)
    assert want[2] > 0
    for spl in (1, 3, 20):
        assert equal(run(L, N, P, 40 + L, rings, 45, steps_per_launch=spl), want), spl


def test_more_rings_than_chain_numbers_run_on_the_generic_kernel():
    for L in (24, 32):
        assert elp.Melt(L=L, N=5, P=2048, seed=1).info().specialised == 1
        assert elp.Melt(L=L, N=5, P=2049, seed=1).info().specialised == 0


@pytest.mark.parametrize("replicas", [2, 40])
def test_a_batch_of_boxes_equals_single_melts(replicas):
    specs = [dict(L=32, N=60, seed=800 + i, steps_per_launch=7) for i in range(replicas)]
    b = elp.Batch(specs)
    b.init_melts()
    b.run(20)
    for j in (0, 1, replicas - 1):
        m = elp.Melt(kernel=1, **specs[j])
        m.init_melt()
        m.run(20)
        want, got = m.state(), b.state(j)
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])


def test_a_wait_that_runs_out_reports_and_leaves_the_context_usable():
    geom = dict(L=32, N=100, seed=9, steps_per_launch=4)
    m = elp.Melt(**geom)
    m.init_melt()
    m.run(8)
    m.sync()
    m.debug_waits(polls=2000, hold_block=0)      # the first slab leaves after a launch's first step
    m.run(4)
    with pytest.raises(elp.ElpError) as e:
        m.sync()
    assert e.value.status == elp.ERR_STATE
    m.debug_waits(0, -1)
    m.init_melt()
    m.run(12)
    ref = elp.Melt(kernel=1, **geom)
    ref.init_melt()
    ref.run(12)
    assert all(np.array_equal(x, y) for x, y in zip(m.state(), ref.state()))
