"""Whole boxes loaded for one step at a time (csrc/elp_sweep2.cu, load_words).

A thread copies every THREADS-th word and then sees to the labelled ones among
them.  Boxes whose words the threads do and do not divide, with none, one and
many labelled words a thread, loaded and stored at every step.
"""
import numpy as np
import pytest

import elp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,N,P", [
    (16, 3, 900), (16, 4000, 1), (18, 4, 1200), (20, 5, 1600), (22, 4, 2048), (24, 6, 2048), (26, 8, 2000), (26, 3000, 0),
    (28, 10, 2048), (30, 12, 2048), (32, 15, 2048),
])
def test_single_step_launches_equal_the_generic_kernel(L, N, P):
    runs = []
    for kw in (dict(), dict(kernel=1)):
        m = elp.Melt(L=L, N=N, P=P, seed=30 + L, steps_per_launch=1, **kw)
        m.init_melt()
        m.run(40)
        assert m.check() == 0
        runs.append((*m.state(), m.accepted()))
    assert all(np.array_equal(a, b) for a, b in zip(*runs))


@pytest.mark.parametrize("L,N,P", [(16, 2, 1500), (24, 8, 1800), (32, 16, 2048)])
def test_linear_chains_do_not_depend_on_the_steps_per_launch(L, N, P):
    runs = []
    for spl in (1, 40):
        m = elp.Melt(L=L, N=max(N, 3), P=P, seed=30 + L, steps_per_launch=spl, linear=1)
        m.init_melt()
        m.run(40)
        assert m.check() == 0
        runs.append((*m.state(), m.accepted()))
    assert all(np.array_equal(a, b) for a, b in zip(*runs))
