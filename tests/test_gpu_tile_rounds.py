"""16^3 tiles at three and at four CTAs an SM (csrc/elp_sweep2.cu).

The kernel is chosen by the number of tiles and SMs.  On 148 SMs, three take
444 tiles in one round and four 592; batches of boxes of 64 tiles on both sides
of each line, rings and linear chains, launches of one step and of several,
equal single melts on the generic kernel (rings) or alone (linear chains).
"""
import numpy as np
import pytest

import elp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("linear", [0, 1])
@pytest.mark.parametrize("members,spl", [(6, 4), (7, 4), (7, 1), (9, 4), (10, 4), (14, 4), (14, 1), (28, 4), (36, 4)])
def test_batches_of_any_number_of_tiles_equal_single_melts(members, spl, linear):
    specs = [dict(L=64, N=60 + i, seed=500 + i, steps_per_launch=spl, linear=linear) for i in range(members)]
    b = elp.Batch(specs)
    b.init_melts()
    b.run(9)
    for j in sorted({0, members // 2, members - 1}):
        kw = dict(specs[j]) if linear else dict(specs[j], kernel=1)
        m = elp.Melt(**kw)
        m.init_melt()
        m.run(9)
        assert all(np.array_equal(x, y) for x, y in zip(b.state(j), m.state()))
        assert b.check(j) == 0 and b.accepted(j) == m.accepted()


def test_a_box_of_512_tiles_equals_the_generic_kernel():
    geom = dict(L=128, N=200, seed=7, periodic=0, tile=(16, 16, 16))
    got = []
    for kw in (dict(steps_per_launch=5), dict(kernel=1)):
        m = elp.Melt(**geom, **kw)
        m.init_melt()
        m.run(10)
        got.append((*m.state(), m.accepted()))
    assert all(np.array_equal(x, y) for x, y in zip(*got))
