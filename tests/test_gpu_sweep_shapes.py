"""Every specialised domain shape against the generic kernel, bit for bit.

The specialised kernels (csrc/elp_sweep2.cu) run from the same loaded rings as
the generic one (csrc/elp_sweep.cu, itself equal to the host replay,
test_gpu_parity.py) in launches of one and of several steps: site words, chain
records and accepted moves must agree.  Shapes whose last warp is not full,
colour moduli that are no power of two, substeps that do not come in fours,
tiles at every origin modulo 4, rings short enough to put hundreds of
monomer-0 runs into a domain.
"""
import numpy as np
import pytest

import elp

pytestmark = pytest.mark.gpu

SHAPES = [
    (16, {}), (18, {}), (20, {}), (22, {}), (24, {}), (26, {}), (28, {}), (30, {}), (32, {}),
    (40, {}), (60, {}), (72, {}), (48, {}), (80, {}),
    (48, dict(periodic=0, tile=(24, 24, 24))), (96, dict(periodic=0, tile=(48, 24, 24))),
    (64, dict(periodic=0, tile=(32, 16, 16))), (64, dict(periodic=0, tile=(32, 32, 16))),
    (64, dict(periodic=0, tile=(32, 32, 32))),
]


# slot tables that N = 25 outgrows (mean + 8 sigma + 16): the generic kernel runs
SLOTS = {(32, 32, 16): 1024, (32, 32, 32): 1792}


def has_kernel(m, kw):
    i = m.info()
    runs = i.P * i.tile[0] * i.tile[1] * i.tile[2] / i.L ** 3
    cap = SLOTS.get(tuple(kw.get("tile", ())), 1 << 30)
    return i.periodic or runs + 8 * runs ** 0.5 + 16 <= cap


@pytest.mark.parametrize("N", [25, 160])
@pytest.mark.parametrize("L,kw", SHAPES)
def test_shape_equals_generic_kernel(L, kw, N):
    seed = 7000 + L + N
    start = elp.Melt(L=L, N=N, seed=seed, steps_per_launch=50, **kw)
    start.init_melt()
    start.run(400)                       # away from the collapsed initial melt
    rings = start.fetch()
    assert start.check() == 0
    want = None
    for kernel, spl in ((1, 1), (0, 1), (0, 7)):
        m = elp.Melt(L=L, N=N, seed=seed, kernel=kernel, steps_per_launch=spl, **kw)
        assert m.info().specialised == (0 if kernel else int(has_kernel(m, kw)))
        m.load_chains(*rings, 400)
        m.run(15)
        got = (*m.state(), m.accepted())
        if want is None:
            want = got
            assert got[2] > 0
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1]) and got[2] == want[2], (kernel, spl)
        assert m.check() == 0


def test_ring_only_shapes_still_refuse_linear_chains():
    for L in (18, 20, 28, 40, 72):
        with pytest.raises(elp.ElpError) as e:
            elp.Melt(L=L, N=50, linear=1)
        assert e.value.status == elp.ERR_ARG, L
