"""The slabs' handshake at the end of a substep (csrc/elp_sweep2.cu).

One lane of a warp arrives at the neighbour's mbarrier for all 32.  What the
lanes read and wrote of the words that the neighbour may change next must be
ordered before that arrival: a barrier over the warp, and a release at cluster
scope, as the neighbour's waits acquire.  No run can be relied on to show a
missing order, so the source is looked at, and dense melts of short rings,
which send at every substep, are compared with the generic kernel over many
steps.
"""
import os
import re

import numpy as np
import pytest

import elp

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mc-polymer-simulation_b200", "csrc",
                   "elp_sweep2.cu")


def test_arrivals_for_a_warp_release_what_its_lanes_did():
    src = open(SRC).read()
    waits = re.findall(r"mbarrier\.try_wait[\w.:]*", src)
    assert waits and all(".acquire.cluster." in w for w in waits)
    arrivals = [m for m in re.finditer(r"mbarrier\.arrive[\w.:]*", src) if "shared::cluster" in m.group(0)]
    assert len(arrivals) == 1 and ".cluster." in arrivals[0].group(0).replace(".shared::cluster", "")
    body = src[src.index("auto announce = [&]()"):arrivals[0].end()]
    warp, release = body.find("__syncwarp();"), body.find("fence.release.sync_restrict::shared::cta.cluster;")
    assert 0 < body.index("__reduce_add_sync") < warp < release


@pytest.mark.gpu
@pytest.mark.parametrize("L,N,P", [(28, 6, 2048), (30, 9, 2000), (32, 16, 2000), (32, 600, 0)])
def test_dense_melts_equal_the_generic_kernel_over_many_steps(L, N, P):
    runs = []
    for kw in (dict(steps_per_launch=50), dict(kernel=1)):
        m = elp.Melt(L=L, N=N, P=P, seed=70 + L, **kw)
        m.init_melt()
        m.run(1000)
        assert m.check() == 0
        runs.append((*m.state(), m.accepted()))
    assert all(np.array_equal(a, b) for a, b in zip(*runs))
