"""The server's scratch for dumps comes from the device's memory pool.

The I/O threads rebuild the chains of snapshots in scratch of their own: a few
bytes a site and a byte a bond each.  It is taken from the pool that the jobs'
memory comes from (an allocation outside it stops the other threads) and given
back when the server ends, so that servers one after another hold no more than
the jobs' own memory.
"""
import os
import subprocess
import sys

import pytest

import elp

pytestmark = pytest.mark.gpu

PROGRAM = """
import sys
sys.path.insert(0, sys.argv[1])
import elp, torch
L, N, jobs = 192, 500, 8
used = lambda: (lambda f, t: t - f)(*torch.cuda.mem_get_info())
torch.zeros(1, device="cuda")
out = []
for _ in range(3):
    s = elp.Server(quantum=10, io_threads=8)
    before = used()
    for i in range(jobs):
        s.submit(20, 10, L=L, N=N, seed=i)
    s.drain(60.0)
    got = s.poll(jobs)
    assert [r["status"] for r in got] == [0] * jobs and [r["integrity"] for r in got] == [0] * jobs
    s.close()
    out.append(used() - before)
print(*out)
"""


def test_scratch_is_given_back_when_the_server_ends():
    python = os.path.join(elp.PKG, "python")
    r = subprocess.run([sys.executable, "-c", PROGRAM, python], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr[-2000:]
    held = [int(x) for x in r.stdout.split()]
    state = 8 * 2 * 4 * 192**3                       # the jobs' states and snapshots
    scratch = 8 * (6 * 192**3 + 12 * 192**3 // 10)   # ranking and bonds of eight threads
    assert scratch > state * 0.6
    assert max(held) < state + scratch // 2, (held, state, scratch)
    assert held[1] + held[2] < scratch // 2, (held, state, scratch)
