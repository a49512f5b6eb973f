"""What a user of the engine has it do, as cases that can be timed and compared.

Every case goes through the public binding (``elp.Melt``, ``elp.Batch``,
``elp.Server``).  Kinds:

  dump      one interval of a production run, as the drop-in programs run it:
            ``steps`` time steps, then the chains back on the host, checked
  restart   a run resumed from a dump in pinned host memory: load, ``steps``
            time steps, the chains back into pinned host memory
  observe   in-situ observables of a resident melt
  batch     an ensemble of small melts of uneven size advanced together for
            ``steps`` steps, then every member's chains back on the host
  serve     a burst of jobs through the serving loop, from submit to results

The single melts start from rings (or linear chains) grown by ``melt`` below:
self-avoiding, interpenetrating, with stored length, at the occupancy of a
relaxed melt, so that a pass meets what a production run spends its time in.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "mc-polymer-simulation_b200", "python"))
import elp  # noqa: E402


# ---- the cases ---------------------------------------------------------------
def listed():
    return [
        # a test-sized box watched closely: the smallest call, launches and copies
        dict(name="ring_L16_dump10", kind="dump", L=16, N=50, density=1.2, linear=0, steps=10),
        # the plain ring melt with its dump every 100 steps (whole box on chip)
        dict(name="ring_L32_dump100", kind="dump", L=32, N=100, density=1.2, linear=0, steps=100),
        # linear chains in a small tiled box
        dict(name="linear_L64_dump100", kind="dump", L=64, N=200, density=1.2, linear=1, steps=100),
        # a box edge that no power of two divides well
        dict(name="ring_L40_dump50", kind="dump", L=40, N=100, density=1.2, linear=0, steps=50),
        # a small tiled box: fewer tiles than the GPU has SMs
        dict(name="ring_L64_dump100", kind="dump", L=64, N=300, density=1.2, linear=0, steps=100),
        # a middling box of an odd number of tiles per edge, short rings, lower density
        dict(name="ring_L80_dump100", kind="dump", L=80, N=64, density=1.0, linear=0, steps=100),
        # the single large melt resumed from a dump, one launch of 100 steps
        dict(name="ring_L128_restart100", kind="restart", L=128, N=1000, density=1.2, linear=0, steps=100, spl=100),
        # the same melt with one kernel per time step and a checked dump
        dict(name="ring_L128_dump50_single", kind="dump", L=128, N=1000, density=1.2, linear=0, steps=50, spl=1),
        # the very large melt
        dict(name="ring_L256_dump50", kind="dump", L=256, N=5000, density=1.2, linear=0, steps=50),
        # observables of the large melt between two intervals
        dict(name="observe_L128", kind="observe", L=128, N=1000, density=1.2, linear=0),
        # replicas and parameter sweeps: box 16 to 64, chains 50 to 1000
        dict(name="batch_mix128", kind="batch", replicas=128, steps=100, spl=10),
        # a burst of jobs of the same mix through the serving loop
        dict(name="serve_mix48", kind="serve", jobs=48, steps=200, dump=100, quantum=50),
    ]


EDGES = (14, 16, 20, 24, 28, 32, 40, 48, 64, 72, 80, 96, 112, 128, 160, 192, 256)
SPECIAL = (16, 24, 32, 48, 64, 80, 96, 128)      # boxes that run linear chains
WORK = 256 ** 3 * 50                             # site steps of the largest listed case


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("dump", "dump", "dump", "restart", "restart", "observe", "batch", "serve"))
    if kind == "batch":
        return dict(kind=kind, replicas=_log(rng, 8, 128), steps=_log(rng, 10, 100), spl=rng.choice((1, 10, 10)))
    if kind == "serve":
        return dict(kind=kind, jobs=_log(rng, 4, 48), steps=50 * rng.randint(1, 4), dump=50 * rng.randint(0, 2), quantum=50)
    linear = int(rng.random() < 0.25)
    L = rng.choice(SPECIAL if linear else EDGES)
    density = rng.choice((0.8, 1.0, 1.2, 1.2, 1.2))
    c = dict(kind=kind, L=L, N=_log(rng, 20, min(5000, density * L ** 3 / 16)), density=density, linear=linear)
    if kind != "observe":
        c["steps"] = _log(rng, 5, max(6, min(200, 0.5 * WORK / L ** 3)))
        c["spl"] = rng.choice((1, 10, 100, 100))
    return c


def npol(c):
    return max(1, int(c["density"] * c["L"] ** 3 / c["N"] + 0.5))


def mix(count, seed):
    """Members of an ensemble: L of {16, 24, 32, 48, 64}, N log-uniform on 50..1000
    (at least two rings fit); the sizes belong to the case, the random streams
    to the seed."""
    sizes, streams = np.random.RandomState(count), np.random.RandomState(seed % (1 << 32))
    out = []
    for i in range(count):
        L = (16, 24, 32, 48, 64)[i % 5]
        N = int(round(math.exp(sizes.uniform(math.log(50), math.log(1000)))))
        out.append(dict(L=L, N=min(N, int(0.6 * L ** 3)), density=1.2, seed=int(streams.randint(1, 1 << 30))))
    return out


# ---- inputs ------------------------------------------------------------------
BONDS = [b for b in range(1, 15) if b not in (3, 12)]
VEC = [((b & 1) - (b >> 3), (b >> 1 & 1) - (b >> 3), (b >> 2 & 1) - (b >> 3)) for b in range(16)]


def _splits():
    """For each bond the four ways to go there in two bonds (the common
    neighbours of its two sites): [16][4][2]."""
    out = [[[0, 0]] * 4 for _ in range(16)]
    for b in BONDS:
        out[b] = [[x, y] for x in BONDS for y in BONDS if all(VEC[x][k] + VEC[y][k] == VEC[b][k] for k in range(3))]
        assert len(out[b]) == 4
    return out


def melt(L, N, P, linear, occupancy, seed, device):
    """P chains of N monomers on the periodic FCC lattice of edge L: (start
    (P, 3) int32, bonds (P, N) uint8), on `device`.  Pairs of neighbouring
    sites grow into self-avoiding chains: in each round bonds are replaced by
    two bonds through a free common neighbour, until about `occupancy` of the
    sites hold a run; the monomers left are stored in runs at random."""
    g = torch.Generator(device=device)
    g.manual_seed(seed)
    S = L ** 3
    i64 = dict(dtype=torch.int64, device=device)
    split = torch.tensor(_splits(), **i64)
    vec = torch.tensor(VEC, **i64)

    def rand(n):
        return torch.rand(n, generator=g, device=device, dtype=torch.float64)

    target = int(min(N, max(2, round(occupancy * S / P))))
    first = 2 * torch.randperm(S // 2, generator=g, device=device)[:P]
    pos = torch.cat([first, first + 1])
    ring = torch.arange(P, **i64).repeat(2)
    nxt = torch.cat([torch.arange(P, 2 * P, **i64), torch.arange(P, **i64)])
    bond = torch.cat([torch.full((P,), 1, **i64), torch.full((P,), 15 if linear else 14, **i64)])
    used = torch.zeros(S, dtype=torch.bool, device=device)
    used[pos] = True
    for _ in range(60):
        size = torch.bincount(ring, minlength=P)
        # half of what is missing at most, so that no chain outgrows N
        p = 0.5 * ((target - size).clamp(min=0).double() / size).clamp(max=1.0)
        cand = torch.nonzero((rand(ring.numel()) < p[ring]) & (bond != 15)).squeeze(1)
        way = split[bond[cand], (rand(cand.numel()) * 4).long()]
        at = pos[cand]
        d = vec[way[:, 0]]
        t, u, v = (at % L + d[:, 0]) % L, (at // L % L + d[:, 1]) % L, (at // (L * L) + d[:, 2]) % L
        site = t + L * (u + L * v)
        claim = torch.full((S,), 1 << 40, **i64).scatter_reduce_(0, site, cand, "amin")
        won = torch.nonzero(~used[site] & (claim[site] == cand)).squeeze(1)
        old, new, way = cand[won], ring.numel() + torch.arange(won.numel(), **i64), way[won]
        used[site[won]] = True
        pos, ring = torch.cat([pos, site[won]]), torch.cat([ring, ring[old]])
        nxt = torch.cat([nxt, nxt[old]])
        bond = torch.cat([bond, way[:, 1]])
        nxt[old], bond[old] = new, way[:, 0]
        if ring.numel() >= 0.98 * target * P:
            break
    # place of each site in its chain, by doubling jumps to the chain's last site
    size = torch.bincount(ring, minlength=P)
    assert int(size.max()) <= N
    me = torch.arange(ring.numel(), **i64)
    last = nxt < P
    link, dist = torch.where(last, me, nxt), (~last).long()
    for _ in range(max(1, int(size.max()).bit_length())):
        dist, link = dist + dist[link], link[link]
    base = torch.cumsum(size, 0) - size
    place = base[ring] + size[ring] - 1 - dist
    # stored length: the monomers left go to runs at random
    extra = torch.repeat_interleave(torch.arange(P, **i64), N - size)
    at = base[extra] + (rand(extra.numel()) * size[extra]).long()
    length = 1 + torch.bincount(at, minlength=ring.numel())
    bonds = torch.zeros(P * N, dtype=torch.uint8, device=device)
    ends = torch.cumsum(length, 0) - 1
    bonds[ends[place]] = bond.to(torch.uint8)
    bonds = bonds.view(P, N)
    if not linear:   # monomer 0 anywhere in its run
        off = (rand(P) * length[base]).long()
        bonds = bonds.gather(1, (torch.arange(N, **i64)[None, :] + off[:, None]) % N)
    head = pos[:P]
    start = torch.stack([head % L, head // L % L, head // (L * L)], 1).to(torch.int32)
    return start, bonds


def chains(c, seed):
    occupancy = 0.6 if c["N"] > 300 else 0.7
    return melt(c["L"], c["N"], npol(c), c["linear"], occupancy * min(1.0, c["density"] / 1.2), seed,
                "cuda" if torch.cuda.is_available() else "cpu")


def pinned(t):
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h.numpy()


def prepare(c, seed):
    kind = c["kind"]
    if kind == "batch":
        # an ensemble some way into its run
        b = elp.Batch([dict(m, steps_per_launch=c["spl"]) for m in mix(c["replicas"], seed)])
        b.init_melts()
        b.run(200)
        b.sync()
        return dict(c, batch=b)
    if kind == "serve":
        return dict(c, server=elp.Server(quantum=c["quantum"], io_threads=8), specs=mix(c["jobs"], seed))
    start, bonds = (pinned(x) for x in chains(c, seed))
    spl = min(c["spl"], c["steps"]) if "spl" in c else min(100, c.get("steps", 1))
    m = elp.Melt(L=c["L"], N=c["N"], P=npol(c), seed=seed % (1 << 31), linear=c["linear"], steps_per_launch=max(1, spl))
    s = dict(c, melt=m, start=start, bonds=bonds)
    if kind == "restart":
        s.update(out_start=pinned(torch.zeros(start.shape, dtype=torch.int32)),
                 out_bonds=pinned(torch.zeros(bonds.shape, dtype=torch.uint8)))
        return s
    m.load_chains(start, bonds, 0)
    if kind == "dump":
        m.run(100 if c["L"] > 32 else 500)   # a run under way
        m.sync()
    return s


def run(s):
    kind = s["kind"]
    if kind == "dump":
        s["melt"].run(s["steps"])
        start, bonds, code = s["melt"].fetch_checked()
        return dict(start=start, bonds=bonds, code=code)
    if kind == "restart":
        m = s["melt"]
        m.load_chains(s["start"], s["bonds"], 1000)
        m.run(s["steps"])
        start, bonds = m.fetch(s["out_start"], s["out_bonds"])
        return dict(start=start, bonds=bonds)
    if kind == "observe":
        return s["melt"].observe(32)
    if kind == "batch":
        b = s["batch"]
        b.run(s["steps"])
        got = [b.fetch(j) for j in range(b.n)]
        return dict(start=np.concatenate([x[0].reshape(-1) for x in got]),
                    bonds=np.concatenate([x[1].reshape(-1) for x in got]))
    server = s["server"]
    for m in s["specs"]:
        server.submit(s["steps"], s["dump"], **m)
    server.drain(60.0)
    got = sorted(server.poll(len(s["specs"])), key=lambda r: r["id"])
    return {k: np.array([r[k] for r in got], dtype=np.uint64).view(np.int64)
            for k in ("status", "integrity", "steps", "moves", "dumps", "checksum")}


# ---- what a pass cannot do without --------------------------------------------
# Bytes: the chains in and out once and the 4-byte site words read and written
# once.  Operations: a time step visits every site twice on average; a visit
# cannot do without its share of a Philox call and about 40 integer operations
# (the site word, the next run's, the table entry, the target's, the test and
# the new words).
VISIT = 40


def _melt_work(L, N, P, steps, chains_in):
    return (12 * P + N * P) * (2 if chains_in else 1) + 8 * L ** 3, VISIT * 2 * L ** 3 * steps


def work(c):
    if c["kind"] in ("batch", "serve"):
        b = f = 0
        for m in mix(c["replicas"] if c["kind"] == "batch" else c["jobs"], 1):
            x, y = _melt_work(m["L"], m["N"], npol(m), c["steps"], False)
            b, f = b + x, f + y
        return {"bytes": b, "flops": f}
    if c["kind"] == "observe":
        # the runs' words read once, the per-chain results and the histogram written
        return {"bytes": 4 * c["L"] ** 3 + (16 + 40) * npol(c) + 32 * 8, "flops": 20 * c["N"] * npol(c)}
    b, f = _melt_work(c["L"], c["N"], npol(c), c["steps"], c["kind"] == "restart")
    return {"bytes": b, "flops": f}


def exact(c, seed):
    """Observables in 64 bits from the chains alone; the other kinds return
    whole numbers."""
    if c["kind"] != "observe":
        return None
    start, bonds = chains(c, seed)
    P, N = bonds.shape
    step = torch.tensor(VEC, dtype=torch.int64, device=bonds.device)[bonds.long()]
    if c["linear"]:
        step[:, -1] = 0
    r = torch.cumsum(step, 1) - step          # monomer m relative to monomer 0
    x = torch.stack([r[..., 0] + r[..., 1] - r[..., 2], r[..., 0] - r[..., 1], r[..., 2]], -1)
    num = N * x.square().sum((1, 2)) - x.sum(1).square().sum(1)
    zero = (bonds == 0).sum(1)
    return dict(cms_tuv=start.double() + r.sum(1).double() / N, rg2=num.double() / (2.0 * N * N),
                sl=zero.double() / (N - 1 if c["linear"] else N), run_hist=None)
