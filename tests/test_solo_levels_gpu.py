"""Single-source levels that one block runs by itself: frontiers of just under, at
and over its edge limit (4 per thread: 1,024 and 2,048), hubs that end a stretch,
stretches longer than the 64 levels one may have, the switch to bottom-up and
back, and every one of these within a run of small levels.  Depths are the
oracle's, frontiers and directions cpu_do's, traces account for every vertex."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _spider(gb, legs, length, extra=0):
    """A centre with `legs` paths of `length` vertices; `extra` leaves on the
    middle vertex of the first path."""
    v = np.arange(legs * length).reshape(legs, length) + 1
    u = np.concatenate([np.zeros(legs, np.int64), v[:, :-1].ravel()])
    w = np.concatenate([v[:, 0], v[:, 1:].ravel()])
    n = 1 + legs * length
    if extra:
        u = np.concatenate([u, np.full(extra, v[0, length // 2])])
        w = np.concatenate([w, n + np.arange(extra)])
        n += extra
    return gb.from_edges(n, u.astype(np.uint32), w.astype(np.uint32))


CASES = [(1, 300, 0), (3, 130, 0), (511, 5, 0), (512, 5, 0), (513, 5, 0), (1023, 4, 0), (1024, 4, 0), (1025, 4, 0),
         (2049, 3, 0), (2, 200, 31), (2, 200, 32), (2, 200, 3000), (7, 140, 1022), (7, 140, 5000)]


@pytest.mark.parametrize("legs,length,extra", CASES)
def test_depths_and_traces(gb, oracle, legs, length, extra):
    g = _spider(gb, legs, length, extra)
    bfs = gb.GpuBfs(g)
    for src in sorted({0, 1, length, g.n - 1, g.n // 2}):
        want = oracle.bfs_serial(g, src)
        for block in (256, 512):
            for hub_min in (32, 4096):
                for alpha, beta in ((15.0, 18.0), (1e-9, 18.0), (2.0, 2.0), (1e9, 1e9)):
                    o = gb.BfsOptions(block=block, hub_min=hub_min, alpha=alpha, beta=beta)
                    d, tr = bfs.run("gpu_do_persistent", src, opts=o, trace=True)
                    assert np.array_equal(d, want), (src, block, hub_min, alpha)
                    _, ctr = oracle.bfs_do(g, src, alpha, beta)
                    assert [L["direction"] for L in tr] == [t[1] for t in ctr]
                    assert [L["frontier"] for L in tr] == [t[2] for t in ctr]
                    assert np.array_equal(bfs.run("gpu_do_persistent", src, opts=o), want)
                    assert bfs.lastLevels() == len(tr)


def test_many_in_flight(gb, oracle):
    g = _spider(gb, 40, 150, 3000)
    srcs = np.arange(0, g.n, 433, dtype=np.uint32)[:24]
    want = [oracle.bfs_serial(g, int(s)) for s in srcs]
    bfs = gb.GpuBfs(g)
    for k in (1, 4, 16):
        d, _, _ = bfs.run_many("gpu_do_persistent", srcs, opts=gb.BfsOptions(in_flight=k))
        for i in range(len(srcs)):
            assert np.array_equal(d[i], want[i]), (k, i)
