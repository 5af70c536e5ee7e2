"""gpu_edge and gpu_do, one launch per level: every block size and edges per
thread, owner ranges in and past the staged 2,048, lists whose expansion crosses
blocks, the switch to bottom-up and back, sources without edges, and runs of two
handles in turn (their level numbers are their own).  Depths are the oracle's;
frontiers, edges and directions cpu_do's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graph(gb, kind):
    rng = np.random.default_rng(5)
    if kind == "path":
        v = np.arange(699)
        return gb.from_edges(700, v.astype(np.uint32), (v + 1).astype(np.uint32))
    if kind == "star":  # one list over many blocks, then 70,000 lists of one entry
        return gb.from_edges(70_001, np.zeros(70_000, np.uint32), np.arange(1, 70_001, dtype=np.uint32))
    if kind == "tree":  # a frontier whose chunks have more than 2,048 owners
        n = 40_000
        v = np.arange(1, n)
        return gb.from_edges(n, ((v - 1) // 190).astype(np.uint32), v.astype(np.uint32))
    if kind == "dense":
        return gb.from_edges(300, rng.integers(0, 300, 20_000).astype(np.uint32), rng.integers(0, 300, 20_000).astype(np.uint32))
    # sparse and uneven, with vertices of degree 0 and components apart
    u = (rng.random(30_000) ** 3 * 20_000).astype(np.uint32)
    return gb.from_edges(20_001, u, rng.integers(0, 20_000, 30_000).astype(np.uint32))


@pytest.mark.parametrize("kind", ["path", "star", "tree", "dense", "sparse"])
def test_depths_and_traces(gb, oracle, kind):
    g = _graph(gb, kind)
    bfs, other = gb.GpuBfs(g), gb.GpuBfs(g)
    for src in (0, 1, g.n // 2, g.n - 1):
        want = oracle.bfs_serial(g, src)
        for tg, ept in ((32, 1), (32, 64), (96, 3), (256, 1), (256, 2), (256, 5), (1024, 4), (1024, 64)):
            for alpha in (1e-9, 2.0, 15.0, 1e9):
                o = gb.BfsOptions(tg=tg, ept=ept, alpha=alpha)
                for b in (bfs, other):
                    d, tr = b.run("gpu_do", src, opts=o, trace=True)
                    assert np.array_equal(d, want), (src, tg, ept, alpha)
                _, ctr = oracle.bfs_do(g, src, alpha, 18.0)
                assert [(L["direction"], L["frontier"], L["edges"]) for L in tr] == [tuple(t[1:4]) for t in ctr]
                assert bfs.lastLevels() == len(tr)
            o = gb.BfsOptions(tg=tg, ept=ept)
            d, tr = bfs.run("gpu_edge", src, opts=o, trace=True)
            assert np.array_equal(d, want)
            assert sum(L["frontier"] for L in tr) == np.count_nonzero(want != 0xFFFFFFFF)
            assert bfs.lastGpuMs() > 0
    d, _, _ = bfs.run_many("gpu_do", np.array([0, g.n - 1, 0], np.uint32))
    assert np.array_equal(d[0], d[2]) and np.array_equal(d[1], oracle.bfs_serial(g, g.n - 1))
