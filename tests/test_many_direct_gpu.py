"""Several single-source traversals per call whose kernels return the depths
themselves (up to 2^20 vertices) or not (one more): every packed width, depths past
the widest, isolated sources, more sources than buffers, one output place for all,
and a wait that runs out followed by a call that works."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 33, 300, 66_000, (1 << 20) - 1, 1 << 20, (1 << 20) + 1])
@pytest.mark.parametrize("in_flight", [1, 4, 16])
def test_rows(gb, oracle, n, in_flight):
    edges = min(n - 1, 66_000) if n != 66_000 else n - 1  # a path, then vertices of degree 0
    edges = edges if n < 1 << 20 else 300
    v = np.arange(edges)
    g = gb.from_edges(n, v.astype(np.uint32), (v + 1).astype(np.uint32))
    few = 3 if edges > 10_000 else 40
    src = np.random.default_rng(n).integers(0, min(n, edges + 5), few).astype(np.uint32)
    src[0], src[-1] = 0, n - 1
    bfs = gb.GpuBfs(g)
    o = gb.BfsOptions(in_flight=in_flight)
    d, ms, levels = bfs.run_many("gpu_do_persistent", src, opts=o)
    for i, s in enumerate(src):
        want = oracle.bfs_serial(g, int(s))
        assert np.array_equal(d[i], want), (i, int(s))
        assert levels[i] == want[want != 0xFFFFFFFF].max() + 1
    assert (ms > 0).all() and bfs.lastLevels() == levels[-1]
    one = np.empty(n, np.uint32)
    bfs.run_many("gpu_do_persistent", src, out=one, stride=0, opts=o)
    assert np.array_equal(one, d[-1])
    _, _, on_device = bfs.run_many("gpu_do_persistent", src, opts=o, device=True)
    assert np.array_equal(levels, on_device)


def test_timeout_is_reported_and_left_behind(gb, oracle):
    g = gb.gen.rmat(16, 16, False, 1)
    bfs = gb.GpuBfs(g)
    src = gb.pick_sources(g, 6, 7)
    with pytest.raises(gb.GraphError):  # one poll is never enough for a barrier of 296 blocks
        bfs.run_many("gpu_do_persistent", src, opts=gb.BfsOptions(spin_limit=1))
    with pytest.raises(gb.GraphError):
        bfs.run("gpu_do_persistent", int(src[0]), opts=gb.BfsOptions(spin_limit=1))
    d, _, _ = bfs.run_many("gpu_do_persistent", src)
    for i, s in enumerate(src):
        assert np.array_equal(d[i], oracle.bfs_serial(g, int(s)))
    assert np.array_equal(bfs.run("gpu_do_persistent", int(src[0])), d[0])
