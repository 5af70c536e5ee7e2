"""Bounded-degree graphs through the cluster form (a thread-block cluster per
source): batched runs, and single and many-source runs with the learned
selector, without a trace.  Depths are integers, so the tolerance is exact
equality with the oracle's serial BFS.  The graphs sit at the form's edges:
bitmap words and their spread over the blocks, degrees around the 4 neighbour
slots and up to the 31 the form takes, frontiers that make blocks share their
queues and ones that outgrow them, and each number of blocks per source."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _tree(gb, branch, n):
    """Vertex v's children are branch*v+1 .. branch*v+branch: degree branch + 1."""
    v = np.arange(1, n, dtype=np.uint32)
    return gb.from_edges(n, (v - 1) // branch, v)


def _regular(gb, n, deg, seed):
    """Union of deg random perfect matchings (an expander: wide frontiers)."""
    rng = np.random.default_rng(seed)
    u, v = [], []
    for _ in range(deg):
        p = rng.permutation(n).astype(np.uint32)
        u.append(p[: n // 2]); v.append(p[n // 2: 2 * (n // 2)])
    return gb.from_edges(n, np.concatenate(u), np.concatenate(v))


def _graphs(gb):
    return {
        "one": gb.gen.empty(1), "isolated": gb.gen.empty(1000), "path31": gb.gen.path(31), "path32": gb.gen.path(32),
        "path33": gb.gen.path(33), "path4097": gb.gen.path(4097), "grid": gb.gen.grid2d(97, 211),
        "grid_long": gb.gen.grid2d(3, 40000), "tree3": _tree(gb, 3, 9000), "tree4": _tree(gb, 4, 5001),
        "tree30": _tree(gb, 30, 40000), "road200": gb.gen.road(200, 201, 0.04, 0.005, 1),
        "road600": gb.gen.road(600, 599, 0.04, 0.05, 2), "expander": _regular(gb, 60000, 3, 5),
    }


NAMES = ["one", "isolated", "path31", "path32", "path33", "path4097", "grid", "grid_long", "tree3", "tree4", "tree30",
         "road200", "road600", "expander"]


@pytest.fixture(scope="module")
def graphs(gb):
    return _graphs(gb)


@pytest.mark.parametrize("name", NAMES)
def test_depths_exact(gb, oracle, graphs, name):
    g = graphs[name]
    rng = np.random.default_rng(len(name))
    srcs = np.concatenate([[0, g.n - 1, g.n // 2, 0], rng.integers(0, g.n, 60)]).astype(np.uint32)
    want = {int(s): oracle.bfs_serial(g, int(s)) for s in srcs}
    params = gb.default_selector_params("single")
    o = gb.BfsOptions(selector="learned")
    for hub_first in (False, True):
        bfs = gb.GpuBfs(g)
        bfs.set_selector(params, 0)
        for k in (1, 5, 9, 20, 40, 64):  # 16, 16, 16, 4, 2 and 2 blocks each where the graph is large enough
            d = bfs.run_batch(srcs[:k])
            for i in range(k):
                assert np.array_equal(d[i], want[int(srcs[i])]), (hub_first, k, i)
        for s in srcs[:3]:
            d = bfs.run("gpu_do_persistent", int(s), opts=o)
            assert np.array_equal(d, want[int(s)])
            reached = want[int(s)][want[int(s)] != 0xFFFFFFFF]
            assert bfs.lastLevels() == int(reached.max()) + 1
        many = np.concatenate([srcs, srcs[:6]])  # two launches
        d, ms, lv = bfs.run_many("gpu_do_persistent", many, opts=o)
        for i, s in enumerate(many):
            assert np.array_equal(d[i], want[int(s)])
            assert lv[i] == int(want[int(s)][want[int(s)] != 0xFFFFFFFF].max()) + 1
        assert (ms > 0).all() and bfs.lastLevels() == lv[-1]
        if hub_first:
            break
        bfs.hub_first()  # the neighbour table follows the re-sorted lists
        assert np.array_equal(bfs.run_batch(srcs[:3])[2], want[int(srcs[2])])


def test_large_grid_needs_several_blocks(gb, oracle):
    """A bitmap larger than one block's shared memory, at 64 sources."""
    g = gb.gen.grid2d(1500, 1301)
    srcs = np.random.default_rng(3).integers(0, g.n, 64).astype(np.uint32)
    bfs = gb.GpuBfs(g)
    d = bfs.run_batch(srcs)
    for i in (0, 31, 63):
        assert np.array_equal(d[i], oracle.bfs_serial(g, int(srcs[i])))
