"""The batched kernel keeps depths below 256 in bit planes (from 8 sources on)
and stores deeper ones directly.  Wheels of spokes around hubs keep the batch on
the grid form; the paths hanging off them put the deepest level at and around
each power of two and at the planes' end.  Exact against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _hub_with_path(gb, spokes, length):
    """A star of `spokes` leaves whose hub starts a path of `length` vertices, and
    an isolated vertex."""
    n = 1 + spokes + length + 1
    u = np.concatenate([np.zeros(spokes), [0] if length else [], np.arange(1 + spokes, spokes + length)])
    v = np.concatenate([np.arange(1, 1 + spokes), [1 + spokes] if length else [], np.arange(2 + spokes, 1 + spokes + length)])
    return gb.from_edges(n, u.astype(np.uint32), v.astype(np.uint32))


@pytest.mark.parametrize("length", [0, 1, 2, 3, 6, 7, 8, 14, 30, 126, 253, 254, 255, 256, 257, 600])
@pytest.mark.parametrize("k", [7, 8, 33, 64])
def test_deepest_level_around_the_planes(gb, oracle, length, k):
    g = _hub_with_path(gb, 700, length)
    rng = np.random.default_rng(length)
    srcs = np.concatenate([[g.n - 1, 0, g.n - 2], rng.integers(0, g.n, 61)]).astype(np.uint32)[:k]
    bfs = gb.GpuBfs(g)
    for o in (gb.BfsOptions(), gb.BfsOptions(force_strategy="bu"), gb.BfsOptions(force_strategy="td_warp")):
        d = bfs.run_batch(srcs, opts=o)
        for i, s in enumerate(srcs):
            assert np.array_equal(d[i], oracle.bfs_serial(g, int(s))), (o.force_strategy, i)
