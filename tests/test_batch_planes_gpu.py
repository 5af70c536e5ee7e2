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


@pytest.mark.parametrize("degs", [(319, 320, 321), (4158, 4159, 4160, 4161), (70, 128, 400, 6000)])
def test_deferred_rests_around_their_cuts(gb, oracle, degs):
    """Bottom-up scans that run to the end of lists whose rest (after the first
    64 entries) is just below, at and above the cuts at which a warp or a block
    of the grid takes it: half of the sources are in another component, so no
    list stops early."""
    rng = np.random.default_rng(sum(degs))
    n1, nb = 9000, 300
    eu, ev = [], []
    for hub, deg in enumerate(degs):
        eu.append(np.full(deg, hub)); ev.append(rng.choice(np.arange(len(degs), n1), deg, replace=False))
    eu.append(np.arange(len(degs) - 1)); ev.append(np.arange(1, len(degs)))
    eu.append(np.arange(n1, n1 + nb - 1)); ev.append(np.arange(n1 + 1, n1 + nb))
    g = gb.from_edges(n1 + nb, np.concatenate(eu).astype(np.uint32), np.concatenate(ev).astype(np.uint32))
    srcs = np.concatenate([rng.integers(0, n1, 20), rng.integers(n1, n1 + nb, 20)]).astype(np.uint32)
    bfs = gb.GpuBfs(g)
    for k in (40, 6):
        pick = srcs[:k] if k == 40 else srcs[17:23]
        for o in (gb.BfsOptions(force_strategy="bu"), gb.BfsOptions(force_strategy="bu", block=256, grid_blocks=3)):
            d = bfs.run_batch(pick, opts=o)
            for i, s in enumerate(pick):
                assert np.array_equal(d[i], oracle.bfs_serial(g, int(s))), (k, i)
