"""Depths that the traversal's kernel packs into pinned memory, around the sizes
where its room is for the last run's width (over 2^16) and where it no longer packs
(over 2^23): runs of few, more than 14, 254 and 65,534 levels in every order, sizes
that are not a multiple of 8."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(1 << 20) - 3, 1 << 20, (1 << 20) + 1, (1 << 20) + 13, (1 << 23) - 1, 1 << 23, (1 << 23) + 1])
def test_every_width_after_every_other(gb, n):
    # paths of 10, 200, 1,000 and 66,000 vertices, one after the other; the rest have no edges
    lengths, u, start, at = (10, 200, 1000, 66_000), [], [], 5
    for length in lengths:
        start.append(at)
        u.append(np.arange(at, at + length - 1))
        at += length
    u = np.concatenate(u).astype(np.uint32)
    g = gb.from_edges(n, u, u + 1)
    bfs = gb.GpuBfs(g)
    for i in (2, 0, 1, 0, 2, 1, 3, 0, 3, 1):
        want = np.full(n, 0xFFFFFFFF, np.uint32)
        want[start[i] : start[i] + lengths[i]] = np.arange(lengths[i])
        d = bfs.run("gpu_do_persistent", start[i])
        assert np.array_equal(d, want), lengths[i]
        assert bfs.lastLevels() == lengths[i]
