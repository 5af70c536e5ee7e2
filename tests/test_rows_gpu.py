"""A batch's rows to the host in groups: every packed width, rows that are not a
multiple of 4 or 32 vertices, groups of many rows, of one and a last one that is
partly filled, rows apart by more than their length (what lies between them stays),
and depths past the widest packing."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PATH = "path"  # depths up to n - 1: the width follows from the length


@pytest.mark.parametrize("kind,n,k", [(PATH, 1, 3), (PATH, 13, 13), (PATH, 241, 64), (PATH, 1003, 9), (PATH, 66_001, 3),
                                      ("rmat", 3, 64), ("rmat", 12, 64), ("rmat", 17, 64), ("rmat", 19, 65),
                                      ("rmat", 21, 9)])
@pytest.mark.parametrize("gap", [0, 5])
def test_rows_match_the_oracle(gb, oracle, kind, n, k, gap):
    if kind == PATH:
        v = np.arange(n - 1)
        g = gb.from_edges(n, v.astype(np.uint32), (v + 1).astype(np.uint32))
    else:
        g = gb.gen.rmat(n, 8, False, 4)
    rng = np.random.default_rng(n + k)
    src = rng.integers(0, g.n, k).astype(np.uint32)
    bfs = gb.GpuBfs(g)
    out = np.full(k * (g.n + gap), 7, np.uint32)
    bfs.run_many("batch", src, out=out, stride=g.n + gap)
    rows = out.reshape(k, g.n + gap)
    assert (rows[:, g.n:] == 7).all()
    seen = {}
    for i, s in enumerate(src):
        if int(s) not in seen:
            if len(seen) == 12:
                continue
            seen[int(s)] = oracle.bfs_serial(g, int(s))
        assert np.array_equal(rows[i, : g.n], seen[int(s)]), (i, int(s))
    last = np.full(g.n, 7, np.uint32)
    bfs.run_many("batch", src, out=last, stride=0)  # every row to the same place, in order
    assert np.array_equal(last, rows[k - 1, : g.n])
