"""Results back in host memory: packed depths and staged copies at the edges of
their groups (8 depths on the device, 16 and 32 on the host), of the one-thread
and streaming cuts and of the chunks, into aligned and unaligned arrays, with
the width guessed right, too wide and too narrow; exact against the oracle
(depths) and against the FP64 pull (ranks, checkRanks of the oracle)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _hub_and_path(gb, n, tail):
    """A star over n - tail vertices with a path of `tail` vertices from its hub."""
    hub = n - tail
    u = np.concatenate([np.zeros(max(hub - 1, 0)), [0] if tail and n > 1 else [], np.arange(hub, n - 1) if tail else []])
    v = np.concatenate([np.arange(1, hub), [hub] if tail and n > 1 else [], np.arange(hub + 1, n) if tail else []])
    return gb.from_edges(n, u.astype(np.uint32), v.astype(np.uint32))


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 31, 32, 33, 63, 4097, 65535, 65536, 65537, (1 << 20) - 1, (1 << 20) + 1, (1 << 20) + 33])
def test_depths_at_every_size(gb, oracle, n):
    for tail in sorted({0, min(n // 2, 10), min(n // 2, 40), min(n // 2, 300)}):  # 4 bits, 1 and 2 bytes
        g = _hub_and_path(gb, n, tail)
        want = oracle.bfs_serial(g, 0)
        far = oracle.bfs_serial(g, n - 1)
        bfs = gb.GpuBfs(g)
        buf = np.zeros(n + 3, np.uint32)
        for off in (0, 1, 3):
            for variant in ("gpu_do_persistent", "gpu_do"):
                out = buf[off:off + n]
                out[:] = 77
                bfs.run(variant, 0, out=out)
                assert np.array_equal(out, want), (n, tail, off, variant)
        assert np.array_equal(bfs.run("gpu_do_persistent", n - 1), far)  # deeper than the last run's guess
        assert np.array_equal(bfs.run("gpu_do_persistent", 0), want)     # shallower
        d, _, _ = bfs.run_many("gpu_do_persistent", [0, n - 1, 0], opts=gb.BfsOptions(in_flight=2))
        assert np.array_equal(d[0], want) and np.array_equal(d[1], far) and np.array_equal(d[2], want)


@pytest.mark.parametrize("n", [1, 3, 1000, 262143, 262144, 262145, 1048577, 1400001])
def test_ranks_at_every_size(gb, oracle, n):
    rng = np.random.default_rng(n)
    k = 3 * n
    g = gb.from_edges(n, rng.integers(0, n, k).astype(np.uint32), rng.integers(0, n, k).astype(np.uint32), True)
    pr = gb.pagerank_handle(g)
    pr.run("gpu_pull_f64")
    want = pr.ranks_f64()
    assert abs(want.sum() - 1) < 1e-9
    for variant in ("gpu_pull_adaptive", "gpu_pull_vector"):
        pr.run(variant)
        assert oracle.check_ranks(want, pr.ranks()).ok, (n, variant)
    pr.prepareGS(2)
    pr.run("gpu_pull_gs", gb.PrOptions(iters=100, tol=1e-7))
    pr2 = gb.pagerank_handle(g)
    pr2.run("gpu_pull_f64", gb.PrOptions(iters=200, tol=1e-12))
    assert np.abs(pr.ranks() - pr2.ranks_f64()).sum() < 1e-4
