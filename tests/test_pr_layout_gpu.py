"""The pulls' list layouts at their edges: list lengths around whole vectors, the
interleaved cut (32 entries), the lane groups, the warp-per-list and split cuts
and whole chunks; runs that end inside a block of 32 lists; every cut pair that
changes the classes; and the scalar and vector pulls' split lists.

Against the FP64 pull on the same graph.  Per sweep a rank carries the rounding
of a compensated sum, of the few plain additions across lanes and of the final
expression, under 8 units of 2^-24 relative; errors of earlier sweeps shrink by
0.85, so the L1 distance stays below 8 * 2^-24 / 0.15 = 3.2e-6."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BOUND = 8 * 2.0 ** -24 / 0.15


def _graph(gb, lengths, extra, seed):
    """A directed graph whose in-lists have exactly the given lengths (then
    `extra` vertices with none), from distinct random sources."""
    rng = np.random.default_rng(seed)
    n = max(len(lengths) + extra, max(lengths) + 1)
    u = [rng.choice(n - 1, d, replace=False) for d in lengths]
    u = [np.where(x >= v, x + 1, x) for v, x in enumerate(u)]  # no self-loops
    v = np.repeat(np.arange(len(lengths)), lengths)
    perm = rng.permutation(n).astype(np.uint32)
    return gb.from_edges(n, perm[np.concatenate(u)], perm[v], True)


CASES = {
    "short": list(range(0, 40)) * 3,
    "one": [1], "vec": [3, 4, 5] * 11, "inter": [28, 31, 32, 33, 36] * 33,
    "groups": [15, 16, 17, 63, 64, 65, 127, 128, 129, 130, 131, 132, 255, 256, 257],
    "chunks": [1023, 1024, 1025, 2047, 2048, 2049, 3072, 4096, 4097, 33000],
    "mixed": [40000, 5000, 700, 300] + [60] * 50 + [9] * 500 + [1] * 3000,
}


@pytest.mark.parametrize("name", list(CASES))
@pytest.mark.parametrize("extra", [0, 77])
def test_every_pull_matches_fp64(gb, name, extra):
    g = _graph(gb, CASES[name], extra, len(name) + extra)
    pr = gb.pagerank_handle(g)
    for tol, iters in ((0.0, 20), (1e-7, 300)):
        pr.run("gpu_pull_f64", gb.PrOptions(iters=iters, tol=tol))
        want = pr.ranks_f64()
        runs = [("gpu_pull_scalar", {}), ("gpu_pull_vector", {})]
        runs += [("gpu_pull_adaptive", dict(small_max=s, large_min=l))
                 for s, l in ((16, 256), (0, 0), (0, 1 << 30), (1 << 30, 1 << 31), (2, 3), (33, 1024), (300, 300), (40, 33))]
        for variant, cuts in runs:
            for tg in (32, 256, 1024):
                r = pr.run(variant, gb.PrOptions(iters=iters, tol=tol, tg=tg, **cuts))
                # to a tolerance a sweep more or less is possible: the residual bounds what it changes
                slack = 0.0 if tol == 0 else 10 * tol
                assert np.abs(pr.ranks() - want).sum() < BOUND + slack, (variant, cuts, tg, r.iters)


def test_inplace_pulls_converge(gb):
    g = _graph(gb, CASES["mixed"], 10, 5)
    pr = gb.pagerank_handle(g)
    pr.run("gpu_pull_f64", gb.PrOptions(iters=300, tol=1e-13))
    want = pr.ranks_f64()
    for variant in ("gpu_pull_scalar", "gpu_pull_vector", "gpu_pull_adaptive"):
        pr.run(variant, gb.PrOptions(iters=200, inplace=1))
        assert np.abs(pr.ranks() - want).sum() < 4 * BOUND, variant  # renormalised each sweep: a few roundings more


def test_ranks_after_other_cuts(gb):
    """The layout is rebuilt for other cuts and the ranks stay in the caller's ids."""
    g = gb.gen.rmat(14, 16, True, 9)
    pr = gb.pagerank_handle(g)
    pr.run("gpu_pull_f64")
    want = pr.ranks_f64()
    for s, l in ((16, 256), (4, 64), (16, 256), (64, 4096)):
        pr.prepareAdaptive(s, l)
        pr.run("gpu_pull_adaptive", gb.PrOptions(small_max=s, large_min=l))
        first = pr.ranks()
        assert np.abs(first - want).sum() < BOUND and np.array_equal(first, pr.ranks())
