"""The damping factor belongs to a run: a handle that has run with one value
(and kept that run's captured sweeps) gives with another value what a new
handle gives, for every variant and both stop rules."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

VARIANTS = ["gpu_push", "gpu_pull_scalar", "gpu_pull_vector", "gpu_pull_adaptive", "gpu_pull_gs", "gpu_pull_f64",
            "gpu_pull_blocked"]


@pytest.mark.parametrize("inplace", [0, 1])
@pytest.mark.parametrize("variant", VARIANTS)
def test_another_damping_on_the_same_handle(gb, variant, inplace):
    if inplace and variant in ("gpu_push", "gpu_pull_f64", "gpu_pull_blocked"):
        pytest.skip("this variant has no in-place form")
    g = gb.gen.web(5000, 6.0, 2.1, 3)
    gin = gb.transpose(g)

    def ranks(pr, damping, tol):
        pr.run(variant, gb.PrOptions(iters=60 if tol else 12, tol=tol, damping=damping, inplace=inplace))
        return pr.ranks_f64() if variant == "gpu_pull_f64" else pr.ranks().astype(np.float64)

    pr = gb.GpuPageRank(g.n, g, gin, g.degrees())
    for damping, tol in ((0.85, 0.0), (0.5, 0.0), (0.85, 1e-6), (0.6, 1e-6), (0.85, 0.0)):
        new = ranks(gb.GpuPageRank(g.n, g, gin, g.degrees()), damping, tol)
        got = ranks(pr, damping, tol)
        # the order of atomics and of in-place updates differs from run to run; 0.5 against 0.85 is 40% and more
        assert np.abs(got - new).sum() < 1e-3, (damping, tol)


def test_many_dampings_on_one_handle(gb):
    """More values than a handle keeps captured sweeps for, then the first again."""
    g = gb.gen.web(500, 6.0, 2.1, 4)
    pr = gb.GpuPageRank(g.n, None, gb.transpose(g), g.degrees())
    o = [gb.PrOptions(iters=3, damping=0.3 + 0.005 * i) for i in range(100)]
    first = []
    for i in range(100):
        pr.run("gpu_pull_vector", o[i])
        first.append(pr.ranks())
    for i in (0, 99, 50):
        pr.run("gpu_pull_vector", o[i])
        assert np.array_equal(pr.ranks(), first[i]), i
    assert not np.array_equal(first[0], first[99])


@pytest.mark.parametrize("damping", [0.85, 0.5, 0.8500001, 0.123456789, 0.9999995, 0.99999994])
@pytest.mark.parametrize("variant", [v for v in VARIANTS if v != "gpu_pull_gs"])
def test_the_damping_written_is_the_one_used(gb, oracle, variant, damping):
    """Vertex 0 has no in-links and nothing dangles, so its rank is (1 - d) / n,
    where another damping factor than the one written shows, the more the nearer
    to 1 it is.  d: the shortest decimal of the option's float.  Tolerance: a
    few roundings to float (6e-8 each)."""
    n = 4097
    u = np.arange(n, dtype=np.uint32)
    v = np.where(u + 1 < n, u + 1, 1).astype(np.uint32)  # 0 -> 1 -> ... -> n - 1 -> 1
    g = gb.from_edges(n, u, v, True)
    gin = gb.transpose(g)
    pr = gb.GpuPageRank(n, g, gin, g.degrees())
    pr.run(variant, gb.PrOptions(iters=3, damping=damping))
    got = pr.ranks_f64() if variant == "gpu_pull_f64" else pr.ranks().astype(np.float64)
    decimals = [float(f"{np.float32(damping):.{k}g}") for k in range(6, 10)]
    d = next(x for x in decimals if np.float32(x) == np.float32(damping))
    want, _, _ = oracle.pagerank_serial(gin, g.degrees(), 3, damping=d)
    assert abs(want[0] * n / (1.0 - d) - 1.0) < 1e-7
    assert np.abs(got / want - 1.0).max() < 3e-7
