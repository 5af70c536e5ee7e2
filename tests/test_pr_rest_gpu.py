"""What a vertex gets besides its in-links, (1 - d) / n + d * dangling / n, is
the same for all vertices, so an error in it does not average out: it is rounded
once.  After one sweep from 1 / n (as a float) over a graph whose in-links all
go to one vertex it is known exactly, and every other rank is the float nearest
to it; the tolerance is half an ulp and what FP64 adds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", ["gpu_push", "gpu_pull_scalar", "gpu_pull_vector", "gpu_pull_adaptive", "gpu_pull_blocked"])
def test_ranks_without_in_links_are_rounded_once(gb, variant):
    for n in (3, 10, 33, 97, 100, 331, 1000, 1007, 4099, 10000, 30011, 65537, 100003):
        for links in (1, n // 3, n - 1):
            u = np.arange(1, links + 1, dtype=np.uint32)  # links vertices point to 0, all others dangle
            g = gb.from_edges(n, u, np.zeros_like(u), True)
            pr = gb.GpuPageRank(n, g, gb.transpose(g), g.degrees())
            pr.run(variant, gb.PrOptions(iters=1))
            got = pr.ranks()[1:]
            start = np.float64(np.float32(1.0) / np.float32(n))
            want = 0.15 / n + 0.85 * ((n - links) * start) / n
            assert (got == got[0]).all()
            assert abs(np.float64(got[0]) - want) <= 0.5001 * np.spacing(np.float32(want)), (n, links)
