"""A PageRank layout for which the memory runs out part of the way leaves the
handle as good as before: the other variants, and the same one once there is
memory, give what a new handle gives.  The amounts left run from less than the
first buffers take to more than the layout needs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20


def test_a_layout_that_ran_out_of_memory(gb):
    torch = pytest.importorskip("torch")
    g = gb.gen.rmat(19, 16, False, 5)  # 16M in-edges: its contributions move to make room for the hot ones
    assert g.m > 12 << 20
    o = gb.PrOptions(iters=4)

    def new():
        return gb.GpuPageRank(g.n, None, g, g.degrees())

    def ranks(pr, variant):
        pr.run(variant, o)
        return pr.ranks()

    want = {v: ranks(new(), v) for v in ("gpu_pull_vector", "gpu_pull_adaptive")}
    failed = 0
    for leave in (2, 6, 10, 14, 18, 22, 26, 30, 40, 80, 160, 320, 640):
        pr = new()
        torch.cuda.empty_cache()
        held = []
        while (more := torch.cuda.mem_get_info()[0] - leave * MB) >= 2 * MB:
            piece = min(more // (2 * MB) * 2 * MB, 16 << 30)
            piece -= 1 << 30 if 0 < more - piece < 64 * MB and piece == 16 << 30 else 0  # torch rounds small pieces up
            held.append(torch.empty(piece, dtype=torch.uint8, device="cuda"))
        try:
            pr.prepareAdaptive()
        except gb.GraphError as e:
            assert "memory" in str(e)
            failed += 1
        del held
        torch.cuda.empty_cache()
        assert np.array_equal(ranks(pr, "gpu_pull_vector"), want["gpu_pull_vector"]), leave
        got = ranks(pr, "gpu_pull_adaptive").astype(np.float64)
        # the same sums, in the same order, with or without the hot places
        assert np.array_equal(got, want["gpu_pull_adaptive"].astype(np.float64)), leave
    assert 0 < failed < 13
