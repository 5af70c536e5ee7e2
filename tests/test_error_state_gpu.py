"""A call that fails for want of memory fails alone: the calls after it, on new
handles and on old ones, succeed."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20


def test_out_of_memory_is_reported_once(gb, oracle):
    torch = pytest.importorskip("torch")
    small = gb.gen.rmat(12, 8, False, 1)
    large = gb.gen.rmat(21, 16, False, 2)  # 270 MB
    old = gb.GpuBfs(small)
    want = oracle.bfs_serial(small, 3)
    assert np.array_equal(old.run("gpu_do_persistent", 3), want)
    for after in ("old handle", "new handle", "pagerank", "build"):
        torch.cuda.empty_cache()
        held = []
        while (more := torch.cuda.mem_get_info()[0] - 64 * MB) >= 2 * MB:
            piece = min(more // (2 * MB) * 2 * MB, 16 << 30)
            piece -= 1 << 30 if 0 < more - piece < 64 * MB and piece == 16 << 30 else 0  # torch rounds small pieces up
            held.append(torch.empty(piece, dtype=torch.uint8, device="cuda"))
        with pytest.raises(gb.GraphError, match="memory"):
            gb.GpuBfs(large)
        del held
        torch.cuda.empty_cache()
        if after == "old handle":
            assert np.array_equal(old.run("gpu_do", 3), want)
        elif after == "new handle":
            assert np.array_equal(gb.GpuBfs(small).run("gpu_vertex", 3), want)
        elif after == "pagerank":
            pr = gb.GpuPageRank(small.n, None, small, small.degrees())
            pr.run("gpu_pull_vector", gb.PrOptions(iters=3))
            assert abs(float(pr.ranks().astype(np.float64).sum()) - 1.0) < 1e-6
        else:
            u = np.array([0, 1, 2], np.uint32)
            assert gb.from_edges_gpu(4, u, u + 1).m == 6
