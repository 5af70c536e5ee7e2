"""A graph of small degrees whose frontier outgrows the cluster form's queues
ends on the grid with no more device memory than a handle that never tried: the
neighbour table and the rows of that form are given back.  The grid form's own
buffers are the same for both; 4 MB allow for the allocator's granularity."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("call", ["run", "run_many"])
def test_nothing_is_kept(gb, oracle, call):
    torch = pytest.importorskip("torch")
    n = 1 << 20
    rng = np.random.default_rng(9)
    ends = [rng.permutation(n).astype(np.uint32).reshape(2, -1) for _ in range(3)]  # 3 random matchings: an expander
    g = gb.from_edges(n, np.concatenate([e[0] for e in ends]), np.concatenate([e[1] for e in ends]))
    src = np.array([1, 5, 9], np.uint32)

    def used(selector):
        before = torch.cuda.mem_get_info()[0]
        bfs = gb.GpuBfs(g)
        bfs.set_selector(gb.default_selector_params("single"), 0)
        o = gb.BfsOptions(selector=selector)
        d = bfs.run("gpu_do_persistent", 9, opts=o) if call == "run" else bfs.run_many("gpu_do_persistent", src, opts=o)[0][2]
        return before - torch.cuda.mem_get_info()[0], d

    used("rule")  # modules and streams of the first call
    want = oracle.bfs_serial(g, 9)
    (rule, a), (learned, b) = used("rule"), used("learned")
    assert np.array_equal(a, want) and np.array_equal(b, want)
    assert learned - rule < 4 << 20, (rule, learned)
