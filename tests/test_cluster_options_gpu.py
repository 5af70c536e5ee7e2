"""Options of a call that the cluster form would take: a spin limit that asks
for waits shorter than its own is honoured by the grid forms, as on any other
graph, and the handle is good for the next call."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("call", ["run", "run_many", "run_batch", "batch"])
def test_a_short_spin_limit_runs_out(gb, oracle, call):
    g = gb.gen.road(300, 301, 0.04, 0.005, 4)
    bfs = gb.GpuBfs(g)
    bfs.set_selector(gb.default_selector_params("single"), 0)
    src = np.array([0, 5, 77, g.n - 1], np.uint32)

    def go(limit):
        o = gb.BfsOptions(selector="rule" if "batch" in call else "learned", spin_limit=limit)
        if call == "run":
            return bfs.run("gpu_do_persistent", int(src[-1]), opts=o)
        if call == "run_many":
            return bfs.run_many("gpu_do_persistent", src, opts=o)[0][-1]
        if call == "batch":
            return bfs.run_many("batch", src, opts=o)[0][-1]
        return bfs.run_batch(src, opts=o)[-1]

    want = oracle.bfs_serial(g, int(src[-1]))
    for limit in (0, 1 << 14, 1, 1 << 30):
        if limit == 1:
            with pytest.raises(gb.GraphError, match="spin limit"):
                go(limit)
        else:
            assert np.array_equal(go(limit), want), limit
