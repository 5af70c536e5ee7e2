"""The learned selector in the kernel that consults it.  Untraced calls on road
networks go to the cluster form under the learned selector, whatever its
parameters, so the selectors are compared with the whole grid asked for
(grid_blocks), which keeps both in the same kernel: parameters that always
predict one strategy fastest get it on every top-down level of the grid, and the
shipped ones beat the rule there on a road grid they were not trained on."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SOLO_EDGES = 4 * 512  # levels of fewer edges run in one block, the rule's way
WHOLE = 1 << 16       # more blocks than are resident: all of them


@pytest.mark.parametrize("strategy", ["td_ept1", "td_ept4", "td_warp"])
def test_the_parameters_decide(gb, oracle, strategy):
    g = gb.gen.road(600, 500, 0.04, 0.005, 77)
    _, _, outputs = gb.selector_shape()
    p = np.zeros(gb.lib().gb_selector_param_count(), np.float32)
    p[-outputs:] = 5.0  # the last layer's biases: log2 of the time
    p[len(p) - outputs + gb.STRATEGIES.index(strategy)] = 1.0
    bfs = gb.GpuBfs(g)
    bfs.set_selector(p, 0)
    src = int(gb.pick_sources(g, 1, 3)[0])
    o = gb.BfsOptions(selector="learned", grid_blocks=WHOLE)
    d, tr = bfs.run("gpu_do_persistent", src, opts=o, trace=True)
    large = [l for l in tr if l["direction"] == "T" and l["edges"] > SOLO_EDGES]
    assert len(large) > 20 and {l["strategy"] for l in large} == {strategy}
    want = oracle.bfs_serial(g, src)
    assert np.array_equal(d, want)
    assert np.array_equal(bfs.run("gpu_do_persistent", src, opts=o), want)


def test_the_shipped_selector_beats_the_rule_in_the_same_kernel(gb):
    g = gb.gen.road(1400, 1400, 0.04, 0.005, 902)
    srcs = [int(s) for s in gb.pick_sources(g, 4, 3)]
    bfs = gb.GpuBfs(g)
    bfs.set_selector(gb.default_selector_params("single"), 0)
    best = {}
    for sel in ("rule", "learned"):
        o = gb.BfsOptions(selector=sel, grid_blocks=WHOLE)
        times = []
        for _ in range(4):  # the first one warms up
            t = 0.0
            for s in srcs:
                bfs.run("gpu_do_persistent", s, opts=o)
                t += bfs.lastGpuMs()
            times.append(t)
        best[sel] = min(times)
    gain = best["rule"] / best["learned"]
    print(f"road 1400, same kernel: rule {best['rule']:.2f} ms, learned {best['learned']:.2f} ms, {gain:.2f}x")
    assert gain >= 1.25, best
