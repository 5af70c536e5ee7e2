"""Where the memory that a faster form takes beside the results is not there,
the form without it runs: a batch without bit planes (64 bytes a vertex), a
learned call on a road network without the neighbour table (16) or a row of
depths per source.  The rest of the GPU's memory is held meanwhile."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _held(torch, leave):
    """Holds all of the GPU's free memory but `leave` bytes, in pieces."""
    torch.cuda.empty_cache()
    pieces = []
    while True:
        more = torch.cuda.mem_get_info()[0] - leave
        if more < 4 * MB:
            return pieces
        piece = min(more // (2 * MB) * 2 * MB, 16 << 30)
        piece -= 1 << 30 if 0 < more - piece < 64 * MB and piece == 16 << 30 else 0  # torch rounds small pieces up
        pieces.append(torch.empty(piece, dtype=torch.uint8, device="cuda"))


@pytest.mark.parametrize("call", ["batch", "cluster", "cluster_many"])
def test_less_memory_the_other_form(gb, oracle, call):
    torch = pytest.importorskip("torch")
    if call == "batch":
        g, extra = gb.gen.rmat(22, 4, False, 3), 64 << 22
        srcs = np.asarray(gb.pick_sources(g, 16, 1), np.uint32)
    else:
        g = gb.gen.road(2000, 2000, 0.04, 0.005, 5)
        extra = 16 * g.n if call == "cluster" else 4 * g.n * 61
        srcs = np.arange(64, dtype=np.uint32) * 1000
    params = gb.default_selector_params("single")

    def run(leave=None):
        bfs = gb.GpuBfs(g)
        bfs.set_selector(params, 0)
        # what this form needs in any case is there: the buffers of a first call
        free = torch.cuda.mem_get_info()[0]
        held = _held(torch, leave) if leave else []
        if call == "batch":
            d = bfs.run_batch(srcs)
        elif call == "cluster":
            d = [bfs.run("gpu_do_persistent", int(srcs[0]), opts=gb.BfsOptions(selector="learned"))]
        else:
            d = bfs.run_many("gpu_do_persistent", srcs[: 64], opts=gb.BfsOptions(selector="learned"))[0]
        taken = free - torch.cuda.mem_get_info()[0]
        del held
        torch.cuda.empty_cache()
        return d, taken

    def without():  # what the form without the extra memory takes
        bfs = gb.GpuBfs(g)
        free = torch.cuda.mem_get_info()[0]
        if call == "batch":
            bfs.run_batch(srcs[:7])
            return free - torch.cuda.mem_get_info()[0] + 4 * g.n * (len(srcs) - 7)
        if call == "cluster":
            bfs.run("gpu_do_persistent", int(srcs[0]))
        else:
            bfs.run_many("gpu_do_persistent", srcs)
        return free - torch.cuda.mem_get_info()[0]

    without()
    least = without()
    leave = least + 24 * MB  # granularity, events, streams
    assert extra > 48 * MB
    d, _ = run(leave)
    want = oracle.bfs_serial(g, int(srcs[0]))
    assert np.array_equal(d[0], want)
    d2, _ = run()  # with room: the same depths
    for a, b in zip(d, d2):
        assert np.array_equal(a, b)
