"""Sorted keys to CSR on the GPU (from_edges, transpose, symmetrize, permute) at
the edges of its tiles (2,048 keys) and of the runs of empty rows a thread fills
itself (64), with duplicates and self-loops across tile borders: byte for byte
the host layer's graphs, in arrays that outlive their graph."""
import gc

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _same(a, b):
    assert a.equal(b), (a.n, a.m, b.m)


@pytest.mark.parametrize("ne", [0, 1, 2, 2047, 2048, 2049, 4096, 50001])
@pytest.mark.parametrize("n", [1, 2, 64, 1000, 300000])
def test_from_edges_sizes(gb, n, ne):
    rng = np.random.default_rng(n + ne)
    for lo, hi in ((0, n), (n // 2, n // 2 + 1), (max(n - 3, 0), n)):  # spread, all self-loops, all in the last rows
        u = rng.integers(lo, hi, ne).astype(np.uint32)
        v = rng.integers(lo, hi, ne).astype(np.uint32)
        for directed in (False, True):
            _same(gb.from_edges_gpu(n, u, v, directed), gb.from_edges(n, u, v, directed))


@pytest.mark.parametrize("gap", [62, 63, 64, 65, 66, 1000, 100000])
def test_empty_rows(gb, gap):
    """Rows gap apart, gaps before the first and after the last among them."""
    rows = np.arange(gap, 12 * gap, gap, dtype=np.uint32)
    n = 13 * gap + 1
    u = np.repeat(rows, 7)
    v = np.tile(np.arange(7, dtype=np.uint32) * (gap // 8 + 1), rows.size)
    g = gb.from_edges(n, u, v, True)
    _same(gb.from_edges_gpu(n, u, v, True), g)
    _same(gb.transpose_gpu(g), gb.transpose(g))
    _same(gb.symmetrize_gpu(g), gb.symmetrize(g))
    perm = np.random.default_rng(gap).permutation(n).astype(np.uint32)
    _same(gb.permute_gpu(g, perm), gb.permute(g, perm))


def test_arrays_outlive_their_graph(gb):
    g = gb.from_edges_gpu(5000, np.arange(4999), np.arange(1, 5000))
    rp, ci = g.row_ptr, g.col_idx[100:200]
    want = ci.copy()
    del g
    gc.collect()
    other = [gb.gen.path(5000) for _ in range(20)]  # reuse freed memory, if any was
    assert rp[-1] == 2 * 4999 and np.array_equal(ci, want) and len(other) == 20
    ci[:] = 7  # writable, as before
    assert (ci == 7).all()
