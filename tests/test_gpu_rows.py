"""PageRank over row lists (gs_pr_rows.cu) against the FP64 oracle and, after
one iteration, against exact sums: graphs whose rows fall on the edges of the
layout's segments, slices, panels and units."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PR_TOL = 1e-6


def _rows_of(lengths, V):
    """Edges that give vertex i lengths[i] records with vertices from
    len(lengths) on (cyclically), so those rows have exactly these lengths."""
    n = len(lengths)
    others = V - n
    out, at = [], 0
    for i, k in enumerate(lengths):
        ends = n + (at + np.arange(k, dtype=np.int64)) % others
        out.append(np.stack([np.full(k, i), ends], 1))
        at += k
    return np.concatenate(out).astype(np.uint32)


def _edges(name):
    rng = np.random.default_rng(7)
    if name == "one":
        return np.array([[1, 0]], np.uint32), 2
    if name == "star":               # a hub far longer than a segment, leaves of one entry
        return np.stack([np.full(40_000, 3), 4 + np.arange(40_000)], 1).astype(np.uint32), 1 << 16
    if name == "edges":              # rows around 16-byte, segment and long-row sizes
        return _rows_of([1, 2, 3, 4, 5, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 511, 512, 513, 1025],
                        1 << 12), 1 << 12
    if name == "ragged":             # vertex count no multiple of anything, repeated edges, unused vertices
        return rng.integers(0, 99_991 // 2, (300_000, 2)).astype(np.uint32) * 2, 99_991
    # every row long enough to be split by panel, sources over three panels
    return rng.integers(0, 1 << 16, (1 << 24, 2)).astype(np.uint32), 1 << 16


@pytest.mark.parametrize("directed", [False, True])
@pytest.mark.parametrize("name", ["one", "star", "edges", "ragged", "panels"])
def test_pagerank_row_lists(name, directed, gpu_ctx_factory, oracle_lib):
    edges, V = _edges(name)
    edges = edges[edges[:, 0] != edges[:, 1]]
    g = gpu_ctx_factory(directed).convert(edges, V)
    start, grid, degree = g.download()
    p, _, _ = oracle_lib.geometry(V)
    r1, _ = g.pagerank(1)
    r64, x64 = oracle_lib.pagerank(start, grid, degree, p, directed, V, 4)
    r, x = g.pagerank(4)
    again, _ = g.pagerank(1)
    g.free()
    if V & (V - 1) == 0:
        # x = 1/V is a power of two: every sum of the first iteration is exact
        into = np.bincount(edges[:, 1], minlength=V).astype(np.float64)
        if not directed:
            into += np.bincount(edges[:, 0], minlength=V)
        exact = (0.15 + 0.85 * (into / V)).astype(np.float32)
        assert np.array_equal(r1, exact) and np.array_equal(again, exact)
    for a, b in ((r, r64), (x, x64)):
        assert np.abs(a.astype(np.float64) - b).sum() <= PR_TOL * np.abs(b).sum()
