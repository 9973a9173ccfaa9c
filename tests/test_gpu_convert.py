"""The converter's bucket passes (graphs of one tile group, 2^14 edges and more)
against the oracle's converter, at the sizes where they start, where a stretch
of edges ends, and with tiles sliced and whole."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("directed", [False, True])
@pytest.mark.parametrize("n, V", [((1 << 14) - 1, 1 << 16), (1 << 14, 70_001), ((1 << 20) + 65_537, 2),
                                  (300_001, 150_000), (3_000_001, 1 << 24)])
def test_convert_buckets(n, V, directed, gpu_ctx_factory, oracle_lib):
    rng = np.random.default_rng(n & 0xFFFF)
    edges = rng.integers(0, V, (n, 2)).astype(np.uint32)
    edges[: n // 3, 0] %= 7                       # a few crowded tiles, self-loops among them
    p, _, _ = oracle_lib.geometry(V, directed)
    start_o, grid_o, degree_o = oracle_lib.convert(edges, p, directed, V)
    g = gpu_ctx_factory(directed).convert(edges, V)
    start, grid, degree = g.download()
    g.free()
    assert np.array_equal(start, start_o) and np.array_equal(degree, degree_o)
    # the converter sorts the records of a tile
    tile = np.repeat(np.arange(start.size - 1), np.diff(start).astype(np.int64))
    assert np.array_equal(grid, grid_o[np.lexsort((grid_o, tile))])


@pytest.mark.parametrize("n, V, directed", [((1 << 24) + 5, 60_000, True), ((1 << 24) + 4099, 1 << 20, False)])
def test_convert_scanned_counts(n, V, directed, gpu_ctx_factory, oracle_lib):
    """Enough edges for the stretches' counts to be scanned as one table."""
    test_convert_buckets(n, V, directed, gpu_ctx_factory, oracle_lib)
