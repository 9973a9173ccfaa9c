"""Adjacency lists (gs_adj.cu) where their fixed-size lists run over, and
beside degrees that are not the records' counts."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _listed(graph):
    ctx = graph.ctx
    for _ in range(17):
        graph.wcc()
    with graph.state("bfs", 0) as s:
        before = ctx.launches()
        s.run()
        assert ctx.launches() - before <= 3      # the lists are in use
    return graph


def test_a_frontier_too_large_for_the_queue(gpu_ctx_factory):
    """The root's 100,000 neighbours are found together, and few vertices enough
    are concerned for the next level to go top-down -- but the queue holds some
    72,000 (N / 16 and a few): that level and the next go bottom-up."""
    V, n = 1 << 20, 100_000
    a = 1 + np.arange(n)
    rest = np.arange(1 + 2 * n, V)
    edges = np.concatenate([np.stack([np.zeros(n, np.int64), a], 1), np.stack([a, a + n], 1),
                            np.stack([rest[:-1], rest[1:]], 1)]).astype(np.uint32)
    graph = _listed(gpu_ctx_factory(False).convert(edges, V))
    want = np.zeros(V, np.uint8)
    want[0], want[1:n + 1], want[n + 1:2 * n + 1] = 1, 2, 3
    with graph.state("bfs", 0) as s:
        s.run()
        assert np.array_equal(s.download(), want)
        assert s.bfs_stats()["level_counts"].tolist() == [n, n, 0]
    graph.free()


@pytest.mark.parametrize("k", [4_330, 5_000])
def test_more_long_rows_than_the_chunk_list_holds(k, gpu_ctx_factory, oracle_lib):
    """6,000 rows of some 4,320 entries are five chunks each, a few hundred more
    than the list has room for when a round removes them all."""
    V = 6_000
    edges = np.random.default_rng(12).integers(0, V, (12_960_000, 2)).astype(np.uint32)
    graph = _listed(gpu_ctx_factory(False).convert(edges, V))
    start, grid, degree = graph.download()
    assert 5 * np.count_nonzero(degree > 4_096) > 2 * grid.size // 1_024 + 4_096 + 300
    p, _, _ = oracle_lib.geometry(V)
    deg_o, mem_o, _ = oracle_lib.kcore(start, grid, degree, p, V, k)
    deg, mem = graph.kcore(k)
    assert np.array_equal(deg, deg_o) and mem == mem_o
    graph.free()


def test_degrees_that_are_not_the_counts(gpu_ctx_factory, oracle_lib):
    """A caller's degree array decides k-core and PageRank; the lists are those
    of the records whatever it says."""
    V = 70_001
    rng = np.random.default_rng(13)
    ctx = gpu_ctx_factory(False)
    graph = ctx.convert(rng.integers(0, V, (400_000, 2)).astype(np.uint32), V)
    start, grid, counts = graph.download()
    graph.free()
    degree = (counts + rng.integers(-3, 4, V)).clip(0).astype(np.int32)
    graph = _listed(ctx.upload(start, grid, degree, V))
    p, _, _ = oracle_lib.geometry(V)
    for k in (3, 9, 12):
        deg_o, mem_o, _ = oracle_lib.kcore(start, grid, degree, p, V, k)
        deg, mem = graph.kcore(k)
        assert np.array_equal(deg, deg_o) and mem == mem_o, f"k={k}"
    assert np.array_equal(graph.bfs(7), oracle_lib.bfs(start, grid, p, False, V, 7)[0])
    r64, _ = oracle_lib.pagerank(start, grid, degree, p, False, V, 3)
    r, _ = graph.pagerank(3)
    assert np.abs(r.astype(np.float64) - r64).sum() <= 1e-6 * np.abs(r64).sum()
    graph.free()
