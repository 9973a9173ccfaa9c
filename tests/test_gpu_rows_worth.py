"""Whether a graph gets row lists is decided from histograms of its counts:
the same for counts that the graph made itself and for those counted anew
beside a caller's degrees, with hubs in the coarse bins (4,096 entries and
more), and without reserving or sorting anything for a graph without hubs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _edges(name):
    rng = np.random.default_rng(8)
    if name == "uniform":            # pulled bins: no hubs
        return rng.integers(0, 1 << 19, (8 << 19, 2)).astype(np.uint32), 1 << 19
    V = 200_003                      # row lists: hubs of 4,095 to 60,000 entries
    hubs = [np.stack([np.full(n, i), 100 + rng.integers(0, V - 100, n)], 1)
            for i, n in enumerate([4_095, 4_096, 4_097, 8_191, 8_192, 20_000, 60_000] * 4)]
    hubs += [h[:, ::-1] for h in hubs[:7]]   # (long rows of the directed graph, too)
    return np.concatenate([*hubs, rng.integers(100, V, (100_000, 2))]).astype(np.uint32), V


def _run(graph, iterations=3):
    """(launches to make the state, launches of a run, ranks)"""
    ctx = graph.ctx
    a = ctx.launches()
    with graph.state("pagerank", iterations) as s:
        b = ctx.launches()
        s.run()
        return b - a, ctx.launches() - b, s.download()


@pytest.mark.parametrize("directed", [False, True])
@pytest.mark.parametrize("name,per_iteration", [("uniform", 3), ("hubs", 4)])
def test_choice_from_histograms(name, per_iteration, directed, gpu_ctx_factory, oracle_lib):
    edges, V = _edges(name)
    edges = edges[edges[:, 0] != edges[:, 1]]
    ctx = gpu_ctx_factory(directed)
    graph = ctx.convert(edges, V)
    start, grid, degree = graph.download()
    p, _, _ = oracle_lib.geometry(V)
    r64, _ = oracle_lib.pagerank(start, grid, degree, p, directed, V, 3)
    own = _run(graph)
    graph.free()
    graph = ctx.upload(start, grid, degree, V)
    given = _run(graph)
    graph.free()
    # (pulled bins: gather, pull, finalize; row lists: permute, pull, longest rows, finalize)
    assert own[1] == given[1] == 3 * per_iteration
    for r in (own[2], given[2]):
        assert np.abs(r.astype(np.float64) - r64).sum() <= 1e-6 * np.abs(r64).sum()
    if name == "uniform":
        # 17 on the half grid: the ranks' start, a histogram, 15 for the bins; two
        # more to count for the attempt and for the bins beside a caller's degrees,
        # three on the directed grid, which has two histograms
        assert (own[0], given[0]) == ((20, 20) if directed else (17, 19))
