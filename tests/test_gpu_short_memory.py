"""Device allocations that fail: what a faster layout cannot have, the engine
does without."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NONE = (2**64 - 1, 0)


def fail_allocs(ctx, least, most):
    """From now on ctx's device allocations of `least` to `most` bytes fail."""
    import gstore_b200 as gs

    fn = gs.lib().gs_testing_fail_allocs
    fn.argtypes, fn.restype = [C.c_void_p, C.c_uint64, C.c_uint64], None
    fn(ctx._h, least, most)


@pytest.fixture
def ctx():
    import gstore_b200 as gs

    with gs.Context(0) as c:
        yield c


@pytest.mark.parametrize("shape", ["star", "dense"])
def test_pagerank_without_room_for_row_lists(shape, ctx, oracle_lib):
    """The row lists' build reserves over 12 MB in one block, the other
    layouts of these graphs take less."""
    V = 1 << 16
    if shape == "star":
        edges = np.stack([np.full(40_000, 3), 4 + np.arange(40_000)], 1).astype(np.uint32)
    else:
        edges = np.random.default_rng(2).integers(0, 300, (100_000, 2)).astype(np.uint32)
    graph = ctx.convert(edges, V)
    start, grid, degree = graph.download()
    p, _, _ = oracle_lib.geometry(V)
    r64, x64 = oracle_lib.pagerank(start, grid, degree, p, False, V, 3)
    fail_allocs(ctx, 12 << 20, 2**64 - 1)
    short = [graph.pagerank(3) for _ in range(2)]
    fail_allocs(ctx, *NONE)
    short.append(graph.pagerank(3))
    graph.free()
    for r, x in short:
        assert np.abs(r.astype(np.float64) - r64).sum() <= 1e-6 * np.abs(r64).sum()
        assert np.abs(x.astype(np.float64) - x64).sum() <= 1e-6 * np.abs(x64).sum()


@pytest.mark.parametrize("algo,arg", [("bfs", 5), ("kcore", 3), ("wcc", 0)])
def test_lists_without_room_for_a_query(algo, arg, ctx, oracle_lib):
    """A query on adjacency lists whose own scratch cannot be had runs on the
    tiles, which need none; the lists are dropped first."""
    V = 70_001
    edges = np.random.default_rng(3).integers(0, V, (300_000, 2)).astype(np.uint32)
    edges = edges[edges[:, 0] != edges[:, 1]]
    graph = ctx.convert(edges, V)
    start, grid, degree = graph.download()
    p, _, _ = oracle_lib.geometry(V)
    want = {"bfs": lambda: oracle_lib.bfs(start, grid, p, False, V, arg)[0],
            "kcore": lambda: oracle_lib.kcore(start, grid, degree, p, V, arg)[0],
            "wcc": lambda: oracle_lib.wcc(start, grid, p, False, V)[0]}[algo]()
    with graph.state("kcore", 2) as s:                 # (the tiles' own order)
        s.run()
    for _ in range(17):                                # until the lists are there
        graph.bfs(1) if algo == "wcc" else graph.wcc()
    with graph.state(algo, arg) as s:
        fail_allocs(ctx, 0, 2**64 - 1)
        s.run()
        fail_allocs(ctx, *NONE)
        assert np.array_equal(s.download(), want)
        s.reset(arg)
        s.run()
        assert np.array_equal(s.download(), want)
    graph.free()
