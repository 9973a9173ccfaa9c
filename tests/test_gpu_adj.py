"""BFS, WCC and k-core on adjacency lists (gs_adj.cu), which a graph gets once
its queries have swept it often enough: the same depths, labels, degrees,
level counts and swept records as the tile sweeps and the oracle."""
import numpy as np
import pytest

from conftest import GOLDEN_NAMES, load_golden

pytestmark = pytest.mark.gpu


def _listed(graph):
    """Queries until the graph has its lists (a WCC counts two sweeps of 32)."""
    for _ in range(17):
        graph.wcc()
    return graph


def _bfs(graph, root):
    """(depth, stats, kernels launched) of one run."""
    with graph.state("bfs", int(root)) as s:
        before = graph.ctx.launches()
        s.run()
        n = graph.ctx.launches() - before
        return s.download(), s.bfs_stats(), n


def _check(graph, oracle_lib, roots, ks):
    V, directed = graph.V, graph.directed
    start, grid, degree = graph.download()
    p, _, _ = oracle_lib.geometry(V, directed)
    _listed(graph)
    for root in roots:
        depth_o, counts_o, swept_o = oracle_lib.bfs(start, grid, p, directed, V, int(root))
        depth, st, launches = _bfs(graph, root)
        assert launches <= 3          # one launch for all levels: the lists are in use
        assert np.array_equal(depth, depth_o)
        assert st["level_counts"].tolist() == counts_o.tolist()
        assert st["swept"].tolist() == swept_o.tolist()
    lab_o, n_o = oracle_lib.wcc(start, grid, p, directed, V)
    lab, n = graph.wcc()
    assert np.array_equal(lab, lab_o) and n == n_o
    for k in [] if directed else ks:
        deg_o, mem_o, _ = oracle_lib.kcore(start, grid, degree, p, V, k)
        deg, mem = graph.kcore(k)
        assert np.array_equal(deg, deg_o) and mem == mem_o, f"k={k}"


@pytest.mark.parametrize("name", GOLDEN_NAMES)
def test_adjacency_golden(name, gpu_ctx_factory, oracle_lib):
    g = load_golden(name)
    graph = gpu_ctx_factory(g["directed"]).upload(g["start"], g["grid"], g["degree"], g["V"])
    _check(graph, oracle_lib, g["bfs_roots"], (1, 2, 3, 8, 24))
    graph.free()


def _two_stars(V):
    """Two components, each a hub with long rows: one is searched bottom-up in
    vain while the other is being found."""
    n = V // 2 - 1
    leaves = np.arange(n, dtype=np.uint32)
    a = np.stack([np.zeros(n, np.uint32), 1 + leaves], 1)
    b = np.stack([np.full(n, V // 2, np.uint32), V // 2 + 1 + leaves], 1)
    chains = np.stack([1 + leaves[:-1], 2 + leaves[:-1]], 1)[np.arange(n - 1) % 100 != 99]
    return np.concatenate([a, b, chains]).astype(np.uint32)


def _edges(name, rng):
    if name == "one":
        return np.array([[0, 1]], np.uint32), 2, (0, 1)
    if name == "stars":
        return _two_stars(30_000), 30_000, (0, 1, 29_999)
    if name == "path":                       # one vertex a level, and a clique at its end
        path = np.stack([np.arange(250), np.arange(1, 251)], 1)
        clique = np.array([(a, b) for a in range(250, 290) for b in range(a + 1, 290)])
        return np.concatenate([path, clique]).astype(np.uint32), 70_001, (0, 125, 289)
    if name == "sparse":                     # many components, some vertices unused
        return rng.integers(0, 200_003, (150_000, 2)).astype(np.uint32), 200_003, (int(rng.integers(0, 200_003)),)
    return rng.integers(0, 4_099, (1 << 20, 2)).astype(np.uint32), 4_099, (0, 4_098)


@pytest.mark.parametrize("directed", [False, True])
@pytest.mark.parametrize("name", ["one", "stars", "path", "sparse", "dense"])
def test_adjacency_matches_oracle(name, directed, gpu_ctx_factory, oracle_lib):
    edges, V, roots = _edges(name, np.random.default_rng(11))
    graph = gpu_ctx_factory(directed).convert(edges, V)
    _check(graph, oracle_lib, roots, (1, 2, 3, 5, 40))
    graph.free()


def test_adjacency_level_overflow_and_step_protocol(gs, gpu_ctx_factory):
    """A BFS past 254 levels still fails alone; sweeps taken one by one still
    run on the tiles and agree."""
    ctx = gpu_ctx_factory(False)
    path = np.arange(0, 301, dtype=np.uint32)
    graph = _listed(ctx.convert(np.stack([path[:-1], path[1:]], 1), 1 << 16))
    with pytest.raises(gs.GStoreError, match="GS_ERR_RANGE"):
        graph.bfs(0)
    depth = graph.bfs(150)
    with graph.state("bfs", 150) as s:
        done = False
        while not done:
            s.sweep()
            _, done = s.finalize()
        assert np.array_equal(s.download(), depth)
    graph.free()


@pytest.fixture(scope="module")
def gs():
    import gstore_b200

    return gstore_b200
