"""PageRank over pulled bins (gs_pr_blocked.cu: graphs without hubs) against the
FP64 oracle and, after one iteration, against exact sums; plain and served."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PR_TOL = 1e-6


@pytest.fixture(scope="module")
def gs():
    import gstore_b200
    return gstore_b200


def _edges(name):
    rng = np.random.default_rng(11)
    V = 400_009 if name == "ragged" else 1 << 19
    e = rng.integers(0, V, (8 * V, 2))
    if name == "gaps":               # vertices without records, bins of half the mean
        e |= 1
        e[:, 1] = np.where(e[:, 1] < V // 4, e[:, 1] | 2, e[:, 1])
    elif name == "full":             # bins of twice the mean: too full to be pulled
        e[:, 1] //= 2
    elif name in ("longest", "longer"):   # a row of 128 entries, the longest that is pulled, or of 129
        e = e[(e != 77).all(1)]
        n = 128 if name == "longest" else 129
        e = np.concatenate([e, np.stack([100 + np.arange(n), np.full(n, 77)], 1)])
    return e.astype(np.uint32), V


@pytest.mark.parametrize("name,directed", [("uniform", False), ("uniform", True), ("ragged", False), ("ragged", True),
                                           ("gaps", True), ("full", True), ("longest", True), ("longest", False),
                                           ("longer", True)])
def test_pagerank_bins(name, directed, gs, gpu_ctx_factory, oracle_lib):
    edges, V = _edges(name)
    edges = edges[edges[:, 0] != edges[:, 1]]
    ctx = gpu_ctx_factory(directed)
    g = ctx.convert(edges, V)
    start, grid, degree = g.download()
    p, _, _ = oracle_lib.geometry(V)
    r1, _ = g.pagerank(1)
    r64, x64 = oracle_lib.pagerank(start, grid, degree, p, directed, V, 4)
    r, x = g.pagerank(4)
    again, _ = g.pagerank(1)
    with gs.Server(ctx) as srv:
        rid = srv.submit(srv.add_graph(g), "pagerank", 4)
        while srv.step() != (0, 0):
            pass
        served = srv.result(rid)[0]
    g.free()
    if V & (V - 1) == 0:
        # x = 1/V is a power of two: every sum of the first iteration is exact
        into = np.bincount(edges[:, 1], minlength=V).astype(np.float64)
        if not directed:
            into += np.bincount(edges[:, 0], minlength=V)
        exact = (0.15 + 0.85 * (into / V)).astype(np.float32)
        assert np.array_equal(r1, exact) and np.array_equal(again, exact)
    for a, b in ((r, r64), (x, x64), (served, r64)):
        assert np.abs(a.astype(np.float64) - b).sum() <= PR_TOL * np.abs(b).sum()
