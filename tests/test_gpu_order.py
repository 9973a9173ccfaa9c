"""Sweeps in the L2-blocked orders (gs_order.cu) on graphs of many windows:
blocks at the grid's ragged end, tiles of many units, rows with one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("windows", [1, 64, 65, 131])
def test_blocked_orders(windows, gpu_ctx_factory, oracle_lib):
    import gstore_b200 as gs

    rng = np.random.default_rng(windows)
    V = (windows - 1) * 65536 + 12_345
    spread = rng.integers(0, V, (200_000, 2))
    dense = (V - 12_000) + rng.integers(0, 12_000, (60_000, 2))      # one tile of many units
    edges = np.concatenate([spread, dense]).astype(np.uint32)
    ctx = gpu_ctx_factory(False)
    g = ctx.convert(edges, V)
    start, grid, degree = g.download()
    p, _, _ = oracle_lib.geometry(V)
    lab_o, n_o = oracle_lib.wcc(start, grid, p, False, V)
    lab, n = g.wcc()
    assert np.array_equal(lab, lab_o) and n == n_o
    for k in (2, 5):
        deg_o, mem_o, _ = oracle_lib.kcore(start, grid, degree, p, V, k)
        deg, mem = g.kcore(k)
        assert np.array_equal(deg, deg_o) and mem == mem_o
    roots = [int(edges[0, 0]), int(edges[-1, 1])]
    want = [oracle_lib.bfs(start, grid, p, False, V, r)[0] for r in roots]
    for _ in range(9):                                               # every order the batch tries
        with gs.Batch(ctx) as b:
            ids = [b.add(g, "bfs", r) for r in roots]
            b.run()
            for i, w in zip(ids, want):
                assert np.array_equal(b.download(i), w)
    g.free()
