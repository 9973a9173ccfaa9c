"""Served PageRank is as close to the 64-bit ranks as one rounding to 32 bits:
the sums of the blocked layout are not cut into more pieces, each added in 32
bits, than a bin of a small graph needs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [18, 19, 20])
def test_served_ranks_within_a_rounding(scale, gpu_ctx_factory, oracle_lib):
    import gstore_b200 as gs

    ctx = gpu_ctx_factory(False)
    V = 1 << scale
    graph = ctx.convert(ctx.kron_generate(scale, 16), V)
    start, grid, degree = graph.download()
    p, _, _ = oracle_lib.geometry(V)
    r64, _ = oracle_lib.pagerank(start, grid, degree, p, False, V, 5)
    errors = []
    with gs.Server(ctx) as srv:
        gid = srv.add_graph(graph)
        for _ in range(24):                  # (the order of the additions differs from run to run)
            rid = srv.submit(gid, "pagerank", 5)
            while srv.step() != (0, 0):
                pass
            r = srv.result(rid)[0].astype(np.float64)
            errors.append(np.linalg.norm(r - r64) / np.linalg.norm(r64))
    graph.free()
    # 2-norm, mean of the runs: a quarter over the unit roundoff 2^-24
    assert np.mean(errors) <= 1.25 * 2.0**-24, np.mean(errors)
