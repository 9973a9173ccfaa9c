"""A graph gets adjacency lists once queries have swept it often enough: the
k-core queries of a batch count when they have run, not when they are asked."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_a_batch_counts_after_it_has_run(gpu_ctx_factory, oracle_lib):
    import gstore_b200 as gs

    ctx = gpu_ctx_factory(False)
    V = 80_001
    edges = np.random.default_rng(10).integers(0, V, (250_000, 2)).astype(np.uint32)
    graph = ctx.convert(edges, V)
    start, grid, degree = graph.download()
    p, _, _ = oracle_lib.geometry(V)
    ks = range(2, 11)                            # nine queries of four sweeps each; 32 sweeps make lists worth it
    want = [oracle_lib.kcore(start, grid, degree, p, V, k)[0] for k in ks]

    def launches_of_a_batch():
        with gs.Batch(ctx) as b:
            ids = [b.add(graph, "kcore", k) for k in ks]
            before = ctx.launches()
            b.run()
            n = ctx.launches() - before
            for i, w in zip(ids, want):
                assert np.array_equal(b.download(i), w)
            return n

    first, second, third = (launches_of_a_batch() for _ in range(3))
    assert first <= 9                            # the tiles' blocked order, once, and the batch's one
    assert second > 9                            # the lists' build
    assert third == 1
    with graph.state("bfs", int(edges[0, 0])) as s:
        before = ctx.launches()
        s.run()
        assert ctx.launches() - before <= 3      # on lists
    graph.free()
