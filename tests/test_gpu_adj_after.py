"""Calls on a BFS state after gs_run took the query on adjacency lists, whose
bitmaps are not the sweeps': they answer as after a run on the tiles."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graph(ctx, edges, V, listed):
    graph = ctx.convert(edges, V)
    for _ in range(17 if listed else 0):
        graph.wcc()
    return graph


@pytest.mark.parametrize("listed", [False, True])
def test_finalize_after_a_finished_run(listed, gpu_ctx_factory):
    edges = np.random.default_rng(4).integers(0, 90_000, (200_000, 2)).astype(np.uint32)
    graph = _graph(gpu_ctx_factory(False), edges, 90_000, listed)
    with graph.state("bfs", int(edges[0, 0])) as s:
        s.run()
        depth, levels = s.download(), s.bfs_stats()["level_counts"].tolist()
        assert s.finalize() == (0, True)
        assert np.array_equal(s.download(), depth)
        assert s.bfs_stats()["level_counts"].tolist() == levels + [0]
    graph.free()


@pytest.mark.parametrize("listed", [False, True])
def test_run_again_after_too_many_levels(listed, gpu_ctx_factory):
    import gstore_b200 as gs

    path = np.arange(0, 301, dtype=np.uint32)
    graph = _graph(gpu_ctx_factory(False), np.stack([path[:-1], path[1:]], 1), 1 << 16, listed)
    with graph.state("bfs", 0) as s:
        for _ in range(2):
            with pytest.raises(gs.GStoreError, match="GS_ERR_RANGE"):
                s.run()
        s.reset(150)
        s.run()
        want = np.zeros(1 << 16, np.uint8)
        want[:301] = np.abs(np.arange(301) - 150) + 1
        assert np.array_equal(s.download(), want)
    graph.free()
