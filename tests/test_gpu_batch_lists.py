"""Batched k-core on adjacency lists (wk_batch_kernel), beside batched WCC on
the tiles of the same graph, against the oracle: a graph with fewer runs of
tiles than blocks of vertex words, rows around the lengths that a lane, a warp
and the whole CTA take, and more long rows in one block than a CTA keeps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _edges(name):
    rng = np.random.default_rng(5)
    if name == "few_runs":       # 41 windows, 1,312 blocks of words; records in three tiles
        V = 40 * 65536 + 777
        a, b = rng.integers(0, 700, (2, 3_000))
        far = 40 * 65536
        e = np.concatenate([np.stack([a, b], 1), np.stack([a, far + b], 1), far + np.stack([b, a], 1)])
    else:
        # "rows": hubs of every length; "long_rows": 100 hubs of 1,100 to 1,199 entries side by side
        lengths = [1, 31, 32, 33, 63, 64, 65, 66, 1023, 1024, 1025, 1500] if name == "rows" else list(range(1100, 1200))
        V, at, parts = 70_001, 0, []
        for i, n in enumerate(lengths):
            parts.append(np.stack([np.full(n, i), 4_096 + (at + np.arange(n)) % 30_000], 1))
            at += n
        core = np.array([(a, b) for a in range(3_000, 3_030) for b in range(a + 1, 3_030)])   # 29 neighbours each
        e = np.concatenate([*parts, core])
    return e[e[:, 0] != e[:, 1]].astype(np.uint32), V


@pytest.mark.parametrize("name", ["few_runs", "rows", "long_rows"])
def test_batched_kcore_on_lists(name, gpu_ctx_factory, oracle_lib):
    import gstore_b200 as gs

    edges, V = _edges(name)
    ctx = gpu_ctx_factory(False)
    graph = ctx.convert(edges, V)
    start, grid, degree = graph.download()
    p, _, _ = oracle_lib.geometry(V)
    for _ in range(17):
        graph.wcc()
    with graph.state("bfs", int(edges[0, 0])) as s:
        before = ctx.launches()
        s.run()
        assert ctx.launches() - before <= 3      # the lists are in use
    ks = (1, 2, 5, 20, 29, 30, 1_030, 2_000)
    with gs.Batch(ctx) as b:
        cores = [b.add(graph, "kcore", k) for k in ks]
        wcc = b.add(graph, "wcc")
        b.run()
        assert b.stats()["launches"] == 1
        for qid, k in zip(cores, ks):
            deg_o, mem_o, _ = oracle_lib.kcore(start, grid, degree, p, V, k)
            assert np.array_equal(b.download(qid), deg_o) and b.count(qid) == mem_o, f"k={k}"
        lab_o, n_o = oracle_lib.wcc(start, grid, p, False, V)
        assert np.array_equal(b.download(wcc), lab_o) and b.count(wcc) == n_o
    graph.free()
