"""bench.py books every timed BFS by the path it took, and states no share of
a bandwidth for kernels that did not read the records."""
import numpy as np
import pytest

import bench


def test_roofline_without_bytes_has_no_share():
    none = bench.roofline(6000.0, "measured", "k", 1, 0.5, 0, "-")
    some = bench.roofline(6000.0, "measured", "k", 1, 0.5, 3_000_000, "-")
    assert none["achieved"] is None and none["frac"] is None and none["bound"] != "hbm"
    assert some["bound"] == "hbm" and abs(some["frac"] - 0.001) < 1e-12


@pytest.mark.gpu
def test_paths_of_a_graph_queried_often(gpu_ctx_factory):
    import gstore_b200 as gs

    ctx = gpu_ctx_factory(False)
    graph = ctx.convert(ctx.kron_generate(16, 16), 1 << 16)
    nz = np.nonzero(graph.degree())[0]
    ctx.profile(True)
    paths, timed, levels = [], [], []
    with graph.state("bfs", int(nz[0])) as s:
        for r in nz[:12]:
            launches, n = ctx.launches(), ctx.kernel_time(gs.GS_ALGO_BFS)[0]
            s.reset(int(r))
            s.run()
            timed.append(ctx.kernel_time(gs.GS_ALGO_BFS)[0] - n)
            paths.append(bench.bfs_path(ctx.launches() - launches, timed[-1]))
            levels.append(int(s.bfs_stats()["level_counts"].size))
    # eight queries on the tiles, a timed sweep per level, then the lists
    assert paths == ["tiles"] * 8 + ["build"] + ["lists"] * 3
    assert timed == levels[:8] + [1] * 4
    for algo, arg, gid in (("wcc", 0, gs.GS_ALGO_WCC), ("kcore", 8, gs.GS_ALGO_KCORE)):
        ctx.profile(True)
        with graph.state(algo, arg) as s:
            s.run()
        n, ms, nbytes = ctx.kernel_time(gid)
        assert n == 1 and ms > 0 and nbytes == 0    # on lists: no claim on the records' bytes
    ctx.profile(False)
    graph.free()
