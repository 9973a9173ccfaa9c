"""A graph handed to a server while the device is busy: its blocked order is
finished when gs_serve_add_graph returns (the server's streams do not wait for
the context's), and the requests that follow are answered from it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("windows", [1, 9, 40])
def test_order_is_finished_when_a_served_graph_is_added(windows):
    import torch

    import gstore_b200 as gs

    rng = np.random.default_rng(windows)
    V = (windows - 1) * 65536 + 20_001
    edges = rng.integers(0, V, (300_000, 2)).astype(np.uint32)
    stream, other = torch.cuda.Stream(), torch.cuda.Stream()
    with gs.Context(0) as ctx, gs.Context(0) as alone:
        ctx.set_stream(stream.cuda_stream)
        graph, same = ctx.convert(edges, V), alone.convert(edges, V)
        ks = (2, 4, 9)
        want = [same.kcore(k)[0] for k in ks]
        labels = same.wcc()[0]
        a = torch.randn(8192, 8192, device="cuda", dtype=torch.bfloat16)
        torch.cuda.synchronize()
        with gs.Server(ctx) as srv:
            with torch.cuda.stream(other):
                for _ in range(40):                  # some 30 ms of work that fills every SM
                    torch.mm(a, a)
            gid = srv.add_graph(graph)
            assert stream.query()                    # nothing of the order is still queued
            rids = [srv.submit(gid, "kcore", k) for k in ks] + [srv.submit(gid, "wcc", 0)]
            while srv.step() != (0, 0):
                pass
            got = [srv.result(r)[0] for r in rids]
        torch.cuda.synchronize()
        for g, w in zip(got, [*want, labels]):
            assert np.array_equal(g, w)
        same.free()
        graph.free()
        ctx.set_stream(None)
