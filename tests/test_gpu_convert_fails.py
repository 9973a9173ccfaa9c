"""A conversion that runs out of memory half way: nothing of it is still
queued when the error is returned, since the caller may free the edge list."""
import numpy as np
import pytest

from test_gpu_short_memory import NONE, fail_allocs

pytestmark = pytest.mark.gpu


def test_failed_conversion_has_finished():
    import torch

    import gstore_b200 as gs

    V, n = 1 << 22, 20_000
    pairs = torch.from_numpy(np.random.default_rng(6).integers(0, V, (n, 2)).astype(np.int32)).cuda()
    a = torch.randn(8192, 8192, device="cuda", dtype=torch.bfloat16)
    stream, other = torch.cuda.Stream(), torch.cuda.Stream()
    with gs.Context(0) as ctx:
        ctx.set_stream(stream.cuda_stream)
        want = ctx.convert(pairs.data_ptr(), V, n_pairs=n)
        expect = want.download()
        want.free()
        torch.cuda.synchronize()
    with gs.Context(0) as ctx:
        ctx.set_stream(stream.cuda_stream)
        with torch.cuda.stream(other):
            for _ in range(40):                      # work that fills every SM
                torch.mm(a, a)
        # the records take 80 KB, .start 263 KB, the tiles' sort something between
        fail_allocs(ctx, 82_000, 262_000)
        with pytest.raises(gs.GStoreError, match="GS_ERR_OOM"):
            ctx.convert(pairs.data_ptr(), V, n_pairs=n)
        assert stream.query()
        fail_allocs(ctx, *NONE)
        graph = ctx.convert(pairs.data_ptr(), V, n_pairs=n)
        for got, exp in zip(graph.download(), expect):
            assert np.array_equal(got, exp)
        graph.free()
        torch.cuda.synchronize()
        ctx.set_stream(None)
