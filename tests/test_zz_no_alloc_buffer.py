"""gs_bfs_noalloc writes the V bytes of the caller's buffer and no others,
wherever in memory the buffer starts and ends (it may be a row of a larger
array, whose other rows other streams write)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GUARD = 64


@pytest.mark.parametrize("V", [37, 65_567, 70_001, 131_072])   # V % 32: 5, 31, 17, 0
@pytest.mark.parametrize("offset", [0, 1, 4, 8, 15])
def test_noalloc_stays_inside_the_buffer(V, offset, gpu_ctx_factory):
    import torch

    ctx = gpu_ctx_factory(False)
    root = 3
    others = np.delete(np.arange(V, dtype=np.uint32), root)
    graph = ctx.convert(np.stack([np.full(V - 1, root, np.uint32), others], 1), V)
    want = np.full(V, 2, np.uint8)          # whole words of one level, the last one cut off by V
    want[root] = 1
    space = torch.full((GUARD + offset + V + GUARD,), 0xA5, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    sweeps = graph.bfs_noalloc(root, space.data_ptr() + GUARD + offset)
    got = space.cpu().numpy()
    lo = GUARD + offset
    assert sweeps == 2
    assert np.array_equal(got[lo:lo + V], want)
    assert (got[:lo] == 0xA5).all() and (got[lo + V:] == 0xA5).all()
    assert np.array_equal(graph.bfs(root), want)
    graph.free()
