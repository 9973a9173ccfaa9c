"""Device allocations that fail: what a faster layout cannot have, the engine
does without."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NONE = (2**64 - 1, 0)


def fail_allocs(ctx, least, most):
    """From now on ctx's device allocations of `least` to `most` bytes fail."""
    import gstore_b200 as gs

    fn = gs.lib().gs_testing_fail_allocs
    fn.argtypes, fn.restype = [C.c_void_p, C.c_uint64, C.c_uint64], None
    fn(ctx._h, least, most)


@pytest.fixture
def ctx():
    import gstore_b200 as gs

    with gs.Context(0) as c:
        yield c


@pytest.mark.parametrize("shape", ["star", "dense"])
def test_pagerank_without_room_for_row_lists(shape, ctx, oracle_lib):
    """The row lists' build reserves over 12 MB in one block, the other
    layouts of these graphs take less."""
    V = 1 << 16
    if shape == "star":
        edges = np.stack([np.full(40_000, 3), 4 + np.arange(40_000)], 1).astype(np.uint32)
    else:
        edges = np.random.default_rng(2).integers(0, 300, (100_000, 2)).astype(np.uint32)
    graph = ctx.convert(edges, V)
    start, grid, degree = graph.download()
    p, _, _ = oracle_lib.geometry(V)
    r64, x64 = oracle_lib.pagerank(start, grid, degree, p, False, V, 3)
    fail_allocs(ctx, 12 << 20, 2**64 - 1)
    short = [graph.pagerank(3) for _ in range(2)]
    fail_allocs(ctx, *NONE)
    short.append(graph.pagerank(3))
    graph.free()
    for r, x in short:
        assert np.abs(r.astype(np.float64) - r64).sum() <= 1e-6 * np.abs(r64).sum()
        assert np.abs(x.astype(np.float64) - x64).sum() <= 1e-6 * np.abs(x64).sum()
