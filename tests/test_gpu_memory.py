"""GPU test of the device memory that the library keeps between its allocations:
it is given back on request, and when an allocation of the library's own would
fail without it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _fill_the_pool(eb):
    """A graph made and closed: several blocks of up to 128 MB come back, about 0.5 GB."""
    rng = np.random.RandomState(1)
    src, dst = rng.randint(0, 1 << 18, (2, 8 << 20))
    eb.Graph.from_edges(src, dst, 1 << 18).close()


def test_release_memory(eb):
    _fill_the_pool(eb)
    kept = _free()
    eb.release_memory()
    assert _free() - kept > 256 * MB
    eb.release_memory()  # nothing is kept: no effect
    with eb.Graph.rmat(12, 16, seed=1) as g:  # the pool goes on
        assert g.bfs(0)[2].status == 0
    for gpu in (-1, 1000):
        with pytest.raises(eb.EntError):
            eb.release_memory(gpu)


def test_other_allocators_get_what_is_kept(eb):
    import torch
    eb.release_memory()
    _fill_the_pool(eb)
    held = []
    try:
        while _free() > 170 * MB:
            held.append(torch.empty(min(_free() - 160 * MB, 16 << 30), dtype=torch.uint8, device="cuda"))
        held.append(torch.empty(300 * MB, dtype=torch.uint8, device="cuda"))
    finally:
        held.clear()
        torch.cuda.empty_cache()
    with eb.Graph.rmat(12, 16, seed=1) as g:
        assert g.bfs(0)[2].status == 0
