"""GPU test of ent_bfs_noalloc on levels of few vertices with long rows, which
all CTAs share although one could hold the frontier: degree sums around those
at which CTA 0 starts and stops running alone, and a band graph of 1000-vertex
levels, which must not cost a multiple of the ordinary traversal. Depths equal
the CPU oracle's."""
import ctypes as C
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _band(eb, widths, half, seed):
    """Levels of the given widths, each vertex with about `half` random edges to the level before."""
    rng = np.random.RandomState(seed)
    first = np.concatenate([[0], np.cumsum(widths)])
    u, v = [], []
    for k in range(1, len(widths)):
        ids = np.repeat(np.arange(first[k], first[k + 1]), min(half, widths[k - 1]))
        u.append(ids)
        v.append(first[k - 1] + rng.randint(0, widths[k - 1], len(ids)))
    return eb.Csr.from_edges(np.concatenate(u), np.concatenate(v), int(first[-1]) + 1)


def _run(eb, b, a, V, src, out):
    f = eb.lib().ent_bfs_noalloc
    f.restype = C.c_int
    f.argtypes = [C.c_void_p, C.c_void_p, C.c_int64, C.c_int32, C.c_void_p, C.c_void_p]
    assert f(b, a, V, int(src), out.data_ptr(), None) == 0


@pytest.mark.parametrize("width,half", [(100, 20), (102, 20), (103, 20), (204, 20), (206, 20), (1000, 2), (1024, 4),
                                        (1025, 4), (40, 100), (600, 120), (2047, 3), (2049, 3)])
def test_degree_sums(eb, orc, width, half):
    import torch
    # wide levels between narrow ones: CTA 0 takes over and hands back several times
    csr = _band(eb, [width if k % 5 else 3 for k in range(24)], half, width)
    b, a = torch.from_numpy(csr.beg_pos).cuda(), torch.from_numpy(csr.csr).cuda()
    out = torch.full((csr.vert_count,), 7, dtype=torch.int32, device="cuda")
    for s in (0, csr.vert_count // 2, csr.vert_count - 2, csr.vert_count - 1):
        _run(eb, b.data_ptr(), a.data_ptr(), csr.vert_count, s, out)
        np.testing.assert_array_equal(out.cpu().numpy(), orc.bfs(csr.beg_pos, csr.csr, s)[0])


def test_band_time(eb):
    """One CTA alone took 15.4 ms for this graph, all CTAs 1.2 (ent_bfs_device: 2.3)."""
    import torch
    csr = _band(eb, [1000] * 100, 100, 5)
    with eb.Graph.from_csr(csr) as g:
        out = torch.empty(csr.vert_count, dtype=torch.int32, device="cuda")
        beg, adj = g.device_csr()

        def best(call):
            t = []
            for _ in range(6):
                torch.cuda.synchronize()
                t0 = time.perf_counter()
                call()
                torch.cuda.synchronize()
                t.append(time.perf_counter() - t0)
            return min(t)

        ordinary = best(lambda: g.bfs_device(0, out.data_ptr()))
        alone = best(lambda: _run(eb, beg, adj, csr.vert_count, 0, out))
    assert alone < 3 * ordinary, (alone, ordinary)
