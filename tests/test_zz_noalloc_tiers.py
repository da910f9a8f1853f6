"""GPU test of ent_bfs_noalloc where its level split changes: rows at the
degrees from which a CTA and then all CTAs take them, frontiers around the
sizes that one CTA runs alone, chains longer than it runs at once, and rows
that hold one direction only. Depths equal the CPU oracle's."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _depths(eb, beg, adj, src):
    import torch
    f = eb.lib().ent_bfs_noalloc
    f.restype = C.c_int
    f.argtypes = [C.c_void_p, C.c_void_p, C.c_int64, C.c_int32, C.c_void_p, C.c_void_p]
    b = torch.from_numpy(beg).cuda()
    a = torch.from_numpy(adj if len(adj) else np.zeros(1, np.int32)).cuda()
    out = torch.full((len(beg) - 1,), 7, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    assert f(b.data_ptr(), a.data_ptr(), len(beg) - 1, int(src), out.data_ptr(), None) == 0
    return out.cpu().numpy()


def _check(eb, orc, csr, srcs):
    for s in srcs:
        exp, _ = orc.bfs(csr.beg_pos, csr.csr, int(s))
        np.testing.assert_array_equal(_depths(eb, csr.beg_pos, csr.csr, s), exp)


@pytest.mark.parametrize("degree", [1, 31, 32, 255, 256, 257, 1023, 1024, 1025, 2047, 2048, 2049, 32767, 32768, 32769])
def test_hub_and_frontier_sizes(eb, orc, degree):
    # a hub of `degree` children (the second frontier), a grandchild each, all reached from a grandchild too
    kids = np.arange(1, degree + 1)
    src = np.concatenate([np.zeros(degree, np.int64), kids])
    dst = np.concatenate([kids, kids + degree])
    csr = eb.Csr.from_edges(src, dst, 2 * degree + 2)
    _check(eb, orc, csr, [0, 1, 2 * degree, 2 * degree + 1])


@pytest.mark.parametrize("n", [1, 2, 4095, 4097, 9000])
def test_long_chains(eb, orc, n):
    csr = eb.Csr.from_edges(np.arange(n - 1), np.arange(1, n), n)
    _check(eb, orc, csr, [0, n // 2])


def test_one_directional_rows(eb, orc):
    rng = np.random.RandomState(3)
    deg = rng.randint(0, 9, 5000)
    deg[7], deg[11] = 700, 40000
    beg = np.concatenate([[0], np.cumsum(deg)]).astype(np.int64)
    csr = eb.Csr(beg, rng.randint(0, 5000, beg[-1]).astype(np.int32))
    _check(eb, orc, csr, [7, 11, 0, 4999])
