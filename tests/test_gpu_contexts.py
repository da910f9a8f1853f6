"""GPU test of a program that makes CUDA contexts of its own, one after another,
beside the primary one: graphs live in each, with copies above and below the sizes
at which the library stages them, and nothing kept from a context that is gone is
used again."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture
def driver():
    cu = C.CDLL("libcuda.so.1")

    def call(name, *args):
        rc = getattr(cu, name)(*args)
        assert rc == 0, (name, rc)

    call("cuInit", 0)
    return call


def _work(eb, orc, csr, srcs):
    with eb.Graph.from_csr(csr) as g, eb.Graph.grid(64, 64, 0.1, seed=2) as grid:
        back = g.download()
        np.testing.assert_array_equal(back.beg_pos, csr.beg_pos)
        np.testing.assert_array_equal(back.csr, csr.csr)
        for s in srcs:
            exp = orc.bfs(csr.beg_pos, csr.csr, int(s))[0]
            d, p, _ = g.bfs(int(s), parents=True)
            np.testing.assert_array_equal(d, exp)
            assert orc.check_parents(csr.beg_pos, csr.csr, int(s), d, p)[0] == 0
            np.testing.assert_array_equal(g.bfs(int(s))[0], exp)
        rows, _ = g.bfs_batch(srcs)
        np.testing.assert_array_equal(rows[0], orc.bfs(csr.beg_pos, csr.csr, int(srcs[0]))[0])
        assert grid.bfs(0)[2].status == 0


def test_contexts_in_turn(eb, orc, driver):
    csr = eb.Csr.rmat(16, 16, seed=0x61)  # 8 MB of columns, depths below 1 MB
    srcs = eb.pick_sources(csr.beg_pos, 111, 2)
    dev = C.c_int()
    driver("cuDeviceGet", C.byref(dev), 0)
    _work(eb, orc, csr, srcs)  # the primary context
    for _ in range(3):
        ctx = C.c_void_p()
        driver("cuCtxCreate_v2", C.byref(ctx), 0, dev)
        try:
            _work(eb, orc, csr, srcs)
        finally:
            driver("cuCtxDestroy_v2", ctx)
        _work(eb, orc, csr, srcs)


def test_graphs_of_two_contexts_at_once(eb, orc, driver):
    csr = eb.Csr.rmat(14, 16, seed=0x62)
    s = int(eb.pick_sources(csr.beg_pos, 112, 1)[0])
    exp = orc.bfs(csr.beg_pos, csr.csr, s)[0]
    dev, ctx, out = C.c_int(), C.c_void_p(), C.c_void_p()
    driver("cuDeviceGet", C.byref(dev), 0)
    mine = eb.Graph.from_csr(csr)
    np.testing.assert_array_equal(mine.bfs(s)[0], exp)
    driver("cuCtxCreate_v2", C.byref(ctx), 0, dev)
    try:
        other = eb.Graph.from_csr(csr)
        np.testing.assert_array_equal(other.bfs(s)[0], exp)
        driver("cuCtxPopCurrent_v2", C.byref(out))
        np.testing.assert_array_equal(mine.bfs(s)[0], exp)
        driver("cuCtxPushCurrent_v2", ctx)
        np.testing.assert_array_equal(other.bfs(s)[0], exp)
        other.close()
    finally:
        driver("cuCtxDestroy_v2", ctx)
    np.testing.assert_array_equal(mine.bfs(s)[0], exp)
    mine.close()
