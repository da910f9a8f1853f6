"""GPU test of bottom-up levels of the resident kernels over words full of rows of
small_max entries and more: a warp scans four at a time while there are four,
then one by one. Rows end around the steps of both, words hold any number of such
rows, and graphs lie on both sides of the size from which a warp takes three
words together. Depths equal the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("policy", [0, 3])
@pytest.mark.parametrize("small_max", [1, 8, 32, 48])
@pytest.mark.parametrize("V,degree", [(2011, 31.0), (2011, 64.0), (9001, 20.0), (9001, 40.0), (700001, 12.0)])
def test_rows_and_words(eb, orc, V, degree, small_max, policy):
    csr = eb.Csr.er(V, degree, seed=0xD0 + int(degree))
    with eb.Graph.from_csr(csr) as g:
        o = g.opts
        o.policy, o.small_max, o.large_min = policy, small_max, 1024
        g.opts = o
        for s in eb.pick_sources(csr.beg_pos, 81, 2 if V > 100000 else 4):
            exp = orc.bfs(csr.beg_pos, csr.csr, int(s))[0]
            d, _, st = g.bfs(int(s))
            np.testing.assert_array_equal(d, exp)
            assert st.launches == 1 and st.bu_levels > 0


@pytest.mark.parametrize("long_rows", [1, 3, 4, 5, 31, 32, 33, 200])
@pytest.mark.parametrize("length", [33, 63, 64, 65, 127, 300])
def test_counts_of_long_rows(eb, orc, long_rows, length):
    """`long_rows` vertices of `length` neighbours beside short rows; found through any of their entries, or not at all."""
    rng = np.random.RandomState(length * 1000 + long_rows)
    V = 4000
    src = np.concatenate([np.repeat(np.arange(long_rows), length), rng.randint(500, V - 500, 9 * V)])
    dst = np.concatenate([rng.randint(500, V, long_rows * length), rng.randint(500, V - 500, 9 * V)])
    csr = eb.Csr.from_edges(src, dst, V + 50)
    with eb.Graph.from_csr(csr) as g:
        o = g.opts
        o.policy = 3  # every level bottom-up
        g.opts = o
        for s in (0, 700, V - 1, V + 1):
            d, _, st = g.bfs(s)
            np.testing.assert_array_equal(d, orc.bfs(csr.beg_pos, csr.csr, s)[0])
            assert st.launches == 1


def test_time_of_uniform_rows(eb):
    """Rows one after another: 268 us a traversal of this graph, as long as the level kernels need; four together 158."""
    import torch
    with eb.Graph.er(1 << 20, 40, seed=3) as g:
        d = torch.empty(g.vert_count, dtype=torch.int32, device="cuda")
        srcs = eb.pick_sources(g.download().beg_pos, 83, 8)

        def median():
            t = [g.bfs_device(int(s), d.data_ptr()).device_ms for _ in range(3) for s in srcs]
            return float(np.median(t[len(srcs):]))

        resident = median()
        o = g.opts
        o.narrow_max_frontier = 0  # the level kernels
        g.opts = o
        assert resident < 0.85 * median()
