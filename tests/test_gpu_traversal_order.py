"""GPU tests of what depends on the traversal order and on how top-down batch
levels split rows: hubs whose degrees sit at the edges of a warp's chunk of
entries, sources without a row, and rows that the caller left one-directional.
Every row equals the CPU oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _hub_graph(eb, degree, tail):
    """A hub of exactly `degree` neighbours, each with a leaf for every third, and isolated vertices after them."""
    src, dst = [0] * degree, list(range(1, degree + 1))
    v = degree + 1
    for i in range(1, degree + 1, 3):
        src.append(i)
        dst.append(v)
        v += 1
    return eb.Csr.from_edges(src, dst, v + tail)


@pytest.mark.parametrize("n_src", [1, 65, 300])
@pytest.mark.parametrize("degree", [31, 32, 511, 512, 513, 1024, 1025, 4096])
def test_batch_hub_rows_at_chunk_edges(eb, orc, degree, n_src):
    csr = _hub_graph(eb, degree, 5)
    V = csr.vert_count
    rng = np.random.RandomState(degree)
    srcs = [0, V - 1] + [int(x) for x in rng.randint(0, V, 298)]  # the hub, an isolated vertex, any others
    with eb.Graph.from_csr(csr) as g:
        for alpha in (1e-9, 4.0, 1e9):  # all top-down, the default, all bottom-up
            o = g.opts
            o.batch_alpha, o.batch_deep = alpha, 0
            g.opts = o
            rows, stats = g.bfs_batch(srcs[:n_src])
            for i, s in enumerate(srcs[:n_src]):
                exp, _ = orc.bfs(csr.beg_pos, csr.csr, s)
                np.testing.assert_array_equal(rows[i], exp)
                assert (stats[i].traversed_edges, stats[i].reached_vertices) == orc.report(csr.beg_pos, exp)
                assert stats[i].levels == exp.max() + 1


@pytest.mark.parametrize("small_max", [1, 2, 32])
@pytest.mark.parametrize("policy", ["beamer", "td", "bu"])
def test_single_hub_and_isolated_source(eb, orc, policy, small_max):
    csr = _hub_graph(eb, 777, 40)
    with eb.Graph.from_csr(csr) as g:
        o = g.opts
        o.policy, o.small_max = eb.POLICY[policy], small_max
        g.opts = o
        for s in (0, 1, 777, csr.vert_count - 1, 2):
            depth, parent, _ = g.bfs(s, parents=True)
            exp, _ = orc.bfs(csr.beg_pos, csr.csr, s)
            np.testing.assert_array_equal(depth, exp)
            assert orc.check_parents(csr.beg_pos, csr.csr, s, depth, parent)[0] == 0


def test_one_directional_rows_top_down(eb, orc):
    """A CSR whose rows hold one direction only: vertices without a row are reached, in several calls on one handle."""
    beg = np.array([0, 2, 4, 4, 5, 5, 5, 5], dtype=np.int64)
    adj = np.array([1, 2, 3, 2, 4], dtype=np.int32)
    with eb.Graph.from_arrays(beg, adj) as g:
        o = g.opts
        o.policy = eb.POLICY["td"]
        g.opts = o
        for s in (0, 1, 3, 0, 6, 2, 0):
            depth, _, _ = g.bfs(s)
            exp, _ = orc.bfs(beg, adj, s)
            np.testing.assert_array_equal(depth, exp)
