"""GPU test of resident traversals without parents around the row lengths at which
vertices change hands (256 and 16384 entries), as one kernel and in parts: depths in
int32 and in bytes equal the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(eb, orc, csr, srcs, launches, policy):
    with eb.Graph.from_csr(csr) as g:
        o = g.opts
        o.policy = policy
        g.opts = o
        for s in srcs:
            exp = orc.bfs(csr.beg_pos, csr.csr, s)[0]
            d, _, st = g.bfs(s)
            np.testing.assert_array_equal(d, exp)
            assert st.launches == launches
            assert (st.traversed_edges, st.reached_vertices) == orc.report(csr.beg_pos, exp)
            row = np.zeros(csr.vert_count, np.uint8)
            g.bfs_many([s], [row])
            np.testing.assert_array_equal(row, np.where(exp < 0, 255, exp).astype(np.uint8))


@pytest.mark.parametrize("policy", [0, 1, 3])
@pytest.mark.parametrize("hub", [254, 255, 256, 16382, 16383, 16384])
def test_one_kernel(eb, orc, hub, policy):
    # two hubs that share their `hub` children and an edge (rows of hub + 1 entries), grandchildren, and a denser part
    rng = np.random.RandomState(hub)
    kids = np.arange(2, hub + 2)
    r0, rest = 2 * hub + 2, 60000
    src = np.concatenate([np.zeros(hub, np.int64), np.ones(hub, np.int64), kids, [0, 2],
                          rng.randint(0, rest, 5 * rest) + r0])
    dst = np.concatenate([kids, kids, kids + hub, [1, r0], rng.randint(0, rest, 5 * rest) + r0])
    csr = eb.Csr.from_edges(src, dst, r0 + rest + 3)
    assert np.diff(csr.beg_pos)[:2].tolist() == [hub + 1, hub + 1]
    _check(eb, orc, csr, [0, 2, hub + 2, r0 + 5, r0 + rest + 1], 1, policy)


@pytest.mark.parametrize("policy", [0, 1, 3])
def test_in_parts(eb, orc, policy):
    # rows of about 300, 16384 and 20000 entries beside a sparse uniform graph of more than 2^22 vertices
    rng = np.random.RandomState(11)
    V = (1 << 22) + 101
    src = np.concatenate([rng.randint(0, V - 9, 12 << 20), np.full(20000, 5), np.full(16384, 7), np.full(300, 11)])
    dst = np.concatenate([rng.randint(0, V - 9, 12 << 20), rng.randint(0, V - 9, 36684)])
    csr = eb.Csr.from_edges(src, dst, V)
    _check(eb, orc, csr, [5, 7, 123456, V - 1], 6, policy)
