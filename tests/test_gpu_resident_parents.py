"""GPU test of traversals with parents as resident kernels, which graphs of more than
786432 vertices take: every place where a parent is stored (claims of light, heavy and
huge rows, of one CTA alone, bottom-up finds by lead entry, by lane, by four rows
and by one row of a warp), in one kernel and in parts. Depths equal the oracle's,
and every parent is an edge one level up."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LIMIT = 3 << 18


def _check(eb, orc, csr, srcs, launches, **opts):
    with eb.Graph.from_csr(csr) as g:
        o = g.opts
        for name, value in opts.items():
            setattr(o, name, value)
        g.opts = o
        for s in srcs:
            exp = orc.bfs(csr.beg_pos, csr.csr, int(s))[0]
            d, p, st = g.bfs(int(s), parents=True)
            np.testing.assert_array_equal(d, exp)
            assert orc.check_parents(csr.beg_pos, csr.csr, int(s), d, p)[0] == 0
            assert g.validate(int(s), d, p) == ((0, -1), (0, -1))
            assert (st.launches == launches) if launches else st.launches > 6
            assert (st.traversed_edges, st.reached_vertices) == orc.report(csr.beg_pos, exp)


@pytest.mark.parametrize("policy", [0, 1, 3])
@pytest.mark.parametrize("small_max", [4, 32])
@pytest.mark.parametrize("kind", ["rmat", "er", "uniform"])
def test_one_kernel(eb, orc, kind, small_max, policy):
    csr = {"rmat": lambda: eb.Csr.rmat(20, 8, seed=0xF1), "er": lambda: eb.Csr.er(LIMIT + 1, 9.0, seed=0xF2),
           "uniform": lambda: eb.Csr.er(LIMIT + 77, 36.0, seed=0xF3)}[kind]()
    _check(eb, orc, csr, eb.pick_sources(csr.beg_pos, 101, 2), 1, small_max=small_max, large_min=1024, policy=policy)


@pytest.mark.parametrize("policy", [0, 1, 3])
@pytest.mark.parametrize("hub", [255, 256, 16383, 16384, 40000])
def test_long_rows_and_chains(eb, orc, hub, policy):
    # a hub with children and grandchildren, a path, an isolated vertex, and an ER part that brings the mean degree past 5
    rng = np.random.RandomState(hub)
    kids = np.arange(1, hub + 1)
    at = 2 * hub + 1
    chain = np.arange(at, at + 300)
    rest = LIMIT - at - 300 + 50
    r0 = at + 300
    src = np.concatenate([np.zeros(hub, np.int64), kids, [hub], chain[:-1], rng.randint(0, rest, 3 * LIMIT) + r0, [r0]])
    dst = np.concatenate([kids, kids + hub, [at], chain[1:], rng.randint(0, rest, 3 * LIMIT) + r0, [at + 299]])
    csr = eb.Csr.from_edges(src, dst, LIMIT + 60)
    _check(eb, orc, csr, [0, 1, at + 150, r0 + 5, LIMIT + 59], 1, policy=policy)


@pytest.mark.parametrize("policy", [0, 1, 3])
def test_in_parts(eb, orc, policy):
    # hubs of heavy and huge rows beside a sparse uniform graph above 2^22 vertices
    rng = np.random.RandomState(7)
    V = (1 << 22) + 101
    src = np.concatenate([rng.randint(0, V - 9, 12 << 20), np.full(20000, 5), np.full(300, 11)])
    dst = np.concatenate([rng.randint(0, V - 9, 12 << 20), rng.randint(0, V - 9, 20300)])
    csr = eb.Csr.from_edges(src, dst, V)
    _check(eb, orc, csr, [5, 123456, V - 1], 6, policy=policy)


def test_smaller_graphs_keep_the_level_loop(eb, orc):
    csr = eb.Csr.er(LIMIT, 9.0, seed=0xF4)
    _check(eb, orc, csr, eb.pick_sources(csr.beg_pos, 102, 1), 0)
