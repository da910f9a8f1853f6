"""GPU test of ent_validate where rows change hands (a lane, a warp or a CTA per
row): correct results pass, and a depth damaged at a hub, at one of its
neighbours, far from it or at the source gives the oracle's (rule, vertex)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("degree", [3, 31, 32, 33, 2047, 2048, 2049, 5000])
def test_certificates_at_row_tiers(eb, orc, degree):
    kids = np.arange(1, degree + 1)
    V = 2 * degree + 4
    src = np.concatenate([np.zeros(degree, np.int64), kids, [2 * degree + 1]])
    dst = np.concatenate([kids, kids + degree, [2 * degree + 2]])
    csr = eb.Csr.from_edges(src, dst, V)
    with eb.Graph.from_csr(csr) as g:
        s = degree + 1  # a grandchild of the hub
        depth, parent, _ = g.bfs(s, parents=True)
        assert g.validate(s, depth, parent) == ((0, -1), (0, -1))
        for v, value in [(0, 9), (1, -1), (degree, 7), (2 * degree, -1), (2 * degree, 0), (2 * degree + 1, 4),
                         (V - 1, 3), (s, 1), (0, -2)]:
            bad = depth.copy()
            bad[v] = value
            dc, pc = g.validate(s, bad, parent)
            assert dc == orc.check_depths(csr.beg_pos, csr.csr, s, bad), (v, value)
            assert pc == orc.check_parents(csr.beg_pos, csr.csr, s, bad, parent), (v, value)
        for v, value in [(0, 5), (1, V), (2 * degree, -1), (V - 1, 0), (s, 0)]:
            bad = parent.copy()
            bad[v] = value
            dc, pc = g.validate(s, depth, bad)
            assert dc == (0, -1)
            assert pc == orc.check_parents(csr.beg_pos, csr.csr, s, depth, bad), (v, value)


@pytest.mark.parametrize("build", ["rmat", "er", "edges"])
def test_parent_certificates_of_graphs_built_here(eb, orc, build):
    """Rows with every edge both ways: a parent of the right depth that is no
    neighbour is found at the vertex, as from the parent's row."""
    rng = np.random.RandomState(3)
    g = {"rmat": lambda: eb.Graph.rmat(12, 8, seed=9), "er": lambda: eb.Graph.er(5003, 9.0, seed=9),
         "edges": lambda: eb.Graph.from_edges(rng.randint(0, 5003, 20000), rng.randint(0, 5003, 20000), 5003)}[build]()
    with g:
        csr = g.download()
        s = int(np.argmax(np.diff(csr.beg_pos)))
        depth, parent, _ = g.bfs(s, parents=True)
        assert g.validate(s, depth, parent) == ((0, -1), (0, -1))
        for v in np.flatnonzero(depth >= 2)[:: max(1, (depth >= 2).sum() // 12)]:
            row = csr.csr[csr.beg_pos[v]:csr.beg_pos[v + 1]]
            level = np.flatnonzero(depth == depth[v] - 1)
            for p in [level[-1], level[0], row[0], row[-1], np.setdiff1d(level, row)[0], int(v)]:
                bad = parent.copy()
                bad[v] = p
                assert g.validate(s, depth, bad)[1] == orc.check_parents(csr.beg_pos, csr.csr, s, depth, bad), (v, p)
