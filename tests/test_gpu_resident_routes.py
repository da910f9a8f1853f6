"""GPU test of which graphs of mean degree 5 and more leave the resident kernels
for the level loop: those whose traversals show many small levels (meshes,
bands), known once a first traversal has ended, whether the host waited for it or
not, and within a source list after its first sources. Depths equal the oracle's on both routes; the
launches of the statistics tell the routes apart."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _band(eb, levels, width, half):
    rng = np.random.RandomState(width)
    u = np.repeat(np.arange((levels - 1) * width, dtype=np.int64), half)
    return eb.Csr.from_edges(u, (u // width + 1) * width + rng.randint(0, width, u.size), levels * width)


def _mesh(eb, n):
    i = np.arange(n ** 3, dtype=np.int64)
    x, y, z = i % n, i // n % n, i // n // n
    e = [(i[c], i[c] + st) for c, st in ((x < n - 1, 1), (y < n - 1, n), (z < n - 1, n * n))]
    return eb.Csr.from_edges(np.concatenate([a for a, _ in e]), np.concatenate([b for _, b in e]), n ** 3)


GRAPHS = {
    "mesh": (lambda eb: _mesh(eb, 24), True),
    "narrow band": (lambda eb: _band(eb, 96, 200, 20), True),
    "long thin band": (lambda eb: _band(eb, 400, 50, 10), True),
    "wide band": (lambda eb: _band(eb, 96, 1000, 100), False),  # 190k entries a level
    "short band": (lambda eb: _band(eb, 12, 200, 20), False),
    "rmat": (lambda eb: eb.Csr.rmat(14, 16, seed=0xC1), False),
    "er": (lambda eb: eb.Csr.er(30001, 9.0, seed=0xC2), False),
}


@pytest.mark.parametrize("first", ["waited for", "not waited for", "source list"])
@pytest.mark.parametrize("name", list(GRAPHS))
def test_routes(eb, orc, name, first):
    import torch
    make, deep = GRAPHS[name]
    csr = make(eb)
    srcs = [int(s) for s in eb.pick_sources(csr.beg_pos, 71, 3)]
    exp = [orc.bfs(csr.beg_pos, csr.csr, s)[0] for s in srcs]
    with eb.Graph.from_csr(csr) as g:
        row = torch.full((csr.vert_count,), 7, dtype=torch.int32, device="cuda")
        if first == "source list":
            rows = [np.zeros(csr.vert_count, np.int32) for _ in srcs]
            g.bfs_many(srcs, rows)
            for r, e in zip(rows, exp):
                np.testing.assert_array_equal(r, e)
        else:
            st = g.bfs_device(srcs[0], row.data_ptr(), stats=first == "waited for")
            torch.cuda.synchronize()
            np.testing.assert_array_equal(row.cpu().numpy(), exp[0])
            assert st is None or st.launches == 1
        for s, e in zip(srcs, exp):
            d, _, st = g.bfs(s)
            np.testing.assert_array_equal(d, e)
            assert (st.launches > 1) == deep, st
            assert st.levels == e.max() + 1 == st.td_levels + st.bu_levels
