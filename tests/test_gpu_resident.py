"""GPU test of the one-kernel traversal of small graphs where its work changes
hands: rows at the degrees from which a CTA and all CTAs take them, frontiers
around the sizes that one CTA runs alone, chains longer than it runs at once,
isolated sources and byte rows. Each graph carries a clique beside the part
under test, so that its mean degree lets it run as one kernel (one launch in
the statistics). Depths equal the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _with_clique(eb, src, dst, V):
    """The edges on vertices [0, V), and a clique on as many more as bring the mean degree past 5."""
    k = 8
    while k * (k - 1) + 2 * len(src) < 6 * (V + k + 1):
        k += 8
    i, j = np.triu_indices(k, 1)
    return eb.Csr.from_edges(np.concatenate([src, V + i]), np.concatenate([dst, V + j]), V + k + 1), V, k


def _check(eb, orc, csr, srcs, deep=False, **opts):
    with eb.Graph.from_csr(csr) as g:
        o = g.opts
        for name, value in opts.items():
            setattr(o, name, value)
        g.opts = o
        exp = [orc.bfs(csr.beg_pos, csr.csr, int(s))[0] for s in srcs]
        for s, e in zip(srcs, exp):
            d, _, st = g.bfs(int(s))
            np.testing.assert_array_equal(d, e)
            assert st.launches == 1
            assert (st.traversed_edges, st.reached_vertices) == orc.report(csr.beg_pos, e)
            assert st.levels == e.max() + 1 == st.td_levels + st.bu_levels
        if not deep:
            rows = [np.zeros(csr.vert_count, np.uint8) for _ in srcs]
            g.bfs_many(list(srcs), rows)
            for r, e in zip(rows, exp):
                np.testing.assert_array_equal(r, np.where(e < 0, 255, e).astype(np.uint8))


@pytest.mark.parametrize("policy", [0, 1, 2, 3])
@pytest.mark.parametrize("degree", [1, 31, 32, 255, 256, 257, 2047, 2048, 2049, 4095, 4097, 32767, 32768, 32769])
def test_hub_and_frontier_sizes(eb, orc, degree, policy):
    kids = np.arange(1, degree + 1)
    src = np.concatenate([np.zeros(degree, np.int64), kids])
    dst = np.concatenate([kids, kids + degree])
    csr, V, k = _with_clique(eb, src, dst, 2 * degree + 1)
    # the hub, a child, a grandchild, the clique, the isolated last vertex
    _check(eb, orc, csr, [0, 1, 2 * degree, V, V + k], policy=policy)


@pytest.mark.parametrize("n", [2, 300, 4095, 4097, 9000])
def test_long_chains(eb, orc, n):
    csr, V, k = _with_clique(eb, np.arange(n - 1), np.arange(1, n), n)
    _check(eb, orc, csr, [0, n // 2, V + 1], deep=n > 250)


@pytest.mark.parametrize("alpha,beta", [(1e-6, 256.0), (24.0, 1e-6), (1e6, 2.0), (4.0, 8.0)])
@pytest.mark.parametrize("small_max", [1, 4, 32, 300])
def test_direction_switches(eb, orc, alpha, beta, small_max):
    for csr in (eb.Csr.rmat(13, 16, seed=0xA11), eb.Csr.er(20001, 9.0, seed=0xA12)):
        _check(eb, orc, csr, eb.pick_sources(csr.beg_pos, 31, 4), alpha=alpha, beta=beta, small_max=small_max,
               large_min=1024)


@pytest.mark.parametrize("policy", [0, 2, 3])
def test_in_parts(eb, orc, policy):
    """Above 2^22 vertices the bottom-up levels are kernels of their own between
    a head and a tail (eight bottom-up levels here when all are: the tail runs
    what the kernels between do not)."""
    with eb.Graph.er((1 << 22) + 37, 6, seed=0xA14) as g:
        csr = g.download()
        o = g.opts
        o.policy = policy
        g.opts = o
        iso = int(np.flatnonzero(np.diff(csr.beg_pos) == 0)[0])
        for s in [int(x) for x in eb.pick_sources(csr.beg_pos, 33, 2)] + [iso]:
            d, _, st = g.bfs(s)
            exp, _ = orc.bfs(csr.beg_pos, csr.csr, s)
            np.testing.assert_array_equal(d, exp)
            assert st.launches == 6 and st.levels == exp.max() + 1 == st.td_levels + st.bu_levels
            if policy == 3:
                assert st.bu_levels == st.levels
            row = np.zeros(csr.vert_count, np.uint8)
            g.bfs_many([s], [row])
            np.testing.assert_array_equal(row, np.where(exp < 0, 255, exp).astype(np.uint8))


def test_streams_in_turn(eb, orc):
    """Asynchronous traversals of one handle on two streams keep their order: each row is its own source's."""
    import torch
    csr = eb.Csr.rmat(15, 16, seed=0xA13)
    srcs = [int(s) for s in eb.pick_sources(csr.beg_pos, 32, 12)]
    with eb.Graph.from_csr(csr) as g:
        rows = torch.full((len(srcs), csr.vert_count), 7, dtype=torch.int32, device="cuda")
        streams = [torch.cuda.Stream(), torch.cuda.Stream()]
        torch.cuda.synchronize()
        for i, s in enumerate(srcs):
            g.bfs_device(s, rows[i].data_ptr(), stream=streams[i % 2].cuda_stream, stats=False)
        torch.cuda.synchronize()
        got = rows.cpu().numpy()
    for i, s in enumerate(srcs):
        np.testing.assert_array_equal(got[i], orc.bfs(csr.beg_pos, csr.csr, s)[0])
