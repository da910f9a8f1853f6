"""GPU test of copies between the device and pageable host memory at the sizes
where they change route (1 MB) and chunk (4 MB), forth and back, and of row
copies that pack whole rows into a chunk."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 18  # int32 entries


@pytest.mark.parametrize("E", [1, MB - 1, MB, MB + 1, 4 * MB - 1, 4 * MB, 4 * MB + 1, 8 * MB, 8 * MB + 1, 13 * MB + 5])
def test_csr_round_trip(eb, E):
    rng = np.random.RandomState(E & 0xFFFF)
    V = 1001
    beg = np.concatenate([[0], np.sort(rng.randint(0, E + 1, V - 1)), [E]]).astype(np.int64)
    adj = rng.randint(0, V, E).astype(np.int32)
    with eb.Graph.from_arrays(beg, adj) as g:
        back = g.download()
    np.testing.assert_array_equal(back.beg_pos, beg)
    np.testing.assert_array_equal(back.csr, adj)


@pytest.mark.parametrize("scale,n_src", [(13, 31), (13, 33), (14, 64), (16, 40)])
def test_rows_of_a_plan(eb, scale, n_src):
    with eb.Graph.rmat(scale, 8, seed=5) as a, eb.Graph.er(5003, 9.0, seed=6) as b:
        csr = a.download()
        srcs = eb.pick_sources(csr.beg_pos, 7, n_src)
        with eb.MultiPlan([b, a], [[1, 2], srcs]) as plan:
            plan.run()
            rows = plan.depths(1)
        exp, _ = a.bfs_batch(srcs)
        np.testing.assert_array_equal(rows, exp)
        for i in (0, n_src - 1):
            np.testing.assert_array_equal(rows[i], a.bfs(int(srcs[i]))[0])
