"""GPU test of byte rows where their stores change width (rows in 16s, in 4s,
neither) and where a unit of vertices ends: equal to the int32 rows with -1 as
255, up to the deepest level a byte holds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3, 67, 130, 1025])
@pytest.mark.parametrize("V", [16, 256, 1008, 1024, 1040, 4084, 4095, 4112, 8192])
def test_byte_rows_at_widths_and_unit_edges(eb, V, n):
    rng = np.random.RandomState(V + n)
    m = V * 3 // 2
    csr = eb.Csr.from_edges(rng.randint(0, V, m), rng.randint(0, V, m), V)
    srcs = rng.randint(0, V, n)
    with eb.Graph.from_csr(csr) as g:
        d32, _ = g.bfs_batch(srcs)
        d8, _ = g.bfs_batch_u8(srcs)
    np.testing.assert_array_equal(d8, np.where(d32 < 0, 255, d32).astype(np.uint8))


@pytest.mark.parametrize("length", [16, 240, 241, 255])
def test_byte_rows_of_deep_levels(eb, length):
    V = 272
    csr = eb.Csr.from_edges(np.arange(length - 1), np.arange(1, length), V)
    srcs = [0, length - 1, length // 2, V - 1] * 20
    with eb.Graph.from_csr(csr) as g:
        d8, _ = g.bfs_batch_u8(srcs)
    at = np.arange(V)
    for row, s in zip(d8, srcs):
        exp = np.where(at < length, abs(at - s), 255) if s < length else np.where(at == s, 0, 255)
        np.testing.assert_array_equal(row, exp.astype(np.uint8))
