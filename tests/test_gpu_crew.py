"""GPU test of the kernels whose CTAs go from phase to phase together, beside other
work: kernels on other streams hold some SMs, for longer than a traversal takes or
for moments that end while it runs, so CTAs start late or join between phases. The
traversal does not wait for the held SMs, and depths equal the oracle's."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MS = 1_500_000  # cycles, at most a millisecond


def _noalloc(eb):
    f = eb.lib().ent_bfs_noalloc
    f.restype = C.c_int
    f.argtypes = [C.c_void_p, C.c_void_p, C.c_int64, C.c_int32, C.c_void_p, C.c_void_p]
    return f


class _Runs:
    """The traversals under test, by name: (graph, call(source, row, stream))."""

    def __init__(self, eb):
        self.graphs = {"rmat": eb.Graph.rmat(16, 16, seed=0xE1), "small": eb.Graph.rmat(11, 16, seed=0xE2),
                       "parts": eb.Graph.er((1 << 22) + 37, 6, seed=0xE3), "grid": eb.Graph.grid(150, 150, 0.1, seed=0xE4)}
        f = _noalloc(eb)
        self.calls = {}
        for name, g in self.graphs.items():
            if name != "grid":
                self.calls[name] = (g, lambda s, row, st, g=g: g.bfs_device(s, row.data_ptr(), stream=st.cuda_stream, stats=False))
            if name in ("rmat", "grid"):
                beg, adj = g.device_csr()
                self.calls["noalloc " + name] = (g, lambda s, row, st, g=g, b=beg, a=adj: self._check(
                    f(b, a, g.vert_count, s, row.data_ptr(), C.c_void_p(st.cuda_stream))))

    @staticmethod
    def _check(status):
        assert status == 0


@pytest.fixture(scope="module")
def runs(eb):
    return _Runs(eb)


@pytest.fixture(scope="module")
def expected(runs, eb, orc):
    out = {}
    for name, (g, _) in runs.calls.items():
        csr = g.download()
        out[name] = [(int(s), orc.bfs(csr.beg_pos, csr.csr, int(s))[0]) for s in eb.pick_sources(csr.beg_pos, 91, 3)]
    return out


NAMES = ["rmat", "small", "parts", "noalloc rmat", "noalloc grid"]


@pytest.mark.parametrize("held", [1, 16, 100])
@pytest.mark.parametrize("name", NAMES)
def test_held_sms_are_not_waited_for(runs, expected, name, held):
    import torch
    g, call = runs.calls[name]
    row = torch.empty(g.vert_count, dtype=torch.int32, device="cuda")
    own = torch.cuda.Stream()
    others = [torch.cuda.Stream() for _ in range(held)]
    call(expected[name][0][0], row, own)  # everything that is made on first use
    torch.cuda.synchronize()
    for s, exp in expected[name]:
        done = torch.cuda.Event()
        for o in others:
            with torch.cuda.stream(o):
                torch.cuda._sleep(100 * MS)
        call(s, row, own)
        done.record(own)
        done.synchronize()
        early = not all(o.query() for o in others)
        torch.cuda.synchronize()
        assert early, "the traversal ended after the kernels that held its SMs"
        np.testing.assert_array_equal(row.cpu().numpy(), exp)


@pytest.mark.parametrize("name", NAMES)
def test_sms_come_free_while_it_runs(runs, expected, name):
    import torch
    g, call = runs.calls[name]
    rng = np.random.RandomState(5)
    own = torch.cuda.Stream()
    others = [torch.cuda.Stream() for _ in range(60)]
    rows = [torch.empty(g.vert_count, dtype=torch.int32, device="cuda") for _ in expected[name]]
    for turn in range(12):
        for o in others[: rng.randint(1, 61)]:
            with torch.cuda.stream(o):
                torch.cuda._sleep(int(10 ** rng.uniform(3, 5.7)))
        for (s, _), row in zip(expected[name], rows):
            row.fill_(7)
            own.wait_stream(torch.cuda.current_stream())
            for o in others[: rng.randint(0, 30)]:
                with torch.cuda.stream(o):
                    torch.cuda._sleep(int(10 ** rng.uniform(3, 5.7)))
            call(s, row, own)
        torch.cuda.synchronize()
        for (_, exp), row in zip(expected[name], rows):
            np.testing.assert_array_equal(row.cpu().numpy(), exp)


@pytest.mark.parametrize("lead", [10, 62, 63, 64, 65, 66, 300])
def test_noalloc_goes_on_after_a_long_run_alone(eb, orc, lead):
    """Chains of levels of one vertex between levels that all CTAs share: the others have left, and come back."""
    import torch
    rng = np.random.RandomState(lead)
    widths = ([1] * lead + [3000, 40, 2000]) * 3 + [1] * lead + [1000]
    first = np.concatenate([[0], np.cumsum(widths)])
    u, v = [], []
    for k in range(1, len(widths)):
        n = widths[k] * (1 if widths[k] == 1 else 6)
        ids = np.repeat(np.arange(first[k], first[k + 1]), n // widths[k])
        u += [ids, [first[k]]]
        v += [first[k - 1] + rng.randint(0, widths[k - 1], n), [first[k - 1]]]
    csr = eb.Csr.from_edges(np.concatenate(u), np.concatenate(v), int(first[-1]) + 3)
    b, a = torch.from_numpy(csr.beg_pos).cuda(), torch.from_numpy(csr.csr).cuda()
    out = torch.full((csr.vert_count,), 7, dtype=torch.int32, device="cuda")
    for s in (0, int(first[lead]) + 5, int(first[-1]) - 1, csr.vert_count - 1):
        assert _noalloc(eb)(b.data_ptr(), a.data_ptr(), csr.vert_count, s, out.data_ptr(), None) == 0
        np.testing.assert_array_equal(out.cpu().numpy(), orc.bfs(csr.beg_pos, csr.csr, s)[0])


def test_noalloc_alone_leaves_the_gpu_to_others(eb):
    """A chain of 200000 vertices, half a second of one CTA: another stream's kernel ends long before."""
    import threading
    import time
    import torch
    n = 200_000
    csr = eb.Csr.from_edges(np.arange(n - 1), np.arange(1, n), n)
    beg, adj = csr.beg_pos, csr.csr
    b, a = torch.from_numpy(beg).cuda(), torch.from_numpy(adj).cuda()
    out = torch.empty(n, dtype=torch.int32, device="cuda")
    x = torch.zeros(1 << 20, device="cuda")
    own, other = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(other):
        x += 1
    torch.cuda.synchronize()
    status = []
    call = threading.Thread(target=lambda: status.append(_noalloc(eb)(b.data_ptr(), a.data_ptr(), n, 0, out.data_ptr(),
                                                                      C.c_void_p(own.cuda_stream))))
    call.start()
    time.sleep(0.05)
    with torch.cuda.stream(other):
        x += 1
    other.synchronize()
    running = call.is_alive()
    call.join()
    assert status == [0] and running
    np.testing.assert_array_equal(out.cpu().numpy(), np.arange(n, dtype=np.int32))
