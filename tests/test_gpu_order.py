"""GPU tests of the order between calls that share memory: a plan's seed list
and the kernels that read it, and asynchronous runs of one handle on several
streams. Depths equal the oracle's whatever else the GPU is doing."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_plan_seeds_land_before_they_are_read(eb, orc):
    """A plan made while long copies wait on the legacy stream, its seed list in
    memory that the plan before gave back (so a list that has not landed is the
    other plan's)."""
    import torch
    csrs = [eb.Csr.rmat(12, 8, seed=0xB1), eb.Csr.er(3001, 9.0, seed=0xB2)]
    src = torch.empty(64 << 20, dtype=torch.uint8, pin_memory=True)
    dst = torch.empty(64 << 20, dtype=torch.uint8, device="cuda")
    lists = [[eb.pick_sources(c.beg_pos, 40 + 7 * turn + k, 5 + k) for k, c in enumerate(csrs)] for turn in range(3)]
    exp = [[[orc.bfs(c.beg_pos, c.csr, int(s))[0] for s in ss] for c, ss in zip(csrs, turn)] for turn in lists]
    with eb.Graph.from_csr(csrs[0]) as a, eb.Graph.from_csr(csrs[1]) as b:
        torch.cuda.synchronize()
        for turn, ss in enumerate(lists):
            for _ in range(6):
                dst.copy_(src, non_blocking=True)  # torch's default stream is the legacy one
            with eb.MultiPlan([a, b], ss) as plan:
                plan.run()
                for k in range(2):
                    np.testing.assert_array_equal(plan.depths(k), np.stack(exp[turn][k]))


@pytest.mark.parametrize("bytes_", [False, True])
def test_batches_on_streams_in_turn(eb, orc, bytes_):
    """Asynchronous batches of one handle on two streams, of other sources and
    another number of them each, keep their order: each writes its own rows."""
    import torch
    csr = eb.Csr.rmat(14, 16, seed=0xB3)
    lists = [eb.pick_sources(csr.beg_pos, 50 + i, 60 + 3 * i) for i in range(8)]
    with eb.Graph.from_csr(csr) as g:
        call = g.bfs_batch_device_u8 if bytes_ else g.bfs_batch_device
        rows = [torch.full((len(ss), csr.vert_count), 7, dtype=torch.uint8 if bytes_ else torch.int32, device="cuda")
                for ss in lists]
        streams = [torch.cuda.Stream(), torch.cuda.Stream()]
        call(lists[-1], rows[-1].data_ptr())  # the workspace is as wide as the widest batch from here on
        torch.cuda.synchronize()
        for i, ss in enumerate(lists):
            call(ss, rows[i].data_ptr(), stream=streams[i % 2].cuda_stream, stats=False)
        torch.cuda.synchronize()
        for ss, r in zip(lists, rows):
            got = r.cpu().numpy()
            for s, d in zip(ss, got):
                exp = orc.bfs(csr.beg_pos, csr.csr, int(s))[0]
                np.testing.assert_array_equal(d, np.where(exp < 0, 255, exp).astype(np.uint8) if bytes_ else exp)


def test_batch_trace_after_an_asynchronous_batch(eb, orc):
    import torch
    csr = eb.Csr.rmat(16, 16, seed=0xB4)
    ss, st = eb.pick_sources(csr.beg_pos, 60, 128), eb.pick_sources(csr.beg_pos, 61, 70)
    with eb.Graph.from_csr(csr) as g:
        rows = torch.full((len(ss), csr.vert_count), 7, dtype=torch.int32, device="cuda")
        traced = torch.full((len(st), csr.vert_count), 7, dtype=torch.int32, device="cuda")
        stream = torch.cuda.Stream()
        g.bfs_batch_device(ss, rows.data_ptr())
        torch.cuda.synchronize()
        for _ in range(4):
            g.bfs_batch_device(ss, rows.data_ptr(), stream=stream.cuda_stream, stats=False)
        g.trace_batch(st, traced.data_ptr())
        torch.cuda.synchronize()
        for got, src in ((rows, ss), (traced, st)):
            got = got.cpu().numpy()
            for s, d in zip(src, got):
                np.testing.assert_array_equal(d, orc.bfs(csr.beg_pos, csr.csr, int(s))[0])


@pytest.mark.parametrize("loop", ["graph", "host"])
def test_trace_after_an_asynchronous_traversal(eb, orc, loop):
    import torch
    csr = eb.Csr.rmat(18, 16, seed=0xB5)
    a, b = (int(s) for s in eb.pick_sources(csr.beg_pos, 62, 2))
    with eb.Graph.from_csr(csr) as g:
        o = g.opts
        o.loop = eb.LOOP[loop]
        g.opts = o
        row = torch.full((csr.vert_count,), 7, dtype=torch.int32, device="cuda")
        stream = torch.cuda.Stream()
        g.bfs_device(a, row.data_ptr())
        torch.cuda.synchronize()
        for _ in range(8):
            g.bfs_device(a, row.data_ptr(), stream=stream.cuda_stream, stats=False)
        levels, st = g.trace(b)
        torch.cuda.synchronize()
        np.testing.assert_array_equal(row.cpu().numpy(), orc.bfs(csr.beg_pos, csr.csr, a)[0])
        exp = orc.bfs(csr.beg_pos, csr.csr, b)[0]
        assert (st.traversed_edges, st.reached_vertices) == orc.report(csr.beg_pos, exp) and st.levels == exp.max() + 1
        assert sum(r["frontier_vertices"] for r in levels) <= st.reached_vertices
