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
