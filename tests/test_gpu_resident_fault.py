"""Failure detection of the traversals that run as cooperative kernels, without
a GPU fault: every wait between their CTAs is bounded. With the fault_inject
hook one CTA of the only kernel never arrives at a barrier, so the others'
waits run out; and in a traversal in parts one CTA of the head gives up just as
the head's last barrier opens for the others, which then finish the head. Both
must end with ENT_ERR_TIMEOUT, also right after a traversal that succeeded, and
the same handle must then run exact traversals again."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ENT_ERR_TIMEOUT = 6


@pytest.mark.parametrize("kind", ["one kernel", "in parts"])
def test_wait_runs_out_cleanly(eb, orc, kind):
    make = {"one kernel": lambda: eb.Graph.rmat(14, 16, seed=4321), "in parts": lambda: eb.Graph.er((1 << 22) + 37, 6, seed=0xA14)}
    with make[kind]() as g:
        csr = g.download()
        src = int(eb.pick_sources(csr.beg_pos, 4322, 1)[0])
        exp, _ = orc.bfs(csr.beg_pos, csr.csr, src)
        for _ in range(2):
            for fault in (0, 1):
                o = g.opts
                o.fault_inject = fault
                g.opts = o
                if fault:
                    t0 = time.time()
                    with pytest.raises(eb.EntError) as ei:
                        g.bfs(src)
                    assert ei.value.code == ENT_ERR_TIMEOUT, str(ei.value)
                    assert time.time() - t0 < 60
                else:
                    d, _, st = g.bfs(src)
                    np.testing.assert_array_equal(d, exp)
                    assert st.status == 0 and st.launches == (1 if kind == "one kernel" else 6)
