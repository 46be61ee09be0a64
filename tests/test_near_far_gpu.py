"""SSSP with a near-far step under every way the iterations can be driven."""
import numpy as np
import pytest

import ascetic_gb300 as A
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("delta", [1, 16, 1000])
@pytest.mark.parametrize("flags", ["none", "host_loop", "phase_timing", "fragment_counts", "gather_copy",
                                   "partition_copy"])
@pytest.mark.parametrize("frac", [0.2, 0.1])
def test_near_far(frac, flags, delta):
    """The far set is worked off to the end: distances equal the oracle's."""
    ptr, adj = A.rmat_csr(12, 16, 91, weights=(1, 63))
    flag = 0 if flags == "none" else getattr(A, "RUN_" + flags.upper())
    # two staging buffers of 16 KiB for the partition copies, out of the byte budget
    budget = A.make_budget(frac=frac, stage_bytes=32 << 10)
    with A.Graph.from_csr(ptr, adj, budget=budget) as g:
        g.set_tuning(delta=delta)
        for s in (0, 321):
            got, _ = g.run("sssp", s, params=A.make_params(flags=flag))
            assert np.array_equal(got, oracle.sssp(ptr, adj, s)), s
