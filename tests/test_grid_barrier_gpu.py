"""The wait of the persistent loop's grid barrier, when it runs out."""
import ctypes

import numpy as np
import pytest

import ascetic_gb300 as A
import oracle

pytestmark = pytest.mark.gpu


def test_barrier_gives_up():
    """A grid barrier whose wait runs out ends the launch with a status; the next run
    starts anew. No poll beyond the first: every CTA but the last to arrive leaves."""
    polls = A.lib().asc_test_barrier_polls
    polls.argtypes, polls.restype = [ctypes.c_uint32], None
    V, ef = 70001, 12
    rng = np.random.RandomState(1)
    src = np.sort(rng.randint(0, V, V * ef))
    ptr = np.zeros(V + 1, np.uint64)
    ptr[1:] = np.cumsum(np.bincount(src, minlength=V))
    col = rng.randint(0, V, V * ef).astype(np.uint32)
    w = np.stack([col, rng.randint(1, 64, len(col)).astype(np.uint32)], 1)
    expect = {"bfs": oracle.bfs(ptr, col, 5), "sssp": oracle.sssp(ptr, w, 5), "cc": oracle.cc(ptr, col)}
    with A.Graph.from_csr(ptr, w, budget=A.make_budget(frac=0.3)) as g:
        for algo in expect:
            for _ in range(2):
                polls(0)
                try:
                    with pytest.raises(A.AscError) as e:
                        g.run(algo, 5)
                    assert e.value.status == A.ERR_TIMEOUT and "barrier" in str(e.value)
                finally:
                    polls(1 << 25)
                assert np.array_equal(g.run(algo, 5)[0], expect[algo])
