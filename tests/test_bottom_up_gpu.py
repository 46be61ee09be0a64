"""Bottom-up BFS steps over in-edges in host memory and on the device, at the widths,
list ends and numbers of waiting vertices where their reads can go wrong. Levels are
whole numbers: compared bit for bit with the oracle."""
import numpy as np
import pytest

import ascetic_gb300 as A
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("packing", ["1", "0"])
@pytest.mark.parametrize("V", [2, 3, 17, 33, 300, 5000, 65537])
@pytest.mark.parametrize("frac", [1.0, 0.3, 0.0])
def test_in_lists(V, frac, packing, monkeypatch):
    """Widths of 1 to 17 and of 32 bits. In-lists of 0 to 40 entries, so that words of
    32 vertices hold from none to 32 that scan on; the last list ends with the array."""
    monkeypatch.setenv("ASC_EDGE_PACKING", packing)
    rng = np.random.RandomState(V)
    for shape in ("even", "some", "last"):
        indeg = {"even": np.full(V, 9), "some": rng.randint(0, 41, V) * (rng.rand(V) < 0.6),
                 "last": np.where(np.arange(V) >= V - 3, 40, rng.randint(0, 3, V))}[shape]
        dst = np.repeat(np.arange(V), indeg)
        src = rng.randint(0, V, len(dst))
        if not len(dst):
            continue
        order = np.argsort(src, kind="stable")
        ptr = np.zeros(V + 1, np.uint64)
        ptr[1:] = np.cumsum(np.bincount(src, minlength=V))
        col = dst[order].astype(np.uint32)
        with A.Graph.from_csr(ptr, col, budget=A.make_budget(frac=frac, fragment_edges=16)) as g:
            for bu_div in (0x7fffffff, 8):  # every step, and steps of large frontiers
                g.set_tuning(bu_div=bu_div)
                for s in {0, int(src[0]), V - 1}:
                    exp = oracle.bfs(ptr, col, s)
                    for p in (None, A.make_params(flags=A.RUN_HOST_LOOP)):
                        got, st = g.run("bfs", s, params=p)
                        assert np.array_equal(got, exp), (shape, bu_div, s)
                        assert st["reached_vertices"] == (exp < V + 1).sum()
