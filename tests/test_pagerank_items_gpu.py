"""Edge-balanced PageRank passes at the sizes where their items can go wrong.

An item is 2048 merge positions (rows plus edges): lists much longer than one
item, runs of empty rows longer than one, ends that fall on and around item,
warp (256 edges) and thread (8 edges) boundaries, single vertices, and splits
whose static region ends inside such a run.
"""
import numpy as np
import pytest

import ascetic_gb300 as A
import oracle

pytestmark = pytest.mark.gpu

# Tolerances against the serial FP64 oracle. FP64: its own row sums are up to
# 9,000 serial additions (9,000 x 2^-53 = 1e-12 relative), amplified by at most
# 1 / (1 - 0.85) over the passes. FP32 contributions: 2^-24 each plus 8 additions
# in FP32 (5e-7), amplified likewise.
TOL = {A.F64: 1e-11, A.F32: 1e-5}

SHAPES = {
    "one_vertex": [0],
    "one_loop": [1],
    "one_long_row": [0] * 70 + [9000] + [0] * 3,
    "empty_runs": [3] + [0] * 5000 + [7] + [0] * 2047 + [1] + [0] * 2048 + [2],
    "ends_on_boundaries": [8, 248, 256, 0, 512, 1023, 2048, 2047, 2049, 1, 0, 7, 9, 4096],
    "ramp": list(range(0, 300)),
    "short": [0, 1, 2, 3, 4, 5, 6, 7, 8, 9] * 900,
    "exact_item": [1] * 1024,
}


@pytest.mark.parametrize("layout", ["csc", "csr", "csr_w63", "csr_w99999"])
@pytest.mark.parametrize("frac", [1.0, 0.4, 0.0])
@pytest.mark.parametrize("shape", sorted(SHAPES))
def test_items(shape, frac, layout):
    deg = np.array(SHAPES[shape], np.int64)
    V, E = len(deg), int(deg.sum())
    ptr = np.zeros(V + 1, np.uint64)
    ptr[1:] = np.cumsum(deg)
    rng = np.random.RandomState(7)
    # half of the entries name one of three vertices: hot destinations of a scatter
    other = np.where(rng.rand(E) < 0.5, rng.randint(0, min(V, 3), E), rng.randint(0, V, E)).astype(np.uint32)
    rows = np.repeat(np.arange(V, dtype=np.uint32), deg)
    if layout == "csc":
        cptr, ccol = ptr, other
        od = np.bincount(other, minlength=V).astype(np.uint32)
    else:  # the same lists as out-edges; the oracle takes in-edges
        order = np.argsort(other, kind="stable")
        cptr = np.zeros(V + 1, np.uint64)
        cptr[1:] = np.cumsum(np.bincount(other, minlength=V))
        ccol, od = rows[order], deg.astype(np.uint32)
    exp, _, _ = oracle.pr_std(cptr, ccol, od)
    ref, _ = oracle.pr_ref(cptr, ccol, od)
    budget = A.make_budget(frac=frac, fragment_edges=16)
    kw = {"outdeg": od} if layout == "csc" else {}
    edges = other
    if "_w" in layout:  # packed with the destination, or beside it
        edges = np.stack([other, rng.randint(1, int(layout[5:]) + 1, E).astype(np.uint32)], 1)
    with A.Graph.from_csr(ptr, edges, budget=budget, **kw) as g:
        for prec in (A.F64, A.F32, A.F64):
            got, st = g.run("pr", params=A.make_params(pr_mode=A.PR_STD, precision=prec))
            err = np.abs(got.astype(np.float64) - exp) / exp
            assert err.max() <= TOL[prec], (prec, err.max())
            assert st["edges_processed"] == E * st["iterations"]
            assert st["frontier_vertices"] == V * st["iterations"]
        got, _ = g.run("pr")
        assert np.abs(got - ref).max() <= 1e-6
