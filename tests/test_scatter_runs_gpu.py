"""PageRank by scatter where consecutive edges go to one destination: runs that end
inside a thread's 8 edges, at its ends and at those of rows, warps and items, to
frequent destinations and to rare ones."""
import numpy as np
import pytest

import ascetic_gb300 as A
import oracle

pytestmark = pytest.mark.gpu

# serial FP64 sums of up to 12,000 terms, amplified by at most 1 / (1 - 0.85); FP32
# contributions: 2^-24 each, added exactly, amplified likewise
TOL = {A.F64: 1e-11, A.F32: 1e-5}


def _lists(name):
    rng = np.random.RandomState(2)
    if name == "leaves":  # each vertex one edge, thousands in a row to one hub
        return [[10 + v // 4000] for v in range(12000)] + [[0, 0, 1]]
    if name == "runs":  # runs of 1 to 20 in lists of any length
        return [list(np.repeat(rng.randint(0, 700, n), rng.randint(1, 21, n))) for n in rng.randint(0, 60, 700)]
    if name == "rows":  # a run goes on from row to row with another contribution
        return [[v // 100] * (1 + v % 9) for v in range(3000)]
    return [[(v + k) % 2000 for k in range(40)] for v in range(2000)]  # no run at all


@pytest.mark.parametrize("frac", [1.0, 0.3])
@pytest.mark.parametrize("name", ["leaves", "runs", "rows", "none"])
def test_runs(name, frac):
    lists = _lists(name)
    V = len(lists)
    deg = np.array([len(x) for x in lists])
    ptr = np.zeros(V + 1, np.uint64)
    ptr[1:] = np.cumsum(deg)
    dst = np.concatenate([np.array(x, np.uint32) for x in lists if len(x)])
    order = np.argsort(dst, kind="stable")
    cptr = np.zeros(V + 1, np.uint64)
    cptr[1:] = np.cumsum(np.bincount(dst, minlength=V))
    ccol = np.repeat(np.arange(V, dtype=np.uint32), deg)[order]
    od = deg.astype(np.uint32)
    exp, _, _ = oracle.pr_std(cptr, ccol, od)
    ref, _ = oracle.pr_ref(cptr, ccol, od)
    for edges in (dst, np.stack([dst, 1 + dst % 63], 1)):
        with A.Graph.from_csr(ptr, edges, budget=A.make_budget(frac=frac, fragment_edges=16)) as g:
            for prec in (A.F64, A.F32):
                got, _ = g.run("pr", params=A.make_params(pr_mode=A.PR_STD, precision=prec))
                err = np.abs(got.astype(np.float64) - exp) / exp
                assert err.max() <= TOL[prec], (prec, err.max())
            got, _ = g.run("pr")
            assert np.abs(got - ref).max() <= 1e-6 * max(1.0, np.abs(ref).max())
