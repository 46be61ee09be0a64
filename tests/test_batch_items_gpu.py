"""Batched BFS and staged PageRank over merge items at the sizes where they can go
wrong: lists and runs of empty rows longer than an item, ends on item, warp and thread
boundaries, splits inside them, every stored edge width, and items shortened to fit a
small staging buffer."""
import numpy as np
import pytest

import ascetic_gb300 as A
import oracle

pytestmark = pytest.mark.gpu

SHAPES = {
    "one_vertex": [0],
    "one_loop": [1],
    "one_long_row": [1] * 70 + [9000] + [0] * 3,
    "empty_runs": [3] + [0] * 5000 + [7] + [0] * 2047 + [1] + [0] * 2048 + [2],
    "ends_on_boundaries": [8, 248, 256, 0, 512, 1023, 2048, 2047, 2049, 1, 0, 7, 9, 4096],
    "ramp": list(range(0, 300)),
    "short": [0, 1, 2, 3, 4, 5, 6, 7, 8, 9] * 900,
    "exact_item": [1] * 1024,
    "hubs": ([4000] + [2] * 700) * 4,
}
# serial FP64 sums of up to 9,000 terms, amplified by at most 1 / (1 - 0.85); FP32
# contributions: 2^-24 each plus 8 additions in FP32, amplified likewise
TOL = {A.F64: 1e-11, A.F32: 1e-5}


def _graph(shape):
    deg = np.array(SHAPES[shape], np.int64)
    V, E = len(deg), int(deg.sum())
    ptr = np.zeros(V + 1, np.uint64)
    ptr[1:] = np.cumsum(deg)
    rng = np.random.RandomState(13)
    return ptr, rng.randint(0, V, E).astype(np.uint32), rng, V, E


@pytest.mark.parametrize("frac", [1.0, 0.4, 0.0])
@pytest.mark.parametrize("shape", sorted(SHAPES))
def test_batched_bfs(shape, frac):
    ptr, dst, rng, V, E = _graph(shape)
    srcs = np.concatenate([[0, int(np.argmax(np.diff(ptr))), V - 1], rng.randint(0, V, 61)])
    exp = {int(s): oracle.bfs(ptr, dst, int(s)) for s in srcs}
    for maxw in (0, 63, 90000000):  # bit stream, packed beside the weight, {dst, weight}
        edges = dst
        if maxw:
            edges = np.stack([dst, rng.randint(1, maxw + 1, E).astype(np.uint32)], 1)
        with A.Graph.from_csr(ptr, edges, budget=A.make_budget(frac=frac, fragment_edges=16)) as g:
            for n in (64, 3, 64):
                rows, _ = g.run_batch("bfs", srcs[:n])
                for row, s in zip(rows, srcs):
                    assert np.array_equal(row, exp[int(s)]), (maxw, n, s)


@pytest.mark.parametrize("layout", ["csc", "csr", "csr_w90000000"])
@pytest.mark.parametrize("shape", ["one_long_row", "ends_on_boundaries", "ramp", "hubs"])
def test_short_items(shape, layout, monkeypatch):
    """Two staging buffers of 4 KiB hold items of 512 or 256 positions (of 32 and 64
    bits an edge) in place of 2048: staged passes, and traversals over those items."""
    monkeypatch.setenv("ASC_EDGE_PACKING", "0")
    ptr, other, rng, V, E = _graph(shape)
    rows = np.repeat(np.arange(V, dtype=np.uint32), np.diff(ptr).astype(np.int64))
    budget = A.make_budget(nbytes=8192, stage_bytes=8192, fragment_edges=16)
    if layout == "csc":
        cptr, ccol, od = ptr, other, np.bincount(other, minlength=V).astype(np.uint32)
        args, kw = (ptr, other), {"outdeg": od}
    else:
        order = np.argsort(other, kind="stable")
        cptr = np.zeros(V + 1, np.uint64)
        cptr[1:] = np.cumsum(np.bincount(other, minlength=V))
        ccol, od = rows[order], np.diff(ptr).astype(np.uint32)
        edges = other
        if "_w" in layout:
            edges = np.stack([other, rng.randint(1, 90000000, E).astype(np.uint32)], 1)
        args, kw = (ptr, edges), {}
    exp, _, _ = oracle.pr_std(cptr, ccol, od)
    with A.Graph.from_csr(*args, budget=budget, **kw) as g:
        assert g.info.staging_bytes == 8192
        for prec in (A.F64, A.F32):
            got, st = g.run("pr", params=A.make_params(pr_mode=A.PR_STD, precision=prec))
            assert st["staged_chunks"] >= 2 * st["iterations"]
            err = np.abs(got.astype(np.float64) - exp) / exp
            assert err.max() <= TOL[prec], (prec, err.max())
        if layout == "csc":
            return
        g.set_tuning(dense_div=0xffffffff, bu_div=0)
        src = int(np.argmax(np.diff(ptr)))
        assert np.array_equal(g.run("bfs", src)[0], oracle.bfs(ptr, other, src))
        assert np.array_equal(g.run("cc")[0], oracle.cc(ptr, other))
        if "_w" in layout:
            assert np.array_equal(g.run("sssp", src)[0], oracle.sssp(*args, src))
