"""The persistent traversal loop and its merge items at the sizes where they can
go wrong: lists and runs of empty rows longer than an item (2048 rows plus
edges), ends on item, warp (256 edges) and thread (8 edges) boundaries, splits
inside them, every stored edge width, frontiers walked only through items, only
through lists and as chosen, with and without the near-far thresholds. Values
are whole numbers: compared bit for bit with the oracle and the host-driven loop.
"""
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
}


@pytest.mark.parametrize("walk", ["items", "lists", "default"])
@pytest.mark.parametrize("frac", [1.0, 0.4, 0.0])
@pytest.mark.parametrize("shape", sorted(SHAPES))
def test_loop(shape, frac, walk):
    deg = np.array(SHAPES[shape], np.int64)
    V, E = len(deg), int(deg.sum())
    ptr = np.zeros(V + 1, np.uint64)
    ptr[1:] = np.cumsum(deg)
    rng = np.random.RandomState(11)
    # few-vertex graphs reach everything; "short" and "empty_runs" need several iterations
    dst = rng.randint(0, V, E).astype(np.uint32)
    srcs = sorted({0, int(np.argmax(deg)), V - 1})
    for maxw in (0, 63, 99999):
        edges = dst
        if maxw:
            edges = np.stack([dst, rng.randint(1, maxw + 1, E).astype(np.uint32)], 1)
        with A.Graph.from_csr(ptr, edges, budget=A.make_budget(frac=frac, fragment_edges=16)) as g:
            for delta in (0, 16) if maxw else (0,):
                g.set_tuning(dense_div={"items": 0xffffffff, "lists": 0, "default": 64}[walk], delta=delta,
                             bu_div=0 if walk == "items" else 64)
                for s in srcs:
                    exp = oracle.bfs(ptr, dst, s)
                    got, st = g.run("bfs", s)
                    assert np.array_equal(got, exp), (maxw, s)
                    reached = exp < V + 1
                    assert st["reached_vertices"] == reached.sum() and st["reached_edges"] == deg[reached].sum()
                    if maxw:
                        exp = oracle.sssp(ptr, edges, s)
                        got, st = g.run("sssp", s)
                        assert np.array_equal(got, exp), (maxw, s, delta)
                        assert st["reached_edges"] == deg[exp < V + 1].sum()
                got, st = g.run("cc")
                assert np.array_equal(got, oracle.cc(ptr, dst)), maxw
                host, _ = g.run("cc", params=A.make_params(flags=A.RUN_HOST_LOOP))
                assert np.array_equal(got, host)


def test_iteration_cap():
    """A path needs as many iterations as it has vertices; a lower cap is a timeout."""
    V = 100
    ptr = np.minimum(np.arange(V + 1), V - 1).astype(np.uint64)
    col = np.arange(1, V, dtype=np.uint32)
    with A.Graph.from_csr(ptr, col) as g:
        for algo in ("bfs", "cc"):
            got, st = g.run(algo, 0, params=A.make_params(max_iterations=V))
            assert st["iterations"] <= V
            with pytest.raises(A.AscError) as e:
                g.run(algo, 0, params=A.make_params(max_iterations=V // 2))
            assert e.value.status == A.ERR_TIMEOUT
            assert np.array_equal(g.run(algo, 0)[0], got)


@pytest.mark.parametrize("V,ef", [(64, 3), (2045, 5), (2048, 16), (3001, 1), (5000, 40), (70001, 12)])
@pytest.mark.parametrize("frac", [1.0, 0.3, 0.0])
def test_in_edges(V, ef, frac):
    """In-edges built on the device (in several runs of lists, V entries each) and,
    where a list is longer than V or the degree above 64, on the host: bottom-up
    steps from the first iteration on give the oracle's levels."""
    rng = np.random.RandomState(V)
    for hub in (False, True):
        src = rng.randint(0, V, V * ef)
        dst = np.minimum(rng.randint(0, V, V * ef), rng.randint(0, V, V * ef))
        if hub:  # one in-list longer than V
            dst[: 2 * V] = 7
        order = np.argsort(src, kind="stable")
        ptr = np.zeros(V + 1, np.uint64)
        ptr[1:] = np.cumsum(np.bincount(src, minlength=V))
        col = dst[order].astype(np.uint32)
        for edges in (col, np.stack([col, rng.randint(1, 64, len(col)).astype(np.uint32)], 1)):
            with A.Graph.from_csr(ptr, edges, budget=A.make_budget(frac=frac, fragment_edges=64)) as g:
                g.set_tuning(bu_div=0x7fffffff)  # every step bottom-up
                for s in (int(src[0]), V - 1):
                    got, st = g.run("bfs", s)
                    assert np.array_equal(got, oracle.bfs(ptr, col, s)), (hub, s)
                    host, _ = g.run("bfs", s, params=A.make_params(flags=A.RUN_HOST_LOOP))
                    assert np.array_equal(got, host)


def test_concurrent_graphs():
    """Threads with a graph each: their persistent loops fill the GPU one after the other."""
    import threading

    sizes = [(65536, 16), (1001, 8), (200000, 8), (65536, 16)]
    graphs, expect, failed = [], [], []
    for k, (V, ef) in enumerate(sizes):
        rng = np.random.RandomState(k)
        src = np.sort((V * rng.rand(V * ef) ** 2).astype(np.int64))
        col = (V * rng.rand(V * ef) ** 2).astype(np.uint32)
        ptr = np.zeros(V + 1, np.uint64)
        ptr[1:] = np.cumsum(np.bincount(src, minlength=V))
        w = np.stack([col, rng.randint(1, 64, len(col)).astype(np.uint32)], 1)
        graphs.append(A.Graph.from_csr(ptr, w, budget=A.make_budget(frac=0.3)))
        expect.append({"bfs": oracle.bfs(ptr, col, 0), "sssp": oracle.sssp(ptr, w, 0), "cc": oracle.cc(ptr, col)})

    def work(k):
        try:
            for i in range(20):
                algo = ("bfs", "sssp", "cc")[(i + k) % 3]
                got, _ = graphs[k].run(algo, 0)
                if not np.array_equal(got, expect[k][algo]):
                    failed.append((k, i, algo, "values"))
        except Exception as e:  # reported below: a thread's exception fails no test by itself
            failed.append((k, repr(e)))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(sizes))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for g in graphs:
        g.close()
    assert not failed, failed
