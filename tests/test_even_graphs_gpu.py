"""Traversals of graphs with even degrees and of graphs along a thread: where dense
frontiers go by tiles until they are large, and connected components by more than the
first label early. Values are whole numbers: compared bit for bit with the oracle and
the host-driven loop."""
import numpy as np
import pytest

import ascetic_gb300 as A
import oracle

pytestmark = pytest.mark.gpu


def _csr(src, dst, V):
    order = np.argsort(src, kind="stable")
    ptr = np.zeros(V + 1, np.uint64)
    ptr[1:] = np.cumsum(np.bincount(src, minlength=V))
    return ptr, dst[order].astype(np.uint32)


def _check(ptr, col, sources, frac):
    V, E = len(ptr) - 1, len(col)
    w = np.stack([col, np.random.RandomState(3).randint(1, 64, E).astype(np.uint32)], 1)
    wide = w.copy()
    wide[:, 1] *= 1000000  # beside the destination, not packed with it
    host = A.make_params(flags=A.RUN_HOST_LOOP)
    for edges in (col, w, wide):
        with A.Graph.from_csr(ptr, edges, budget=A.make_budget(frac=frac, fragment_edges=16)) as g:
            for dense_div in (64, 0xffffffff):
                g.set_tuning(dense_div=dense_div, bu_div=0)
                for s in sources:
                    exp = oracle.bfs(ptr, col, s)
                    for p in (None, host):
                        got, st = g.run("bfs", s, params=p)
                        assert np.array_equal(got, exp), (s, dense_div)
                        assert st["edges_processed"] == np.diff(ptr.astype(np.int64))[exp < V + 1].sum()
                        if edges is not col:
                            assert np.array_equal(g.run("sssp", s, params=p)[0], oracle.sssp(ptr, edges, s))
                exp = oracle.cc(ptr, col)
                for p in (None, host):
                    assert np.array_equal(g.run("cc", params=p)[0], exp), dense_div
            rows, _ = g.run_batch("bfs", sources * 8)
            assert all(np.array_equal(r, oracle.bfs(ptr, col, s)) for r, s in zip(rows, sources * 8))


@pytest.mark.parametrize("V", [255, 257, 4097, 30011])
@pytest.mark.parametrize("ef", [2, 4, 16])
@pytest.mark.parametrize("frac", [1.0, 0.4])
def test_uniform(V, ef, frac):
    """Mean degrees on each side of the rule's lines (3 and 8 edges per vertex)."""
    rng = np.random.RandomState(V + ef)
    s, d = rng.randint(0, V, V * ef // 2), rng.randint(0, V, V * ef // 2)
    ptr, col = _csr(np.concatenate([s, d]), np.concatenate([d, s]), V)
    _check(ptr, col, [0, V // 2, V - 1], frac)


def _links(pairs):
    a, b = np.array(pairs).T
    return np.concatenate([a, b]), np.concatenate([b, a])


@pytest.mark.parametrize("frac", [1.0, 0.4])
@pytest.mark.parametrize("name", ["path", "rings", "grid", "spider3", "spider4", "pairs", "late"])
def test_threads(name, frac):
    V = 700
    v = np.arange(V - 1)
    if name == "path":
        pairs = list(zip(v, v + 1))
    elif name == "rings":
        pairs = [(i, i - i % 7 + (i + 1) % 7) for i in range(V)]
    elif name == "grid":
        pairs = [(i, i + 1) for i in range(V - 1) if i % 25 != 24] + [(i, i + 25) for i in range(V - 25)]
    elif name.startswith("spider"):  # the first vertex's second iteration reaches 3 or 4 vertices
        legs = int(name[6:])
        pairs = [(0, 1 + k) for k in range(legs)] + [(i, i + legs) for i in range(1, V - legs)]
    elif name == "pairs":
        pairs = [(i, i + 1) for i in range(0, V, 2)]
    else:  # the first label runs along a thread into a dense part
        pairs = [(i, i + 1) for i in range(40)] + [(40 + i % 60, 100 + i % 600) for i in range(6000)]
    src, dst = _links(pairs)
    ptr, col = _csr(src, dst, V)
    _check(ptr, col, [0, V // 2], frac)
