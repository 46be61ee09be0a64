"""What a batch leaves behind for the next one on the same graph."""
import ctypes

import numpy as np
import pytest

import ascetic_gb300 as A
import oracle

pytestmark = pytest.mark.gpu


def _random_csr(V, ef, seed):
    rng = np.random.RandomState(seed)
    src = np.sort(rng.randint(0, V, V * ef))
    ptr = np.zeros(V + 1, np.uint64)
    ptr[1:] = np.cumsum(np.bincount(src, minlength=V))
    return ptr, rng.randint(0, V, V * ef).astype(np.uint32)


@pytest.mark.parametrize("frac", [1.0, 0.25])
@pytest.mark.parametrize("algo", ["bfs", "sssp"])
def test_capped_batch_leaves_nothing(algo, frac):
    """A batch stopped by its iteration cap drops its sources: the frontier they
    had does not go on in the next batch, under the sources that take their slots
    or beside them."""
    V = 5003
    ptr, col = _random_csr(V, 3, 5)
    edges = col
    if algo == "sssp":
        edges = np.stack([col, np.random.RandomState(6).randint(1, 64, len(col)).astype(np.uint32)], 1)
    ref = oracle.bfs if algo == "bfs" else oracle.sssp
    old = np.arange(64) * 70 + 3
    new = np.arange(64) * 71 + 9
    cap = A.make_params(max_iterations=2)
    with A.Graph.from_csr(ptr, edges, budget=A.make_budget(frac=frac)) as g:
        for first, then in ((64, 2), (3, 3), (40, 64), (64, 1)):
            with pytest.raises(A.AscError) as e:
                g.run_batch(algo, old[:first], params=cap)
            assert e.value.status == A.ERR_TIMEOUT
            for _ in range(2):
                got, st = g.run_batch(algo, new[:then])
                for row, s in zip(got, new):
                    assert np.array_equal(row, ref(ptr, edges, int(s))), (first, then, s)
                if then == 1:  # one source: every vertex it reaches is expanded, and no other
                    reached = got[0] < V + 1
                    deg = np.diff(ptr.astype(np.int64))
                    assert algo == "sssp" or st["edges_processed"] == deg[reached].sum()


@pytest.mark.parametrize("n", [5, 7, 30, 63])
def test_sssp_columns_without_a_source(n):
    """Distance columns that hold no source take no part in a batch, whatever the
    memory held before: with unit weights and every slot at one vertex, each
    reached list is read once. Columns that a cap left unfinished likewise."""
    torch = pytest.importorskip("torch")
    V = 100003
    ptr, col = _random_csr(V, 8, n)
    edges = np.stack([col, np.ones_like(col)], 1)
    exp = oracle.sssp(ptr, edges, 17)
    reads = np.diff(ptr.astype(np.int64))[exp < V + 1].sum()
    with A.Graph.from_csr(ptr, edges) as g:
        g.run("sssp", 17)  # the single-source state is not what takes the memory below
        # device memory full of small numbers, returned for the distance rows to take
        dirty = [torch.randint(1, 2 * V, (64 * V,), dtype=torch.int32, device="cuda") for _ in range(4)]
        torch.cuda.synchronize()
        del dirty
        torch.cuda.empty_cache()
        for _ in range(2):
            got, st = g.run_batch("sssp", [17] * n)
            assert all(np.array_equal(row, exp) for row in got)
            assert st["edges_processed"] == reads
        with pytest.raises(A.AscError):
            g.run_batch("sssp", np.arange(64) * 1500, params=A.make_params(max_iterations=2))
        got, st = g.run_batch("sssp", [17] * n)
        assert all(np.array_equal(row, exp) for row in got)
        assert st["edges_processed"] == reads


@pytest.mark.parametrize("algo", ["bfs", "sssp"])
def test_batch_after_a_failed_one(algo):
    """A batch that ran out of device memory, at its start or on the way, fails with
    a status; the next one starts anew, and writes the rows of its own sources only."""
    V = 5003
    ptr, col = _random_csr(V, 6, 8)
    edges = col
    if algo == "sssp":
        edges = np.stack([col, np.random.RandomState(6).randint(1, 64, len(col)).astype(np.uint32)], 1)
    ref = oracle.bfs if algo == "bfs" else oracle.sssp
    fail_after = A.lib().asc_test_fail_batch_alloc
    fail_after.argtypes, fail_after.restype = [ctypes.c_int], None
    src = np.arange(64) * 70 + 3
    failed = 0
    for after in list(range(0, 10)) + [40, 60, 68]:
        with A.Graph.from_csr(ptr, edges, budget=A.make_budget(frac=0.25)) as g:
            for _ in range(3):
                fail_after(after)
                try:
                    got, _ = g.run_batch(algo, src)
                    assert all(np.array_equal(got[i], ref(ptr, edges, int(src[i]))) for i in (0, 63))
                except A.AscError as e:
                    assert e.status == A.ERR_BUDGET, e
                    failed += 1
                finally:
                    fail_after(-1)
            buf = np.full((6, V), 0xdeadbeef, np.uint32)
            g.run_batch(algo, src[5:7], out=buf[2:4])
            assert np.array_equal(buf[2], ref(ptr, edges, int(src[5]))), after
            assert np.array_equal(buf[3], ref(ptr, edges, int(src[6]))), after
            assert (buf[:2] == 0xdeadbeef).all() and (buf[4:] == 0xdeadbeef).all(), after
    assert failed >= 5


@pytest.mark.parametrize("after", [7, 8])
def test_sssp_rows_without_copy_buffers(after):
    """Where the buffers that several columns leave through do not fit, columns leave
    one at a time: the batch still succeeds. The state's bytes are reported."""
    V = 3001
    ptr, col = _random_csr(V, 6, 8)
    edges = np.stack([col, np.random.RandomState(6).randint(1, 64, len(col)).astype(np.uint32)], 1)
    src = np.arange(64) * 40 + 3
    fail_after = A.lib().asc_test_fail_batch_alloc
    fail_after.argtypes, fail_after.restype = [ctypes.c_int], None
    with A.Graph.from_csr(ptr, edges) as g:
        exp = np.stack([g.run("sssp", int(s))[0] for s in src])
        before = g.refresh_info().device_vertex_bytes
        fail_after(after)  # the state is seven allocations
        try:
            got, _ = g.run_batch("sssp", src)
        finally:
            fail_after(-1)
        assert np.array_equal(got, exp)
        short = g.refresh_info().device_vertex_bytes
        assert short - before >= (256 + 28) * V
        got, _ = g.run_batch("sssp", src)
        assert np.array_equal(got, exp)
        assert g.refresh_info().device_vertex_bytes - short == 64 * V
