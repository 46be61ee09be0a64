"""Measured cases: the calls a user of the engine makes, over the sizes it is used at.

Graphs are RMAT graphs (a = .57, b = .19, c = .19), as in the tests and the benchmark, drawn
on the GPU from the seed and handed to the engine as host CSR/CSC arrays, which is how a
program that has a graph in memory opens it. Vertex counts need not be powers of two (ids
are folded into the range), lists keep the order in which their edges were drawn, self-loops
and duplicates stay. Results come back in host memory: into a page-locked buffer that the
program keeps, or (the small calls) into a fresh array from the call itself.
"""
import numpy as np
import torch

import ascetic_gb300 as A

DEV = "cuda"


def listed():
    return [
        # The smallest call: BFS on a graph of a thousand vertices held whole on the device, where
        # only launches and the host path count. Odd vertex count.
        {"name": "bfs_1k", "call": "bfs", "V": 1001, "ef": 8, "maxw": 0, "frac": 1.0, "out": "fresh"},
        # Plain BFS at RMAT scale 16, edge factor 16, no cap: the reference's ordinary small graph.
        {"name": "bfs_s16", "call": "bfs", "V": 1 << 16, "ef": 16, "maxw": 0, "frac": 1.0, "out": "fresh"},
        # The headline configuration: BFS at RMAT scale 24, edge factor 16, static region at 25%.
        {"name": "bfs_s24", "call": "bfs", "V": 1 << 24, "ef": 16, "maxw": 0, "frac": 0.25, "out": "pinned"},
        # SSSP, weights 1..63 (packed edge words), the out-of-memory configuration at 25%.
        {"name": "sssp_s23", "call": "sssp", "V": 1 << 23, "ef": 16, "maxw": 63, "frac": 0.25, "out": "pinned"},
        # Connected components of a symmetrised graph of ragged size under the same cap.
        {"name": "cc_6m", "call": "cc", "V": 6000011, "ef": 15, "maxw": 0, "frac": 0.25, "sym": True,
         "out": "pinned"},
        # Standard PageRank over in-edges to the 1e-9 residual, FP32 contributions, 30% (the precision study).
        {"name": "pr_f32_s24", "call": "pr", "V": 1 << 24, "ef": 16, "layout": "csc", "mode": "std",
         "prec": "f32", "frac": 0.3, "out": "pinned"},
        # The same in FP64 on a graph of ragged size.
        {"name": "pr_f64_1m5", "call": "pr", "V": 1500007, "ef": 17, "layout": "csc", "mode": "std",
         "prec": "f64", "frac": 0.3, "out": "pinned"},
        # The reference's own PageRank (ptgraph --type pr): per-vertex stop at 0.001.
        {"name": "pr_ref_s20", "call": "pr", "V": 1 << 20, "ef": 16, "layout": "csc", "mode": "ref",
         "prec": "f64", "frac": 0.3, "out": "fresh"},
        # PageRank on a graph stored by out-edges (scatter).
        {"name": "pr_push_1m", "call": "pr", "V": 1000003, "ef": 16, "layout": "csr", "mode": "std",
         "prec": "f32", "frac": 0.5, "out": "pinned"},
        # 64 BFS sources in one batch, as the batched configuration and the query server run them.
        {"name": "batch_bfs_s21", "call": "batch_bfs", "V": 1 << 21, "ef": 16, "maxw": 0, "frac": 0.25,
         "n": 64, "out": "pinned"},
        # 64 SSSP sources in one batch.
        {"name": "batch_sssp_s20", "call": "batch_sssp", "V": 1 << 20, "ef": 16, "maxw": 63, "frac": 0.25,
         "n": 64, "out": "pinned"},
        # A burst of queries (50% BFS, 30% SSSP, 10% CC, 10% PageRank) to the server over two
        # resident graphs.
        {"name": "serve_48", "call": "serve", "V": 1 << 17, "ef": 16, "maxw": 63, "frac": 0.25, "n": 48,
         "out": "fresh"},
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    call = rng.choice(["bfs", "bfs", "bfs", "sssp", "sssp", "cc", "cc", "pr", "pr", "pr", "batch_bfs",
                       "batch_sssp", "serve"])
    top = {"bfs": 1 << 23, "sssp": 1 << 23, "cc": 6 << 20, "pr": 1 << 23, "batch_bfs": 1 << 21,
           "batch_sssp": 1 << 20, "serve": 1 << 17}[call]
    V = _log_int(rng, 1000, top)
    c = {"call": call, "V": V, "ef": rng.randint(4, 16), "frac": rng.choice([1.0, 0.5, 0.3, 0.25, 0.1]),
         "out": "pinned" if V > 200000 else "fresh"}
    if call == "pr":
        c["layout"] = rng.choice(["csc", "csc", "csr"])
        c["mode"] = rng.choice(["std", "std", "ref"])
        c["prec"] = "f64" if c["mode"] == "ref" else rng.choice(["f32", "f64"])
        return c
    # weights up to 63 are packed with the destination, up to 99,999 are stored beside it
    c["maxw"] = 0
    if call in ("sssp", "batch_sssp", "serve"):
        c["maxw"] = rng.choice([63, 63, 20, 99999])
    elif call == "bfs":
        c["maxw"] = rng.choice([0, 0, 63])
    if call == "cc":
        c["sym"] = rng.random() < 0.7
    if call.startswith("batch"):
        c["n"] = rng.choice([64, 64, rng.randint(2, 63)])
    if call == "serve":
        c["n"] = rng.randint(8, 60)
    return c


# ------------------------------------------------------------------ inputs --


def _edges(V, E, seed):
    """E RMAT edges over V vertices: (sources, destinations), int64 on the GPU."""
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    scale = max(1, (V - 1).bit_length())
    src = torch.empty(E, dtype=torch.int64, device=DEV)
    dst = torch.empty(E, dtype=torch.int64, device=DEV)
    for b in range(0, E, 1 << 26):  # in blocks: the largest graphs have hundreds of millions of edges
        n = min(1 << 26, E - b)
        s = torch.zeros(n, dtype=torch.int64, device=DEV)
        d = torch.zeros(n, dtype=torch.int64, device=DEV)
        for _ in range(scale):
            r = torch.rand(n, device=DEV, generator=g)
            down, right = r >= 0.76, (r >= 0.57) & (r < 0.76) | (r >= 0.95)
            s.mul_(2).add_(down)
            d.mul_(2).add_(right)
        src[b:b + n], dst[b:b + n] = s % V, d % V
    return src, dst


def _lists(keys, other, V):
    """Adjacency lists by `keys`: (V + 1 offsets, `other` in list order, the order)."""
    key, order = torch.sort(keys.to(torch.int32), stable=True)
    ptr = torch.zeros(V + 1, dtype=torch.int64, device=DEV)
    ptr[1:] = torch.cumsum(torch.bincount(key, minlength=V), 0)
    return ptr, other[order].to(torch.int32), order


def _host(t):
    return t.cpu().numpy()


def _pr_graph(case, seed):
    """Offsets, list entries and out-degrees of a PageRank graph, on the GPU."""
    V = case["V"]
    src, dst = _edges(V, V * case["ef"], seed)
    outdeg = torch.bincount(src, minlength=V)
    if case["layout"] == "csc":
        ptr, adj, _ = _lists(dst, src, V)
    else:
        ptr, adj, _ = _lists(src, dst, V)
    return ptr, adj, outdeg


def _open(case, V, seed):
    """The engine's handle and out-degrees of one graph of the case."""
    budget = A.make_budget(frac=case["frac"]) if case["frac"] < 1.0 else A.make_budget()
    if case["call"] == "pr":
        ptr, adj, outdeg = _pr_graph(case, seed)
        od = _host(outdeg.to(torch.int32)).view(np.uint32) if case["layout"] == "csc" else None
        return A.Graph.from_csr(_host(ptr).view(np.uint64), _host(adj).view(np.uint32), outdeg=od,
                                budget=budget), outdeg
    src, dst = _edges(V, V * case["ef"], seed)
    if case.get("sym"):
        src, dst = torch.cat([src, dst]), torch.cat([dst, src])
    ptr, adj, _ = _lists(src, dst, V)
    if case["maxw"]:
        g = torch.Generator(device=DEV)
        g.manual_seed(seed + 1)
        w = torch.randint(1, case["maxw"] + 1, (adj.numel(),), device=DEV, generator=g, dtype=torch.int32)
        adj = torch.stack([adj, w], 1)
    deg = ptr[1:] - ptr[:-1]
    return A.Graph.from_csr(_host(ptr).view(np.uint64), _host(adj).view(np.uint32), budget=budget), deg


def _sources(deg, n, seed):
    """n vertices with out-edges, drawn uniformly."""
    live = _host(torch.nonzero(deg).flatten())
    rng = np.random.RandomState(seed % (1 << 31))
    return live[rng.randint(0, len(live), n)].astype(np.uint32)


def _params(case):
    if case["call"] != "pr":
        return A.make_params()
    return A.make_params(pr_mode=A.PR_REF if case["mode"] == "ref" else A.PR_STD,
                         precision=A.F32 if case["prec"] == "f32" else A.F64)


class _State:
    pass


class _Held(np.ndarray):
    """A result buffer in page-locked memory; `keep` holds the memory as long as the array is in use."""


def _pinned(shape, dtype):
    keep = A.PinnedArray(int(np.prod(shape)), dtype)
    a = keep.array.reshape(shape).view(_Held)
    a.keep = keep
    return a


def prepare(case, seed):
    s = _State()
    s.case, call = case, case["call"]
    if call == "serve":
        s.graphs, s.queries = [], []
        s.server = A.Server(budget_bytes=4 << 30)
        degs = []
        for k, V in enumerate((case["V"], max(64, case["V"] // 4))):
            g, deg = _open(case, V, 1000 * seed + 7 * k + 1)
            s.graphs.append(g)
            s.server.add_graph(g)
            degs.append(_sources(deg, case["n"], seed + k))
        mix = np.random.RandomState(case["n"])
        pr = A.make_params(pr_mode=A.PR_STD, precision=A.F32)
        for i in range(case["n"]):
            k, x = int(mix.randint(2)), mix.rand()
            algo = "bfs" if x < 0.5 else "sssp" if x < 0.8 else "cc" if x < 0.9 else "pr"
            s.queries.append((k, algo, int(degs[k][i]) if algo in ("bfs", "sssp") else 0,
                              pr if algo == "pr" else None))
        return s
    s.graph, deg = _open(case, case["V"], seed)
    s.params = _params(case)
    s.out = None
    n = case["n"] if call.startswith("batch") else 1
    s.sources = _sources(deg, n, seed)
    if case["out"] == "pinned":
        dt = np.uint32
        if call == "pr":
            dt = np.float32 if case["prec"] == "f32" else np.float64
        s.out = _pinned((n, case["V"]) if call.startswith("batch") else (case["V"],), dt)
    return s


def run(s):
    call = s.case["call"]
    if call == "serve":
        tickets = [s.server.submit(k, algo, src, params=p) for k, algo, src, p in s.queries]
        got = [s.server.wait(t)[0] for t in tickets]
        return [x if q[1] == "pr" else x.view(np.int32) for x, q in zip(got, s.queries)]
    if call == "pr":
        return s.graph.run(call, params=s.params, out=s.out)[0]
    if call.startswith("batch"):
        x = s.graph.run_batch(call[6:], s.sources, params=s.params, out=s.out)[0]
    else:
        x = s.graph.run(call, 0 if call == "cc" else int(s.sources[0]), params=s.params, out=s.out)[0]
    return x.view(np.int32)  # levels, distances and labels are at most V + 1


# ---------------------------------------------------------- work and truth --


def work(case):
    """The graph read once (4-byte ids, offsets, and weights or out-degrees where the call
    reads them) and every result written once. PageRank: the sums of one pass over the edges."""
    V, call = case["V"], case["call"]
    E = V * case["ef"] * (2 if case.get("sym") else 1)
    weighted = call in ("sssp", "batch_sssp", "serve")
    read = (8 if weighted else 4) * E + 4 * (V + 1)
    n = case["n"] if call.startswith("batch") else 1
    if call == "serve":
        return {"bytes": 1.25 * read + 4.0 * case["n"] * 0.625 * V, "flops": 0}
    if call == "pr":
        width = 4 if case["prec"] == "f32" else 8
        return {"bytes": read + (4 * V if case["layout"] == "csc" else 0) + width * V, "flops": 2.0 * E}
    return {"bytes": read + 4.0 * n * V, "flops": 0}


def exact(case, seed):
    """PageRank in 64 bits (the traversals' results are whole numbers)."""
    if case["call"] != "pr":
        return None
    ptr, adj, outdeg = _pr_graph(case, seed)
    V = case["V"]
    rows = torch.repeat_interleave(torch.arange(V, device=DEV), ptr[1:] - ptr[:-1])
    adj = adj.to(torch.int64)
    src, dst = (adj, rows) if case["layout"] == "csc" else (rows, adj)
    od = outdeg.to(torch.float64)
    dangling = outdeg == 0
    rank = torch.full((V,), 1.0 / V, dtype=torch.float64, device=DEV)
    share = torch.where(dangling, torch.zeros_like(od), rank / od)
    active = torch.ones(V, dtype=torch.bool, device=DEV)
    for _ in range(100 if case["mode"] == "std" else 100000):
        sums = torch.zeros(V, dtype=torch.float64, device=DEV).index_add_(0, dst, share[src])
        if case["mode"] == "std":
            new = 0.15 / V + 0.85 * rank[dangling].sum() / V + 0.85 * sums
            residual = float((new - rank).abs().sum())
            rank = new
            share = torch.where(dangling, torch.zeros_like(od), rank / od)
            if residual < 1e-9:
                break
        else:  # a vertex takes its new rank while it changes by more than 0.001, then stays as it is
            new = 0.15 + 0.85 * sums
            active = active & ((new - rank).abs() > 0.001)
            rank = torch.where(active, new, rank)
            share = torch.where(active & ~dangling, rank / od, share)
            if not bool(active.any()):
                break
    return _host(rank)
