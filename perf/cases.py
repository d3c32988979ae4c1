"""The performance cases: what a program that counts and enumerates subgraphs has this library do, through its
public entry points, over the range of sizes that the benchmark's workloads and the tests span.

A case is one way of using the library ("use") on seeded synthetic graphs of one family:

  load       a host CSR in pinned memory: build the graph, count the patterns, drop the graph
  step       the same from a CSR in device memory, all patterns in one batched call
  edges      a raw host edge list (loops, duplicates, unordered): build the graph and count
  query      a resident graph: one count per pattern, each call planned anew
  noalloc    the allocation-free entry point on a device CSR
  enumerate  a resident graph: every match (up to a limit above their number), as tuples
  batch      (graph, pattern) pairs over several resident graphs, planned once and replayed
  serve      requests to a running server over resident graphs

Graph families: "er" (G(n, p)), "rmat" ((.57, .19, .19, .05), n = 2^scale), "chung_lu" (power law, exponent 2.1),
each symmetrised, without loops and duplicates, rows sorted, int32 CSR; degree is the average directed degree that
is sampled, before duplicates go.
"""
import numpy as np
import torch

import beep_b200 as B
from beep_b200 import patterns as P

MODES = {"sgm": B.SGM, "sgc": B.SGC}
# cliques larger than the named ones: the deepest walks that the tests count on graphs of this kind
PATTERNS = {**P.NAMED, **P.NON_CENTRAL,
            **{"k%d" % k: P._undirected([(a, b) for b in range(k) for a in range(b)]) for k in (6, 7)}}
SERVED = ["triangle", "diamond", "k4", "tailed_triangle", "w5", "k5"]  # the served workload's mix
SERVED_K = 10000  # tuples of a first-k request
ENUMERATED = 1 << 20  # tuples asked for where every match is wanted (the cases have fewer)
_ctx = None


def listed():
    return [
        # the smallest call: a small graph from host memory, triangles (the benchmark's small workload)
        {"name": "load_er_triangle", "use": "load", "family": "er", "n": 4096, "degree": 16.4, "patterns": "triangle", "mode": "sgc"},
        # the headline step: build, peel, order and count, 4-clique and diamond, on a mid-size skewed graph
        {"name": "step_rmat20", "use": "step", "family": "rmat", "n": 1 << 20, "degree": 6.0, "patterns": "k4,diamond", "mode": "sgm"},
        # a file's edges as they come, sorted and deduplicated on the device, one pattern counted
        {"name": "edges_chunglu18", "use": "edges", "family": "chung_lu", "n": 1 << 18, "degree": 16.0, "patterns": "tailed_triangle", "mode": "sgm"},
        # an ordinary query on a resident graph of odd size
        {"name": "query_k4_chunglu", "use": "query", "family": "chung_lu", "n": 100003, "degree": 24.0, "patterns": "k4", "mode": "sgm"},
        # the large workload's two patterns on its graph shape (edge factor 28), at smaller scales
        {"name": "query_w5_rmat16", "use": "query", "family": "rmat", "n": 1 << 16, "degree": 56.0, "patterns": "w5", "mode": "sgm"},
        {"name": "query_k5_rmat17", "use": "query", "family": "rmat", "n": 1 << 17, "degree": 56.0, "patterns": "k5", "mode": "sgm"},
        # deep walks
        {"name": "query_k7_rmat14", "use": "query", "family": "rmat", "n": 1 << 14, "degree": 24.0, "patterns": "k6,k7", "mode": "sgm"},
        # queries without a central vertex, which walk lists: on graphs without hubs
        {"name": "query_noncentral", "use": "query", "family": "er", "n": 20011, "degree": 10.0, "patterns": "cycle4,house,bull", "mode": "sgm"},
        # a caller that owns all device memory
        {"name": "noalloc_rmat15", "use": "noalloc", "family": "rmat", "n": 1 << 15, "degree": 12.0, "patterns": "diamond", "mode": "sgm"},
        # every match, handed over as tuples
        {"name": "enumerate_k4", "use": "enumerate", "family": "chung_lu", "n": 8009, "degree": 10.0, "patterns": "k4", "mode": "sgm"},
        # the batched workload: graphs of 2^10 to 2^15 vertices, degree 8 to 48, all 15 central patterns of 4 and 5 vertices
        {"name": "batch_chunglu", "use": "batch", "family": "chung_lu", "n": 1 << 15, "degree": 48.0, "graphs": 12, "mode": "sgm"},
        # the served workload: requests for counts, one in five for the first 10,000 tuples too
        {"name": "serve_chunglu", "use": "serve", "family": "chung_lu", "n": 1 << 15, "degree": 16.0, "graphs": 6, "requests": 96, "mode": "sgm"},
    ]


def draw(rng):
    """One more case: sizes spread over the logarithm of their range, odd ones among them."""

    def size(lo, hi):
        return int(round(2 ** rng.uniform(lo, hi)))

    use = rng.choice(["load", "step", "edges", "query", "query", "query", "noalloc", "enumerate", "batch", "serve"])
    case = {"use": use, "mode": "sgm"}
    if use in ("load", "step", "edges"):
        family = rng.choice(["er", "rmat", "chung_lu"])
        n = 1 << rng.randint(12, 20) if family == "rmat" else size(11, 19)
        degree = rng.uniform(4.0, 16.0) if n <= 1 << 18 else rng.uniform(4.0, 6.0)
        pats = rng.choice(["triangle", "k4", "diamond", "k4,diamond", "triangle,tailed_triangle", "k5"])
        case.update(family=family, n=n, degree=degree, patterns=pats, mode=rng.choice(["sgm", "sgc"]) if pats == "triangle" else "sgm")
    elif use == "query":
        kind = rng.choice(["small", "small", "w5", "k5", "deep", "noncentral"])
        if kind == "small":
            case.update(family=rng.choice(["er", "chung_lu"]), n=size(10, 18), degree=rng.uniform(6.0, 32.0),
                        patterns=rng.choice(["triangle", "diamond", "k4", "tailed_triangle", "claw", "k5", "diamond,k4"]))
        elif kind == "w5":
            case.update(family="rmat", n=1 << rng.randint(11, 15), degree=rng.uniform(12.0, 56.0), patterns="w5")
        elif kind == "k5":
            case.update(family="rmat", n=1 << rng.randint(12, 16), degree=rng.uniform(16.0, 56.0), patterns="k5")
        elif kind == "deep":
            case.update(family="rmat", n=1 << rng.randint(10, 13), degree=rng.uniform(12.0, 24.0), patterns=rng.choice(["k6", "k7"]))
        else:
            case.update(family="er", n=size(9, 14), degree=rng.uniform(3.0, 10.0), patterns=rng.choice(sorted(P.NON_CENTRAL)))
    elif use == "noalloc":
        case.update(family=rng.choice(["er", "rmat"]), n=1 << rng.randint(11, 15), degree=rng.uniform(6.0, 12.0),
                    patterns=rng.choice(["triangle", "diamond", "k4"]))
    elif use == "enumerate":
        case.update(family="chung_lu", n=size(10, 12.9), degree=rng.uniform(6.0, 10.0), patterns=rng.choice(["triangle", "k4"]))
    elif use == "batch":
        case.update(family="chung_lu", n=size(11, 15), degree=rng.uniform(16.0, 48.0), graphs=rng.randint(2, 11))
    else:
        case.update(family="chung_lu", n=size(12, 15), degree=rng.uniform(8.0, 16.0), graphs=rng.randint(2, 6),
                    requests=rng.randint(16, 95))
    return case


# ---- inputs ----------------------------------------------------------------


def _endpoints(family, n, degree, g):
    """Sampled edges (src, dst) on the device: n * degree / 2 of them, loops and duplicates among them."""
    ne = int(n * degree / 2)
    if family == "rmat":
        u = torch.zeros(ne, dtype=torch.int64, device="cuda")
        v = torch.zeros(ne, dtype=torch.int64, device="cuda")
        for _ in range(n.bit_length() - 1):
            r = torch.rand(ne, device="cuda", generator=g)
            down = r >= 0.76  # quadrants a, b, c, d = .57, .19, .19, .05
            right = ((r >= 0.57) & ~down) | (r >= 0.95)
            u = u * 2 + down
            v = v * 2 + right
        return u, v
    if family == "er":
        return (torch.randint(0, n, (ne,), device="cuda", generator=g), torch.randint(0, n, (ne,), device="cuda", generator=g))
    w = torch.arange(1, n + 1, dtype=torch.float64, device="cuda") ** (-1.0 / 1.1)
    cum = torch.cumsum(w, 0)
    both = [torch.searchsorted(cum, torch.rand(ne, dtype=torch.float64, device="cuda", generator=g) * cum[-1]).clamp_(max=n - 1)
            for _ in range(2)]
    return both[0], both[1]


def _csr(family, n, degree, seed):
    """(row_ptr, col) int32 on the device: both directions, sorted rows, no loops, no duplicates."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    u, v = _endpoints(family, n, degree, g)
    keep = u != v
    u, v = u[keep], v[keep]
    key = torch.unique(torch.cat([u * n + v, v * n + u]))
    row_ptr = torch.zeros(n + 1, dtype=torch.int32, device="cuda")
    row_ptr[1:] = torch.cumsum(torch.bincount(key // n, minlength=n), 0).to(torch.int32)
    return row_ptr, (key % n).to(torch.int32)


def _raw_edges(case, seed):
    """Both directions of the sampled edges in shuffled order, loops and duplicates kept: uint32 arrays on the host."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    u, v = _endpoints(case["family"], case["n"], case["degree"], g)
    src, dst = torch.cat([u, v]), torch.cat([v, u])
    order = torch.randperm(len(src), device="cuda", generator=g)
    return [x[order].to(torch.int32).cpu().numpy().view(np.uint32) for x in (src, dst)]


def _graph_sizes(case):
    """The graphs of a batch or a server: from 1/32 of the largest size up, the degree from a sixth of the largest up."""
    k = case["graphs"]
    f = [i / max(k - 1, 1) for i in range(k)]
    return [(max(64, int(case["n"] * 2.0 ** (-5 * (1 - x)))), case["degree"] * (1 / 6 + 5 / 6 * ((7 * i) % k) / max(k - 1, 1)))
            for i, x in enumerate(f)]


def _requests(case, seed):
    """(graph, pattern, k) of every request, as the served workload draws them."""
    rng = np.random.default_rng(seed)
    return [(int(rng.integers(0, case["graphs"])), SERVED[int(rng.integers(0, len(SERVED)))], SERVED_K if rng.random() < 0.2 else 0)
            for _ in range(case["requests"])]


def _context():
    """A program's one context."""
    global _ctx
    if _ctx is None:
        _ctx = B.Context(0)
    return _ctx


def _resident(row_ptr, col):
    torch.cuda.synchronize()  # the library has a stream of its own
    return B.Graph.from_device_csr(_context(), len(row_ptr) - 1, len(col), row_ptr.data_ptr(), col.data_ptr())


def prepare(case, seed):
    use, mode = case["use"], MODES[case["mode"]]
    state = {"use": use, "mode": mode, "ctx": _context(), "names": case.get("patterns", "").split(",")}
    if use in ("batch", "serve"):
        graphs = [_resident(*_csr(case["family"], n, d, seed * 100 + i)) for i, (n, d) in enumerate(_graph_sizes(case))]
        state["graphs"] = graphs
        if use == "batch":
            state["batch"] = B.Batch(_context())
            queries = [B.Query.from_edges(q) for q in P.central_patterns(4) + P.central_patterns(5)]
            for g in graphs:
                for q in queries:
                    state["batch"].add(g, q, mode)
        else:
            state["server"] = B.Server(_context())
            queries = {name: B.Query.from_edges(PATTERNS[name]) for name in SERVED}
            ids = [state["server"].add_graph(g) for g in graphs]
            state["requests"] = [(ids[g], queries[name], k) for g, name, k in _requests(case, seed)]
        return state
    state["queries"] = [B.Query.from_edges(PATTERNS[name]) for name in state["names"]]
    if use == "edges":
        state["src"], state["dst"] = _raw_edges(case, seed)
        return state
    row_ptr, col = _csr(case["family"], case["n"], case["degree"], seed)
    state["n"], state["m"] = len(row_ptr) - 1, len(col)
    if use == "load":
        state["pinned"] = [x.cpu().pin_memory() for x in (row_ptr, col)]
        state["row_ptr"], state["col"] = [x.numpy() for x in state["pinned"]]
    elif use in ("query", "enumerate"):
        state["graph"] = _resident(row_ptr, col)
    else:
        state["row_ptr"], state["col"] = row_ptr, col
        torch.cuda.synchronize()
    return state


# ---- one pass --------------------------------------------------------------


def run(state):
    use, mode = state["use"], state["mode"]
    if use == "query":
        return [B.count(state["graph"], q, mode) for q in state["queries"]]
    if use == "load":
        g = B.Graph.from_csr(state["ctx"], state["row_ptr"], state["col"])
        counts = [B.count(g, q, mode) for q in state["queries"]]
        g.close()
        return counts
    if use == "step":
        g = B.Graph.from_device_csr(state["ctx"], state["n"], state["m"], state["row_ptr"].data_ptr(), state["col"].data_ptr())
        batch = B.Batch(state["ctx"])
        for q in state["queries"]:
            batch.add(g, q, mode)
        counts = batch.run(B.OPT_NO_GRAPH)
        batch.close()
        g.close()
        return counts
    if use == "edges":
        g = B.Graph.from_edges(state["ctx"], state["src"], state["dst"])
        counts = [B.count(g, q, mode) for q in state["queries"]] + [g.info()["m"], g.info()["max_degree"]]
        g.close()
        return counts
    if use == "noalloc":
        return [B.count_noalloc(0, state["n"], state["m"], state["row_ptr"].data_ptr(), state["col"].data_ptr(), q, mode)
                for q in state["queries"]]
    if use == "enumerate":
        tuples, total = B.enumerate_matches(state["graph"], state["queries"][0], ENUMERATED)
        # the order of matches is unspecified: a table on the device, by their vertices, -1 in the rows that are left
        rows = torch.from_numpy(tuples).cuda()
        key = torch.zeros(len(rows), dtype=torch.int64, device="cuda")
        for i in range(rows.shape[1]):
            key = key * state["n"] + rows[:, i]
        table = torch.full((ENUMERATED, rows.shape[1]), -1, dtype=torch.int32, device="cuda")
        table[: len(rows)] = rows[torch.argsort(key)]
        return [total, table]
    if use == "batch":
        return np.array(state["batch"].run(), dtype=np.int64)
    server = state["server"]
    asked = [(server.submit(g, q, mode, k), k) for g, q, k in state["requests"]]
    got = [server.wait(rid, k) for rid, k in asked]
    # which tuples a first-k request returns is unspecified, their number is not
    return [np.array([r["count"] for r in got], dtype=np.int64),
            np.array([len(r["tuples"]) if "tuples" in r else 0 for r in got], dtype=np.int64)]


# ---- what a pass cannot do without, and what it has to give ------------------


def _csr_bytes(n, degree):
    return 4.0 * (n + 1) + 4.0 * n * degree


def work(case):
    use = case["use"]
    if use in ("batch", "serve"):
        sizes = _graph_sizes(case)
        per_graph = 15 if use == "batch" else case["requests"] / len(sizes)
        return {"bytes": sum(_csr_bytes(n, d) * per_graph for n, d in sizes), "flops": 0.0}
    n, d, k = case["n"], case["degree"], len(case["patterns"].split(","))
    if use == "edges":
        return {"bytes": 8.0 * n * d + _csr_bytes(n, d) * (1 + k), "flops": 0.0}
    return {"bytes": _csr_bytes(n, d) * (1 + k if use in ("load", "step") else k), "flops": 0.0}


def tolerance(case):
    return "exact"


def exact(case, seed):
    """Counts by torch in 64 bits: cliques level by level over the edges oriented by (degree, id), the others from the
    triangles of every edge and vertex. None where a pattern has no such form here, or for the larger cases."""
    use = case["use"]
    if use in ("batch", "serve") or case["n"] * case["degree"] > 8e6:
        return None
    if use == "edges":
        src, dst = (torch.from_numpy(x.view(np.int32)).cuda().to(torch.int64) for x in _raw_edges(case, seed))
        n = int(max(src.max(), dst.max())) + 1
        keep = src != dst
        key = torch.unique(src[keep] * n + dst[keep])
    else:
        row_ptr, col = _csr(case["family"], case["n"], case["degree"], seed)
        n = case["n"]
        deg = (row_ptr[1:] - row_ptr[:-1]).to(torch.int64)
        key = torch.repeat_interleave(torch.arange(n, device="cuda"), deg) * n + col
    deg = torch.bincount(key // n, minlength=n)
    rank = torch.empty(n, dtype=torch.int64, device="cuda")
    rank[torch.argsort(deg * n + torch.arange(n, device="cuda"))] = torch.arange(n, device="cuda")
    a, b = rank[key // n], rank[key % n]
    by_rank = torch.empty(n, dtype=torch.int64, device="cuda")
    by_rank[rank] = deg
    edge = torch.sort((a * n + b)[a < b]).values  # oriented edges (low rank, high rank)

    def extend(cliques, prefix, last):
        """Cliques (rows of ranks, sorted) one vertex larger; prefix: group of equal first vertices, last: their last."""
        end = torch.searchsorted(prefix, prefix, right=True)
        later = end - 1 - torch.arange(len(prefix), device="cuda")
        if int(later.sum()) > 100_000_000:
            return None
        i = torch.repeat_interleave(torch.arange(len(prefix), device="cuda"), later)
        j = i + 1 + torch.arange(len(i), device="cuda") - torch.repeat_interleave(torch.cumsum(later, 0) - later, later)
        want = last[i] * n + last[j]
        at = torch.searchsorted(edge, want).clamp_(max=len(edge) - 1)
        ok = edge[at] == want
        return torch.cat([cliques[i[ok]], last[j[ok]][:, None]], 1), i[ok], last[j[ok]]

    level = {2: (torch.stack([edge // n, edge % n], 1), edge // n, edge % n)}
    for k in range(3, 8):
        level[k] = extend(*level[k - 1]) if level[k - 1] is not None and len(edge) else None

    def count(name):
        if name == "claw":
            return int((by_rank * (by_rank - 1) * (by_rank - 2) // 6).sum())
        k = {"triangle": 3, "k4": 4, "k5": 5, "k6": 6, "k7": 7}.get(name)
        if k:
            return len(level[k][0]) if level[k] is not None else None
        if level[3] is None:
            return None
        t = level[3][0]
        if name == "tailed_triangle":
            return int((torch.bincount(t.reshape(-1), minlength=n) * (by_rank - 2)).sum())
        if name == "diamond":
            on = torch.cat([t[:, 0] * n + t[:, 1], t[:, 0] * n + t[:, 2], t[:, 1] * n + t[:, 2]])
            c = torch.unique(on, return_counts=True)[1]
            return int((c * (c - 1) // 2).sum())
        return None

    counts = [count(name) for name in case["patterns"].split(",")]
    if all(c is None for c in counts):
        return None
    if use == "edges":
        return counts + [len(key), int(deg.max())]
    return [counts[0], None] if use == "enumerate" else counts
