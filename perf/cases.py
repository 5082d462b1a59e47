"""The work this framework is measured on: BYO's run_all applications and its
batch-update schedule through the public entry points (the Python package and
the C ABI's device forms, as bench.py and the tests call them).

A case is one application on one seeded graph:
  op         bfs, bfs_multi, cc, pagerank, pagerank_edgemap, triangles,
             update (insert, traverse, remove), mixed (a stream of batches and
             64-source queries) or bytepd (load and write a compressed graph)
  graph      rmat (skewed), er (uniform), grid (high diameter), chung_lu
             (power law); symmetric, sorted, no duplicates or self loops
  container  csr, pma, pcsr or vos
Graphs and batches are drawn with torch on the GPU from the seed alone and
handed over as a loader would (host CSR, device keys).
"""
import ctypes
import math

import numpy as np
import torch

import byo_gb300 as byo
from byo_gb300 import _abi

RMAT = (0.57, 0.19, 0.19)  # quadrant probabilities of every RMAT configuration
DAMPING = 0.85
ITERS = 20                 # PageRank iterations (eps 0: exactly these)
QUERY_SOURCES = 64         # sources of one bit-lane BFS

_ctx = None


def _context():
    """One context per process, as a program keeps it."""
    global _ctx
    if _ctx is None:
        _ctx = byo.Context(0)
    return _ctx


def listed():
    return [
        # the smallest call: one BFS on a graph that fits in L1, all latency (a service's point query)
        dict(name="bfs_small", op="bfs", graph="rmat", n=1 << 12, draws=1 << 15, container="csr"),
        # BFS on a skewed graph larger than L2, a handful of rounds of very different widths
        dict(name="bfs_rmat", op="bfs", graph="rmat", n=1 << 22, draws=1 << 26, container="csr"),
        # BFS over thousands of narrow rounds (road-like graph, odd side lengths)
        dict(name="bfs_grid", op="bfs", graph="grid", n=1277 * 1531, draws=1531, container="csr"),
        # connectivity of a uniform sparse graph, odd size, many small components beside the giant one
        dict(name="cc_er", op="cc", graph="er", n=3000017, draws=9000001, container="csr"),
        # PageRank in FP64, the plain method's configuration
        dict(name="pagerank_fp64", op="pagerank", graph="rmat", n=1 << 20, draws=1 << 24, container="csr",
             precision=_abi.PR_FP64),
        # the reference's loop through edgeMap and vertexMap (the API that other applications are written on)
        dict(name="edgemap_chung_lu", op="pagerank_edgemap", graph="chung_lu", n=1000003, draws=8000000,
             container="csr"),
        # triangle counting, degree ordered, average degree 32
        dict(name="triangles", op="triangles", graph="rmat", n=1 << 22, draws=1 << 26, container="csr"),
        # 64 BFS queries answered by one traversal, average degree 16, on the updatable container
        dict(name="bfs_multi", op="bfs_multi", graph="rmat", n=1 << 20, draws=1 << 23, container="pma"),
        # a small batch between traversals: launches and latency of the update path
        dict(name="update_small", op="update", graph="rmat", n=1 << 18, draws=1 << 21, container="pcsr", pairs=1000,
             pagerank=False),
        # the largest: the dynamic step, 10^7 pairs in, BFS + CC + PageRank (FP32, compensated), pairs out
        dict(name="update_large", op="update", graph="rmat", n=1 << 22, draws=1 << 26, container="pma",
             pairs=10 ** 7, pagerank=True),
        # serving a dynamic graph: uneven batches (10^2..10^4 pairs) between 64-source queries, one call
        dict(name="mixed_stream", op="mixed", graph="rmat", n=1 << 20, draws=1 << 23, container="pma", batches=8,
             queries=4),
        # a compressed graph file's arrays decoded, summed over and encoded again
        dict(name="bytepd", op="bytepd", graph="rmat", n=1 << 20, draws=1 << 24, container="csr", block=1000),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["bfs", "bfs", "cc", "pagerank", "pagerank_edgemap", "triangles", "bfs_multi", "update", "update",
                     "mixed", "bytepd"])
    top = {"bfs_multi": 1 << 20, "mixed": 1 << 20, "bytepd": 1 << 20, "pagerank_edgemap": 1 << 20}.get(op, 1 << 22)
    kinds = {"triangles": ["rmat", "er", "chung_lu"], "bfs": ["rmat", "er", "grid", "chung_lu"]}
    graph = rng.choice(kinds.get(op, ["rmat", "rmat", "er", "chung_lu"]))
    n = _log_int(rng, 1 << 10, top)
    if graph == "rmat":
        n = 1 << int(round(math.log2(n)))
    draws = int(n * rng.uniform(2, 16)) | 1  # average degree 4 to 32
    if op == "cc" and graph == "er":
        draws = int(n * rng.uniform(0.5, 3)) | 1  # denser uniform graphs are one component, with nothing to tell apart
    case = dict(op=op, graph=graph, n=n, draws=draws, container="csr")
    if graph == "grid":
        rows = _log_int(rng, 3, min(n // 3, 1500))
        case.update(n=rows * max(3, min(n // rows, 1500)), draws=rows)
    if op == "update":
        case["container"] = rng.choice(["pma", "pcsr", "vos"])
        case["pairs"] = _log_int(rng, 100, max(200, min(10 ** 7, 4 * n)))
        case["pagerank"] = rng.random() < 0.5
    elif op == "mixed":
        case.update(container="pma", batches=rng.randint(2, 8), queries=rng.randint(1, 4))
    elif op in ("bfs", "cc", "bfs_multi", "pagerank"):
        case["container"] = rng.choice(["csr", "csr", "pma", "pcsr", "vos"])
    if op == "pagerank":
        case["precision"] = rng.choice([_abi.PR_FP32_KAHAN, _abi.PR_FP64, _abi.PR_FP32])
    if op == "bytepd":
        case["block"] = rng.choice([64, 1000])
    return case


# ---------------------------------------------------------------- inputs

def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(1000003 * int(seed) + 17)


def _uniform_ids(gen, n, count):
    return torch.randint(0, n, (count,), generator=gen, device="cuda", dtype=torch.int64)


def _pairs(case, gen):
    n, draws = case["n"], case["draws"]
    if case["graph"] == "grid":  # draws: rows; a 4-neighbour grid
        rows, cols = draws, n // draws
        v = torch.arange(n, device="cuda", dtype=torch.int64)
        right, down = v[v % cols != cols - 1], v[: n - cols]
        return torch.cat([right, down]), torch.cat([right + 1, down + cols])
    if case["graph"] == "er":
        return _uniform_ids(gen, n, draws), _uniform_ids(gen, n, draws)
    if case["graph"] == "chung_lu":  # endpoints by weight i^(-1/1.1): power-law exponent 2.1
        w = torch.arange(1, n + 1, device="cuda", dtype=torch.float64).pow(-1 / 1.1)
        cum = torch.cumsum(w, 0)
        ids = [torch.searchsorted(cum, torch.rand(draws, generator=gen, device="cuda", dtype=torch.float64) * cum[-1])
               for _ in range(2)]
        return ids[0].clamp_(max=n - 1), ids[1].clamp_(max=n - 1)
    a, b, c = RMAT
    u = torch.zeros(draws, device="cuda", dtype=torch.int64)
    v = torch.zeros(draws, device="cuda", dtype=torch.int64)
    for _ in range(n.bit_length() - 1):
        r = torch.rand(draws, generator=gen, device="cuda")
        lower = r >= a + b
        u.mul_(2).add_(lower)
        v.mul_(2).add_(torch.where(lower, r >= a + b + c, r >= a))
    return u, v


def _keys(u, v):
    """Both directions as src << 32 | dst, self loops dropped."""
    keep = u != v
    u, v = u[keep], v[keep]
    return torch.cat([(u << 32) | v, (v << 32) | u])


def _edges(case, gen):
    """The graph's keys, sorted and without duplicates."""
    k = _keys(*_pairs(case, gen)).sort().values
    return k[torch.cat([torch.ones(1, device="cuda", dtype=torch.bool), k[1:] != k[:-1]])]


def _csr(keys, n):
    off = torch.zeros(n + 1, device="cuda", dtype=torch.int64)
    torch.cumsum(torch.bincount(keys >> 32, minlength=n), 0, out=off[1:])
    return off, keys & 0xFFFFFFFF


def _batch(gen, n, pairs, present):
    """A symmetrised, unsorted batch of uniform pairs that the graph does not hold, so that removing it restores the
    graph."""
    k = _keys(_uniform_ids(gen, n, pairs), _uniform_ids(gen, n, pairs))
    at = torch.searchsorted(present, k).clamp_(max=present.numel() - 1)
    k = k[present[at] != k]
    return k[torch.randperm(k.numel(), generator=gen, device="cuda")]


def _mixed_sizes(case):
    """Batch sizes in pairs, log-uniform over 10^2..10^4."""
    b = case["batches"]
    return [int(10 ** (2 + 2 * (i + 0.5) / b)) for i in range(b)]


def _stream(case, gen, present):
    """ops, key offsets and keys of a stream: each batch goes in, a query runs, an earlier batch goes out."""
    batches = [_batch(gen, case["n"], s, present) for s in _mixed_sizes(case)]
    order = torch.randperm(len(batches), generator=gen, device="cuda").tolist()
    ops, keys, queries = [], [], case["queries"]
    for i, b in enumerate(order):
        ops.append(_abi.OP_INSERT)
        keys.append(batches[b])
        if queries * (i + 1) // len(order) > queries * i // len(order):
            ops.append(_abi.OP_QUERY)
            keys.append(batches[b][:0])
        if i >= 1:
            ops.append(_abi.OP_REMOVE)
            keys.append(batches[order[i - 1]])
    ops.append(_abi.OP_REMOVE)
    keys.append(batches[order[-1]])
    off = np.zeros(len(ops) + 1, np.uint64)
    off[1:] = np.cumsum([k.numel() for k in keys])
    return np.array(ops, np.uint8), off, torch.cat(keys)


def _inputs(case, seed):
    gen = _generator(seed)
    keys = _edges(case, gen)
    return gen, keys


def _sources(gen, keys, count):
    """Ends of uniformly drawn edges: sources that reach something, hubs more often."""
    return (keys[_uniform_ids(gen, keys.numel(), count)] >> 32).to(torch.int32)


def prepare(case, seed):
    ctx, n = _context(), case["n"]
    gen, keys = _inputs(case, seed)
    s = {"case": case, "ctx": ctx, "n": n}
    if case["op"] == "update":
        s["batch"] = _batch(gen, n, case["pairs"], keys)
    if case["op"] == "mixed":
        s["ops"], s["off"], s["keys"] = _stream(case, gen, keys)
        s["sources"] = _sources(gen, keys, QUERY_SOURCES * case["queries"]).cpu().numpy().view(np.uint32)
        s["levels"] = torch.empty(case["queries"], QUERY_SOURCES, n, dtype=torch.int32, device="cuda")
        s["changed"] = np.zeros(len(s["ops"]), np.uint64)
    if case["op"] == "bfs_multi":
        s["sources"] = _sources(gen, keys, QUERY_SOURCES).cpu().numpy().view(np.uint32)
        s["levels"] = torch.empty(QUERY_SOURCES, n, dtype=torch.int32, device="cuda")
    if case["op"] in ("bfs", "update"):
        s["src"] = int(_sources(gen, keys, 1).item())
        s["parent"] = torch.empty(n, dtype=torch.int32, device="cuda")
        s["level"] = torch.empty(n, dtype=torch.int32, device="cuda")
    if case["op"] in ("cc", "update"):
        s["label"] = torch.empty(n, dtype=torch.int32, device="cuda")
    if case["op"] == "pagerank" or case.get("pagerank"):
        s["p"] = torch.empty(n, dtype=torch.float64, device="cuda")
    off, nbr = _csr(keys, n)
    off, nbr = off.cpu().numpy().view(np.uint64), nbr.to(torch.int32).cpu().numpy().view(np.uint32)
    torch.cuda.synchronize()  # the library's stream does not wait for torch's
    g = byo.Graph.from_csr(ctx, off, nbr, container=case["container"])
    if case["op"] == "bytepd":
        s["encoded"] = g.to_bytepd(block=case["block"])
        g.close()
        s["offsets"], s["degrees"] = np.zeros(n + 1, np.int64), np.zeros(n, np.int32)
        # room for the encoded bytes: about 2 an edge in practice
        s["bytes"] = np.zeros(4 * 2 * case["draws"] + 64 * n, np.uint8)
    else:
        s["graph"] = g
    return s


# ---------------------------------------------------------------- one pass

def _bfs(s):
    _abi.check(_abi.lib().byo_bfs_device(s["graph"].h, s["src"], s["parent"].data_ptr(), s["level"].data_ptr(),
                                         _abi.POLICY_M20, None), s["ctx"].h)
    return [s["parent"], s["level"]]


def _cc(s):
    _abi.check(_abi.lib().byo_cc_device(s["graph"].h, s["label"].data_ptr()), s["ctx"].h)
    return [s["label"]]


def _pagerank(s, precision):
    _abi.check(_abi.lib().byo_pagerank_device(s["graph"].h, 0.0, ITERS, precision, s["p"].data_ptr(), None, None),
               s["ctx"].h)
    return [s["p"]]


def _update(s):
    lib, g, batch = _abi.lib(), s["graph"], s["batch"]
    added, removed = ctypes.c_uint64(0), ctypes.c_uint64(0)
    _abi.check(lib.byo_graph_insert_batch_device(g.h, batch.data_ptr(), batch.numel(), 0, ctypes.byref(added)),
               s["ctx"].h)
    out = _bfs(s) + _cc(s)
    if s["case"]["pagerank"]:
        out += _pagerank(s, _abi.PR_FP32_KAHAN)
    _abi.check(lib.byo_graph_remove_batch_device(g.h, batch.data_ptr(), batch.numel(), 0, ctypes.byref(removed)),
               s["ctx"].h)
    return out + [added.value, removed.value, g.M()]


def _mixed(s):
    _abi.check(_abi.lib().byo_graph_mixed_stream_device(
        s["graph"].h, s["keys"].data_ptr(), s["off"].ctypes.data, s["ops"].ctypes.data, len(s["ops"]),
        s["sources"].ctypes.data, QUERY_SOURCES, s["levels"].data_ptr(), s["changed"].ctypes.data, None), s["ctx"].h)
    return [s["levels"], s["changed"].astype(np.int64), s["graph"].degrees().astype(np.int64)]


def _bytepd(s):
    block, size = s["case"]["block"], ctypes.c_uint64(s["bytes"].size)
    g = byo.Graph.from_bytepd(s["ctx"], *s["encoded"], block=block)
    total = byo.Test_Map(g)
    _abi.check(_abi.lib().byo_graph_encode_bytepd(g.h, block, s["offsets"].ctypes.data, s["degrees"].ctypes.data,
                                                  s["bytes"].ctypes.data, ctypes.byref(size)), s["ctx"].h)
    g.close()
    return [total, s["offsets"], s["degrees"], s["bytes"], size.value]


def run(state):
    op = state["case"]["op"]
    if op == "bfs":
        return _bfs(state)
    if op == "bfs_multi":
        _abi.check(_abi.lib().byo_bfs_multi_device(state["graph"].h, state["sources"].ctypes.data, QUERY_SOURCES,
                                                   state["levels"].data_ptr(), None), state["ctx"].h)
        return [state["levels"]]
    if op == "cc":
        return _cc(state)
    if op == "pagerank":
        return _pagerank(state, state["case"]["precision"])
    if op == "pagerank_edgemap":
        return [byo.PageRank_edgeMap(state["graph"], eps=0.0, max_iters=ITERS)]
    if op == "triangles":
        return [byo.Triangle_degree_ordering(state["graph"])]
    if op == "update":
        return _update(state)
    if op == "mixed":
        return _mixed(state)
    return _bytepd(state)


# ---------------------------------------------------------------- what a pass cannot do without

def work(case):
    """Bytes with every input read once and every output written once (a PageRank iteration reads the graph and the
    iterate, and writes the iterate); operations are additions over edges."""
    n, op = case["n"], case["op"]
    m = 4 * n if case["graph"] == "grid" else 2 * case["draws"]  # before duplicates go: an upper estimate
    graph = 8 * n + 4 * m
    if op == "bfs":
        return dict(bytes=graph + 8 * n, flops=0)
    if op == "cc":
        return dict(bytes=graph + 4 * n, flops=0)
    if op == "bfs_multi":
        return dict(bytes=graph + 4 * QUERY_SOURCES * n, flops=0)
    if op in ("pagerank", "pagerank_edgemap"):
        word = 8 if op == "pagerank_edgemap" or case["precision"] == _abi.PR_FP64 else 4
        return dict(bytes=ITERS * (graph + 2 * word * n), flops=ITERS * m)
    if op == "triangles":
        return dict(bytes=graph, flops=0)
    if op == "update":
        b = 2 * case["pairs"]
        after = 8 * n + 4 * (m + b)
        total = 2 * (8 * b + 2 * 4 * min(m, 512 * b)) + 2 * after + 12 * n
        if case["pagerank"]:
            total += ITERS * (after + 8 * n)
        return dict(bytes=total, flops=ITERS * (m + b) if case["pagerank"] else 0)
    if op == "mixed":
        b = 2 * sum(2 * s for s in _mixed_sizes(case))
        return dict(bytes=16 * b + case["queries"] * (graph + 4 * QUERY_SOURCES * n) + 4 * n, flops=0)
    return dict(bytes=2 * (2 * m + 12 * n) + 8 * m, flops=0)  # bytepd: about two bytes an edge, in and out


# ---------------------------------------------------------------- 64-bit results

def _exact_pagerank(keys, n):
    off, nbr = _csr(keys, n)
    adj = torch.sparse_csr_tensor(off, nbr, torch.ones(nbr.numel(), device="cuda", dtype=torch.float64), size=(n, n))
    deg = (off[1:] - off[:-1]).double()
    p = torch.full((n,), 1 / n, device="cuda", dtype=torch.float64)
    for _ in range(ITERS):
        share = torch.where(deg > 0, p / deg.clamp(min=1), torch.zeros_like(p))
        p = DAMPING * (adj @ share) + (1 - DAMPING) / n
    return p


def exact(case, seed):
    """PageRank by torch in FP64; the other outputs are whole numbers."""
    op, n = case["op"], case["n"]
    if op not in ("pagerank", "pagerank_edgemap") and not case.get("pagerank"):
        return None
    gen, keys = _inputs(case, seed)
    if op == "update":
        keys = torch.cat([keys, _batch(gen, n, case["pairs"], keys)]).unique()
        return [None, None, None, _exact_pagerank(keys, n), None, None, None]
    p = _exact_pagerank(keys, n)
    return [p.cpu().numpy() if op == "pagerank_edgemap" else p]
