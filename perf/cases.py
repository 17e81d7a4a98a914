"""Workloads of the engine, one dict of plain values each: what its users run.

A graph comes from the package's own generators, with sizes and parameters of
the test suite, the benchmark and the configurations: G(n, p), Chung-Lu
(exponent 2.5, mean degree 16), R-MAT (0.57/0.19/0.19/0.05), cliques of up to
200 vertices planted in a sparse G(n, p), and the many-instance batch members.  The kinds:

  solve   full enumeration of a resident graph (Graph.solve)
  roots   all cliques under a sample of edge roots of a resident graph
          (Graph.solve_root_list), the benchmark's headline
  coo     pairs in host memory to the result in one call (solve_coo)
  build   pairs in pinned host memory to a resident graph, then a light sample
          of roots on it (Graph.from_coo, Graph.solve_root_list)
  text    a COO text file to a resident graph, then the same sample
          (Graph.load_file, the command line's path)
  batch   many graphs in one captured launch, replayed (Batch.solve)
  serve   requests submitted to a running server until it has drained (Server)

Every result is exact: count, checksum and clique-size histogram.
"""
import os
import tempfile

import numpy as np
import torch

import rdmce_b200 as mce

# Roots are numbered along the degeneracy order.  Below this share of them the
# roots of an R-MAT graph are light (ego networks of a few vertices); the band
# above it reaches into the dense core, with up to some 10^6 cliques a root.
LIGHT = 0.8
BAND = (0.84, 0.955)


def listed():
    return [
        # the smallest call: a tiny resident graph, where latency is all
        {"name": "solve_gnp_64", "kind": "solve", "family": "gnp", "n": 64, "degree": 8.0},
        # the sparse power-law graph that every start-up check enumerates
        {"name": "solve_chunglu_1e4", "kind": "solve", "family": "chunglu", "n": 10000, "degree": 16.0, "gamma": 2.5},
        # full enumerations of skewed graphs: the usual comparison size, and
        # one with 10^9 cliques
        {"name": "solve_rmat_14_16", "kind": "solve", "family": "rmat", "scale": 14, "ef": 16},
        {"name": "solve_rmat_15_16", "kind": "solve", "family": "rmat", "scale": 15, "ef": 16},
        # wide ego networks: planted cliques of 40 to 200 vertices
        {"name": "solve_planted_1e5", "kind": "solve", "family": "planted", "n": 100000, "cliques": 256, "lo": 40,
         "hi": 200},
        # the headline's shape: a sample of core roots of the scale-20 graph
        {"name": "roots_rmat_20", "kind": "roots", "family": "rmat", "scale": 20, "ef": 16, "roots": 1024},
        # one call from host pairs: a small odd-sized graph, and a large sparse one
        {"name": "coo_gnp_1001", "kind": "coo", "family": "gnp", "n": 1001, "degree": 16.0},
        {"name": "coo_chunglu_1e6", "kind": "coo", "family": "chunglu", "n": 1000000, "degree": 16.0, "gamma": 2.5},
        # loading: 16.8 M pairs from memory, 2.1 M pairs as text
        {"name": "build_rmat_20", "kind": "build", "family": "rmat", "scale": 20, "ef": 16, "roots": 256},
        {"name": "text_rmat_17", "kind": "text", "family": "rmat", "scale": 17, "ef": 16, "roots": 256},
        # many instances: a captured batch, and a burst of requests to the server
        {"name": "batch_300", "kind": "batch", "graphs": 300},
        {"name": "serve_31", "kind": "serve", "requests": 31},
    ]


def _log_int(rng, lo, hi):
    return int(round(np.exp(rng.uniform(np.log(lo), np.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "roots", "coo", "build", "text", "batch", "serve"])
    if kind == "batch":
        return {"kind": kind, "graphs": _log_int(rng, 3, 300)}
    if kind == "serve":  # scale 10 to 13, edge factor 8 to 32, as the request stream has them
        return {"kind": kind, "requests": _log_int(rng, 1, 40)}
    if kind == "roots":
        return {"kind": kind, "family": "rmat", "scale": rng.randint(17, 20), "ef": rng.randint(8, 16),
                "roots": _log_int(rng, 60, 1024)}
    if kind in ("build", "text"):
        return {"kind": kind, "family": "rmat", "scale": rng.randint(11, 20 if kind == "build" else 17),
                "ef": rng.randint(4, 16), "roots": _log_int(rng, 16, 256)}
    family = rng.choice(["gnp", "chunglu", "rmat", "planted"])
    case = {"kind": kind, "family": family}
    if family == "gnp":
        case.update(n=_log_int(rng, 64, 4096), degree=round(rng.uniform(8, 64), 1))
    elif family == "chunglu":
        case.update(n=_log_int(rng, 1000, 1000000), degree=round(rng.uniform(4, 16), 1),
                    gamma=round(rng.uniform(2.5, 3.0), 2))
    elif family == "rmat":
        scale = rng.randint(10, 15)
        case.update(scale=scale, ef=rng.randint(4, 32 if scale <= 13 else 14))
    else:
        lo = rng.randint(8, 40)
        case.update(n=_log_int(rng, 5000, 100000), cliques=_log_int(rng, 8, 256), lo=lo,
                    hi=rng.randint(lo + 1, 200))
    return case


def _pairs(case, seed):
    seed = int(seed) + 1
    if case["family"] == "gnp":
        return mce.gen_gnp(case["n"], case["degree"], seed)
    if case["family"] == "chunglu":
        return mce.gen_chung_lu(case["n"], case["degree"], case["gamma"], seed)
    if case["family"] == "rmat":
        return mce.gen_rmat(case["scale"], case["ef"], seed)
    planted = mce.gen_planted(case["n"], case["cliques"], case["lo"], case["hi"], seed)
    background = mce.gen_gnp(case["n"], 12.0, seed)
    return tuple(np.concatenate(uv) for uv in zip(planted, background))


def _requests(case, seed):
    rng = np.random.default_rng(seed)
    return [mce.gen_rmat(int(rng.integers(10, 14)), int(rng.integers(8, 33)), int(rng.integers(1, 1 << 30)))
            for _ in range(case["requests"])]


def _sample(case, num_edges, lo, hi, seed):
    """A seeded sample of distinct root indices in [lo, hi) of the ordered edge list, ascending."""
    a, b = int(lo * num_edges), max(int(hi * num_edges), int(lo * num_edges) + 1)
    k = min(case["roots"], b - a)
    return np.sort(np.random.default_rng(seed).choice(b - a, k, replace=False)).astype(np.uint64) + np.uint64(a)


def _pinned(a):
    return torch.from_numpy(a.view(np.int32)).pin_memory().numpy().view(np.uint32)


def _write_text(u, v, path):
    """One "u v" line for each pair, without padding."""
    cols = []
    for a, sep in ((u, 32), (v, 10)):
        x = torch.from_numpy(a.astype(np.int64)).cuda()
        digits = len(str(int(x.max())))
        for d in range(digits - 1, -1, -1):
            p = 10 ** d
            cols.append(torch.where((x >= p) | (d == 0), x // p % 10 + 48, 0).to(torch.uint8))
        cols.append(torch.full_like(cols[-1], sep))
    text = torch.stack(cols, 1).reshape(-1)
    text[text != 0].cpu().numpy().tofile(path)


def prepare(case, seed):
    kind = case["kind"]
    o = mce.options()
    state = {"kind": kind, "opts": o}
    if kind == "batch":
        state["batch"] = mce.Batch([mce.gen_batch_member(i, (int(seed) + 1) * 10007)[:2] for i in range(case["graphs"])], o)
        return state
    if kind == "serve":
        state["server"] = mce.Server()
        state["requests"] = _requests(case, seed)
        return state
    u, v = _pairs(case, seed)
    if kind in ("solve", "roots"):
        state["graph"] = mce.Graph.from_coo(u, v, o)
        if kind == "roots":
            state["roots"] = _sample(case, state["graph"].info()["num_edges"], BAND[0], BAND[1], seed)
        return state
    if kind in ("build", "text"):
        with mce.Graph.from_coo(u, v, o) as g:
            state["roots"] = _sample(case, g.info()["num_edges"], 0.0, LIGHT, seed)
    if kind == "text":
        state["dir"] = tempfile.TemporaryDirectory(prefix="rdmce_cases_")
        state["path"] = os.path.join(state["dir"].name, "graph.txt")
        _write_text(u, v, state["path"])
    elif kind == "build":
        state["u"], state["v"] = _pinned(u), _pinned(v)
    else:
        state["u"], state["v"] = u, v
    return state


def _signed(x):
    return np.asarray(x, np.uint64).view(np.int64)


def _out(count, checksum, hist):
    """Count, checksum and the number of cliques of every size."""
    bins = np.zeros(mce.HIST_LEN, np.int64)
    bins[list(hist)] = list(hist.values())
    return {"count": _signed([count]), "checksum": _signed([checksum]), "hist": bins}


def _result(r):
    return dict(_out(r.count, r.checksum, r.hist), vertices=r.num_vertices, edges=r.num_edges,
                degeneracy=r.degeneracy, max_degree=r.max_degree)


def run(state):
    kind, o = state["kind"], state["opts"]
    if kind == "solve":
        return _result(state["graph"].solve(o))
    if kind == "roots":
        return _result(state["graph"].solve_root_list(state["roots"], o))
    if kind == "coo":
        return _result(mce.solve_coo(state["u"], state["v"], o))
    if kind == "build":
        with mce.Graph.from_coo(state["u"], state["v"], o) as g:
            return _result(g.solve_root_list(state["roots"], o))
    if kind == "text":
        with mce.Graph.load_file(state["path"], o) as g:
            return _result(g.solve_root_list(state["roots"], o))
    if kind == "batch":
        graphs, hist, _ms = state["batch"].solve(o)
        keys = ("count", "checksum", "max_size", "num_vertices", "num_edges")
        return dict({k: _signed([g[k] for g in graphs]) for k in keys}, hist=_signed(hist))
    server = state["server"]
    ids = [server.submit(u, v) for u, v in state["requests"]]
    server.drain()
    results = [server.poll(i)[0] for i in ids]
    return {"count": _signed([r.count for r in results]), "checksum": _signed([r.checksum for r in results]),
            "hist": np.stack([_out(0, 0, r.hist)["hist"] for r in results])}


def _expected_pairs(case):
    if case["kind"] == "batch":  # n log-uniform in [64, 4096], mean degree uniform in [8, 64]
        return case["graphs"] * 17800
    if case["kind"] == "serve":  # 2^10 to 2^13 vertices, 20 edges each
        return case["requests"] * 3840 * 20
    if case["family"] == "rmat":
        return case["ef"] << case["scale"]
    if case["family"] == "planted":
        lo, hi = case["lo"], case["hi"]
        return 6 * case["n"] + case["cliques"] * sum(s * (s - 1) // 2 for s in range(lo, hi + 1)) // (hi - lo + 1)
    return int(case["n"] * case["degree"] / 2)


def work(case):
    """The graph read once: 8 bytes a pair where pairs come in, 8 bytes an edge
    of the CSR (both directions); a line of text is two labels of up to six
    digits with their separators.  A sample of roots reads its own ego
    networks, some hundreds of neighbours for each of some hundreds of members
    in the core band.  Written: the histogram."""
    pairs, out = _expected_pairs(case), 65536
    if case["kind"] == "roots":
        return {"bytes": case["roots"] * 300 * 300 * 4 + out, "flops": 0}
    if case["kind"] == "text":
        return {"bytes": pairs * 14 + 8 * pairs + out, "flops": 0}
    if case["kind"] in ("coo", "build", "serve"):
        return {"bytes": 16 * pairs + out, "flops": 0}
    return {"bytes": 8 * pairs + out, "flops": 0}


# ------------------------------------------------ plain answers, on the CPU

M64 = (1 << 64) - 1
GOLDEN = 0x9E3779B97F4A7C15


def _mix(x):
    """The SplitMix64 output function."""
    x = (x + GOLDEN) & M64
    x = ((x ^ (x >> 30)) * 0xBF58476D1CE4E5B9) & M64
    x = ((x ^ (x >> 27)) * 0x94D049BB133111EB) & M64
    return x ^ (x >> 31)


def _cliques(u, v):
    """Every maximal clique of the simple graph, as lists of labels, and the graph's figures."""
    adj = {}
    for a, b in zip(u.tolist(), v.tolist()):
        if a != b:
            adj.setdefault(a, set()).add(b)
            adj.setdefault(b, set()).add(a)
    degree = {x: len(s) for x, s in adj.items()}
    buckets = [set() for _ in range(max(degree.values(), default=0) + 1)]
    for x, d in degree.items():
        buckets[d].add(x)
    rank, k, degeneracy = {}, 0, 0
    while len(rank) < len(adj):
        k = next(i for i in range(max(k - 1, 0), len(buckets)) if buckets[i])
        degeneracy = max(degeneracy, k)
        x = buckets[k].pop()
        rank[x] = len(rank)
        for y in adj[x]:
            if y not in rank:
                buckets[degree[y]].discard(y)
                degree[y] -= 1
                buckets[degree[y]].add(y)
    found = []

    def expand(r, p, x):
        if not p:
            if not x:
                found.append(r)
            return
        pivot = max(p | x, key=lambda y: len(adj[y] & p))
        for y in list(p - adj[pivot]):
            expand(r + [y], p & adj[y], x & adj[y])
            p = p - {y}
            x = x | {y}

    for y in sorted(adj, key=rank.get):
        later = {z for z in adj[y] if rank[z] > rank[y]}
        expand([y], later, adj[y] - later)
    edges = sum(len(s) for s in adj.values()) // 2
    return found, (len(adj), edges, degeneracy, max((len(s) for s in adj.values()), default=0))


def exact(case, seed):
    """What run() returns, by a plain search over Python sets where that takes seconds."""
    if case["kind"] not in ("solve", "coo") or case["family"] == "planted" or _expected_pairs(case) > 90000:
        return None
    if case["family"] == "rmat" and case["scale"] * case["ef"] > 140:
        return None
    found, (n, m, degeneracy, max_degree) = _cliques(*_pairs(case, seed))
    labels = {x for c in found for x in c}
    h1 = {x: _mix(x) for x in labels}
    h2 = {x: _mix(x ^ GOLDEN) for x in labels}
    checksum, hist = 0, {}
    for c in found:
        s1, s2 = sum(h1[x] for x in c) & M64, sum(h2[x] for x in c) & M64
        rot = ((s2 << 31) | (s2 >> 33)) & M64
        checksum += _mix(s1 ^ rot ^ ((len(c) << 56) & M64))
        hist[len(c)] = hist.get(len(c), 0) + 1
    return dict(_out(len(found), checksum & M64, hist), vertices=n, edges=m, degeneracy=degeneracy,
                max_degree=max_degree)
