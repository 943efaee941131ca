"""The queries that a user of libcac sends, as cases that a timing program can prepare, run and compare.

Every pass is one call (or one burst of calls) of the public Python mirror of the C ABI, cac.py: connected components
of a resident graph and of host edge arrays, square_root minimum cuts one by one and in a batch, plain Karger-Stein,
approximate cuts, and a burst of mixed queries to the serving loop. Inputs come from the seed alone. All outputs are
whole numbers (cuts, component counts, labels), so they are compared as they are and `exact` has nothing to add.

A program keeps one context (and one server) and sends it queries on many graphs, so the context is shared by all
states of a process; a state holds the graphs and the label buffer.
"""
import importlib
import math

import numpy as np
import torch

cac = importlib.import_module("comm-avoiding-cuts-cc_gb300.cac")

_kept = {}


def _context():
    if "ctx" not in _kept:
        _kept["ctx"] = cac.Context(0)
    return _kept["ctx"]


def _server():
    if "server" not in _kept:
        _kept["server"] = cac.Server(0, 120 << 30)
    return _kept["server"]


# ---------------------------------------------------------------- the cases

def listed():
    return [
        # the smallest query: components of a graph of some thousand edges, labels into a host array
        {"name": "cc_small", "kind": "cc", "family": "rmat", "scale": 10, "edge_factor": 8, "ranks": 4, "labels": "host"},
        # an ordinary sparse graph of odd size near the threshold of its giant component: thousands of components
        {"name": "cc_sparse", "kind": "cc", "family": "er_m", "n": 300007, "degree": 2.5, "ranks": 16, "labels": "device"},
        # the benchmark's graph: preferential attachment, 16.2 M edges in random order, 16 virtual ranks; one id in a
        # hundred is unused, as in id spaces that users come and go in, so the labels are not all alike
        {"name": "cc_ba_1m", "kind": "cc", "family": "ba", "n": 1024000, "k": 16, "ranks": 16, "labels": "device"},
        # the largest graph: R-MAT scale 22, edge factor 16, isolated vertices kept
        {"name": "cc_rmat_22", "kind": "cc", "family": "rmat", "scale": 22, "edge_factor": 16, "ranks": 16, "labels": "device"},
        # one call from pinned host edges to host labels on the benchmark's graph
        {"name": "cc_host_ba", "kind": "cc_host", "family": "ba", "n": 1024000, "k": 16, "ranks": 16},
        # square_root on G(1000, 0.05), weights 1..42, 4 virtual ranks: 60 trials of moderate size
        {"name": "sr_er_1000", "kind": "cut", "family": "er", "n": 1000, "p": 0.05, "wmax": 42, "success": 0.95, "ranks": 4},
        # square_root on the complete graph with 4000 vertices: few trials, large matrices
        {"name": "sr_k4000", "kind": "cut", "family": "complete", "n": 4000, "wmax": 42, "success": 0.95, "ranks": 1},
        # a batch of small and middling graphs of uneven sizes, half Watts-Strogatz, half G(n, M)
        {"name": "sr_batch_64", "kind": "batch", "count": 64, "n_lo": 64, "n_hi": 8192, "success": 0.9},
        # plain karger_stein on a sparse small-world graph of 32,000 vertices
        {"name": "ks_ws_32k", "kind": "ks", "n": 32000, "k": 32, "wmax": 100, "success": 0.9},
        # approx_cut on the reference's draws (the command line's default on unit weights), 15 M edges; each case's
        # density is the one where the answer lies between the `level` and the one after it
        {"name": "approx_er_1m", "kind": "approx", "n": 1000000, "level": 1, "wmax": 1, "replay": True, "ranks": 4,
         "success": 0.9, "repeats": 8},
        # approx_cut on a weighted graph of odd size, 1.4 M edges, some more levels
        {"name": "approx_er_100k", "kind": "approx", "n": 100003, "level": 5, "wmax": 42, "replay": False, "ranks": 1,
         "success": 0.9, "repeats": 8},
        # a burst of mixed queries (2:1:1) on resident graphs of 10^3 to 10^5 edges
        {"name": "serve_mix_64", "kind": "serve", "graphs": 16, "m_lo": 1000.0, "m_hi": 100000.0, "queries": 64},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _cc_graph(rng, m_lo, m_hi):
    m = _log(rng, m_lo, m_hi)
    family = rng.choice(["er_m", "rmat", "ba"])
    if family == "er_m":  # below the degree from which on a random graph is connected and all labels are 0
        degree = _log(rng, 1.5, 0.35 * math.log(m))
        return {"family": family, "n": int(2 * m / degree), "degree": degree}
    k = rng.randint(4, 16)
    if family == "rmat":
        return {"family": family, "scale": max(4, int(math.log2(m / k))), "edge_factor": k}
    return {"family": family, "n": max(4 * k, int(m / k)), "k": k}


def draw(rng):
    kind = rng.choice(["cc", "cc", "cc", "cc_host", "cut", "cut", "batch", "ks", "approx", "approx", "serve"])
    if kind == "cc":
        c = _cc_graph(rng, 1e3, 6.7e7)
        c.update(ranks=rng.randint(1, 16), labels=rng.choice(["device", "device", "host"]))
    elif kind == "cc_host":
        c = _cc_graph(rng, 1e4, 2e7)
        c.update(ranks=rng.randint(1, 16))
    elif kind == "cut":
        family = rng.choice(["er", "ws", "complete"])
        c = {"family": family, "wmax": rng.choice([42, 100]), "success": rng.choice([0.9, 0.95]), "ranks": rng.randint(1, 8)}
        if family == "er":
            n = int(_log(rng, 120, 3000))
            c.update(n=n, p=min(0.9, _log(rng, 24, 200) / n))
        elif family == "ws":
            c.update(n=int(_log(rng, 120, 4000)), k=2 * rng.randint(6, 16))
        else:
            c.update(n=int(_log(rng, 129, 4000)))
    elif kind == "batch":
        c = {"count": rng.randint(8, 96), "n_lo": 64, "n_hi": int(_log(rng, 500, 8192)), "success": rng.choice([0.9, 0.95])}
    elif kind == "ks":
        c = {"n": int(_log(rng, 2200, 32000)), "k": 2 * rng.randint(8, 16), "wmax": rng.choice([42, 100]), "success": 0.9}
    elif kind == "approx":
        c = {"n": int(_log(rng, 3e3, 1e6)), "ranks": rng.randint(1, 8), "success": 0.9, "repeats": 8}
        if rng.random() < 0.5:
            c.update(replay=True, wmax=1, level=rng.randint(1, 2) if c["n"] < 5e5 else 1)
        else:
            c.update(replay=False, wmax=42, level=rng.randint(2, 6) if c["n"] < 5e5 else rng.randint(2, 4))
    else:
        c = {"graphs": rng.randint(8, 24), "m_lo": 1000.0, "m_hi": _log(rng, 2e4, 3e5), "queries": rng.randint(24, 96)}
    return dict(c, kind=kind)


# ---------------------------------------------------------------- inputs

def _barabasi_albert(ids, k, seed):
    """Preferential attachment on the GPU, edges in random order: edge e joins vertex k + e // k to the value of a uniform
    earlier slot of the endpoint list (Batagelj & Brandes 2005). A hundredth of the ids, at random, is unused.
    -> (u, v) int32 tensors."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    n = ids - max(2, ids // 100)
    used = torch.randperm(ids, generator=gen, device="cuda")[:n].sort().values
    ne = (n - k) * k
    e = torch.arange(ne, device="cuda")
    src = k + e // k
    slot = (torch.rand(ne, generator=gen, device="cuda", dtype=torch.float64) * (2 * e)).long()
    dst = e % k  # the first k edges attach to the k seed vertices
    todo = e[k:]
    cur = slot[k:]
    while todo.numel():
        owner = cur // 2
        even = cur % 2 == 0
        first = ~even & (owner < k)
        dst[todo[even]] = src[owner[even]]
        dst[todo[first]] = owner[first] % k
        rest = ~even & ~first
        todo, cur = todo[rest], slot[owner[rest]]
    order = torch.randperm(ne, generator=gen, device="cuda")
    return used[src[order]].int(), used[dst[order]].int()


def _spec(c, seed):
    """The arguments of cac's device generators."""
    w = c.get("wmax", 1)
    if c["family"] == "er_m":
        return "erdos_renyi_m", dict(seed=seed, n=c["n"], avg_degree=c["degree"], wmax=w)
    if c["family"] == "er":
        return "erdos_renyi", dict(seed=seed, n=c["n"], p=c["p"], wmax=w)
    if c["family"] == "ws":
        return "watts_strogatz", dict(seed=seed, n=c["n"], k=c["k"], p=0.4, wmax=w)
    if c["family"] == "rmat":
        return "rmat", dict(seed=seed, scale=c["scale"], edge_factor=c["edge_factor"], wmax=w)
    return "complete", dict(seed=seed, n=c["n"], wmax=w)


def _graph(c, seed):
    ctx = _context()
    if c["family"] == "ba":
        u, v = _barabasi_albert(c["n"], c["k"], seed)
        torch.cuda.synchronize()
        return ctx.graph(c["n"], u, v)
    family, args = _spec(c, seed)
    return ctx.generate(family, **args)


def _approx_graph(c):
    """G(n, M) where a vertex is cut off at the level with probability about 1 / (4 n) (4 copies of n vertices are tried): every
    edge of weight w is dropped with probability (1 - 2^-level)^w, g on average."""
    q = 1 - 0.5 ** c["level"]
    g = sum(q ** w for w in range(1, c["wmax"] + 1)) / c["wmax"]
    return dict(c, family="er_m", degree=math.log(4 * c["n"]) / (1 - g))


def _batch_cases(c):
    rng = np.random.default_rng(c["count"])
    for i in range(c["count"]):
        n = int(math.exp(rng.uniform(math.log(c["n_lo"]), math.log(c["n_hi"]))))
        k, degree = 2 * int(rng.integers(3, 17)), float(rng.uniform(8, 64))
        yield {"family": "ws", "n": n, "k": k, "wmax": 100} if i % 2 == 0 else {"family": "er_m", "n": n, "degree": degree, "wmax": 100}


def _served_cases(c):
    rng = np.random.default_rng(c["graphs"])
    for i in range(c["graphs"]):
        m = math.exp(rng.uniform(math.log(c["m_lo"]), math.log(c["m_hi"])))
        if i % 2 == 0:
            n = max(4, int(2 * math.sqrt(m)))
            yield {"family": "er", "n": n, "p": min(1.0, m / (n * (n - 1) / 2)), "wmax": 42}
        else:
            scale = max(2, int(math.log2(2 * math.sqrt(m))))
            yield {"family": "rmat", "scale": scale, "edge_factor": max(1, round(m / (1 << scale))), "wmax": 42}


def prepare(case, seed):
    seed %= 1 << 31
    kind = case["kind"]
    s = {"case": case, "seed": seed}
    if kind == "batch":
        s["graphs"] = [_graph(g, seed + i) for i, g in enumerate(_batch_cases(case))]
        s["seeds"] = list(range(seed, seed + case["count"]))
    elif kind == "serve":
        server = _server()
        s["graphs"] = []
        for i, g in enumerate(_served_cases(case)):
            family, args = _spec(g, seed + i)
            s["graphs"].append(server.generate(family, **args))
        rng = np.random.default_rng(case["queries"])
        kinds = ["square_root", "square_root", "approx_cut", "parallel_cc"]
        s["queries"] = [(kinds[int(rng.integers(4))], int(rng.integers(case["graphs"])), seed + i)
                        for i in range(case["queries"])]
    elif kind == "cc_host":
        if case["family"] == "ba":
            n = case["n"]
            u, v = _barabasi_albert(n, case["k"], seed)
        else:
            g = _graph(case, seed)
            n = g.n
            u, v, _ = (torch.from_numpy(x.view(np.int32)) for x in g.edges())
        s["n"] = n
        s["u"], s["v"] = (torch.empty(x.numel(), dtype=torch.int32, pin_memory=True).copy_(x) for x in (u, v))
        s["labels"] = torch.empty(n, dtype=torch.int32, pin_memory=True)
    elif kind == "ks":
        s["graph"] = _graph(dict(case, family="ws"), seed)
    elif kind == "approx":
        s["graph"] = _graph(_approx_graph(case), seed)
    else:
        s["graph"] = _graph(case, seed)
        if kind == "cc" and case["labels"] == "device":
            s["labels"] = torch.empty(s["graph"].n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    return s


# ---------------------------------------------------------------- one pass

def run(state):
    c, seed = state["case"], state["seed"]
    kind = c["kind"]
    if kind == "cc":
        count, labels, _ = state["graph"].connected_components(seed=seed, virtual_ranks=c["ranks"], out=state.get("labels"))
        return {"count": count, "labels": labels}
    if kind == "cc_host":
        u, v, labels = (state[x].numpy().view(np.uint32) for x in ("u", "v", "labels"))
        r = _context().cc_edges(state["n"], u, v, seed=seed, virtual_ranks=c["ranks"], labels=labels)
        return {"count": r.num_components, "labels": state["labels"]}
    if kind == "cut":
        r = state["graph"].square_root(c["success"], seed=seed, virtual_ranks=c["ranks"])
        return {"cut": r.cut, "trials": r.total_trials}
    if kind == "batch":
        rs = _context().mincut_batch(state["graphs"], c["success"], seeds=state["seeds"])
        return {"cuts": np.array([r.cut for r in rs], np.int64), "trials": np.array([r.total_trials for r in rs], np.int64)}
    if kind == "ks":
        r = state["graph"].karger_stein(c["success"], seed=seed)
        return {"cut": r.cut, "trials": r.total_trials}
    if kind == "approx":  # a factor-O(log n) estimate: repeated over seeds, the median is taken
        rs = [state["graph"].approx_cut(c["success"], seed=seed + i, virtual_ranks=c["ranks"], seed_replay=c["replay"])
              for i in range(c["repeats"])]
        return {"cuts": np.array([r.cut for r in rs], np.int64), "levels": np.array([r.level for r in rs], np.int64)}
    server, graphs = _server(), state["graphs"]
    tickets = [server.submit(k, graphs[g], 0.9, seed=qs, virtual_ranks=1, labels=k == "parallel_cc")
               for k, g, qs in state["queries"]]
    answers, labels = [], []
    for t in tickets:
        r, lab = server.poll(t)
        answers.append((r.cut, r.trials, r.num_components))
        if lab is not None:
            labels.append(lab.astype(np.int64))
    return {"answers": np.array(answers, np.int64), "labels": np.concatenate(labels) if labels else np.zeros(1, np.int64)}


# ---------------------------------------------------------------- what a pass cannot do without

def _edges(c):
    """(n, expected m) of a graph case."""
    f = c.get("family", "ws")
    if f == "er_m":
        return c["n"], c["n"] * c["degree"] / 2
    if f == "er":
        return c["n"], c["p"] * c["n"] * (c["n"] - 1) / 2
    if f == "ws":
        return c["n"], c["n"] * c["k"] / 2
    if f == "rmat":
        return 1 << c["scale"], float(c["edge_factor"] << c["scale"])
    if f == "ba":
        return c["n"], (0.99 * c["n"] - c["k"]) * c["k"]
    return c["n"], c["n"] * (c["n"] - 1) / 2


def _target(n):
    return max(128, math.ceil(n / math.sqrt(2)) + 1)


def _success(n):
    return 1.0 if n <= 128 else 1 - (1 - 0.5 * _success(_target(n))) ** 2


def _recursion(n):
    """Additions of one Karger-Stein trial: every child sums its parent's matrix (half of it, by symmetry); a leaf takes
    one maximum adjacency ordering."""
    ops, nodes = 0.0, 1
    while n > 128:
        nodes *= 2
        ops += nodes * n * n / 2
        n = _target(n)
    return ops + nodes * n * n / 2


def _cut_work(c):
    """(bytes, additions) of one square_root query: its edges once; per trial its edges summed and one recursion."""
    n, m = _edges(c)
    t = min(n, math.ceil(2 * math.sqrt(m) + 1))
    trials = math.ceil(n * n * math.log(1 / (1 - c["success"])) / (4 * m * _success(t)))
    return 12 * m, trials * (m + _recursion(t))


def _cc_work(c):
    n, m = _edges(c)
    return 8 * m + 4 * n


def work(case):
    kind = case["kind"]
    if kind in ("cc", "cc_host"):
        return {"bytes": _cc_work(case), "flops": 0}
    if kind == "cut":
        b, f = _cut_work(case)
    elif kind == "batch":
        parts = [_cut_work(dict(g, success=case["success"])) for g in _batch_cases(case)]
        b, f = sum(p[0] for p in parts), sum(p[1] for p in parts)
    elif kind == "ks":
        n, m = _edges(case)
        one = _success(n)
        b, f = 12 * m, math.ceil(math.log(1 - case["success"]) / math.log(1 - one)) * _recursion(n)
    elif kind == "approx":  # every repeat reads the edges at least once
        b, f = case["repeats"] * 12 * _edges(_approx_graph(case))[1], 0
    else:
        parts = list(_served_cases(case))
        cut = [_cut_work(dict(g, success=0.9)) for g in parts]
        share = case["queries"] / case["graphs"]
        b = share * sum(0.5 * p[0] + 0.25 * 12 * _edges(g)[1] + 0.25 * _cc_work(g) for p, g in zip(cut, parts))
        f = share * 0.5 * sum(p[1] for p in cut)
    return {"bytes": b, "flops": f}


def exact(case, seed):
    """All outputs are whole numbers, compared as they are."""
    return None
