"""The calls whose speed is followed: betweenness centrality through the public entry points of ck-bc_b200/bcg.py.

A case is a plain dict. "kind" names the entry point, the rest is the seeded graph and the sources:

  run      a resident Graph: reset, run over k sources (k = 0: every vertex), bc to the host
  oneshot  bc_csr: host CSR in, bc out (upload, preparation, search, download)
  noalloc  bc_noalloc: CSR and sources already on the device, bc into the caller's device buffer
  batch    Batch: exact bc of many small graphs in one call
  serve    Server: a mix of exact and k-source requests on a resident pool, all queued at once

Graphs are R-MAT (0.57, 0.19, 0.19, 0.05), Erdos-Renyi G(n, M) and 4-neighbour grids with 5 % of the edges dropped,
as the repository's workloads use them, optionally with random recursive trees hung on 10 % of the vertices. They are
built here with torch from the case and the seed, so that exact() needs nothing of the package.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.abspath("ck-bc_b200"))
import bcg  # noqa: E402

PRUNE = {"none": 0, "layer": bcg.PRUNE_DEGREE1, "trees": bcg.PRUNE_TREES}


def listed():
    return [
        # one query against a small resident graph: latency of a single search
        {"name": "one_source_rmat1k", "kind": "run", "graph": "rmat", "n": 1024, "ef": 16, "k": 1, "prune": "none"},
        # a library call inside another framework's step, its memory owned by that framework
        {"name": "noalloc_rmat4k_k100", "kind": "noalloc", "graph": "rmat", "n": 4000, "ef": 16, "k": 100},
        # exact bc of a small graph, the reference program's own test size, with its -H 1
        {"name": "exact_rmat4k_layer", "kind": "run", "graph": "rmat", "n": 4096, "ef": 16, "k": 0, "prune": "layer"},
        # a command-line user's call: edge list in host memory, 64 sampled sources, one layer of pruning
        {"name": "oneshot_rmat50k_k64", "kind": "oneshot", "graph": "rmat", "n": 50000, "ef": 16, "k": 64, "prune": "layer"},
        # directed input (bc2d -U): push sweeps only
        {"name": "directed_rmat64k_k48", "kind": "run", "graph": "rmat", "n": 65536, "ef": 16, "k": 48, "prune": "none",
         "directed": True},
        # approximate bc of a mid-size social-network-like graph, not pruned: the serving pool's middle
        {"name": "sampled_rmat260k_k255", "kind": "run", "graph": "rmat", "n": 262144, "ef": 16, "k": 255, "prune": "none"},
        # the benchmark's graph and mode at a quarter of its sources
        {"name": "sampled_rmat1m_trees", "kind": "run", "graph": "rmat", "n": 1048576, "ef": 16, "k": 1024, "prune": "trees",
         "pendants": True},
        # the serving pool's largest graph: state far beyond L2
        {"name": "sampled_rmat4m_k24", "kind": "run", "graph": "rmat", "n": 4194304, "ef": 16, "k": 24, "prune": "none"},
        # the road-network stand-in: thousands of levels, path counts beyond any integer
        {"name": "grid2048_extended_k6", "kind": "run", "graph": "grid", "n": 2048 * 2048, "w": 2048, "k": 6, "prune": "none",
         "sigma": "extended"},
        # a smaller mesh with nothing set: counts overflow uint64 and the run is redone by itself
        {"name": "grid300_auto_k24", "kind": "run", "graph": "grid", "n": 300 * 290, "w": 300, "k": 24, "prune": "layer"},
        # many small independent graphs, R-MAT and Erdos-Renyi alternating
        {"name": "batch_48_graphs", "kind": "batch", "graphs": 48, "nmin": 250, "nmax": 2500},
        # a queue of requests on a resident pool: half exact, half sampled
        {"name": "serve_24_requests", "kind": "serve", "graphs": 10, "nmin": 1000, "nmax": 30000, "requests": 24,
         "exact_to": 2500},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "run", "run", "run", "oneshot", "noalloc", "grid", "grid", "directed", "exact", "batch", "serve"])
    if kind == "batch":
        return {"kind": "batch", "graphs": rng.randint(6, 48), "nmin": _log(rng, 60, 400), "nmax": _log(rng, 500, 2500)}
    if kind == "serve":
        return {"kind": "serve", "graphs": rng.randint(3, 10), "nmin": _log(rng, 300, 2000), "nmax": _log(rng, 2500, 20000),
                "requests": rng.randint(3, 16), "exact_to": rng.randint(500, 1500)}
    if kind == "noalloc":
        return {"kind": "noalloc", "graph": rng.choice(["rmat", "er"]), "n": _log(rng, 100, 20000), "ef": rng.randint(8, 20),
                "k": _log(rng, 1, 500)}
    if kind == "grid":
        w, h = _log(rng, 40, 2048), _log(rng, 40, 2048)
        # levels cost time one by one, whatever they hold: fewer sources on the larger grids
        k = _log(rng, 1, max(1, min(48, 3 * 4096 // (w + h))))
        return {"kind": "run", "graph": "grid", "n": w * h, "w": w, "k": k, "prune": rng.choice(["none", "layer"]),
                "sigma": "extended"}
    if kind == "exact":
        return {"kind": "run", "graph": rng.choice(["rmat", "er"]), "n": _log(rng, 200, 4096), "ef": rng.randint(8, 24), "k": 0,
                "prune": rng.choice(["none", "layer", "trees"])}
    if kind == "directed":
        return {"kind": "run", "graph": rng.choice(["rmat", "er"]), "n": _log(rng, 1000, 100000), "ef": rng.randint(8, 16),
                "k": _log(rng, 1, 48), "prune": "none", "directed": True}
    n, ef = _log(rng, 1000, 1048576), rng.randint(8, 20)
    if kind == "oneshot":
        n = min(n, 400000)
    k = max(1, min(_log(rng, 1, 1024), int(1.2e10 / (n * ef))))
    c = {"kind": kind, "graph": rng.choice(["rmat", "rmat", "er"]), "n": n, "ef": ef, "k": k,
         "prune": rng.choice(["none", "layer", "trees"])}
    if rng.random() < 0.5:
        c["pendants"] = True
    return c


# ---- seeded graphs: (offsets, adjacency) as int64 tensors on the GPU, lists sorted, no loops, no duplicates

def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed & 0x7FFFFFFFFFFF)


def _csr(u, v, n, mirror=True):
    keep = u != v
    u, v = u[keep], v[keep]
    key = torch.cat([u * n + v, v * n + u]) if mirror else u * n + v
    key = torch.unique(key)
    row = torch.div(key, n, rounding_mode="floor")
    offs = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    offs[1:] = torch.cumsum(torch.bincount(row, minlength=n), 0)
    return offs, key - row * n


def _endpoints(graph, n, m, g):
    if graph == "er":
        return (torch.randint(0, n, (m,), generator=g, device="cuda"), torch.randint(0, n, (m,), generator=g, device="cuda"))
    u = torch.zeros(m, dtype=torch.int64, device="cuda")
    v = torch.zeros(m, dtype=torch.int64, device="cuda")
    for _ in range(max(1, (n - 1).bit_length())):
        r = torch.rand(m, generator=g, device="cuda")
        down = r >= 0.76
        u = u * 2 + down
        v = v * 2 + (((r >= 0.57) & ~down) | (r >= 0.95))
    inside = (u < n) & (v < n)
    return u[inside], v[inside]


def _pendants(u, v, n, g):
    """Random recursive trees on a tenth of the vertices, mean size 4: geometric sizes given their sum."""
    anchors = torch.randperm(n, generator=g, device="cuda")[: max(1, n // 10)]
    total = 4 * len(anchors)
    cuts = torch.sort(torch.randperm(total - 1, generator=g, device="cuda")[: len(anchors) - 1]).values + 1
    size = torch.diff(cuts, prepend=cuts.new_zeros(1), append=cuts.new_full((1,), total))
    first = n + torch.cumsum(size, 0) - size
    tree = torch.repeat_interleave(torch.arange(len(anchors), device="cuda"), size)
    new = n + torch.arange(total, device="cuda")
    j = new - first[tree]  # the tree's j-th new vertex hangs on one of the j + 1 before it
    p = torch.floor(torch.rand(total, generator=g, device="cuda", dtype=torch.float64) * (j + 1)).to(torch.int64)
    parent = torch.where(p == 0, anchors[tree], first[tree] + p - 1)
    return torch.cat([u, parent]), torch.cat([v, new]), n + total


def _grid(w, h, g):
    at = torch.arange(w * h, device="cuda").reshape(h, w)
    u = torch.cat([at[:, :-1].reshape(-1), at[:-1].reshape(-1)])
    v = torch.cat([at[:, 1:].reshape(-1), at[1:].reshape(-1)])
    keep = torch.rand(len(u), generator=g, device="cuda") >= 0.05
    return u[keep], v[keep]


def _graph(c, seed):
    g = _generator(seed)
    n = c["n"]
    if c["graph"] == "grid":
        u, v = _grid(c["w"], n // c["w"], g)
    else:
        u, v = _endpoints(c["graph"], n, c["ef"] * n, g)
    if c.get("pendants"):
        u, v, n = _pendants(u, v, n, g)
    return _csr(u, v, n, not c.get("directed"))


def _sources(k, offs, seed):
    """k distinct vertices drawn uniformly (0: every vertex), as a uint32 array; a few sources from those with an edge."""
    n = len(offs) - 1
    if k == 0:
        return np.arange(n, dtype=np.uint32)
    rng = np.random.Generator(np.random.PCG64(seed + 77))
    among = torch.nonzero(offs[1:] > offs[:-1]).reshape(-1).cpu().numpy() if k < 8 else n
    return np.sort(rng.choice(among, size=min(k, n), replace=False)).astype(np.uint32)


def _host(t):
    return t.to(torch.int32).cpu().numpy().view(np.uint32)


def _pool(c, seed):
    """The graphs of a batch or a serving pool: sizes spread over their logarithm, kinds alternating."""
    rng = np.random.Generator(np.random.PCG64(c["graphs"]))  # the sizes are the case's, the edges the seed's
    out = []
    for i in range(c["graphs"]):
        n = int(round(math.exp(rng.uniform(math.log(c["nmin"]), math.log(c["nmax"])))))
        one = {"graph": "rmat" if i % 2 == 0 else "er", "n": n, "ef": int(rng.integers(8, 25))}
        out.append(_graph(one, seed * 1000 + i))
    return out


def _requests(c, seed, sizes):
    """(graph, sources or None for exact): half exact, on graphs of up to exact_to vertices; half of 64 to 1024 sources."""
    rng = np.random.Generator(np.random.PCG64(c["requests"]))
    pick = np.random.Generator(np.random.PCG64(seed + 5))
    small = [i for i, n in enumerate(sizes) if n <= c["exact_to"]]
    reqs = []
    for i in range(c["requests"]):
        if i % 2 == 0 and small:
            reqs.append((int(rng.choice(small)), None))
            continue
        g = int(rng.integers(0, len(sizes)))
        k = min(int(round(math.exp(rng.uniform(math.log(64), math.log(1024))))), sizes[g])
        reqs.append((g, np.sort(pick.choice(sizes[g], size=k, replace=False)).astype(np.uint32)))
    return reqs


# ---- the calls

def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return {"kind": kind, "batch": bcg.Batch([(_host(o), _host(a)) for o, a in _pool(case, seed)])}
    if kind == "serve":
        pool = _pool(case, seed)
        sizes = [len(o) - 1 for o, _ in pool]
        return {"kind": kind, "server": bcg.Server([(_host(o), _host(a)) for o, a in pool], 8 << 30),
                "requests": _requests(case, seed, sizes)}
    offs, adj = _graph(case, seed)
    src = _sources(case["k"], offs, seed)
    if kind == "noalloc":
        as_ids = lambda t: t.to(torch.int32).contiguous()  # noqa: E731
        return {"kind": kind, "offs": as_ids(offs), "adj": as_ids(adj),
                "src": torch.from_numpy(src.view(np.int32)).cuda(),
                "bc": torch.zeros(len(offs) - 1, dtype=torch.float64, device="cuda")}
    flags = PRUNE[case["prune"]] | (bcg.DIRECTED if case.get("directed") else 0)
    offs, adj = _host(offs), _host(adj)
    torch.cuda.empty_cache()  # the generator's scratch is not part of what a user keeps
    if kind == "oneshot":
        return {"kind": kind, "offs": offs, "adj": adj, "src": src, "flags": flags}
    g = bcg.Graph(offs, adj, flags)
    if case.get("sigma") == "extended":
        g.set_sigma_mode(bcg.SIGMA_EXTENDED)
    return {"kind": kind, "graph": g, "src": src}


def run(state):
    kind = state["kind"]
    if kind == "run":
        g = state["graph"]
        g.reset()
        st = g.run(state["src"])
        return {"bc": g.bc(), "teps_edges": int(st.teps_edges), "skipped": int(st.skipped)}
    if kind == "oneshot":
        bc, st = bcg.bc_csr(state["offs"], state["adj"], state["src"], state["flags"])
        return {"bc": bc, "teps_edges": int(st.teps_edges), "skipped": int(st.skipped)}
    if kind == "noalloc":
        s = state
        bcg.bc_noalloc(s["offs"].data_ptr(), s["adj"].data_ptr(), len(s["offs"]) - 1, len(s["adj"]), s["src"].data_ptr(),
                       len(s["src"]), s["bc"].data_ptr(), stream=torch.cuda.current_stream().cuda_stream)
        return {"bc": s["bc"]}
    if kind == "batch":
        b = state["batch"]
        b.reset()
        st = b.run()
        return {"bc": [b.bc(i) for i in range(len(b.sizes))], "teps_edges": int(st.teps_edges)}
    server = state["server"]
    ids = [server.submit(g, src) for g, src in state["requests"]]
    out = {}
    while len(out) < len(ids):
        for rid in server.wait():
            out[rid] = server.result(rid)
    return {"bc": [out[i] for i in ids]}


def work(case):
    """The graph read once, bc written once, and two operations (a path-count add and a dependency add) per adjacency
    entry and source. Entries are counted as drawn (duplicates and loops, some per cent, still among them)."""
    kind = case["kind"]
    if kind in ("batch", "serve"):
        mean = math.sqrt(case["nmin"] * case["nmax"])
        n, nnz = case["graphs"] * mean, case["graphs"] * mean * 2 * 16
        if kind == "batch":
            return {"bytes": 12 * n + 4 * nnz, "flops": 2 * nnz * mean}
        return {"bytes": 4 * n + 4 * nnz + 8 * case["requests"] * mean, "flops": 2 * case["requests"] * 256 * mean * 32}
    n = case["n"]
    if case["graph"] == "grid":
        nnz = 2 * 2 * 0.95 * n
    else:
        nnz = (1 if case.get("directed") else 2) * case["ef"] * n
    if case.get("pendants"):
        n, nnz = n + 4 * (n // 10), nnz + 8 * (n // 10)
    k = case["k"] or n
    return {"bytes": 12 * n + 4 * nnz + 4 * k, "flops": 2 * nnz * k}


# ---- the same in 64 bits

def _spmm_bc(offs, adj, src):
    """Brandes over blocks of sources as sparse-matrix times dense-matrix products in float64."""
    n = len(offs) - 1
    deg = offs[1:] - offs[:-1]
    row = torch.repeat_interleave(torch.arange(n, device="cuda"), deg)
    def matrix(o, a):
        return torch.sparse_csr_tensor(o.to(torch.int32), a.to(torch.int32),
                                       torch.ones(len(a), dtype=torch.float64, device="cuda"), size=(n, n))
    out = matrix(offs, adj)
    key = torch.sort(adj * n + row).values  # the transpose: where an undirected graph's lists lead back
    r = torch.div(key, n, rounding_mode="floor")
    toffs = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    toffs[1:] = torch.cumsum(torch.bincount(r, minlength=n), 0)
    into = matrix(toffs, key - r * n)
    del key, r, row, toffs
    src = torch.from_numpy(src.astype(np.int64)).cuda()
    src = src[deg[src] > 0]
    bc = torch.zeros(n, dtype=torch.float64, device="cuda")
    block = max(1, min(512, (1 << 27) // n))
    for i in range(0, len(src), block):
        s = src[i:i + block]
        cols = torch.arange(len(s), device="cuda")
        lvl = torch.full((n, len(s)), -1, dtype=torch.int16, device="cuda")
        sig = torch.zeros(n, len(s), dtype=torch.float64, device="cuda")
        lvl[s, cols] = 0
        sig[s, cols] = 1.0
        d = 0
        while True:
            nxt = into @ torch.where(lvl == d, sig, 0.0)
            fresh = (lvl < 0) & (nxt > 0)
            if not bool(fresh.any()):
                break
            d += 1
            lvl[fresh] = d
            sig = torch.where(fresh, nxt, sig)
        delta = torch.zeros_like(sig)
        for e in range(d - 1, 0, -1):
            x = out @ torch.where(lvl == e + 1, (1.0 + delta) / sig.clamp(min=1.0), 0.0)
            delta = torch.where(lvl == e, sig * x, delta)
        bc += torch.where(lvl > 0, delta, 0.0).sum(1)
    return bc


def _pow2(e):
    return torch.where(e > -1000, (e.clamp(min=-1000) + 1023) << 52, 0).view(torch.float64)


def _norm(m, e):
    """m * 2^e with m back in [1, 2), m > 0."""
    s = (m.view(torch.int64) >> 52) - 1023
    return m * _pow2(-s), e + s


def _grid_bc(offs, adj, src):
    """Brandes on a graph of degree <= 4, all sources level by level together, path counts as float64 times 2^int64."""
    n = len(offs) - 1
    deg = offs[1:] - offs[:-1]
    slot = torch.arange(4, device="cuda")
    has = slot[None, :] < deg[:, None]
    tab = torch.where(has, adj[(offs[:-1, None] + slot[None, :]).clamp(max=len(adj) - 1)], -1)
    src = torch.from_numpy(src.astype(np.int64)).cuda()
    src = src[deg[src] > 0]
    k = len(src)
    lvl = torch.full((k * n + 1,), -1, dtype=torch.int16, device="cuda")  # the last entry stands for "no neighbour"
    lvl[-1] = 32767
    man = torch.zeros(k * n + 1, dtype=torch.float64, device="cuda")
    ex = torch.zeros(k * n + 1, dtype=torch.int64, device="cuda")

    def around(f):
        b = torch.div(f, n, rounding_mode="floor") * n
        t = tab[f - b]
        return torch.where(t >= 0, t + b[:, None], k * n)

    def total(nb, take):
        """The sum over the taken neighbours of man * 2^ex, as (m, e); m = 0 where there is none."""
        e = torch.where(take, ex[nb], -(1 << 40))
        top = e.max(1).values
        return (torch.where(take, man[nb], 0.0) * _pow2(e - top[:, None])).sum(1), top

    f = torch.arange(k, device="cuda") * n + src
    lvl[f], man[f] = 0, 1.0
    levels = [f]
    while True:
        d = len(levels)
        nb = around(levels[-1])
        f = torch.unique(nb[lvl[nb] < 0])
        if len(f) == 0:
            break
        nb = around(f)
        m, e = total(nb, lvl[nb] == d - 1)
        man[f], ex[f] = _norm(m, e)
        lvl[f] = d
        levels.append(f)
    bc = torch.zeros(n, dtype=torch.float64, device="cuda")
    for d in range(len(levels) - 1, 0, -1):
        f = levels[d]
        nb = around(f)
        x, e = total(nb, lvl[nb] == d + 1)
        sm, se = man[f], ex[f]
        delta = sm * x * _pow2(torch.where(x > 0, se + e, -2000).clamp(max=1000))
        bc.index_add_(0, f % n, delta)
        man[f], ex[f] = _norm((1.0 + delta) / sm, -se)
    return bc


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return {"bc": [_spmm_bc(o, a, np.arange(len(o) - 1)).cpu().numpy() for o, a in _pool(case, seed)], "teps_edges": None}
    if kind == "serve":
        pool = _pool(case, seed)
        reqs = _requests(case, seed, [len(o) - 1 for o, _ in pool])
        return {"bc": [_spmm_bc(*pool[g], np.arange(len(pool[g][0]) - 1) if s is None else s).cpu().numpy() for g, s in reqs]}
    offs, adj = _graph(case, seed)
    src = _sources(case["k"], offs, seed)
    bc = (_grid_bc if case["graph"] == "grid" else _spmm_bc)(offs, adj, src)
    if kind == "noalloc":
        return {"bc": bc}
    return {"bc": bc.cpu().numpy(), "teps_edges": None, "skipped": None}
