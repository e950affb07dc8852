"""The wide-batch searches (16 or 32 sources a job, teams of CTAs) against the oracle.

Plain runs go there on graphs of mean degree 6 and up that are not small (a
large component beside them makes the small ones here large enough).
The cases sit at the edges of its work split: vertices of 31 to 33, 64, 256
and several thousand entries (four lanes, a warp, chunks), vertex counts
around 32-vertex words, 1 to 65 roots (one job of 16 to several of 32), several components, every
pruning mode, directed lists, counts of 2^28 and more (the 32-bit rows do not
hold them), counts past 2^64 and searches of more than 62 levels (both leave
the kernel: the run is redone).  The bar is the suite's 1e-9; path counts are
exact, so only the order of FP64 sums differs."""
import numpy as np
import pytest

import bcg
import oracle
from test_gpu_parity import assert_bc_close

pytestmark = pytest.mark.gpu
WIDE = (16, 32)  # sources of a job


def _rows(n, degrees, seed):
    """Vertices 0, 1, ... with the given numbers of random neighbours, among n."""
    rng = np.random.default_rng(seed)
    pairs = [np.stack([np.full(d, v), rng.choice(n, size=d, replace=False)], 1) for v, d in enumerate(degrees)]
    fill = rng.integers(0, n, (4 * n, 2))
    return bcg.from_pairs(np.concatenate(pairs + [fill]), n)


def _beside(offs, adj, undirected=True):
    """The graph (vertices 0 .. n - 1) and a random component of 20,000 vertices."""
    n = len(offs) - 1
    own = np.stack([np.repeat(np.arange(n), np.diff(offs.astype(np.int64))), adj], 1)
    far = np.random.default_rng(31).integers(n, n + 20000, (130000, 2))
    return bcg.from_pairs(np.concatenate([own, far]), n + 20000, undirected=undirected)


GRAPHS = {
    "degrees": lambda: _beside(*_rows(5000, [4000, 3000, 1025, 1024, 513, 512, 300, 257, 256, 255, 129, 128, 65, 64, 63, 33, 32, 31, 1], 3)),
    "word31": lambda: _beside(*bcg.generate("er:scale=5,ef=6,seed=8")),
    "word33": lambda: _beside(*_rows(33, [30, 20], 4)),
    "rmat13": lambda: bcg.generate("rmat:scale=13,ef=16,a=0.57,b=0.19,c=0.19,seed=3"),
    "pendants": lambda: _beside(*bcg.generate("rmat:scale=11,ef=16,seed=9,pendant_frac=0.1,pendant_mean=4")),
    "er15": lambda: bcg.generate("er:scale=15,ef=12,seed=6"),
}


@pytest.fixture(scope="module")
def graphs():
    return {k: f() for k, f in GRAPHS.items()}


@pytest.mark.parametrize("flags", [0, bcg.PRUNE_DEGREE1, bcg.PRUNE_TREES])
@pytest.mark.parametrize("gname", list(GRAPHS))
def test_matches_oracle(graphs, gname, flags):
    offs, adj = graphs[gname]
    n = len(offs) - 1
    live = np.nonzero(np.diff(offs))[0].astype(np.uint32)
    for k in (1, 4, 16, 17, 33, 65):
        src = live[np.linspace(0, len(live) - 1, min(k, len(live))).astype(int)]
        ref, ost = oracle.bc(offs, adj, src, nthreads=oracle.max_threads())
        with bcg.Graph(offs, adj, flags) as G:
            st = G.run(src)
            got = G.bc()
            G.run(src)
            twice = G.bc()
        assert flags or st.batch_width in WIDE
        assert_bc_close(got, ref, f"{gname} k={k} flags={flags}")
        assert_bc_close(twice, 2 * ref, f"{gname} k={k} flags={flags} accumulated")
        assert st.teps_edges == ost["teps_edges"] and st.skipped == ost["skipped"]
        assert flags or (st.max_depth == ost["max_depth"] and st.visited == ost["visited"])


def test_all_sources_many_teams(graphs):
    """More jobs than CTAs: a team is one CTA and draws job after job."""
    offs, adj = graphs["rmat13"]
    src = np.arange(len(offs) - 1, dtype=np.uint32)
    ref, _ = oracle.bc(offs, adj, src, nthreads=oracle.max_threads())
    with bcg.Graph(offs, adj) as G:
        G.run(src)
        first = G.bc()
        G.reset()
        G.run(src)
        assert np.array_equal(first.view(np.uint64), G.bc().view(np.uint64))
    assert_bc_close(first, ref, "rmat13 all sources")


def test_directed():
    rng = np.random.default_rng(12)
    n = 3000
    hub = np.stack([np.zeros(2000, int), rng.choice(np.arange(1, n), 2000, replace=False)], 1)
    into = np.stack([rng.choice(np.arange(2, n), 700, replace=False), np.ones(700, int)], 1)
    offs, adj = bcg.from_pairs(np.concatenate([rng.integers(0, n, (40000, 2)), hub, into]), n, undirected=False)
    offs, adj = _beside(offs, adj, undirected=False)
    src = bcg.sample_sources(n, 100, 1)
    ref, ost = oracle.bc(offs, adj, src)
    with bcg.Graph(offs, adj, bcg.DIRECTED) as G:
        st = G.run(src)
        assert st.batch_width in WIDE
        assert_bc_close(G.bc(), ref, "directed")


def _layers(width, depth):
    """Complete bipartite layers: width^i paths to layer i + 1."""
    ids = np.arange(width * depth).reshape(depth, width)
    pairs = [np.stack(np.meshgrid(ids[i], ids[i + 1]), -1).reshape(-1, 2) for i in range(depth - 1)]
    return bcg.from_pairs(np.concatenate(pairs), width * depth)


@pytest.mark.parametrize("depth,ext", [(9, 0), (12, 0), (15, 0), (30, 1)])
def test_large_counts(depth, ext):
    """16 paths more a layer: 2^28 is passed from depth 9 on, 2^64 at 18."""
    offs, adj = _beside(*_layers(16, depth))
    src = np.arange(0, 16 * depth, 3, dtype=np.uint32)
    ref, _ = oracle.bc_q(offs, adj, src)
    with bcg.Graph(offs, adj) as G:
        st = G.run(src)
        assert st.extended_sigma == ext and (ext or st.batch_width in WIDE)
        assert_bc_close(G.bc(), ref, f"layers {depth}")


def test_deep_search_leaves():
    """Mean degree above 6, 120 levels: the run is redone by the sweep kernel,
    and what was in bc before stays."""
    offs, adj = _beside(*_layers(4, 120))
    src = np.arange(0, 480, 30, dtype=np.uint32)
    ref, _ = oracle.bc_q(offs, adj, src)
    with bcg.Graph(offs, adj) as G:
        st = G.run(src)
        assert st.max_depth > 62 and st.batch_width not in WIDE
        assert_bc_close(G.bc(), ref, "deep")
        G.run(src)
        assert_bc_close(G.bc(), 2 * ref, "deep twice")


def test_batch_of_shallow_graphs():
    """A set that runs as wide searches: one to several jobs a graph, graphs of
    one sorting block and of several, with an edgeless one, twice in a row."""
    specs = ["rmat:scale=12,ef=16,a=0.57,b=0.19,c=0.19,seed=5", "er:scale=8,ef=8,seed=6", "er:scale=6,ef=6,seed=9",
             "rmat:scale=9,ef=16,seed=11"]
    graphs = [bcg.generate(s) for s in specs]
    graphs += [bcg.from_pairs([[0, 1], [1, 2], [2, 3]], 5), (np.zeros(4, np.uint32), np.zeros(0, np.uint32))]
    with bcg.Batch(graphs) as B:
        for runs in (1, 2):
            st = B.run()
            assert st.batch_width in WIDE and B.info()["captured"]
            edges = 0
            for i, (offs, adj) in enumerate(graphs):
                ref, ost = oracle.bc(offs, adj, np.arange(len(offs) - 1), nthreads=oracle.max_threads())
                assert_bc_close(B.bc(i), runs * ref, f"graph {i}")
                edges += ost["teps_edges"]
            assert st.teps_edges == edges


def _cliques(size, count):
    """Cliques in a row, neighbours joined by one edge: deep, one path a pair."""
    pairs = []
    for c in range(count):
        b = c * size
        pairs += [[b + i, b + j] for i in range(size) for j in range(i)]
        if c:
            pairs.append([b - 1, b])
    return bcg.from_pairs(pairs, size * count)


def test_batch_with_a_deep_graph():
    """One graph of mean degree 7 and more than 62 levels: the packed schedule runs the set."""
    graphs = [bcg.generate("er:scale=8,ef=8,seed=6"), _cliques(8, 60)]
    with bcg.Batch(graphs) as B:
        for runs in (1, 2):
            st = B.run()
            assert st.batch_width not in WIDE and st.max_depth > 62
            for i, (offs, adj) in enumerate(graphs):
                ref, _ = oracle.bc(offs, adj, np.arange(len(offs) - 1), nthreads=oracle.max_threads())
                assert_bc_close(B.bc(i), runs * ref, f"graph {i}")


def _served(pool, reqs, wave_batches=4):
    out = {}
    with bcg.Server(pool, 8 << 30, wave_batches) as S:
        ids = [S.submit(g, src) for g, src in reqs]
        while len(out) < len(ids):
            for rid in S.wait():
                out[rid] = S.result(rid)
    return [out[i] for i in ids]


@pytest.mark.parametrize("deep", [False, True])
def test_served_waves(deep):
    """Requests of one source to all, cut into several waves of 4 jobs a graph,
    on graphs of unlike size (several launches a wave): against the oracle, and
    bit for bit alone.  With a deep graph in the pool a wave stops, is taken
    back and runs in packed waves, and nothing is added twice."""
    pool = [bcg.generate("rmat:scale=12,ef=16,a=0.57,b=0.19,c=0.19,seed=5"), bcg.generate("er:scale=8,ef=8,seed=6"),
            bcg.generate("er:scale=6,ef=6,seed=9")]
    if deep:
        pool.append(_cliques(8, 60))
    rng = np.random.default_rng(2)
    reqs = [(1, None), (0, np.array([5], dtype=np.uint32)), (2, None), (0, bcg.sample_sources(4096, 300, 3))]
    reqs += [(int(g), np.sort(rng.choice(60, size=int(rng.integers(1, 60)), replace=False)).astype(np.uint32))
             for g in rng.integers(0, len(pool), 8)]
    if deep:
        reqs.insert(3, (3, None))
    served = _served(pool, reqs)
    for i, (g, src) in enumerate(reqs):
        offs, adj = pool[g]
        s = np.arange(len(offs) - 1, dtype=np.uint32) if src is None else src
        ref, _ = oracle.bc(offs, adj, s, nthreads=oracle.max_threads())
        assert_bc_close(served[i], ref, f"request {i}")
    if not deep:
        for i in (0, 3, 6):
            assert np.array_equal(served[i].view(np.uint64), _served(pool, [reqs[i]])[0].view(np.uint64)), i


@pytest.mark.parametrize("n", [524287, 524288, 2000003])
@pytest.mark.parametrize("shift", [0, 1, 511])
def test_large_result_into_fresh_and_odd_buffers(n, shift):
    """Results from about 4 MB on, at any 8-byte place of a fresh buffer or of
    one in use: the same values, and nothing beside them."""
    offs, adj = bcg.from_pairs([[i, i + 1] for i in range(50)] + [[n - 2, n - 1], [n - 3, n - 2]], n)
    with bcg.Graph(offs, adj) as G:
        G.run([0, 20, n - 1])
        want = np.zeros(n)
        want[1:50] = 49.0 - np.arange(49)  # from vertex 0
        want[1:20] += np.arange(1, 20)     # from vertex 20
        want[21:50] += 49.0 - np.arange(20, 49)
        want[n - 2] = 1.0
        for fill in (0.0, 3.5):
            buf = np.zeros(n + 1024) if fill == 0.0 else np.full(n + 1024, fill)
            out = buf[shift:shift + n]
            assert bcg.lib().bcg_get_bc(G.h, out.ctypes.data_as(bcg._f64p)) == 0
            assert np.array_equal(out, want)
            assert np.all(buf[:shift] == fill) and np.all(buf[shift + n:] == fill)


@pytest.mark.parametrize("k", [1, 31, 33, 300, 8191, 8192, 8193, 20000])
def test_sources_out_of_order(k):
    """Jobs take their sources in an order of their own: weights and totals
    must follow.  Repeated sources (weights above 1), sources without an edge,
    one and several windows of 8,192, against the same sources one by one in
    the totals and the oracle in the values."""
    offs, adj = bcg.generate("rmat:scale=15,ef=8,seed=9")
    n = len(offs) - 1
    rng = np.random.default_rng(k)
    src = rng.permutation(n)[:k].astype(np.uint32)
    if k > 32:
        src[::7] = src[1]
    few = min(k, 40)
    ref, ost = oracle.bc_q(offs, adj, src[:few])
    with bcg.Graph(offs, adj) as G:
        G.run(src[:few])
        assert_bc_close(G.bc(), ref, f"first {few}")
        G.reset()
        st = G.run(src)
        whole = G.bc()
        G.reset()
        parts = [G.run(p) for p in np.array_split(src, max(1, k // 1000))]  # other jobs, other companions
        assert_bc_close(whole, G.bc(), f"k={k}")
        assert st.teps_edges == sum(p.teps_edges for p in parts) and st.skipped == sum(p.skipped for p in parts)


@pytest.mark.parametrize("nsrc", [1, 16, 33])
def test_sums_over_level_one(nsrc):
    """Vertices with 1 to 4,500 neighbours next to a source, whose counts are added bit by bit: a lane of four or of 32
    takes up to 64 of them, at the edges of a block, of a light vertex, a warp's and a chunk."""
    mids = 4600
    sinks = [1, 2, 3, 4, 5, 15, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 511, 512, 513, 2047, 2048, 2049, 4500]
    pairs = [np.stack([np.zeros(mids, int), np.arange(1, mids + 1)], 1)]
    for i, k in enumerate(sinks):
        pairs.append(np.stack([np.full(k, mids + 1 + i), np.arange(1, k + 1)], 1))
    offs, adj = _beside(*bcg.from_pairs(np.concatenate(pairs), mids + 1 + len(sinks)))
    src = np.concatenate([[0], np.arange(mids + len(sinks), mids + len(sinks) + 1 - nsrc, -1)]).astype(np.uint32)
    ref, ost = oracle.bc(offs, adj, src)
    with bcg.Graph(offs, adj) as G:
        st = G.run(src)
        assert st.batch_width in WIDE and st.visited == ost["visited"]
        assert_bc_close(G.bc(), ref, f"{nsrc} sources")


@pytest.mark.parametrize("repeats", [0, 1])
def test_lists_that_name_a_neighbour_twice(repeats):
    """A source's list with a repeated neighbour: a count of 2 at level 1, which no bit holds."""
    rng = np.random.default_rng(5)
    n = 30000
    pairs = np.concatenate([rng.integers(0, n, (300000, 2))] + [np.stack([np.zeros(900, int), rng.integers(1, 400, 900)], 1)] * repeats)
    key = pairs[:, 0] * n + pairs[:, 1]
    pairs = pairs[np.argsort(pairs[:, 0], kind="stable")] if repeats else pairs[np.unique(key, return_index=True)[1]]
    pairs = pairs[np.argsort(pairs[:, 0], kind="stable")]
    offs = np.zeros(n + 1, dtype=np.uint32)
    np.cumsum(np.bincount(pairs[:, 0], minlength=n), out=offs[1:])
    adj = pairs[:, 1].astype(np.uint32)
    src = np.arange(0, 40, dtype=np.uint32)
    with bcg.Graph(offs, adj, bcg.DIRECTED) as G:
        G.set_batch_width(6)
        a = G.run(src)
        want = G.bc()
        G.reset()
        G.set_batch_width(0)
        b = G.run(src)
        got = G.bc()
    assert a.batch_width == 6 and b.batch_width in WIDE
    assert a.teps_edges == b.teps_edges and a.visited == b.visited and a.max_depth == b.max_depth
    assert_bc_close(got, want, "repeated neighbours")
