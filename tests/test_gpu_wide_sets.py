"""Batched and serving forms on the wide searches, where a set or pool is unlike the usual one: a single graph, most of
whose vertices have no edge; path counts just below and just past 2^64; graphs with searches too deep for wide waves;
waves whose memory is full; budgets that hold little beside the pool;
loops in the lists.  Against the oracle, within the suite's 1e-9;
what no path passes is exactly 0."""
import numpy as np
import pytest

import bcg
import oracle
from test_gpu_parity import assert_bc_close

pytestmark = pytest.mark.gpu
WIDE = (16, 32)  # sources of a job


def _serve(pool, reqs, budget=8 << 30, wave_batches=64):
    out = {}
    with bcg.Server(pool, budget, wave_batches) as S:
        ids = [S.submit(g, src) for g, src in reqs]
        while len(out) < len(ids):
            for rid in S.wait():
                out[rid] = S.result(rid)
    return [out[i] for i in ids]


def _dirty_pool():
    """Leaves values other than 0 in the memory that the next buffers take."""
    offs, adj = bcg.generate("rmat:scale=17,ef=16,a=0.57,b=0.19,c=0.19,seed=5")
    with bcg.Graph(offs, adj) as G:
        G.run(bcg.sample_sources(len(offs) - 1, 400, 1))


def _sparse(n, active, seed):
    """A random graph on the last `active` of n vertices."""
    pairs = np.random.default_rng(seed).integers(n - active, n, (12 * active, 2))
    return bcg.from_pairs(pairs, n)


ONE = {
    "rmat": lambda: bcg.generate("rmat:scale=12,ef=8,a=0.57,b=0.19,c=0.19,seed=7"),
    "few": lambda: _sparse(60000, 300, 8),
    "none isolated": lambda: _sparse(700, 700, 9),
    "past the bounds' size": lambda: _sparse(70000, 900, 10),
}


@pytest.mark.parametrize("gname", list(ONE))
def test_one_graph(gname):
    """A set or pool of one graph: only its vertices with an edge have a place in a job's vector."""
    offs, adj = ONE[gname]()
    n = len(offs) - 1
    alone = np.diff(offs) == 0
    ref, ost = oracle.bc(offs, adj, np.arange(n, dtype=np.uint32), nthreads=oracle.max_threads())
    _dirty_pool()
    with bcg.Batch([(offs, adj)]) as B:
        for runs in (1, 2):
            st = B.run()
            assert st.batch_width in WIDE and st.teps_edges == ost["teps_edges"]
            got = B.bc(0)
            assert_bc_close(got, runs * ref, f"batch of {gname}")
            assert not np.any(got[alone])
    _dirty_pool()
    k = bcg.sample_sources(n, 200, 4)
    part, _ = oracle.bc(offs, adj, k, nthreads=oracle.max_threads())
    for got, want in zip(_serve([(offs, adj)], [(0, None), (0, k)]), (ref, part)):
        assert_bc_close(got, want, f"served {gname}")
        assert not np.any(got[alone])


def _layers(width, depth):
    """Complete bipartite layers (width^i paths to layer i + 1) and a triangle beside them, which keeps every vertex
    unfinished: no source reaches both."""
    ids = np.arange(width * depth).reshape(depth, width)
    pairs = [np.stack(np.meshgrid(ids[i], ids[i + 1]), -1).reshape(-1, 2) for i in range(depth - 1)]
    b = width * depth
    return bcg.from_pairs(np.concatenate(pairs + [[[b, b + 1], [b + 1, b + 2], [b + 2, b]]]), b + 3)


def _noalloc(offs, adj, src):
    torch = pytest.importorskip("torch")
    n = len(offs) - 1
    o, a, s = (torch.from_numpy(x.view(np.int32)).cuda() for x in (offs, adj, src))
    bc = torch.zeros(n, dtype=torch.float64, device="cuda")
    bcg.bc_noalloc(o.data_ptr(), a.data_ptr(), n, len(adj), s.data_ptr(), len(src), bc.data_ptr())
    return bc.cpu().numpy()


@pytest.mark.parametrize("depth", [16, 17, 18])
def test_counts_around_two_to_the_64(depth):
    """16 paths more a layer: 2^60 is the largest count at depth 17, and a layer's sums of the one behind it, which are no
    counts, reach 2^64.  At depth 18 a count does."""
    offs, adj = _layers(16, depth)
    n = len(offs) - 1
    src = np.arange(n, dtype=np.uint32)
    ref, ost = oracle.bc_q(offs, adj, src)
    with bcg.Graph(offs, adj) as G:
        st = G.run(src)
        assert st.extended_sigma == (depth == 18)
        assert_bc_close(G.bc(), ref, f"run, {depth} layers")
    beside = bcg.from_pairs(np.concatenate([np.stack([np.repeat(np.arange(n), np.diff(offs.astype(np.int64))), adj], 1),
                                            np.random.default_rng(31).integers(n, n + 20000, (130000, 2))]), n + 20000)
    with bcg.Graph(*beside) as G:  # (too large for the small kernel)
        st = G.run(src)
        assert st.extended_sigma == (depth == 18) and (depth == 18 or st.batch_width in WIDE)
        assert_bc_close(G.bc()[:n], ref, f"run, {depth} layers beside a component")
    assert_bc_close(_noalloc(offs, adj, src), ref, f"no allocation, {depth} layers")
    pool = [bcg.generate("er:scale=8,ef=8,seed=6"), (offs, adj)]
    with bcg.Batch(pool) as B:
        if depth < 18:
            assert B.run().batch_width in WIDE
            assert_bc_close(B.bc(1), ref, f"batch, {depth} layers")
        else:
            with pytest.raises(bcg.BcgError) as e:
                B.run()
            assert e.value.code == bcg.ERR_OVERFLOW
    if depth < 18:
        assert_bc_close(_serve(pool, [(1, None)])[0], ref, f"served, {depth} layers")
    else:
        with pytest.raises(bcg.BcgError) as e:
            _serve(pool, [(1, None)])
        assert e.value.code == bcg.ERR_OVERFLOW


def _cliques(size, count):
    """Cliques in a row, neighbours joined by one edge: two levels a clique, one path a pair."""
    pairs = []
    for c in range(count):
        b = c * size
        pairs += [[b + i, b + j] for i in range(size) for j in range(i)]
        if c:
            pairs.append([b - 1, b])
    return bcg.from_pairs(pairs, size * count)


@pytest.mark.parametrize("wave_batches", [1, 4, 64])
def test_deep_searches_of_a_served_pool(wave_batches):
    """A graph whose searches from the middle have 60 levels and from the ends 119, so some of its requests run in wide
    waves and some in packed ones, found out in the first or only in a later wave; the other graph's requests beside
    them.  Every request gives the bits that it gives alone."""
    deep = _cliques(8, 60)
    pool = [deep, bcg.generate("rmat:scale=10,ef=16,a=0.57,b=0.19,c=0.19,seed=5")]
    middle, ends = np.arange(236, 244, dtype=np.uint32), np.array([0, 1, 478], dtype=np.uint32)
    last = np.concatenate([np.tile(middle, 12), ends]).astype(np.uint32)  # 99 sources, the deep ones in the fourth job
    reqs = [(1, None), (0, middle), (0, ends), (1, np.arange(0, 900, 7, dtype=np.uint32)), (0, None), (0, last),
            (1, np.array([3], dtype=np.uint32)), (0, middle[:1]), (0, ends[:1])]
    served = _serve(pool, reqs, wave_batches=wave_batches)
    for i, (g, src) in enumerate(reqs):
        offs, adj = pool[g]
        ref, _ = oracle.bc(offs, adj, np.arange(len(offs) - 1) if src is None else src, nthreads=oracle.max_threads())
        assert_bc_close(served[i], ref, f"request {i}")
        alone = _serve(pool, [reqs[i]], wave_batches=wave_batches)[0]
        assert np.array_equal(served[i].view(np.uint64), alone.view(np.uint64)), i


def test_a_full_wave_advances_every_graph():
    """More jobs of the larger graph than a wave's memory holds (148 x 8 of its vectors): the smaller graph's request, the
    last to be submitted, ends with the first wave all the same."""
    pool = [bcg.generate("rmat:scale=11,ef=16,a=0.57,b=0.19,c=0.19,seed=5"), bcg.generate("er:scale=8,ef=8,seed=6")]
    refs = [oracle.bc(o, a, np.arange(len(o) - 1), nthreads=oracle.max_threads())[0] for o, a in pool]
    jobs = -(-np.count_nonzero(np.diff(pool[0][0])) // 32)
    with bcg.Server(pool, 8 << 30, 60000) as S:
        ids = [S.submit(0) for _ in range(5 * 148 * 8 // jobs)]  # five waves
        small = S.submit(1)
        first, out = None, {}
        while len(out) <= len(ids):
            done = S.wait()
            first = first or done
            for rid in done:
                out[rid] = S.result(rid)
    assert small in first and not set(ids) <= set(first)
    assert_bc_close(out[small], refs[1], "small")
    for rid in ids:
        assert_bc_close(out[rid], refs[0], "large")
        assert np.array_equal(out[rid].view(np.uint64), out[ids[0]].view(np.uint64))


def test_budgets_close_to_the_pool():
    """Whatever the budget leaves beside the pool's buffers, a request whose result fits beside the pool is taken and ends;
    several end before the first is fetched."""
    offs, adj = bcg.generate("er:scale=13,ef=8,seed=6")
    n = len(offs) - 1
    src = bcg.sample_sources(n, 70, 1)
    ref, _ = oracle.bc(offs, adj, src, nthreads=oracle.max_threads())
    with bcg.Server([(offs, adj)], 8 << 30) as S:
        full = S.info()["resident_bytes"]
    for budget in list(range(full - 8 * n, full + 3 * 8 * n, 2 * n)) + [full + 8 * n - 1, full + 8 * n, full + 8 * n + 1]:
        with bcg.Server([(offs, adj)], budget) as S:
            ids = [S.submit(0, src) for _ in range(4)]
            done = set()
            for _ in range(1000):
                done |= set(S.wait())
                if len(done) == 4:
                    break
                info = S.info()
                assert info["resident_bytes"] + info["admitted_bytes"] <= budget
            assert done == set(ids), budget - full
            for rid in ids:
                assert_bc_close(S.result(rid), ref, f"budget {budget - full} bytes from the wide buffers")
            assert S.info()["admitted_bytes"] == 0


def test_totals_with_loops():
    """A list that names its own vertex makes a component's entries odd: the edges of a set are halved source by source,
    as in a run."""
    offs, adj = bcg.generate("rmat:scale=10,ef=16,a=0.57,b=0.19,c=0.19,seed=5")
    rows = [list(adj[offs[v]:offs[v + 1]]) for v in range(1024)]
    rows[7].append(7)
    o = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.uint32)
    a = np.array([w for r in rows for w in r], dtype=np.uint32)
    src = np.nonzero(np.diff(o))[0].astype(np.uint32)
    with bcg.Graph(o, a) as G:
        G.set_batch_width(6)
        want = G.run(src)
        bc = G.bc()
    with bcg.Batch([(o, a)]) as B:
        for runs in (1, 2):
            st = B.run()
            assert st.teps_edges == want.teps_edges and st.visited == want.visited
            assert_bc_close(B.bc(0), runs * bc, "a loop")
