"""A CTA a source in shared memory (small graphs, up to two sources an SM)
against the oracle and the wide searches.

The cases sit at the edges of its work split and of its rule: one vertex of
some degree and 127 to 129 entries (eight lanes, a warp), lists of 0 to 3
entries past a multiple of 4, 1 to more than two rounds of sources, graphs that
just fit a CTA's shared memory and that just do not, several components, every
pruning mode, directed lists, repeated edges, path counts that pass 2^32 (two
words) and 2^64 (the run is redone with extended counts).  The bar is the
suite's 1e-9: path counts are exact, only FP64 sums differ."""
import numpy as np
import pytest

import bcg
import oracle
from test_gpu_parity import assert_bc_close
from test_gpu_wide import WIDE, _layers, _rows

pytestmark = pytest.mark.gpu
SHARED = 220 << 10  # bytes a source may take


def _bytes(n, nnz):
    return n * 8 + (n + 1) * 4 + (nnz + 3) // 4 * 8 + n * 4 + (n + 2) * 2


def _dense(n, nnz):
    """n vertices in a ring, nnz entries (even) in all."""
    rng = np.random.default_rng(n)
    ring = np.stack([np.arange(n), (np.arange(n) + 1) % n], 1)
    code = rng.choice(n * (n - 1) // 2, size=nnz, replace=False)
    j = ((1 + np.sqrt(1 + 8.0 * code)) // 2).astype(np.int64)
    i = code - j * (j - 1) // 2
    ok = (i >= 0) & (i < j) & (j < n) & (j - i > 1) & (j - i < n - 1)
    rest = np.stack([i, j], 1)[ok][: nnz // 2 - n]
    return bcg.from_pairs(np.concatenate([ring, rest]), n)


GRAPHS = {
    "edge": lambda: bcg.from_pairs([[0, 1]], 2),
    "triangle": lambda: bcg.from_pairs([[0, 1], [1, 2], [2, 0]], 4),
    "heavy": lambda: _rows(900, [800, 600, 257, 256, 255, 129, 128, 127, 126, 66, 65, 64, 63], 7),
    "components": lambda: bcg.from_pairs(np.concatenate([np.random.default_rng(c).integers(40 * c, 40 * c + 37, (300, 2))
                                                         for c in range(9)]), 360),
    "rmat10": lambda: bcg.generate("rmat:scale=10,ef=16,seed=3"),
    "pendants": lambda: bcg.generate("rmat:scale=10,ef=16,seed=9,pendant_frac=0.1,pendant_mean=4"),
    "er": lambda: bcg.generate("er:scale=11,ef=10,seed=6"),
}


@pytest.mark.parametrize("flags", [0, bcg.PRUNE_DEGREE1, bcg.PRUNE_TREES])
@pytest.mark.parametrize("gname", list(GRAPHS))
def test_matches_oracle(gname, flags):
    offs, adj = GRAPHS[gname]()
    n = len(offs) - 1
    live = np.nonzero(np.diff(offs))[0].astype(np.uint32)
    for k in (1, 2, 149, 296, 297):
        src = live[np.linspace(0, len(live) - 1, min(k, len(live))).astype(int)]
        ref, ost = oracle.bc_q(offs, adj, src)
        with bcg.Graph(offs, adj, flags) as G:
            st = G.run(src)
            got = G.bc()
            G.reset()
            G.run(src)
            assert np.array_equal(got.view(np.uint64), G.bc().view(np.uint64))
            G.run(np.concatenate([src, src[:1]]))  # a weight of 2; accumulated
            more = G.bc()
        one, _ = oracle.bc_q(offs, adj, src[:1])
        assert_bc_close(got, ref, f"{gname} k={k} flags={flags}")
        assert_bc_close(more, 2 * ref + one, f"{gname} k={k} flags={flags} accumulated")
        assert st.teps_edges == ost["teps_edges"] and st.skipped == ost["skipped"]
        assert flags or (st.max_depth == ost["max_depth"] and st.visited == ost["visited"])
        if not flags and gname in ("heavy", "rmat10", "er"):
            assert (st.batch_width == 1) == (len(src) <= 296)


@pytest.mark.parametrize("n", [700, 3000, 6000])
def test_size_of_the_shared_memory(n):
    """The largest list that fits beside n vertices, and the next ones."""
    limit = (SHARED - 15 - _bytes(n, 0)) // 2 // 4 * 4
    for entries, fits in ((limit - 2, True), (limit, True), (limit + 40, False)):
        offs, adj = _dense(n, entries)
        assert len(adj) == entries
        src = bcg.sample_sources(n, 5, 1)
        ref, _ = oracle.bc_q(offs, adj, src)
        with bcg.Graph(offs, adj) as G:
            st = G.run(src)
            assert_bc_close(G.bc(), ref, f"{n} {entries}")
        assert st.batch_width == 1 if fits else st.batch_width in WIDE


def test_directed_with_repeated_edges():
    rng = np.random.default_rng(12)
    n = 600
    pairs = np.concatenate([rng.integers(0, n, (8000, 2)), np.stack([np.zeros(300, int), rng.integers(1, n, 300)], 1)])
    pairs = pairs[np.argsort(pairs[:, 0], kind="stable")]
    offs = np.zeros(n + 1, dtype=np.uint32)
    np.cumsum(np.bincount(pairs[:, 0], minlength=n), out=offs[1:])
    adj = pairs[:, 1].astype(np.uint32)  # loops and repeated edges stay
    src = bcg.sample_sources(n, 100, 1)
    with bcg.Graph(offs, adj, bcg.DIRECTED) as G:
        G.set_batch_width(6)
        a = G.run(src)
        want = G.bc()
        G.reset()
        G.set_batch_width(0)
        b = G.run(src)
        got = G.bc()
        assert a.batch_width == 6 and b.batch_width == 1
        assert a.teps_edges == b.teps_edges and a.visited == b.visited and a.max_depth == b.max_depth
    assert_bc_close(got, want, "repeated edges")


@pytest.mark.parametrize("width,depth,ext", [(4, 16, 0), (4, 18, 0), (4, 32, 0), (16, 9, 0), (16, 16, 0), (16, 17, 0),
                                             (16, 18, 1), (4, 34, 1), (5, 26, 0), (5, 60, 1)])
def test_large_counts(width, depth, ext):
    """width paths more a layer: sums that pass 2^32 and, last, 2^64."""
    offs, adj = _layers(width, depth)
    src = np.arange(0, width * depth, 3, dtype=np.uint32)
    ref, _ = oracle.bc_q(offs, adj, src)
    with bcg.Graph(offs, adj) as G:
        st = G.run(src)
        assert st.extended_sigma == ext and (ext or st.batch_width == 1)
        assert_bc_close(G.bc(), ref, f"layers {width} {depth}")


def test_threads_with_graphs_of_different_sizes():
    """The kernel's shared-memory limit is the process's: a thread with a small graph must not lower it for another."""
    import threading

    sets = [_dense(n, nnz) for n, nnz in ((64, 400), (1000, 30000), (300, 8000), (1500, 60000))]
    want = [oracle.bc_q(o, a, np.arange(4, dtype=np.uint32))[0] for o, a in sets]
    got, errors = [None] * len(sets), []

    def work(k):
        try:
            with bcg.Graph(*sets[k]) as g:
                for _ in range(200):
                    g.reset()
                    g.run(np.arange(4, dtype=np.uint32))
                got[k] = g.bc()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(sets))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for w, b in zip(want, got):
        assert_bc_close(b, w)
