"""Which searches take a run, and that the result does not depend on it: low-degree graphs with broad frontiers (random
regular graphs, trees) against meshes of any numbering; and what a run whose searches or counts leave the wide searches
spares the next attempt.  Against the oracle within the suite's 1e-9, and in bits against the same run once more."""
import numpy as np
import pytest

import bcg
import oracle
from test_gpu_parity import assert_bc_close

pytestmark = pytest.mark.gpu


def _regular3(n, seed=7):
    rng = np.random.default_rng(seed)
    pairs = [(lambda p: np.stack([p[:n // 2], p[n // 2:]], 1))(rng.permutation(n)) for _ in range(3)]
    return bcg.from_pairs(np.concatenate(pairs), n)


def _tree(n, children):
    return bcg.from_pairs(np.stack([(np.arange(1, n) - 1) // children, np.arange(1, n)], 1), n)


def _lattice(side, dims, shuffle=False):
    at = np.arange(side**dims).reshape((side,) * dims)
    if shuffle:
        at = np.random.default_rng(3).permutation(side**dims).reshape(at.shape)
    pairs = [np.stack([np.take(at, range(side - 1), k).ravel(), np.take(at, range(1, side), k).ravel()], 1) for k in range(dims)]
    return bcg.from_pairs(np.concatenate(pairs), side**dims)


def _sparse_mesh():
    """A mesh on the last 10,000 of 300,000 vertices."""
    offs, adj = _lattice(100, 2)
    own = np.stack([np.repeat(np.arange(10000), np.diff(offs.astype(np.int64))), adj], 1) + 290000
    return bcg.from_pairs(own, 300000)


# graph, sources, sources of a batch that the run must report (1: a CTA or cluster a source)
CASES = {
    "regular, queues hold it": (lambda: _regular3(1 << 16), 6, 1),
    "regular, queues just hold it": (lambda: _regular3(1 << 18), 6, 1),
    "regular, too broad": (lambda: _regular3(1 << 19), 6, 6),
    "regular, too broad, three": (lambda: _regular3(1 << 19), 3, 3),
    "regular, one CTA a source": (lambda: _regular3(1 << 17), 100, 1),
    "tree of 7, too broad": (lambda: _tree(1 << 18, 7), 12, 6),
    "tree of 2, one CTA a source": (lambda: _tree(1 << 16, 2), 48, 1),
    "tree of 2, too broad": (lambda: _tree(1 << 19, 2), 6, 6),
    "mesh": (lambda: bcg.generate("grid:w=400,h=300,drop=0.05,seed=5"), 24, 1),
    "mesh in any order": (lambda: _lattice(300, 2, shuffle=True), 24, 1),
    "lattice in three dimensions": (lambda: _lattice(45, 3, shuffle=True), 24, 1),
    "mesh among isolated vertices": (_sparse_mesh, 12, 1),
}


@pytest.mark.parametrize("name", list(CASES))
def test_low_degree_graphs(name):
    make, k, width = CASES[name]
    offs, adj = make()
    live = np.nonzero(np.diff(offs))[0].astype(np.uint32)
    src = live[np.sort(np.random.default_rng(k).choice(len(live), k, replace=False))]
    ref, ost = oracle.bc_q(offs, adj, src) if "mesh" in name or "lattice" in name else \
        oracle.bc(offs, adj, src, nthreads=oracle.max_threads())
    with bcg.Graph(offs, adj) as G:
        st = G.run(src)
        got = G.bc()
        G.reset()
        G.run(src)
        assert np.array_equal(got.view(np.uint64), G.bc().view(np.uint64))
    assert st.batch_width == width, name
    assert st.teps_edges == ost["teps_edges"] and st.max_depth == ost["max_depth"]
    assert_bc_close(got, ref, name)


def _cliques_beside(size, count):
    """Cliques in a row (two levels each, 119 from end to end of 60) and a random component of 20,000 vertices."""
    pairs = []
    for c in range(count):
        b = c * size
        pairs += [[b + i, b + j] for i in range(size) for j in range(i)]
        if c:
            pairs.append([b - 1, b])
    n = size * count
    far = np.random.default_rng(31).integers(n, n + 20000, (130000, 2))
    return bcg.from_pairs(np.concatenate([pairs, far]), n + 20000)


def _attempts(path, what):
    return path.read_text().count(what) if path.exists() else 0


def test_deep_runs_are_tried_once(tmp_path, monkeypatch):
    """The wide searches stop at the first run from the ends of a long component; later ones from anywhere that is known
    to be too far from one of its ends are not tried there.  Others are, before and after, with the same bits."""
    offs, adj = _cliques_beside(8, 60)
    ends, near, middle = [0, 1, 478], [20, 470, 9], [238, 240, 241]
    other = list(range(5000, 5040))
    with bcg.Graph(offs, adj) as G:
        def run(src):
            G.reset()
            st = G.run(np.array(src, dtype=np.uint32))
            return st, G.bc()
        before = [run(middle), run(other)]
        trace = tmp_path / "trace"
        monkeypatch.setenv("BCG_TRACE_FILE", str(trace))
        seen = []
        for src in (ends, ends, near, ends + other):
            st, got = run(src)
            seen.append(_attempts(trace, "# wide"))
            assert st.batch_width in (3, 6) and st.max_depth > 100
            assert_bc_close(got, oracle.bc(offs, adj, np.array(src, dtype=np.uint32))[0], f"{len(src)} sources")
        assert seen == [1, 1, 1, 1]
        monkeypatch.delenv("BCG_TRACE_FILE")
        for src, (st0, want) in zip((middle, other), before):
            st, got = run(src)
            assert st.batch_width in (16, 32) and st0.batch_width == st.batch_width
            assert np.array_equal(got.view(np.uint64), want.view(np.uint64))


def _king(w):
    """A mesh of eight neighbours, mean degree 7.8: counts pass 2^64 at level 41."""
    at = np.arange(w * w).reshape(w, w)
    pairs = [np.stack([a.ravel(), b.ravel()], 1) for a, b in ((at[:, :-1], at[:, 1:]), (at[:-1], at[1:]),
                                                             (at[:-1, :-1], at[1:, 1:]), (at[:-1, 1:], at[1:, :-1]))]
    pairs = np.concatenate(pairs)
    return bcg.from_pairs(pairs[(pairs[:, 0] * 7 + pairs[:, 1]) % 50 != 0], w * w)


def _cliques(size, count):
    pairs = []
    for c in range(count):
        b = c * size
        pairs += [[b + i, b + j] for i in range(size) for j in range(i)]
        if c:
            pairs.append([b - 1, b])
    return bcg.from_pairs(pairs, size * count)


@pytest.mark.parametrize("name", ["cliques", "king"])
def test_deep_runs_of_eight_neighbours(tmp_path, monkeypatch, name):
    """The same where a CTA or cluster a source takes what the wide searches leave: for their depth (cliques in a row,
    one path a pair), which is known from then on, or for their counts, which are found again in every run."""
    offs, adj = _cliques(8, 3000) if name == "cliques" else _king(150)
    src = np.array([3, 149, 22000, 11000], dtype=np.uint32)
    trace = tmp_path / "trace"
    monkeypatch.setenv("BCG_TRACE_FILE", str(trace))
    ref, _ = oracle.bc_q(offs, adj, src)
    with bcg.Graph(offs, adj) as G:
        for runs in (1, 2, 3):
            st = G.run(src)
            assert st.batch_width == 1 and st.extended_sigma == (name == "king")
            assert_bc_close(G.bc(), runs * ref, f"run {runs}")
    assert _attempts(trace, "# wide") == (1 if name == "cliques" else 3)


def test_a_count_past_two_to_the_64_is_found_once(tmp_path, monkeypatch):
    """Layers of 16 vertices beside a random component: the wide searches find the overflow, and the sweep kernel runs
    with extended counts at once; where overflow is an error, it is one at once."""
    ids = np.arange(16 * 30).reshape(30, 16)
    pairs = [np.stack(np.meshgrid(ids[i], ids[i + 1]), -1).reshape(-1, 2) for i in range(29)]
    pairs.append(np.random.default_rng(31).integers(480, 20480, (130000, 2)))
    offs, adj = bcg.from_pairs(np.concatenate(pairs), 20480)
    src = np.arange(0, 480, 40, dtype=np.uint32)
    trace = tmp_path / "trace"
    monkeypatch.setenv("BCG_TRACE_FILE", str(trace))
    ref, _ = oracle.bc_q(offs, adj, src)
    with bcg.Graph(offs, adj) as G:
        st = G.run(src)
        assert st.extended_sigma == 1
        assert_bc_close(G.bc(), ref, "layers")
        assert _attempts(trace, "# wide") == 1 and _attempts(trace, "# width") == 1
        G.reset()
        G.set_sigma_mode(bcg.SIGMA_EXACT)
        with pytest.raises(bcg.BcgError) as e:
            G.run(src)
        assert e.value.code == bcg.ERR_OVERFLOW and not np.any(G.bc())
        assert _attempts(trace, "# wide") == 2 and _attempts(trace, "# width") == 1


def test_a_run_of_several_launches():
    """Job vectors of more than 512 MB: the launches add one after the other, and when the last one meets a deep search
    (ordered last by what it reaches), what the others added is taken back and the sweep kernel runs it all."""
    rmat = bcg.generate("rmat:scale=18,ef=8,a=0.57,b=0.19,c=0.19,seed=3")
    n = len(rmat[0]) - 1
    own = np.stack([np.repeat(np.arange(n), np.diff(rmat[0].astype(np.int64))), rmat[1]], 1)
    o, a = _cliques(8, 60)
    tail = np.stack([np.repeat(np.arange(480), np.diff(o.astype(np.int64))), a], 1) + n
    offs, adj = bcg.from_pairs(np.concatenate([own, tail]), n + 480)
    live = np.nonzero(np.diff(rmat[0]))[0].astype(np.uint32)
    jobs = (512 << 20) // (8 * (len(live) + 480)) + 20
    src = live[np.sort(np.random.default_rng(1).choice(len(live), 32 * jobs, replace=False))]
    ends = np.array([n, n + 479], dtype=np.uint32)
    with bcg.Graph(offs, adj) as G:
        parts = [G.run(p) for p in np.array_split(src, 4)]
        want = G.bc()
        G.reset()
        st = G.run(src)
        assert st.batch_width == 32 and st.batches == jobs
        assert st.teps_edges == sum(p.teps_edges for p in parts) and st.visited == sum(p.visited for p in parts)
        assert_bc_close(G.bc(), want, "one call")
        G.run(ends)
        both = G.bc()
        G.reset()
        st = G.run(np.concatenate([src, ends]))
        assert st.batch_width == 6 and st.max_depth > 100
        assert_bc_close(G.bc(), both, "with a deep search")
