"""Which searches take a run, and that the result does not depend on it: low-degree graphs with broad frontiers (random
regular graphs, trees) against meshes of any numbering.  Against the oracle within the suite's 1e-9, and in bits against
the same run once more."""
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
