"""One CTA or cluster a source (graphs of at most 8 neighbours a vertex)
against the oracle: both row widths (4 and 8 neighbours), frontiers from one
vertex to more than a cluster's queues hold, few sources (clusters of 16) and
more than the chip has SMs, path counts that fit uint64, that overflow it
midway, and that are extended from the start, in every pruning mode.  The bar
is the suite's 1e-9; the sums run in list order, so two runs give the same bits."""
import numpy as np
import pytest

import bcg
import oracle
from test_gpu_parity import assert_bc_close

pytestmark = pytest.mark.gpu


def _triangles(w, h):
    """A triangulated mesh: six neighbours a vertex."""
    p = [[y * w + x, (y + dy) * w + x + dx] for y in range(h - 1) for x in range(w - 1)
         for dx, dy in ((1, 0), (0, 1), (1, 1))]
    return bcg.from_pairs(p, w * h)


GRAPHS = {
    "path": lambda: bcg.from_pairs([[i, i + 1] for i in range(299)], 300),
    "star8": lambda: bcg.from_pairs([[0, i] for i in range(1, 9)] + [[9, 10]], 12),
    "grid31": lambda: bcg.generate("grid:w=31,h=33,drop=0.05,seed=5"),
    "strip": lambda: bcg.generate("grid:w=3,h=400,drop=0.02,seed=6"),
    "triangles": lambda: _triangles(45, 40),
}


@pytest.mark.parametrize("flags", [0, bcg.PRUNE_DEGREE1, bcg.PRUNE_TREES])
@pytest.mark.parametrize("gname", list(GRAPHS))
def test_matches_oracle(gname, flags):
    offs, adj = GRAPHS[gname]()
    n = len(offs) - 1
    for k, mode in ((1, bcg.SIGMA_AUTO), (5, bcg.SIGMA_EXTENDED), (40, bcg.SIGMA_AUTO), (min(n, 200), bcg.SIGMA_AUTO)):
        src = bcg.sample_sources(n, min(k, n), 3)
        ref, ost = oracle.bc_q(offs, adj, src)
        with bcg.Graph(offs, adj, flags) as G:
            G.set_sigma_mode(mode)
            st = G.run(src)
            got = G.bc()
            G.reset()
            G.run(src)
            assert np.array_equal(got.view(np.uint64), G.bc().view(np.uint64))
        assert_bc_close(got, ref, f"{gname} k={k} flags={flags}")
        assert st.teps_edges == ost["teps_edges"] and st.skipped == ost["skipped"]
        assert flags or (st.batch_width == 1 and st.max_depth == ost["max_depth"])


def test_exact_mode_refuses_overflow():
    offs, adj = bcg.generate("grid:w=60,h=60,drop=0.0,seed=1")
    with bcg.Graph(offs, adj) as G:
        G.set_sigma_mode(bcg.SIGMA_EXACT)
        with pytest.raises(bcg.BcgError) as e:
            G.run([0, 7])
        assert e.value.code == bcg.ERR_OVERFLOW


@pytest.mark.parametrize("k", [2, 80])
def test_frontier_beyond_the_queues(k):
    """A complete tree of 8 neighbours a vertex, 7 children each: its last
    level has 117,649 vertices, more than a cluster's queues hold (2 sources;
    run again with one CTA a source) and than one CTA's (80 sources)."""
    n = (7**7 - 1) // 6
    offs, adj = bcg.from_pairs(np.stack([(np.arange(1, n) - 1) // 7, np.arange(1, n)], 1), n)
    src = np.concatenate([[0], bcg.sample_sources(n, k - 1, 5)]).astype(np.uint32)
    ref, ost = oracle.bc(offs, adj, src, nthreads=oracle.max_threads())
    with bcg.Graph(offs, adj) as G:
        G.run([3])
        before = G.bc()
        st = G.run(src)
        assert st.teps_edges == ost["teps_edges"] and st.visited == ost["visited"]
        assert_bc_close(G.bc() - before, ref, f"tree k={k}")
