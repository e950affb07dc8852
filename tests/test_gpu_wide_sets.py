"""Batched and serving forms on the wide searches, where a set or pool is unlike the usual one: a single graph, most of
whose vertices have no edge.  Against the oracle, within the suite's 1e-9; what no path passes is exactly 0."""
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
