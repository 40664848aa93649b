"""The library's count of the kernels of a solve (bench.py reports it)."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


def test_supersteps_in_one_cta_and_in_the_chain():
    import olive_b200 as ob
    rp, cl = oracle.grid_csr(16, 16)
    with ob.Graph.from_csr(rp, cl, oracle.uint_weights(len(cl), 7)) as g:
        g.bfs(0)
        assert g.last_launches() == 1                 # levels cleared, run and ended in one
        g.sssp(0)                                     # clear, run, map back; heavy steps by the chain
        chains = (g.last_launches() - 3) // 4
        assert g.last_launches() == 3 + 4 * chains and chains < g.last_stats.iterations // 4
        g.tune(use_graphs=0, levels_per_sync=2)
        g.bfs(0)
        assert g.last_launches() == 1 + 7 * 2
        g.sssp(0)                                     # two chains between looks at the device
        assert g.last_launches() == 3 + 4 * 2 * max(1, -(-chains // 2))
    with ob.Graph.rmat(16, 16, seed=1, weights=True) as g:
        src = g.max_degree_vertex()[0]
        g.bfs(src)
        n, st = g.last_launches(), g.last_stats
        chains = (n - 2) // 7
        assert n == 2 + 7 * chains and 1 <= chains < st.iterations
        assert chains >= st.pull_steps
        g.sssp(src)
        n, st = g.last_launches(), g.last_stats
        assert (n - 3) % 4 == 0 and 1 <= (n - 3) // 4 < st.iterations
        g.msbfs([src, 1])
        assert g.last_launches() == 2 + 5 * g.last_stats.iterations


def test_other_solves():
    import olive_b200 as ob
    rng = np.random.default_rng(1)
    V = 300000
    src, dst = np.sort(rng.integers(0, V, V)), rng.integers(0, V, V)
    rp = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=V))]).astype(np.uint32)
    with ob.Graph.from_csr(rp, dst.astype(np.uint32)) as g:   # a pass an iteration, no long rows
        g.pagerank(max_it=7, tol=0.0)
        assert g.last_launches() == 3 + 2 * 7
        g.ppr([1, 2], max_it=5, tol=0.0)
        assert g.last_launches() == 3 + 2 * 5
        p = np.full(V, 1 / V, np.float32)
        g.wpr_forward(p, w=np.ones(V, np.float32), max_it=3)
        assert g.last_launches() == 6
        g.wpr_backward(p, max_it=3)
        assert g.last_launches() == 4
    with ob.Graph.rmat(12, 16, seed=1) as g:                  # one launch
        g.pagerank(max_it=7, tol=0.0)
        assert g.last_launches() == 3
