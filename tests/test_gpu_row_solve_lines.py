"""PageRank and weighted PageRank on both sides of the lines between their forms: one
cluster (8192 rows, 196,608 entries), one launch on the whole GPU, and a pass per
iteration (past 2^18 vertices or 2^21 edges with a row over 2048 entries, or with fewer
than 3.5 edges a vertex).  References and tolerances are those of test_gpu_row_solve."""
import numpy as np
import pytest

from oracle import oracle
from test_gpu_row_solve import pagerank64

pytestmark = pytest.mark.gpu


def graph(V, E, hub, seed):
    """E edges between drawn vertices, `hub` of them into vertex 3."""
    rng = np.random.default_rng(seed)
    src, dst = np.sort(rng.integers(0, V, E)), rng.integers(0, V, E)
    if hub:
        dst[rng.permutation(E)[:hub]] = 3
    rp = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=V))]).astype(np.uint32)
    return rp, dst.astype(np.uint32)


CASES = [
    (8192, 50000, 0), (8193, 50000, 0),
    (8000, 196608, 3000), (8000, 196609, 3000),
    (1 << 18, 300000, 2100), ((1 << 18) + 1, 300000, 2100),
    (100001, (1 << 21) - 1, 2100), (100001, 1 << 21, 2100),
    (300000, 1050000, 1900), (300000, 1049999, 1900),
    (300000, 1050000, 2100),
]


@pytest.mark.parametrize("case", range(len(CASES)))
def test_pagerank(case):
    import olive_b200 as ob
    rp, cl = graph(*CASES[case], seed=case)
    with ob.Graph.from_csr(rp, cl) as g:
        for mode in ("uniform", "leak"):
            r = g.pagerank(0.85, 9, 0.0, mode)
            assert r.tobytes() == g.pagerank(0.85, 9, 0.0, mode).tobytes()
            ref = pagerank64(rp, cl, 0.85, 9, mode)
            assert np.max(np.abs(r - ref) / ref) < 1e-6


@pytest.mark.parametrize("case", range(4))
def test_weighted_pagerank(case):
    import olive_b200 as ob
    rp, cl = graph(*CASES[case], seed=case)
    V, E = len(rp) - 1, len(cl)
    rng = np.random.default_rng(case)
    w = rng.lognormal(0.0, 1.0, E).astype(np.float32)
    p = rng.random(V)
    p = (p / p.sum()).astype(np.float32)
    gv = rng.standard_normal(V).astype(np.float32)
    with ob.Graph.from_csr(rp, cl) as g:
        r = g.wpr_forward(p, w=w, alpha=0.85, max_it=9)
        dw, dp = g.wpr_backward(gv, max_it=9)
    w64, p64, g64 = w.astype(np.float64), p.astype(np.float64), gv.astype(np.float64)
    ref = oracle.wpr_forward(rp, cl, w64, p64, 0.85, 9)
    assert np.max(np.abs(r - ref)) < 1e-5 * np.max(ref)
    _, dw_ref, dp_ref = oracle.wpr_backward(rp, cl, w64, ref, g64, 0.85, 9)
    for got, want in ((dw, dw_ref), (dp, dp_ref)):
        assert np.linalg.norm(got - want) <= 1e-5 * np.linalg.norm(want)
