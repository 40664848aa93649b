"""The iterated row sums behind PageRank and weighted PageRank at the edges of
their layout: row lengths on both sides of every lanes-per-row class, of the
segmented rows (2048) and their segments (512), on one cluster (up to 54,272
vertices) and on the whole GPU, against FP64 after the same iterations.  Tolerances are those of the full-size tests: 1e-6 relative per
rank (compensated sums: about one FP32 rounding each), 1e-5 for weighted ranks
and normwise for gradients."""
import numpy as np
import pytest

from oracle import oracle
from test_gpu_wpr import GRAD_FLOOR, GRAD_RTOL, operand_scales

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ob():
    import torch
    assert torch.cuda.is_available()
    import olive_b200
    return olive_b200


def graph(V, lengths, hubs, seed):
    """CSR whose first in-degrees are `lengths` (the rest 0..3), sources drawn
    from all vertices (hubs = 0) or mostly from `hubs` of them."""
    rng = np.random.default_rng(seed)
    din = rng.integers(0, 4, V)
    din[:len(lengths)] = lengths
    dst = np.repeat(np.arange(V), din)
    src = rng.integers(0, V, len(dst))
    if hubs:
        m = rng.random(len(dst)) < 0.8
        src[m] = rng.integers(0, hubs, int(m.sum())) * (V // hubs)
    o = np.argsort(src, kind="stable")
    rp = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=V))]).astype(np.uint32)
    return rp, dst[o].astype(np.uint32)


def pagerank64(rp, cl, alpha, it, mode):
    V = len(rp) - 1
    deg = np.diff(rp.astype(np.int64))
    src = np.repeat(np.arange(V), deg)
    r = np.full(V, 1.0 / V)
    for _ in range(it):
        lost = r[deg == 0].sum() if mode == "uniform" else 0.0
        r = (1 - alpha) / V + alpha * lost / V + alpha * np.bincount(
            cl, (r / np.maximum(deg, 1))[src], V)
    return r


EDGES = [1, 2, 3, 4, 5, 7, 8, 9, 15, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257,
         511, 512, 513, 1023, 1024, 1025, 2047, 2048, 2049, 2560, 2561, 4096, 20000]
CASES = [
    (1, [], 0),
    (33, [5], 0),
    (1000, [], 0),                 # no long rows
    (3000, EDGES, 0),
    (9001, EDGES, 64),             # a few sources of most edges
    (70001, EDGES + [40] * 20000, 60000),   # past one cluster
    (54272, EDGES, 0), (54273, EDGES, 0),   # the last of one cluster, the first past it
    (200003, [30] * 150000, 0),    # past 3 M edges without a segmented row
    (200003, EDGES + [30] * 150000, 0),     # and with some: a pass per iteration
]


@pytest.mark.parametrize("case", range(len(CASES)))
@pytest.mark.parametrize("mode", ["uniform", "leak"])
def test_pagerank_layout(ob, case, mode):
    rp, cl = graph(*CASES[case], seed=case)
    with ob.Graph.from_csr(rp, cl) as g:
        for alpha, it in ((0.85, 1), (0.85, 12), (0.6, 7)):
            r = g.pagerank(alpha, it, 0.0, mode)
            again = g.pagerank(alpha, it, 0.0, mode)
            assert r.tobytes() == again.tobytes()
            assert g.last_stats.iterations == it
            ref = pagerank64(rp, cl, alpha, it, mode)
            assert np.max(np.abs(r - ref) / ref) < 1e-6
        r0 = g.pagerank(0.85, 0, 0.0, mode)
        assert np.all(r0 == np.float32(1) / np.float32(len(rp) - 1))


@pytest.mark.parametrize("case", range(len(CASES)))
def test_weighted_pagerank_layout(ob, case):
    rp, cl = graph(*CASES[case], seed=case + 20)
    V, E = len(rp) - 1, len(cl)
    rng = np.random.default_rng(case)
    w = rng.lognormal(0.0, 1.0, E).astype(np.float32)
    p = rng.exponential(1.0, V)
    p = (p / p.sum()).astype(np.float32)
    gv = rng.standard_normal(V).astype(np.float32)
    w64, p64, g64 = w.astype(np.float64), p.astype(np.float64), gv.astype(np.float64)
    with ob.Graph.from_csr(rp, cl) as g:
        for alpha, it in ((0.85, 15), (0.6, 1), (0.85, 15)):
            r = g.wpr_forward(p, w=w, alpha=alpha, max_it=it)
            assert g.last_stats.iterations == it
            dw, dp = g.wpr_backward(gv, max_it=it)
            ref = oracle.wpr_forward(rp, cl, w64, p64, alpha, it)
            assert np.max(np.abs(r - ref)) < 1e-5 * np.max(ref)
            lam, dw_ref, dp_ref = oracle.wpr_backward(rp, cl, w64, ref, g64, alpha, it)
            # gradients as in test_gpu_wpr.py: 1e-5 of the norm, and of each entry
            # and the terms whose difference it is (exact zeros among them)
            s_w, s_p = operand_scales(rp, cl, w, ref, gv, lam)
            for got, want, scale in ((dw, dw_ref, s_w), (dp, dp_ref, s_p)):
                if np.any(want):
                    assert np.linalg.norm(got - want) <= GRAD_RTOL * np.linalg.norm(want)
                assert np.all(np.abs(got - want) <= GRAD_RTOL * (np.abs(want) + scale) +
                              GRAD_FLOOR * np.max(np.abs(want), initial=0.0))
