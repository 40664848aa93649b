"""Handles of different sizes used by several host threads at once: every call
succeeds and gives the bits that one thread alone gives.  The sizes are those of
the one-cluster solves (up to 8192 vertices), whose shared memory depends on the
graph, and some past them."""
import time
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu

SIZES = [700, 3001, 8192, 30011, 60007]


def inputs(V):
    rng = np.random.default_rng(V)
    src, dst = np.sort(rng.integers(0, V, 6 * V)), rng.integers(0, V, 6 * V)
    rp = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=V))]).astype(np.uint32)
    p = rng.random(V).astype(np.float32)
    return dict(rp=rp, cl=dst.astype(np.uint32), p=p / p.sum(),
                w=rng.lognormal(0.0, 1.0, len(dst)).astype(np.float32),
                g=rng.standard_normal(V).astype(np.float32),
                seeds=rng.integers(0, V, 8).astype(np.uint32))


def calls(ob, d):
    V = len(d["rp"]) - 1
    with ob.Graph.from_csr(d["rp"], d["cl"]) as g:
        out = [g.bfs(1), g.pagerank(0.85, 12, 0.0), g.pagerank(0.85, 5, 0.0, "leak"),
               g.wpr_forward(d["p"], w=d["w"], max_it=9), *g.wpr_backward(d["g"], max_it=9),
               g.ppr(d["seeds"], max_it=4, tol=0.0), g.msbfs(d["seeds"])]
        if V <= 30011:
            lv, pr, _ = g.batch(np.array([0, V], np.uint32), d["seeds"][None, :], max_it=4, tol=0.0)
            out += [lv, pr]
        return [np.ascontiguousarray(x).tobytes() for x in out]


def test_same_bits_from_several_threads():
    import olive_b200 as ob
    data = [inputs(V) for V in SIZES]
    want = [calls(ob, d) for d in data]
    assert np.array_equal(np.frombuffer(want[0][0], np.int32),
                          oracle.bfs(data[0]["rp"], data[0]["cl"], 1)[0])

    def work(t):
        for r in range(12):
            i = (t + r * (1 + t % 2)) % len(SIZES)
            got = calls(ob, data[i])
            assert got == want[i], (t, r, [a == b for a, b in zip(got, want[i])])

    with ThreadPoolExecutor(6) as pool:
        for f in [pool.submit(work, t) for t in range(6)]:
            f.result()                       # an error in a thread is the test's


def test_short_solves_from_several_threads():
    """Solves of a few microseconds on kept handles for ten seconds, so that launches
    of different sizes come between each other's steps.  (With a kernel attribute set
    to each handle's size before its launch, one in 20,000 of those of 13,000 to 54,272
    vertices failed.)"""
    import torch
    import olive_b200 as ob
    data = [inputs(V) for V in (8192, 3001, 54272, 1500, 7001, 20011, 6001, 45001)]
    graphs = [ob.Graph.from_csr(d["rp"], d["cl"]) for d in data]
    want = [g.pagerank(0.85, 1, 0.0).tobytes() for g in graphs]
    end = time.monotonic() + 10

    def work(i):
        out = torch.empty(graphs[i].V, device="cuda")
        while time.monotonic() < end:
            for _ in range(500):
                graphs[i].pagerank(0.85, 1, 0.0, out=out)
            assert out.cpu().numpy().tobytes() == want[i]

    with ThreadPoolExecutor(len(graphs)) as pool:
        for f in [pool.submit(work, i) for i in range(len(graphs))]:
            f.result()
    for g in graphs:
        g.close()
