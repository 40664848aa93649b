"""What a handle leaves under way on its stream when a call returns, and what happens
to it when the handle is moved to another stream or closed."""
import time

import numpy as np
import pytest

from oracle import oracle
from test_gpu_alloc_failure import leave

pytestmark = pytest.mark.gpu

CYCLES = 400_000_000   # about 200 ms of a one-thread kernel


@pytest.fixture(scope="module")
def torch():
    import torch
    assert torch.cuda.is_available()
    torch.cuda._sleep(1000)
    torch.cuda.synchronize()
    return torch


def test_weights_are_stream_ordered(torch):
    import olive_b200 as ob
    rp, cl = oracle.rmat_csr(12, 8, 1)
    V, E = len(rp) - 1, len(cl)
    rng = np.random.default_rng(1)
    p = np.full(V, 1.0 / V, np.float32)
    w0, w1 = (rng.random(E).astype(np.float32) + 0.5 for _ in range(2))
    d1 = torch.from_numpy(w1).cuda()
    busy = torch.cuda.Stream()
    with ob.Graph.from_csr(rp, cl) as g:
        g.wpr_forward(p, w=w0, max_it=5)
        g.set_stream(busy)
        torch.cuda.synchronize()
        with torch.cuda.stream(busy):
            torch.cuda._sleep(CYCLES)
        t = time.perf_counter()
        g.set_weights_f32(d1)
        assert time.perf_counter() - t < 0.05       # it waits for nothing
        assert not busy.query()
        g.set_stream(None)                          # its own: after the copy all the same
        r = g.wpr_forward(p, max_it=5)
    ref = oracle.wpr_forward(rp, cl, w1.astype(np.float64), p.astype(np.float64), 0.85, 5)
    assert np.max(np.abs(r - ref)) < 1e-5 * np.max(ref)


def test_moved_to_a_stream_under_capture(torch):
    """Binding a handle neither ends nor joins the stream's capture."""
    import olive_b200 as ob
    rp, cl = oracle.rmat_csr(10, 8, 1)
    x = torch.zeros(8, device="cuda")
    with ob.Graph.from_csr(rp, cl) as g:
        g.set_weights_f32(np.ones(len(cl), np.float32))
        graph, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=s):
            g.set_stream(s)
            x += 1
        g.set_stream(None)
        graph.replay()
        torch.cuda.synchronize()
        assert float(x[0]) == 1.0
        assert np.array_equal(g.bfs(1), oracle.bfs(rp, cl, 1)[0])


def test_closed_behind_a_busy_stream(torch):
    """The buffers of a handle that is moved away from a busy stream and closed are not
    handed out while the copy there is still to come."""
    import olive_b200 as ob
    rp, cl = oracle.rmat_csr(12, 8, 1)
    ones = torch.ones(len(cl), device="cuda")
    busy = torch.cuda.Stream()
    g = ob.Graph.from_csr(rp, cl)
    g.set_stream(busy)
    torch.cuda.synchronize()
    with torch.cuda.stream(busy):
        torch.cuda._sleep(CYCLES)
    g.set_weights_f32(ones)
    g.set_stream(None)
    g.close()
    assert busy.query()
    with ob.Graph.from_csr(rp, cl, np.arange(len(cl), dtype=np.uint32)) as h:
        torch.cuda.synchronize()
        assert np.array_equal(h.csr()[2], np.arange(len(cl), dtype=np.uint32))


def test_a_failed_call_leaves_nothing_under_way(torch):
    import olive_b200 as ob
    with ob.Graph.er_batch(64, 2000, 4000, 8, 1)[0] as g:
        V = g.V
        off = np.arange(0, V + 1, 1000, dtype=np.uint32)
        off = off[off <= V]
        seeds = np.zeros((len(off) - 1, 32), np.uint32)
        out = torch.empty((V, 32), device="cuda")
        busy = torch.cuda.Stream()
        g.set_stream(busy)
        ballast = leave(torch, 4 << 20)      # not enough for the second copy of the vectors
        with torch.cuda.stream(busy):
            torch.cuda._sleep(CYCLES)
        with pytest.raises(ob.OliveError):
            g.batch(off, seeds, max_it=1, bfs=False, ppr_out=out)
        assert busy.query()
        del ballast
        torch.cuda.empty_cache()


def test_a_graph_that_does_not_fit(torch):
    """Creation fails half way, with the handle's own stream going away."""
    import olive_b200 as ob
    ballast = leave(torch, 64 << 20)
    for _ in range(3):
        with pytest.raises(ob.OliveError):
            ob.Graph.rmat(20, 16, seed=3)
        with pytest.raises(ob.OliveError):
            ob.Graph.from_csr(np.zeros(1 << 25, np.uint32), np.zeros(0, np.uint32))
    del ballast
    torch.cuda.empty_cache()
    rp, cl = oracle.grid_csr(20, 20)
    with pytest.raises(ob.OliveError):
        ob.Graph.from_csr(rp, cl + np.uint32(1))
    with ob.Graph.from_csr(rp, cl) as g:
        assert np.array_equal(g.bfs(0), oracle.bfs(rp, cl, 0)[0])
