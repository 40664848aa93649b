"""Calls that run out of device memory part of the way through building what a
handle keeps: the call reports it, and the next one on the handle, with memory
to spare, gives the right answer instead of running on half-built state."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu

MB = 1 << 20


@pytest.fixture(scope="module")
def torch():
    import torch
    assert torch.cuda.is_available()
    return torch


def leave(torch, want):
    """Device memory allocated (not touched) until about `want` bytes are left."""
    import olive_b200 as ob
    torch.cuda.synchronize()
    ob.release_memory()
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    return torch.empty(max(free - want, 1), dtype=torch.uint8, device="cuda")


# a graph of 2^20 vertices and 16 M edges: the lists take about 24 MB of sort
# arrays, 20 MB of vertex lists, 64 MB of in-edges, two 128 MB key arrays and the
# sort's scratch, so that each of these sizes stops it somewhere else
@pytest.mark.parametrize("left", [8, 40, 120, 220, 400])
def test_bfs_lists(torch, left):
    import olive_b200 as ob
    with ob.Graph.rmat(20, 16, seed=3) as g:
        g.pagerank(max_it=1)             # device code loaded
        rp, cl, _ = g.csr()
        src = g.max_degree_vertex()[0]
        ballast = leave(torch, left * MB)
        failed = False
        for call in (lambda: g.bfs(src), lambda: g.msbfs([src, 1])):
            try:
                call()
            except ob.OliveError as e:
                assert "memory" in str(e), e
                failed = True
        assert failed
        del ballast
        torch.cuda.empty_cache()
        want = oracle.bfs(rp, cl, src)[0]
        assert np.array_equal(g.bfs(src), want)
        assert np.array_equal(g.msbfs([src, 1])[0], want)
