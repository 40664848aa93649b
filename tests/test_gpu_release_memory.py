"""The device memory kept from closed graphs: given back on request, and never
handed out in another context than the one it was allocated in."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch
    assert torch.cuda.is_available()
    torch.zeros(1, device="cuda")
    return torch


def test_release_gives_it_back(torch):
    import olive_b200 as ob
    ob.release_memory()
    assert ob.release_memory() == 0
    with ob.Graph.rmat(20, 16, seed=1) as g:
        g.bfs(0)
    before, total = torch.cuda.mem_get_info()
    n = ob.release_memory()
    after, _ = torch.cuda.mem_get_info()
    assert 64 << 20 < n <= total // 64   # the in-edges alone are 64 MB
    # blocks below 1 MB (some 30 of a handle) lie in the driver's pages with other allocations
    assert after - before >= n - (30 << 20)
    assert ob.release_memory() == 0
    rp, cl = oracle.grid_csr(50, 40)
    with ob.Graph.from_csr(rp, cl) as g:
        assert np.array_equal(g.bfs(7), oracle.bfs(rp, cl, 7)[0])


def test_blocks_stay_in_their_context(torch):
    import olive_b200 as ob
    driver = pytest.importorskip("cuda.bindings.driver")

    def ok(r):
        assert r[0] == driver.CUresult.CUDA_SUCCESS, r[0]
        return r[1] if len(r) == 2 else None

    rp, cl = oracle.rmat_csr(14, 8, 5)
    w = oracle.uint_weights(len(cl), 3)
    want = oracle.bfs(rp, cl, 1)[0], oracle.dijkstra(rp, cl, w, 1)[0]

    def solve():
        with ob.Graph.from_csr(rp, cl, w) as g:
            assert np.array_equal(g.bfs(1), want[0])
            assert np.array_equal(g.sssp(1), want[1])

    ob.release_memory()
    ctx = ok(driver.cuCtxCreate(0, ok(driver.cuDeviceGet(torch.cuda.current_device()))))
    try:
        solve()
    finally:
        ok(driver.cuCtxPopCurrent())
    assert ob.release_memory() == 0      # what is kept belongs to the other context
    solve()
    ok(driver.cuCtxDestroy(ctx))
    for _ in range(2):
        solve()
    assert ob.release_memory() > 0
