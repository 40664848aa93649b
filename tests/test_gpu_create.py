"""The checks of a caller's CSR (done on the device) and the first solve of a new
handle, from host and from device arrays."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ob():
    import torch
    assert torch.cuda.is_available()
    import olive_b200
    return olive_b200


BAD = [
    (lambda rp, cl: rp.__setitem__(0, 1), r"rowptr\[0\]=1 rowptr\[V\]=\d+, expected 0"),
    (lambda rp, cl: rp.__setitem__(-1, rp[-1] - 1), r"rowptr\[V\]=\d+, expected 0 and E="),
    (lambda rp, cl: rp.__setitem__(700, 0), r"rowptr decreases at vertex 699"),
    (lambda rp, cl: (cl.__setitem__(5000, 1 << 30), cl.__setitem__(4321, 1024)),
     r"col\[4321\]=1024 out of range \(V=1024\)"),
    (lambda rp, cl: cl.__setitem__(-1, 0xffffffff), r"col\[\d+\]=4294967295 out of range"),
]


@pytest.mark.parametrize("bad", range(len(BAD)))
@pytest.mark.parametrize("device", [False, True])
def test_invalid_csr_is_refused(ob, bad, device):
    import torch
    rp, cl = oracle.rmat_csr(10, 16, 3)
    rp, cl = rp.copy(), cl.copy()
    BAD[bad][0](rp, cl)
    if device:
        rp, cl = (torch.from_numpy(a.view(np.int32)).cuda() for a in (rp, cl))
    with pytest.raises(ob.OliveError, match=BAD[bad][1]):
        ob.Graph.from_csr(rp, cl)


@pytest.mark.parametrize("V", [1, 2, 31, 33, 1025])
def test_first_sssp_of_a_new_handle(ob, V):
    rng = np.random.default_rng(V)
    deg = rng.integers(0, 40, V) * (rng.random(V) < 0.6)
    rp = np.concatenate([[0], np.cumsum(deg)]).astype(np.uint32)
    cl = rng.integers(0, max(1, V // 2), int(deg.sum())).astype(np.uint32)
    w = rng.integers(0, 300, len(cl)).astype(np.uint32)
    for s in (0, V - 1):
        with ob.Graph.from_csr(rp, cl, w) as g:
            np.testing.assert_array_equal(g.sssp(s), oracle.dijkstra(rp, cl, w, s)[0])
