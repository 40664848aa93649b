"""PageRank and weighted PageRank where their grid does not find the whole GPU free:
on a stream of a few SMs (a green context), and beside other streams' kernels.  The
solves end, and those past one cluster give the bits that they give alone; those of a
cluster take the other form on part of a GPU, within the rounding of the sums."""
import numpy as np
import pytest

from test_gpu_threads import inputs

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch
    assert torch.cuda.is_available()
    torch.zeros(1, device="cuda")
    return torch


def solves(g, d):
    return [g.pagerank(0.85, 12, 0.0), g.pagerank(0.85, 30, 1e-5, "leak"),
            g.wpr_forward(d["p"], w=d["w"], max_it=11), *g.wpr_backward(d["g"], max_it=11)]


@pytest.fixture
def few_sms(torch):
    """A stream limited to 8 or 16 SMs."""
    driver = pytest.importorskip("cuda.bindings.driver")

    def ok(r):
        assert r[0] == driver.CUresult.CUDA_SUCCESS, r[0]
        return r[1:] if len(r) > 2 else (r[1] if len(r) == 2 else None)

    dev = ok(driver.cuDeviceGet(torch.cuda.current_device()))
    sms = ok(driver.cuDeviceGetDevResource(dev, driver.CUdevResourceType.CU_DEV_RESOURCE_TYPE_SM))
    parts, n, _ = ok(driver.cuDevSmResourceSplitByCount(1, sms, 0, 8))
    assert n == 1 and parts[0].sm.smCount <= 16
    desc = ok(driver.cuDevResourceGenerateDesc(parts, 1))
    ctx = ok(driver.cuGreenCtxCreate(
        desc, dev, driver.CUgreenCtxCreate_flags.CU_GREEN_CTX_DEFAULT_STREAM))
    stream = ok(driver.cuGreenCtxStreamCreate(
        ctx, driver.CUstream_flags.CU_STREAM_NON_BLOCKING, 0))
    yield int(stream)
    ok(driver.cuStreamDestroy(stream))
    ok(driver.cuGreenCtxDestroy(ctx))


@pytest.mark.parametrize("V", [61, 8001, 54273, 150001])
def test_on_few_sms(few_sms, V):
    import olive_b200 as ob
    d = inputs(V)
    with ob.Graph.from_csr(d["rp"], d["cl"]) as g:
        want = solves(g, d)
        g.set_stream(few_sms)
        got = solves(g, d)
        g.set_stream(None)
        for a, b in zip(got, want):
            if V > 8192:
                assert a.tobytes() == b.tobytes()
            else:   # the order of FP64 sums and of FP32 ones inside a row's lanes
                assert np.max(np.abs(a - b)) <= 1e-6 * np.max(np.abs(b))
        assert [x.tobytes() for x in solves(g, d)] == [x.tobytes() for x in want]


def test_beside_other_kernels(torch):
    """Two streams keep every SM busy with matrix products while the solves run."""
    import olive_b200 as ob
    d = inputs(150001)
    x = torch.randn(2048, 2048, device="cuda")
    side = [torch.cuda.Stream() for _ in range(2)]
    with ob.Graph.from_csr(d["rp"], d["cl"]) as g:
        want = [a.tobytes() for a in solves(g, d)]
        for _ in range(6):
            for s in side:
                with torch.cuda.stream(s):
                    for _ in range(20):
                        torch.mm(x, x)
            assert [a.tobytes() for a in solves(g, d)] == want
        torch.cuda.synchronize()
