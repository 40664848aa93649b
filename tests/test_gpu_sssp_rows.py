"""SSSP's renumbering and light/heavy partition at the edges of their rounds:
rows (and in-edge lists) one short of, at and one past 32 and 256 entries."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu
LENGTHS = [0, 1, 31, 32, 33, 255, 256, 257, 287, 288, 289, 511, 512, 513, 2049]


@pytest.mark.parametrize("relabel", [0, 1])
@pytest.mark.parametrize("reverse", [False, True])
def test_row_lengths(relabel, reverse):
    import olive_b200 as ob
    rng = np.random.default_rng(7 + reverse)
    V = 3001
    src = np.concatenate([np.full(n, 1 + i) for i, n in enumerate(LENGTHS * 3)])
    dst = rng.integers(0, V, len(src))
    if reverse:   # the same lengths as in-edge lists
        src, dst = dst, src
    # a way from the source to every vertex, and back
    src = np.concatenate([np.zeros(V - 1, np.int64), np.arange(V), src])
    dst = np.concatenate([np.arange(1, V), np.roll(np.arange(V), -7), dst])
    order = np.argsort(src, kind="stable")
    rp = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=V))]).astype(np.uint32)
    cl = dst[order].astype(np.uint32)
    w = rng.integers(1, 129, len(cl)).astype(np.uint32)   # both sides of the bucket width
    want = oracle.dijkstra(rp, cl, w, 0)[0]
    with ob.Graph.from_csr(rp, cl, w) as g:
        g.tune(sssp_relabel=relabel)
        np.testing.assert_array_equal(g.sssp(0), want)
