"""Batched PPR-K at the edges of its routes: widths of one to eight lanes a
vertex and those that take a lane per vector, instance sizes on both sides of
the line between one CTA and a cluster, single vertices, and vertices without
out-edges or without in-edges."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu
SIZES = [1, 2, 3, 31, 33, 257, 1999, 2047, 2048, 2049, 5003]


def block_digraphs(rng):
    """Rows of 0..9 out-edges, a hub whose in-edges come from half the vertices."""
    off = np.concatenate([[0], np.cumsum(SIZES)]).astype(np.uint32)
    src, dst = [], []
    for i, n in enumerate(SIZES):
        deg = rng.integers(0, 10, n) * (rng.random(n) < 0.8)
        s = np.repeat(np.arange(n), deg)
        d = rng.integers(0, n, len(s))
        hub = np.flatnonzero(rng.random(n) < 0.5)
        src.append(np.concatenate([s, hub]) + off[i])
        dst.append(np.concatenate([d, np.zeros(len(hub), np.int64)]) + off[i])
    src, dst = np.concatenate(src), np.concatenate(dst)
    order = np.argsort(src, kind="stable")
    rp = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=off[-1]))]).astype(np.uint32)
    return off, rp, dst[order].astype(np.uint32)


@pytest.mark.parametrize("tol", [0.0, 1e-5])
@pytest.mark.parametrize("K", [1, 4, 5, 8, 12, 16, 32])
def test_widths_and_sizes(K, tol):
    import olive_b200 as ob
    rng = np.random.default_rng(K)
    off, rp, cl = block_digraphs(rng)
    seeds = np.stack([rng.integers(0, n, K) for n in SIZES]).astype(np.uint32)
    with ob.Graph.from_csr(rp, cl) as g:
        runs = {}
        for cluster in (0, 8, 16):
            g.tune(batch_cluster=cluster)
            _, pr, iters = g.batch(off, seeds, alpha=0.85, max_it=12, tol=tol, bfs=False)
            runs[cluster] = pr.copy()
            for i in range(len(SIZES)):
                b, e = int(off[i]), int(off[i + 1])
                lrp = (rp[b:e + 1] - rp[b]).astype(np.uint32)
                lcl = (cl[rp[b]:rp[e]] - b).astype(np.uint32)
                # the FP64 definition at the count of sweeps that was run
                ref, _ = oracle.ppr(lrp, lcl, seeds[i], 0.85, int(iters[i]), 0.0)
                assert tol or iters[i] == 12
                # FP32 sums of up to 2500 positive terms: sqrt(2500) * 2^-24 a sweep, seven
                # sweeps' worth at alpha 0.85, times ten
                np.testing.assert_allclose(pr[b:e], ref, rtol=2e-4, atol=2e-6, err_msg=f"{i}")
            for i in (0, 7, 10):   # below, on and above the line: bitwise a solo run
                b, e = int(off[i]), int(off[i + 1])
                lrp = (rp[b:e + 1] - rp[b]).astype(np.uint32)
                lcl = (cl[rp[b]:rp[e]] - b).astype(np.uint32)
                if not len(lcl):
                    continue
                with ob.Graph.from_csr(lrp, lcl) as solo:
                    solo.tune(batch_cluster=cluster)
                    _, spr, sit = solo.batch(np.array([0, e - b], np.uint32), seeds[i:i + 1],
                                             alpha=0.85, max_it=12, tol=tol, bfs=False)
                assert sit[0] == iters[i]
                np.testing.assert_array_equal(spr, pr[b:e])
        # a second run of the call is bitwise the same
        _, again, _ = g.batch(off, seeds, alpha=0.85, max_it=12, tol=tol, bfs=False)
        np.testing.assert_array_equal(again, runs[16])
