"""Batched PPR of instances that a CTA or a cluster can run: which one does depends on
how many there are, the result does not.  Every instance of a large call equals its solo
run bit for bit, the sweep it stops at included."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


def instances(count, lo, hi, deg, rng):
    n = rng.integers(lo, hi + 1, count)
    off = np.concatenate([[0], np.cumsum(n)]).astype(np.uint32)
    rps, cols = [np.zeros(1, np.int64)], []
    for i in range(count):
        src = np.sort(rng.integers(0, n[i], n[i] * deg))
        rps.append(rps[-1][-1] + np.cumsum(np.bincount(src, minlength=n[i])))
        cols.append(rng.integers(0, n[i], len(src)) + int(off[i]))
    return n, off, np.concatenate(rps).astype(np.uint32), np.concatenate(cols).astype(np.uint32)


@pytest.mark.parametrize("K,deg", [(4, 3), (8, 24), (16, 8), (32, 3), (32, 8)])
@pytest.mark.parametrize("cluster", [1, 8])
def test_large_calls_equal_solo_runs(K, deg, cluster):
    import olive_b200 as ob
    rng = np.random.default_rng(100 * K + deg)
    n, off, rp, cl = instances(130, 200, 2048, deg, rng)
    seeds = np.stack([rng.integers(0, m, K) for m in n]).astype(np.uint32)
    with ob.Graph.from_csr(rp, cl) as g:
        g.tune(batch_cluster=cluster)
        for tol in (0.0, 1e-4, 3e-6):
            _, pr, it = g.batch(off, seeds, alpha=0.85, max_it=40, tol=tol, bfs=False)
            assert tol or np.all(it == 40)
            for i in list(range(0, 130, 13)) + [int(np.argmax(n)), int(np.argmin(n))]:
                b, e = int(off[i]), int(off[i + 1])
                lrp, lcl = (rp[b:e + 1] - rp[b]), cl[rp[b]:rp[e]] - np.uint32(b)
                with ob.Graph.from_csr(lrp, lcl) as solo:
                    solo.tune(batch_cluster=cluster)
                    _, spr, sit = solo.batch(np.array([0, e - b], np.uint32), seeds[i:i + 1],
                                             alpha=0.85, max_it=40, tol=tol, bfs=False)
                assert sit[0] == it[i]
                np.testing.assert_array_equal(spr, pr[b:e])
                if tol == 3e-6 and i % 26 == 0:
                    ref, _ = oracle.ppr(lrp, lcl, seeds[i], 0.85, int(it[i]), 0.0)
                    # FP32 sums of at most 64 positive terms (in-degrees of these digraphs):
                    # 66 * 2^-24 a sweep, over 1 - alpha
                    np.testing.assert_allclose(pr[b:e], ref, rtol=2.7e-5, atol=1e-7)
