"""BFS pull levels at the edges of their three passes: candidate counts around
a warp's 32, in-degrees around the first probe, the eight of the candidate pass
and the rounds of 32 of the overflow pass, with and without a parent."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu
FRONTIER = 3000      # too many for the one-CTA levels
DEGREES = [0, 1, 7, 8, 9, 39, 40, 41, 71, 72, 73, 104, 105, 106, 200]   # decoy in-edges


@pytest.mark.parametrize("targets", [1, 4, 31, 32, 33, 127, 1025, 40003])
@pytest.mark.parametrize("extra", [0, 1])
def test_pull_passes(targets, extra):
    import olive_b200 as ob
    rng = np.random.default_rng(targets)
    # 0 -> the frontier -> the targets; unreached decoys, of higher out-degree than
    # the frontier, come first among a target's in-edges
    t0 = 1 + FRONTIER
    d0 = t0 + targets
    deg = rng.choice(DEGREES, targets)
    parent = rng.random(targets) < 0.7
    parent[0] = True     # the frontier has an edge: the level is pulled
    V = d0 + max(DEGREES) + extra
    src = [np.zeros(FRONTIER, np.int64)]
    dst = [np.arange(1, t0)]
    for k in range(max(DEGREES)):
        hit = np.flatnonzero(deg > k)
        pad = np.full(2 * FRONTIER + 64, d0, np.int64)   # an out-degree above the frontier's
        src.append(np.full(len(hit) + len(pad), d0 + k))
        dst.append(np.concatenate([t0 + hit, pad]))
    hit = np.flatnonzero(parent)
    src.append(1 + rng.integers(0, FRONTIER, len(hit)))
    dst.append(t0 + hit)
    src, dst = np.concatenate(src), np.concatenate(dst)
    order = np.argsort(src, kind="stable")
    rp = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=V))]).astype(np.uint32)
    cl = dst[order].astype(np.uint32)
    ref, _ = oracle.bfs(rp, cl, 0)
    with ob.Graph.from_csr(rp, cl) as g:
        g.tune(alpha=1e9)
        got = g.bfs(0)
        assert g.last_stats.pull_steps >= 1
        np.testing.assert_array_equal(got, ref)
        assert g.last_stats.vertices_reached == int(np.sum(ref != oracle.INF))
