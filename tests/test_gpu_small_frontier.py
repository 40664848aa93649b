"""Levels and supersteps that one CTA runs by itself (frontiers of at most 2048
vertices and 16384 edges): layered graphs whose layers sit on both sides of
those limits, so that a run enters and leaves that path on the way, against the
serial oracle (whole numbers: exact)."""
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


def layered(widths, edges, seed):
    """CSR of a graph whose BFS layers from vertex 0 are the given widths: layer
    i has exactly edges[i] out-edges (at least one into every vertex of the next
    layer, the rest back to earlier layers or itself)."""
    rng = np.random.default_rng(seed)
    start = np.concatenate([[0], np.cumsum(widths)])
    src, dst = [], []
    for i, w in enumerate(widths):
        nxt = np.arange(start[i + 1], start[i + 2]) if i + 1 < len(widths) else np.empty(0, int)
        n = max(edges[i], len(nxt))
        src.append(start[i] + rng.integers(0, w, n))
        dst.append(np.concatenate([nxt, rng.integers(0, start[i + 1], n - len(nxt))]))
    src, dst = np.concatenate(src), np.concatenate(dst)
    o = np.argsort(src, kind="stable")
    V = int(start[-1])
    perm = rng.permutation(V)          # ids carry no layer order
    src, dst = perm[src], perm[dst]
    o = np.argsort(src, kind="stable")
    rp = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=V))]).astype(np.uint32)
    return rp, dst[o].astype(np.uint32), int(perm[0])


SHAPES = [
    ([1], [0]),                                              # a lone source
    ([1, 1, 1, 5, 3], [1, 1, 5, 9, 0]),
    ([1, 2047, 2048, 2049, 2048, 31], [2047, 2048, 4000, 2048, 31, 7]),
    ([1, 16384, 10], [16384, 10, 0]),                        # out of the path and back
    ([1, 16385, 10, 700], [16385, 10, 700, 0]),
    ([1, 1024, 1025, 2000, 900], [1024, 16384, 16385, 900, 16000]),
    ([1] + [33] * 40 + [40000] + [3] * 30, [33] * 40 + [40000, 90000] + [3] * 30),
]


@pytest.mark.parametrize("shape", range(len(SHAPES)))
@pytest.mark.parametrize("graphs", [1, 0])
def test_bfs_layers(ob, shape, graphs):
    rp, cl, src = layered(*SHAPES[shape], seed=shape)
    ref, e_ref = oracle.bfs(rp, cl, src)
    with ob.Graph.from_csr(rp, cl) as g:
        g.tune(use_graphs=graphs)
        for s in (src, src):           # a second run on the same handle
            np.testing.assert_array_equal(g.bfs(s), ref)
            assert g.last_stats.edges_traversed == e_ref
            assert g.last_stats.iterations == len(SHAPES[shape][0])


@pytest.mark.parametrize("wmax", [1, 255, 5000])
@pytest.mark.parametrize("shape", range(len(SHAPES)))
def test_sssp_layers(ob, shape, wmax):
    rp, cl, src = layered(*SHAPES[shape], seed=shape + 50)
    w = np.random.default_rng(wmax).integers(1, wmax + 1, len(cl)).astype(np.uint32)
    ref, e_ref, _, nset = oracle.dijkstra(rp, cl, w, src)
    with ob.Graph.from_csr(rp, cl, w) as g:
        for kw in ({}, {"use_graphs": 0}, {"sssp_tail_delta": 0}, {"sssp_relabel": 0},
                   {"sssp_sub": 4}, {"sssp_pull": 0}):
            base = g.tune()
            g.tune(**kw)
            np.testing.assert_array_equal(g.sssp(src), ref, err_msg=str(kw))
            st = g.last_stats
            assert st.edges_traversed == e_ref and st.vertices_reached == nset
            g.tune(**{k: base[k] for k in kw})


@pytest.mark.parametrize("rows,cols", [(1, 1), (3, 700), (90, 101)])
def test_sssp_grid(ob, rows, cols):
    rp, cl = oracle.grid_csr(rows, cols)
    w = np.random.default_rng(rows).integers(0, 256, len(cl)).astype(np.uint32)
    with ob.Graph.from_csr(rp, cl, w) as g:
        for s in (0, rows * cols // 2):
            np.testing.assert_array_equal(g.sssp(s), oracle.dijkstra(rp, cl, w, s)[0])
