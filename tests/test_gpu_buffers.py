"""Device buffers kept from one graph for the next: bounded, and safe when
several threads create, run and close graphs of different sizes at once."""
import threading

import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


def test_kept_memory_is_bounded():
    import torch
    import olive_b200 as ob
    with ob.Graph.rmat(10, 8, seed=1) as g:     # device code and context
        g.bfs(0)
        g.pagerank(max_it=3)
    torch.cuda.synchronize()
    free0, total = torch.cuda.mem_get_info()
    for scale in (16, 20, 22, 19):
        with ob.Graph.rmat(scale, 16, seed=scale) as g:
            g.bfs(0)
            g.pagerank(max_it=3)
    free1, _ = torch.cuda.mem_get_info()
    # the bound, and room for what the driver itself keeps (loaded code, small blocks)
    assert free0 - free1 <= total // 64 + (256 << 20)


def test_graphs_from_several_threads():
    import olive_b200 as ob
    inputs = [oracle.rmat_csr(s, 8, s) for s in (8, 11, 13, 14)]
    want = [oracle.bfs(rp, cl, 1)[0] for rp, cl in inputs]
    bad = []

    def work(t):
        for r in range(8):
            i = (t + r) % len(inputs)
            with ob.Graph.from_csr(*inputs[i]) as g:
                if not np.array_equal(g.bfs(1), want[i]):
                    bad.append((t, r))

    threads = [threading.Thread(target=work, args=(t,)) for t in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
