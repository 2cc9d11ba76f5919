"""Vertex counts at the edges of the scans' tiles (one CTA, tiles that add up
the sums before theirs, a scan of the sums between the two passes): adjacency,
flattened rows and a batch of searches against numpy."""
import numpy as np
import pytest

from llama_b200 import Store

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V", [1, 31, 511, 513, 4095, 4097, 8191, 8192, 8193, 12288, 12289, 70001,
                               4096 * 8192, 4096 * 8192 + 1])
def test_rows(V):
    rng = np.random.default_rng(V)
    n = min(V * 3, 60_000) if V > 1 else 0
    key = np.unique(rng.integers(0, V * V, n))
    s, d = key // V, key % V
    hub = np.unique(rng.integers(0, V, min(V, 3000)))          # one long row, one long column
    s = np.concatenate([s, np.full(len(hub), V - 1), hub])
    d = np.concatenate([d, hub, np.full(len(hub), V // 2)])
    key = np.unique(s * V + d)
    s, d = key // V, key % V
    off = np.zeros(V + 1, np.int64)
    np.cumsum(np.bincount(s, minlength=V), out=off[1:])
    with Store() as st:
        st.build_level(V, s.astype(np.uint32), d.astype(np.uint32), None)
        with st.snapshot(0) as sn:
            o, nb = sn.adjacency(0)
            assert np.array_equal(o.astype(np.int64), off)
            assert np.array_equal(nb, d.astype(nb.dtype))
            if V > 1 << 20:
                return
            before = sn.pagerank_pull(3)
            hops = sn.bfs(V - 1)[0]                            # queues of every length
            sn.flatten()
            assert np.array_equal(sn.pagerank_pull(3), before)
            assert np.array_equal(sn.bfs(V - 1)[0], hops)
    far = 2 ** 31 - 2                                          # an unreached vertex
    dist = np.full(V, far)
    dist[V - 1], front = 0, np.array([V - 1])
    while len(front):
        nxt = np.unique(np.concatenate([d[off[v]:off[v + 1]] for v in front]))
        nxt = nxt[dist[nxt] == far]
        dist[nxt] = dist[front[0]] + 1
        front = nxt
    assert np.array_equal(hops, dist)
