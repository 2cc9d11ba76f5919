"""Strongly connected components on graphs that reach each part of the search:
one giant component, several of a size, chains and cycles, rows cut into
pieces, nothing to trim and nothing left; against scipy."""
import numpy as np
import pytest
from scipy.sparse import csr_matrix
from scipy.sparse.csgraph import connected_components

from llama_b200 import Store

pytestmark = pytest.mark.gpu


def _graph(shape):
    rng = np.random.default_rng(len(shape))
    if shape == "path":                       # no cycle at all
        V = 3000
        p = rng.permutation(V)
        return V, p[:-1], p[1:]
    if shape == "cycles":                     # of every length from 2 to 90, joined in a chain
        s, d, at = [], [], 0
        for n in range(2, 91):
            c = at + np.arange(n)
            s += [c, [c[-1]]]
            d += [np.roll(c, -1), [at + n]]
            at += n
        V = at + 1
        p = rng.permutation(V)
        return V, p[np.concatenate(s)], p[np.concatenate(d)]
    if shape == "hubs":                       # hub rows of V edges, both ways
        V = 9001
        a = np.arange(2, V)
        half = a[a % 2 == 0]
        return V, np.concatenate([np.zeros(V - 2, int), half, half, [1]]), \
            np.concatenate([a, np.zeros(len(half), int), np.ones(len(half), int), [0]])
    if shape == "blocks":                     # five random digraphs, edges only forward between
        n, s, d = 2000, [], []
        for b in range(5):
            s += [b * n + rng.integers(0, n, 5 * n), b * n + rng.integers(0, n, 300)]
            d += [b * n + rng.integers(0, n, 5 * n), min(b + 1, 4) * n + rng.integers(0, n, 300)]
        p = rng.permutation(5 * n)
        return 5 * n, p[np.concatenate(s)], p[np.concatenate(d)]
    if shape == "sparse":                     # many small components
        V = 60000
        return V, rng.integers(0, V, 66000), rng.integers(0, V, 66000)
    V = 40000                                 # giant: one component and its surroundings
    return V, rng.integers(0, V, 120000), rng.integers(0, V, 120000)


@pytest.mark.parametrize("shape", ["path", "cycles", "hubs", "blocks", "sparse", "giant"])
def test_partition(shape):
    V, s, d = _graph(shape)
    k = np.unique(np.asarray(s, np.int64) * V + d)
    s, d = k // V, k % V
    rng = np.random.default_rng(3)
    late = rng.random(len(k)) < 0.2
    dead = ~late & (rng.random(len(k)) < (0.0 if shape in ("path", "cycles") else 0.05))
    live = ~dead
    _, comp = connected_components(csr_matrix((np.ones(live.sum()), (s[live], d[live])), (V, V)),
                                   connection="strong")
    first = np.full(comp.max() + 1, V)
    np.minimum.at(first, comp, np.arange(V))
    with Store() as st:
        st.build_level(V, s[~late], d[~late])
        st.build_level(V, s[late], d[late], None, s[dead], d[dead])
        with st.snapshot() as sn:
            for flat in (False, True):
                if flat:
                    sn.flatten(0).flatten(1)
                lab, r = sn.scc()
                assert np.array_equal(lab, first[comp])
                assert r.components == len(first)
                both = (np.bincount(s[live], minlength=V) > 0) & (
                    np.bincount(d[live], minlength=V) > 0)
                assert r.trimmed == V - both.sum()


def test_chain_settles_a_vertex_per_round():
    """Ids that ascend along a chain: n rounds of up to n steps.  No launch
    takes them all, so that none holds the GPU for as long as they take: a
    launch ends after 50 ms, and half a million steps with a barrier each
    (a microsecond at the least) do not fit into five of them."""
    V = 1000
    a = np.arange(V - 1)
    with Store() as st:
        st.build_level(V, a, a + 1)
        with st.snapshot() as sn:
            sn.flatten(0).flatten(1)
            before = st.launch_count
            lab, r = sn.scc()
            assert np.array_equal(lab, np.arange(V)) and r.components == V
            assert r.rounds >= V - 4 and r.steps >= (V - 4) ** 2 // 2
            assert st.launch_count - before > 14         # 10 with one launch of scc_rest
