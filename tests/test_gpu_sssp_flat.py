"""Delta-stepping over the flat out-CSR in one launch, on graphs that reach
each of its ways to take a step: one CTA alone (paths, small graphs), the whole
grid, rows cut into pieces (hubs), light and heavy passes (large first
buckets), buckets jumped over (heavy weights); against Dijkstra."""
import numpy as np
import pytest
from scipy.sparse import csr_matrix
from scipy.sparse.csgraph import dijkstra

from llama_b200 import LG_UNREACHED, Store
from llama_b200.graph import tune_reset, tune_set

pytestmark = pytest.mark.gpu


def _graph(shape, seed):
    rng = np.random.default_rng(seed)
    if shape == "path":
        V = 6000
        s = np.arange(V - 1)
        d, w = s + 1, rng.integers(1, 300, V - 1)
    elif shape == "hubs":                    # two hubs joined to all, and back
        V = 60001
        a = np.arange(2, V)
        s = np.concatenate([np.zeros(V - 2, int), a, np.ones(V - 2, int), [0, 1]])
        d = np.concatenate([a, np.ones(V - 2, int), a, [1, 0]])
        w = rng.integers(1, 60, len(s))
    elif shape == "far":                     # few edges, distances far apart
        V = 3000
        key = rng.choice(V * V, 9000, replace=False)
        s, d, w = key // V, key % V, rng.integers(1, 1 << 20, 9000)
    elif shape == "sinks":                   # most vertices have no out-edges
        V = 20000
        key = np.unique(rng.integers(0, 100, 30000) * V + rng.integers(0, V, 30000))
        s, d = key // V, key % V
        w = rng.integers(1, 100, len(s))
    else:                                    # dense enough for long queues in a bucket
        V = 150000
        key = np.unique(rng.integers(0, V, 2400000) * V + rng.integers(0, V, 2400000))
        s, d = key // V, key % V
        w = rng.integers(1, 256, len(s))
    return V, s, d, w


@pytest.mark.parametrize("flat", [False, True])
@pytest.mark.parametrize("shape,deltas", [
    ("path", (1, 100, 1 << 22)), ("hubs", (3, 32, 1000)), ("far", (1, 5000, 1 << 30)),
    ("sinks", (8, 32)), ("dense", (16, 64, 300, 100000))])
def test_distances(shape, deltas, flat):
    V, s, d, w = _graph(shape, 11)
    g = csr_matrix((w.astype(np.float64), (s, d)), (V, V))
    want = dijkstra(g, indices=[0, 1])
    deg = np.bincount(s, minlength=V)
    rng = np.random.default_rng(1)
    late = rng.random(len(s)) < 0.2
    with Store(reverse_edges=False) as st:
        for m in (~late, late):
            st.build_level(V, s[m], d[m], w[m])
        with st.snapshot() as sn:
            if flat:
                sn.flatten(0)
            try:
                for rng_len in (1024, 256):
                    tune_set(0, "sssp_range", rng_len)
                    for root in (0, 1):
                        ref = np.where(np.isinf(want[root]), LG_UNREACHED, want[root])
                        for delta in deltas:
                            got, r = sn.sssp(root, delta)
                            assert np.array_equal(got, ref.astype(np.uint32)), (root, delta)
                            near = got < LG_UNREACHED
                            assert (r.reached, r.reach_edges, r.max_dist) == (
                                near.sum(), deg[near].sum(), got[near].max())
            finally:
                tune_reset(0)


def test_single_vertex_and_no_edges():
    with Store(reverse_edges=False) as st:
        st.build_level(1, np.zeros(0, np.uint32), np.zeros(0, np.uint32), np.zeros(0, np.uint32))
        with st.snapshot() as sn:
            got, r = sn.sssp(0, 32)
            assert list(got) == [0] and (r.reached, r.reach_edges, r.max_dist) == (1, 0, 0)


@pytest.mark.parametrize("heavy", ["none", "last rows", "one", "first rows"])
def test_few_heavy_edges(heavy):
    """Edges of at least delta nowhere, or where a first look may not meet them;
    queues long enough for rounds over the light edges alone."""
    rng = np.random.default_rng(len(heavy))
    V = 150000
    key = np.unique(rng.integers(0, V, 2400000) * V + rng.integers(0, V, 2400000))
    s, d = key // V, key % V
    w = rng.integers(1, 31, len(s))
    delta = 40
    at = {"none": s < 0, "last rows": s >= V - 300, "first rows": s < 300,
          "one": np.arange(len(s)) == len(s) - 7}[heavy]
    w[at] = rng.integers(delta, 4 * delta, at.sum())
    # long ways round: rows that only heavy edges improve
    want = dijkstra(csr_matrix((w.astype(np.float64), (s, d)), (V, V)), indices=[0, int(s[-7])])
    with Store(reverse_edges=False) as st:
        st.build_level(V, s, d, w)
        with st.snapshot() as sn:
            for flat in (False, True):
                if flat:
                    sn.flatten(0)
                for i, root in enumerate((0, int(s[-7]))):
                    ref = np.where(np.isinf(want[i]), LG_UNREACHED, want[i]).astype(np.uint32)
                    for dl in (delta, delta + 1, 31, 15):
                        assert np.array_equal(sn.sssp(root, dl)[0], ref), (root, dl)
