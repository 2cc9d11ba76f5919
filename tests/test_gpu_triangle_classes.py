"""Triangle counting over graphs that reach each of its ways to intersect:
pairs of short lists, one-warp, four-warp and whole-SM bitmaps, hash tables of
up to 64 ids, and the searches of labels no bitmap holds.  The graphs are circulants (vertex i joined
to i + 1 .. i + k) under a random renaming, whose triangles are known."""
import numpy as np
import pytest

from llama_b200 import Store

pytestmark = pytest.mark.gpu


def _circulant(n, k, seed, wheel):
    """Arcs of the circulant in random direction, some in both directions,
    self-loops among them, split in two levels; its triangles and edges."""
    rng = np.random.default_rng(seed)
    name = rng.permutation(n + (1 if wheel else 0)).astype(np.int64)
    i = np.repeat(np.arange(n, dtype=np.int64), k)
    j = (i + np.tile(np.arange(1, k + 1, dtype=np.int64), n)) % n
    if wheel:                                   # one vertex joined to all others
        i = np.concatenate([i, np.arange(n)])
        j = np.concatenate([j, np.full(n, n)])
    edges = len(i)
    tri = n * k * (k - 1) // 2 + (n * k if wheel else 0)
    flip = rng.random(edges) < 0.5
    s, d = np.where(flip, j, i), np.where(flip, i, j)
    both = rng.random(edges) < 0.1
    s, d = np.concatenate([s, d[both], np.arange(0, n, 97)]), \
        np.concatenate([d, s[both], np.arange(0, n, 97)])
    s, d = name[s], name[d]
    first = rng.random(len(s)) < 0.8
    arcs = edges + int(both.sum())
    return (s.astype(np.uint32), d.astype(np.uint32), first, tri, edges, arcs, len(name))


@pytest.mark.parametrize("n,k,wheel", [
    (9, 2, False), (257, 4, True), (4099, 12, True), (70001, 5, False), (70001, 14, True),
    (300007, 12, False), (1900003, 10, False), (70001, 90, False), (280001, 80, False),
    (1900003, 70, False)])
def test_circulants(n, k, wheel):
    s, d, first, tri, edges, arcs, V = _circulant(n, k, 7 + n, wheel)
    with Store(reverse_edges=n % 2 == 0) as st:
        st.build_level(V, s[first], d[first])
        st.build_level(V, s[~first], d[~first])
        with st.snapshot() as sn:
            for flat in (False, True):
                if flat:
                    sn.flatten(0)
                r = sn.triangle_count()
                assert (r.triangles, r.undirected_edges, r.arcs) == (tri, edges, arcs)


def test_no_edges():
    with Store() as st:
        st.build_level(5, np.zeros(0, np.uint32), np.zeros(0, np.uint32))
        with st.snapshot() as sn:
            r = sn.triangle_count()
            assert (r.triangles, r.undirected_edges, r.arcs) == (0, 0, 0)
