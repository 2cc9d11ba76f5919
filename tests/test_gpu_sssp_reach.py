"""Shortest paths from roots that reach little of a large snapshot nobody has
flattened: found by a search of bounded size, at whose bounds the calls below
are, and solved over the levels; the others over a flat copy."""
import numpy as np
import pytest
from scipy.sparse import csr_matrix
from scipy.sparse.csgraph import dijkstra

from llama_b200 import LG_UNREACHED, Store

pytestmark = pytest.mark.gpu


def test_roots_of_every_reach():
    rng = np.random.default_rng(6)
    big = 300_000                                # a graph of 4.4 M edges, from 0 on
    key = np.unique(rng.integers(0, big * big, 4_400_000))
    parts, at = [], big
    roots = {"graph": 0}

    def part(name, n, s, d):
        nonlocal at
        roots[name] = at
        parts.append((at + np.asarray(s), at + np.asarray(d)))
        at += n
    one = np.zeros(0, int)
    part("alone", 1, one, one)
    part("loop", 1, [0], [0])
    for n in (20, 32, 33, 200):                  # hops up to the bound and beyond
        part(f"path {n}", n, np.arange(n - 1), np.arange(1, n))
    for n in (255, 256, 257, 1023, 1300, 5000):  # vertices
        part(f"star {n}", n, np.zeros(n - 1, int), np.arange(1, n))
    for n in (44, 45, 46, 128):                  # slots: n (n - 1)
        i, j = np.divmod(np.arange(n * n), n)
        part(f"clique {n}", n, i[i != j], j[i != j])
    a = np.arange(1, 250)                        # a tree, and back edges
    part("tree", 250, np.concatenate([(a - 1) // 3, a]), np.concatenate([a, a // 2]))
    part("cut", 10, [0, 1, 2], [1, 2, 3])        # 1 -> 2 is deleted later
    part("late", 10, one, one)                   # gets its edge later
    small = np.concatenate([p[0] for p in parts]), np.concatenate([p[1] for p in parts])
    V = at + 1_000_000                           # (the rule counts vertices too)
    s = np.concatenate([key // big, small[0]])
    d = np.concatenate([key % big, small[1]])
    w = rng.integers(1, 70, len(s))
    cut, late = roots["cut"], roots["late"]
    bridge = [late, late + 1], [late + 1, 5]     # to a vertex of the big graph
    s2 = np.concatenate([s, bridge[0]])
    d2 = np.concatenate([d, bridge[1]])
    w2 = np.concatenate([w, [4, 9]])
    live = ~((s2 == cut + 1) & (d2 == cut + 2))
    order = list(roots.values())
    want = dijkstra(csr_matrix((w2[live].astype(float), (s2[live], d2[live])), (V, V)),
                    indices=order)
    deg = np.bincount(s2[live], minlength=V)
    with Store(reverse_edges=False) as st:
        st.build_level(V, s, d, w)
        st.build_level(V, *bridge, [4, 9], [cut + 1], [cut + 2])
        with st.snapshot() as sn:
            for i, (name, root) in enumerate(roots.items()):
                before = st.launch_count
                got, r = sn.sssp(root, 32)
                ref = np.where(np.isinf(want[i]), LG_UNREACHED, want[i]).astype(np.uint32)
                assert np.array_equal(got, ref), name
                near = got < LG_UNREACHED
                assert (r.reached, r.reach_edges, r.max_dist) == (
                    near.sum(), deg[near].sum(), got[near].max()), name
                many = name in ("graph", "path 33", "path 200", "star 257", "star 1023",
                                "star 1300", "star 5000", "clique 46", "clique 128", "late")
                # the search, init, the two launches of the steps and the sums;
                # or (the search and) a flat copy
                assert (st.launch_count - before > 5) == many, name
