"""Flattening at the edges of its tiles: rows of one slot and of thousands,
fragments of every level, deletions on either side of a tile boundary, against
the snapshot's adjacency; and calls that take a flat copy of a snapshot whose
vertex-table degrees are wrong."""
import ctypes as C

import numpy as np
import pytest

from llama_b200 import HostGraph, LgError, Store
from llama_b200._lib import VT_DTYPE
from llama_b200.graph import ppr

pytestmark = pytest.mark.gpu


def _levels(V, n, levels, hub, dele, seed):
    """Per level (src, dst, del_src, del_dst) of a random multiversion graph."""
    rng = np.random.default_rng(seed)
    key = rng.choice(V * V, size=n, replace=False)
    s, d = key // V, key % V
    if hub:                                     # a row of V edges at both ends
        s = np.concatenate([s, np.full(V, 3), np.arange(V)])
        d = np.concatenate([d, np.arange(V), np.full(V, 5)])
        k = np.unique(s * V + d)
        s, d = k // V, k % V
    lev = rng.integers(0, levels, len(s))
    live = np.full(len(s), True)
    out = []
    for l in range(levels):
        new = lev == l
        dead = np.zeros(len(s), bool)
        if l and dele:
            dead = live & (lev < l) & (rng.random(len(s)) < dele)
            live &= ~dead
        out.append((s[new], d[new], s[dead], d[dead]))
    return out


@pytest.mark.parametrize("dele", [0.0, 0.3])
@pytest.mark.parametrize("V,n,levels,hub", [
    (3, 5, 1, False), (60, 511, 1, False), (60, 512, 3, False), (60, 513, 5, False),
    (900, 1025, 8, False), (5000, 3000, 40, False), (3001, 9000, 6, True)])
def test_flat_equals_adjacency(V, n, levels, hub, dele):
    hg = HostGraph(V)
    rng = np.random.default_rng(n)
    for s, d, xs, xd in _levels(V, n, levels, hub, dele, n + V):
        hg.add_level(s, d, xs, xd, rng.integers(1, 200, len(s)).astype(np.uint32))
    with Store() as st:
        st.ingest(hg)
        for l in sorted({0, levels // 2, levels - 1}):
            with st.snapshot(l) as sn:
                pr, (dist, _) = sn.pagerank_pull(3), sn.sssp(1, 32)
                bfs = sn.bfs(1)[0]
                age = rng.integers(0, 40, V).astype(np.int32)
                src = [np.repeat(np.arange(V), np.diff(sn.adjacency(k)[0]).astype(np.int64))
                       for k in (0, 1)]
                nbr = [sn.adjacency(k)[1] for k in (0, 1)]
                # teen counts read ids, heads, rows and tile starts
                teen = np.bincount(src[1], ((age >= 10) & (age < 20))[nbr[1]].astype(float), V)
                assert np.array_equal(sn.avg_teen_cnt(age)[0], teen.astype(np.int32))
                sn.flatten(0).flatten(1)
                assert np.array_equal(sn.pagerank_pull(3), pr)
                assert np.array_equal(sn.sssp(1, 32)[0], dist)
                assert np.array_equal(sn.bfs(1)[0], bfs)
                assert np.array_equal(sn.avg_teen_cnt(age)[0], teen.astype(np.int32))


def test_wrong_degrees():
    """A vertex table whose degrees are not the live edge counts: calls that
    need them refuse it, calls that count the edges themselves do not."""
    V, rng = 300, np.random.default_rng(2)
    key = rng.choice(V * V, size=4000, replace=False)
    key = key[key // V != key % V]
    s, d = (key // V).astype(np.uint32), (key % V).astype(np.uint32)
    seeds = np.arange(32)
    want = None
    for wrong in (0, 7):
        hg = HostGraph(V)
        hg.add_level(s, d)
        desc = hg.level_desc(0)
        for dr, c in enumerate((desc.out, desc.in_)):
            vt = np.ctypeslib.as_array(C.cast(c.vt, C.POINTER(C.c_uint8)),
                                       ((V + 1) * 16,)).view(VT_DTYPE)
            if wrong and dr == 1:
                vt["degree"][11] += wrong
            if wrong and dr == 0:
                vt["degree"][V - 1] += wrong       # no seed reaches a wrong division
        with Store() as st:
            st.ingest(hg)
            with st.snapshot() as sn:
                r = sn.triangle_count()
                x = ppr([sn], seeds, iterations=1)
                got = (r.triangles, r.undirected_edges, r.arcs, x)
                if wrong:
                    assert got[:3] == want[:3] and np.array_equal(x, want[3])
                    with pytest.raises(LgError):
                        sn.flatten(1)
                    with pytest.raises(LgError):
                        sn.pagerank_pull(2)
                else:
                    want = got


def _store(V, s, d, w, patch):
    """A store of one level whose vertex tables (out, in) patch(vt, direction)
    has changed."""
    hg = HostGraph(V)
    hg.add_level(s, d, weights=w)
    desc = hg.level_desc(0)
    for dr, c in enumerate((desc.out, desc.in_)):
        patch(np.ctypeslib.as_array(C.cast(c.vt, C.POINTER(C.c_uint8)),
                                    ((V + 1) * 16,)).view(VT_DTYPE), dr)
    st = Store()
    st.ingest(hg)
    return st


@pytest.mark.parametrize("wrong", ["pair", "pair at the end", "huge"])
def test_degrees_that_make_up_for_each_other(wrong):
    """A degree too small by what the next vertex, which has no edges, has too
    much: every other row starts where it should.  And degrees far above the
    number of slots."""
    V, rng = 300, np.random.default_rng(4)
    key = rng.choice(V * V, size=4000, replace=False)
    bare = V - 1 if wrong.endswith("end") else 12           # no edges in or out
    key = key[(key // V != bare) & (key % V != bare) & (key // V != key % V)]
    s, d = (key // V).astype(np.uint32), (key % V).astype(np.uint32)
    w = rng.integers(1, 99, len(s)).astype(np.uint32)
    seeds = np.arange(32)

    def patch(vt, dr):
        if wrong == "huge":
            if dr == 1:
                vt["degree"][[5, 6, 7]] = 1 << 31
        else:
            assert vt["degree"][bare] == 0 and vt["degree"][bare - 1] > 3
            vt["degree"][bare - 1] -= 2
            vt["degree"][bare] += 2
    with _store(V, s, d, w, lambda vt, dr: None) as st, st.snapshot() as sn:
        want = (sn.triangle_count().triangles, sn.scc()[0], sn.sssp(3, 32)[0])
        right = ppr([sn], seeds, iterations=1)
    with _store(V, s, d, w, patch) as st, st.snapshot() as sn:
        got = (sn.triangle_count().triangles, sn.scc()[0], sn.sssp(3, 32)[0])
        x = ppr([sn], seeds, iterations=1)
        if wrong != "huge":                                 # (divided by the wrong degree)
            out = np.setdiff1d(np.arange(V), d[s == bare - 1])
            x, right = x[:, out], right[:, out]
        assert np.array_equal(x, right)
        for a, b in zip(got, want):
            assert np.array_equal(a, b)
        with pytest.raises(LgError):
            sn.flatten(1)
        with pytest.raises(LgError):
            sn.pagerank_pull(2)
        if wrong != "huge":
            with pytest.raises(LgError):
                sn.flatten(0)
